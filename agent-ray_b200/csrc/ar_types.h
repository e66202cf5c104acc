// Device-visible data layout of a scene in HBM (shared by host and device code).
//
// Wide BVH node (80 bytes, five 16-byte words so one node is five coalesced
// 128-bit loads): 8 children with 8-bit quantised boxes on a per-node grid.
//   word0: origin px, py, pz (f32), packed biased exponents ex|ey<<8|ez<<16
//   word1: child_base, tri_base, child_mask, tri_mask
//   word2: qlo_x[0..7], qlo_y[0..7]
//   word3: qlo_z[0..7], qhi_x[0..7]
//   word4: qhi_y[0..7], qhi_z[0..7]
// Child slot s owns bits 4s..4s+3 of the two masks.  child_mask bit 4s: an
// internal child at child_base + (its rank among the internal children);
// tri_mask bits 4s..4s+c-1: a leaf of c primitives, the one of mask bit b at
// tri_base + popc(tri_mask & ((1 << b) - 1)), counted in triangle (BLAS) or
// instance (TLAS) records from the first node.  Neither: an empty slot.
// Slots are assigned by octant (bit k of s set: child lies on the + side of
// axis k), so traversal visits slot (i ^ ray_octant) for i = 0..7, an
// approximately front-to-back order with no sorting.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define AR_HD __host__ __device__
#else
#define AR_HD
#endif

namespace ar {

struct alignas(16) WideNode {
    float px, py, pz;
    uint32_t exps;  // ex | ey << 8 | ez << 16
    uint32_t child_base, tri_base;
    uint32_t child_mask, tri_mask;
    uint8_t qlo_x[8], qlo_y[8], qlo_z[8];
    uint8_t qhi_x[8], qhi_y[8], qhi_z[8];
};
static_assert(sizeof(WideNode) == 80, "wide node is 80 bytes");

// Triangle in BLAS leaf order: v0 (w = original prim id bits), e1 = v1 - v0,
// e2 = v2 - v0, precomputed in f32 exactly as Triangle::new does.
struct alignas(16) TriRecord {
    float v0x, v0y, v0z;
    uint32_t prim;
    float e1x, e1y, e1z;
    uint32_t mesh;
    float e2x, e2y, e2z;
    uint32_t slot;  // this record's index
};
static_assert(sizeof(TriRecord) == 48, "triangle record is 48 bytes");

// TLAS leaf entry: world->local transform columns (xyz of c0..c3) + BLAS root.
struct alignas(16) InstanceRecord {
    float c[12];
    uint32_t blas_root;   // node index of the mesh BLAS root
    uint32_t object;      // SceneObject index (RayHit::instance_id)
    uint32_t valid_blas;  // 0 when the mesh has no triangles
    uint32_t pad;
};
static_assert(sizeof(InstanceRecord) == 64, "instance record is 64 bytes");

struct alignas(16) ObjectRecord {
    float nmat[9];        // normal matrix columns (inverse-transpose of the linear part)
    uint32_t mesh;
    uint32_t mat_offset;  // into material_table
    uint32_t num_mats;    // 1: mat0, whatever the triangle's slot
    uint32_t flags;       // kMeshNormals, kMeshUv
    uint32_t mat0;
    uint32_t shade_off;   // triangle record -> shading record, modulo 2^32
    uint32_t pad;
};
static_assert(sizeof(ObjectRecord) == 64, "object record is 64 bytes");
constexpr uint32_t kMeshNormals = 1u, kMeshUv = 2u;

// What shading reads of a triangle beside its TriRecord, gathered when the
// acceleration structure is built: its vertices' normals and uv and its material
// slot.  Only meshes that have one of these for the triangle have such records.
struct alignas(16) TriShade {
    float n[9];     // normals of the three vertices
    uint32_t slot;  // material slot
    float uv[6];
};
static_assert(sizeof(TriShade) == 64, "shading record is 64 bytes");

struct alignas(16) MaterialRecord {
    uint32_t kind;
    int32_t emitter;
    float albedo[3];
    float f0[3];
    float alpha;
    float eta;  // dielectric interior IOR
    int32_t tex;  // Lambertian albedo texture, -1: constant albedo
    float pad;
};

// ImageTexture (src/texture.rs:65-151) texels [offset, offset + width * height)
// of DevScene::texels, linear RGB, row-major from the top row.
struct TextureRecord {
    uint32_t offset, width, height, pad;
};

struct alignas(16) LightRecord {
    uint32_t kind;
    float area;
    float pad0[2];
    float pos[4];    // point: position;  quad: corner
    float inten[4];  // point: intensity; quad: radiance
    float e1[4], e2[4], n[4];
};

// Read-only view of a device-resident scene, passed by value to kernels.
struct DevScene {
    const WideNode* nodes;  // nodes, triangle and instance records in one buffer
    const TriRecord* tris;  // the triangle records of that buffer
    const TriShade* shade;  // at triangle record + its object's shade_off
    const ObjectRecord* objects;
    const uint32_t* material_table;
    const MaterialRecord* materials;
    const LightRecord* lights;
    const float* light_cdf;
    const float* light_pmf;
    const float4* texels;
    const TextureRecord* textures;
    uint32_t tlas_root;       // 0xFFFFFFFF: empty scene
    uint32_t num_lights;
    uint32_t light_dist;      // ar_light_distribution
    uint32_t pad;
};

constexpr uint32_t kInvalid = 0xFFFFFFFFu;

// Pixel and sample of sample number g of an image of npix pixels: runs of samples
// of one pixel, pixels row by row, run after run of the whole image.  A run keeps a
// warp's camera rays and what they first hit together (16 samples, against one of
// every pixel after the other: extension -7%, render -4.5% at 512x512x16 on 139k
// triangles; 32x32 blocks of pixels in Z order instead of rows gave 0.2% more, 8x4
// tiles of one sample each 1.4%).  It ends after 64, since samples that finish
// together add to one pixel one after the other: without an end 64x64x1024 of a
// small scene at depth 1 took 1.21 ms (one sample of every pixel after the other
// 1.02, runs of 64 0.86), 512x512x64 of 139k triangles 36.9 (49.0, 36.9; runs of 32
// 37.1, of 8 37.7).  Up to 1024 pixels, few enough to stay together anyway, 4 are
// faster: 16x16x4096 at depth 1 0.94 ms without an end (0.51; runs of 64 0.73, of 4
// 0.47), 4x4x65536 3.08 (1.74; 2.64, 1.74).
struct PixelSample {
    uint32_t pixel, sample;
};
AR_HD inline PixelSample pixel_sample(unsigned long long g, uint32_t npix, uint32_t samples) {
    const uint32_t most = npix > 1024u ? 64u : 4u;
    uint32_t first = 0, run = samples;
    if (samples > most) {
        const unsigned long long pass = (unsigned long long)npix * most, k = g / pass;
        g -= k * pass;
        first = uint32_t(k) * most;
        run = samples - first < most ? samples - first : most;
    }
    const uint32_t pixel = uint32_t(g / run);
    return {pixel, first + uint32_t(g % run)};
}
constexpr int kTraversalStack = 32;

}  // namespace ar

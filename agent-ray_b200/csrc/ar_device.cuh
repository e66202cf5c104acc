// Device-side math, sampler and BVH8 traversal for the light-transport kernels.
//
// Parity-critical arithmetic (ray normalisation, instance transforms and the
// Möller–Trumbore test) uses explicitly rounded intrinsics so that no multiply
// is fused into an add: the reference (Rust + glam SSE2) computes these with
// separate roundings, and the closest-hit t/u/v must match it bit for bit.
#pragma once
#include <cfloat>
#include <cstdint>
#include "ar_types.h"

// Traversal kernels: 128 threads, at least 8 blocks per SM (<= 64 registers),
// i.e. half the SM's warps resident to hide node-fetch latency.
#ifndef AR_TRAVERSAL_MIN_BLOCKS
#define AR_TRAVERSAL_MIN_BLOCKS 8
#endif
#define AR_TRAVERSAL_BOUNDS __launch_bounds__(128, AR_TRAVERSAL_MIN_BLOCKS)
constexpr int kTraversalThreads = 128;  // threads per block of every kernel that traverses
// Traversal steps a lane runs between two ray-fetch rounds of its warp: 4 for
// any hit, whose rays end sooner, 6 for closest hit (1M-triangle soup 19.8 ms at
// 4, 19.35 at 6, 19.2 at 8; BDPT room's extension 19.0, 19.1, 19.5; shadow rays
// slow down from 6 on).  One copy of the step body: unrolled twice or four
// times it no longer fits the instruction cache (steps of 2, unrolled: 2x slower).
constexpr int kStepsClosest = 6, kStepsAny = 4;
// Resident blocks per SM under AR_TRAVERSAL_BOUNDS: the persistent grid of a ray-fetch launch.
constexpr int kTraversalBlocksPerSm = AR_TRAVERSAL_MIN_BLOCKS;

namespace ar {

struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator-(f3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ f3 operator*(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ f3 operator*(float s, f3 a) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ f3 operator*(f3 a, f3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ f3 operator/(f3 a, float s) { return {a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float length(f3 a) { return sqrtf(dot(a, a)); }
__device__ __forceinline__ f3 normalize(f3 a) { return a * (1.0f / length(a)); }
__device__ __forceinline__ float max3(f3 a) { return fmaxf(fmaxf(a.x, a.y), a.z); }
__device__ __forceinline__ bool is_zero(f3 a) { return a.x == 0.f && a.y == 0.f && a.z == 0.f; }

// ---- exactly rounded (no contraction) variants: reference arithmetic order ----
__device__ __forceinline__ f3 sub_rn(f3 a, f3 b) {
    return {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
}
__device__ __forceinline__ f3 add_rn(f3 a, f3 b) {
    return {__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)};
}
__device__ __forceinline__ f3 scale_rn(f3 a, float s) {
    return {__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s)};
}
// glam dot3: (x*x' + y*y') + z*z'
__device__ __forceinline__ float dot_rn(f3 a, f3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ f3 cross_rn(f3 a, f3 b) {
    return {__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
            __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x))};
}
// glam normalize: v * (1 / sqrt(dot(v, v)))
__device__ __forceinline__ f3 normalize_rn(f3 a) {
    return scale_rn(a, __frcp_rn(__fsqrt_rn(dot_rn(a, a))));
}
__device__ __forceinline__ f3 ld3(const float* p) { return {p[0], p[1], p[2]}; }

// Queue records that a stage touches once (batched rays and their hits, shadow
// queues): loaded and stored evict-first, so that streaming them through L2
// does not push out the BVH and the traversal stacks, which every ray reuses
// (measured: closest hit on the 1M-triangle soup +0.5%, BDPT +1.3%).
template <class T>
__device__ __forceinline__ T ld_once(const T* p) {
    return __ldcs(p);
}
template <class T>
__device__ __forceinline__ void st_once(T* p, T v) {
    __stcs(p, v);
}

// ---- counter-based sampler (SplitMix64 finalizer, Steele et al. 2014) ----
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t counter_key(uint64_t seed, uint32_t pixel, uint32_t sample) {
    return mix64(seed ^ mix64((uint64_t(pixel) << 32) | uint64_t(sample)));
}
__device__ __forceinline__ float counter_u01(uint64_t key, uint32_t dim) {
    uint64_t z = mix64(key + uint64_t(dim + 1) * 0x9e3779b97f4a7c15ull);
    return float(uint32_t(z >> 40)) * (1.0f / 16777216.0f);
}
constexpr uint32_t kLightSubpathDim = 4096;

// ---- traversal ----
struct Ray {
    f3 o, d;
    float tmin, tmax;
};

struct HitRec {
    float t, u, v;
    uint32_t slot;  // triangle record index (leaf order), kInvalid on miss
    uint32_t inst;  // SceneObject index
};

// Ray::new applied to a world ray (direction normalised as glam does).
__device__ __forceinline__ Ray make_ray(f3 o, f3 d, float tmin, float tmax) { return {o, normalize_rn(d), tmin, tmax}; }

// Triangle::hit (src/geometry.rs:172-206) with the reference's operation order.
__device__ __forceinline__ bool tri_test(const TriRecord& tr, f3 o, f3 d, float tmin, float tmax, float& t, float& u,
                                         float& v) {
    f3 v0 = mk(tr.v0x, tr.v0y, tr.v0z), e1 = mk(tr.e1x, tr.e1y, tr.e1z), e2 = mk(tr.e2x, tr.e2y, tr.e2z);
    f3 h = cross_rn(d, e2);
    float a = dot_rn(e1, h);
    if (fabsf(a) < 1e-8f) return false;
    float f = __frcp_rn(a);
    f3 s = sub_rn(o, v0);
    float uu = __fmul_rn(f, dot_rn(s, h));
    if (uu < 0.0f || uu > 1.0f) return false;
    f3 q = cross_rn(s, e1);
    float vv = __fmul_rn(f, dot_rn(d, q));
    if (vv < 0.0f || __fadd_rn(uu, vv) > 1.0f) return false;
    float tt = __fmul_rn(f, dot_rn(e2, q));
    if (tt < tmin || tt > tmax) return false;
    t = tt;
    u = uu;
    v = vv;
    return true;
}

__device__ __forceinline__ TriRecord load_tri(const TriRecord* rec) {
    const float4* p = reinterpret_cast<const float4*>(rec);
    float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    TriRecord r;
    r.v0x = a.x; r.v0y = a.y; r.v0z = a.z; r.prim = __float_as_uint(a.w);
    r.e1x = b.x; r.e1y = b.y; r.e1z = b.z; r.mesh = __float_as_uint(b.w);
    r.e2x = c.x; r.e2y = c.y; r.e2z = c.z; r.slot = __float_as_uint(c.w);
    return r;
}

// Per-ray constants of the slab test.
struct RayPre {
    f3 inv;
    uint32_t oct;  // bit k set when direction k is negative
};
// Slab reciprocal: the hardware approximation, +-1e20 at most (a zero keeps its
// sign).  It only culls child boxes, which the builder quantised outward; t, u,
// v and the hit itself come from the exactly rounded triangle test.  One
// approximation and two clamps an axis instead of a test, a select and a
// division; with __frcp_rn for the exact reciprocals (1/a of the triangle test,
// 1/length of the local direction: the same correctly rounded value as the
// division in about half its instructions) 1M visibility rays 451 -> 441 us, a
// 139k-triangle scene at 512x512x16 11.0 -> 10.8 ms, BDPT room 57.5 -> 56.6 ms.
__device__ __forceinline__ float slab_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return fminf(fmaxf(r, -1e20f), 1e20f);
}
__device__ __forceinline__ RayPre precompute(f3 d) {
    RayPre r;
    r.inv = mk(slab_rcp(d.x), slab_rcp(d.y), slab_rcp(d.z));
    // the octant follows the reciprocal's sign, -0.0 included (its reciprocal
    // is -1e20): near and far planes must swap exactly when inv is negative
    r.oct = (signbit(d.x) ? 1u : 0u) | (signbit(d.y) ? 2u : 0u) | (signbit(d.z) ? 4u : 0u);
    return r;
}

// Packed pairs of f32 (Blackwell's f32x2 arithmetic: one instruction per
// pair, each half rounded exactly as the scalar instruction would).
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// max / min of three (NaN operands ignored, as fmaxf / fminf do)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Byte j of w as the float 2^23 + byte: the bits 0x4B0000qq encode 2^23 + qq,
// and subtracting 2^23 afterwards is exact (a byte-permute and an add
// instead of an I2F).
__device__ __forceinline__ float biased_byte(uint32_t w, uint32_t j) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u + j));
}

// Child masks: slot s of a node has bits 4s..4s+3 of a 32-bit word, so one word
// holds a flag per child (bit 4s) and room for up to four primitives per leaf.
constexpr uint32_t kSlotBits = 0x11111111u;

// Reorders a word of slot flags from slot s to traversal position i = s ^ oct
// (bytes by one permute, the two slots of a byte by a masked swap).
__device__ __forceinline__ uint32_t to_traversal_order(uint32_t v, uint32_t oct) {
    v = __byte_perm(v, 0u, 0x3210u ^ (0x1111u * ((oct >> 1) & 3u)));
    const uint32_t w = (v ^ (v >> 4)) & ((oct & 1u) * 0x01010101u);
    return v ^ (w * 17u);
}

// Intersects the 8 children of node `ni`; returns a flag per child slot whose
// box the ray meets (empty slots may be flagged: the node's masks exclude them).
// Each child's six slab distances come from three packed multiply-adds, each
// half the scalar fmaf(byte, a, b) of the same operands (measured against the
// scalar form: served-scene traversal stages -2%, two children per pair instead
// of the (x, y) / (near z, far z) pairs used here: -0.3..+0.5%, more spills).
// A child is missed when far - near is negative: exactly when near > far, since
// the rounded difference of two floats keeps its sign, but for far = -0 against
// near = +0, whose difference is -0.  The offsets b are therefore formed as
// x y + 0, which is never -0, so no plane lies at -0 (a ray that starts on a
// node's low face and leaves through it, t_min = 0, would lose its hit at t = 0;
// a multiply-add costs what the multiply did).  A funnel shift gathers that
// sign bit, two instructions a child where a compare, a byte of leaf data and
// its shifts took about seven.  The traversal kernels issue on 0.75 of the
// cycles, so instructions are what counts: 16M rays on the 1M-triangle soup
// 26.4 -> 24.1 ms, extension of a 512x512x16 render of a 139k-triangle scene
// 6.71 -> 6.37 ms, its shadow rays 4.43 -> 4.13 ms.
__device__ __forceinline__ uint32_t intersect_node(const WideNode* node, f3 o, f3 inv, uint32_t oct,
                                                   float tmin, float tmax, uint4& links) {
    const uint4* np = reinterpret_cast<const uint4*>(node);
    const uint4 w0 = __ldg(np), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    links = __ldg(np + 1);
    const float px = __uint_as_float(w0.x), py = __uint_as_float(w0.y), pz = __uint_as_float(w0.z);
    const uint32_t ex = w0.w & 0xffu, ey = (w0.w >> 8) & 0xffu, ez = w0.w >> 16;
    const float ax = __uint_as_float(ex << 23) * inv.x;
    const float ay = __uint_as_float(ey << 23) * inv.y;
    const float az = __uint_as_float(ez << 23) * inv.z;
    const float bx = __fmaf_rn(px - o.x, inv.x, 0.0f);
    const float by = __fmaf_rn(py - o.y, inv.y, 0.0f);
    const float bz = __fmaf_rn(pz - o.z, inv.z, 0.0f);
    // pairs: (x, y) of the near and of the far planes, and (near z, far z)
    const uint64_t AXY = f2_pack(ax, ay), BXY = f2_pack(bx, by), AZZ = f2_pack(az, az), BZZ = f2_pack(bz, bz);
    const uint64_t UNBIAS = f2_pack(-8388608.0f, -8388608.0f);
    // near/far plane bytes per axis, chosen by the ray octant
    const bool nx = oct & 1u, ny = oct & 2u, nz = oct & 4u;
    uint32_t miss = 0;
    const float tfar_limit = tmax * 1.0000004f;
#pragma unroll
    for (int half = 1; half >= 0; --half) {
        const uint32_t lox = half ? w2.y : w2.x, loy = half ? w2.w : w2.z, loz = half ? w3.y : w3.x;
        const uint32_t hix = half ? w3.w : w3.z, hiy = half ? w4.y : w4.x, hiz = half ? w4.w : w4.z;
        const uint32_t nxw = nx ? hix : lox, fxw = nx ? lox : hix;
        const uint32_t nyw = ny ? hiy : loy, fyw = ny ? loy : hiy;
        const uint32_t nzw = nz ? hiz : loz, fzw = nz ? loz : hiz;
#pragma unroll
        for (int j = 3; j >= 0; --j) {
            float tnx, tny, tfx, tfy, tnz, tfz;
            f2_unpack(f2_fma(f2_add(f2_pack(biased_byte(nxw, j), biased_byte(nyw, j)), UNBIAS), AXY, BXY), tnx, tny);
            f2_unpack(f2_fma(f2_add(f2_pack(biased_byte(fxw, j), biased_byte(fyw, j)), UNBIAS), AXY, BXY), tfx, tfy);
            f2_unpack(f2_fma(f2_add(f2_pack(biased_byte(nzw, j), biased_byte(fzw, j)), UNBIAS), AZZ, BZZ), tnz, tfz);
            const float tn = fmax3(tnx, tny, fmaxf(tnz, tmin));
            const float tf = fmin3(tfx, tfy, fminf(tfz, tfar_limit));
            miss = __funnelshift_l(__float_as_uint(tf - tn), miss, 4);
        }
    }
    return (~miss >> 3) & kSlotBits;
}

// Two-level closest-hit / any-hit traversal (TLAS::intersect + BLASAccel::intersect,
// src/accel/bvh.rs:247-296, :413-447) as a resumable state machine.  One
// stack serves both levels: entering an instance pushes a marker so that
// popping it restores the world ray.  start() loads a ray, step() performs one
// node visit with its leaf tests and the stack work up to the next node, and
// returns true when the ray is done; stack overflow or a runaway loop sets *err and
// ends the ray.  Kernels drive it with dynamic ray fetch (run_traversal
// below): a lane whose ray finishes takes the next ray at once, so a warp is
// not held by its slowest ray.
//
// Registers hold only what a node visit and a triangle test read (the current
// ray, its t limit, the next node, the stack pointer).  What is read once per
// instance or once per ray lies in named slots of cold state: the world ray, the
// best hit so far.  With all of it in scalars the compiler spilled 120-200 bytes
// inside the node visit, more local traffic than the stack's; now nothing spills at
// the 64 registers of 8 blocks per SM: 16M rays on the 1M-triangle soup 24.1 ->
// 20.1 ms, a 139k-triangle scene's extension rays 6.35 -> 5.70 ms and shadow rays
// 4.11 -> 3.73 ms per 512x512x16 render; 7 blocks (72 registers) 2-12 % slower, 9,
// 10 and 12 blocks (56, 48, 40 registers, spilling again) 2-5, 5-25 and 13-40 %.
// Any hit keeps its cold state in local memory, closest hit (which touches more
// of it) in shared memory, 80 bytes a thread, whose accesses do not go through to
// L2: soup 19.4 -> 17.6 ms, BDPT room's extension 18.1 -> 17.7; for any hit that
// was 0.4-1.8 % slower, the stack in either place costs L1 (7-11 %).
template <bool kAnyHit>
struct Traverser {
    static constexpr uint32_t kNodeGroup = 0x80000000u, kMarker = 0x40000000u;
    static constexpr uint32_t kInBlas = 8u;  // in `oct`: the current ray is an instance's local ray
    // slots of the cold state: world origin and t_min, world direction and
    // t limit (its best hit), world reciprocals and octant, then the best hit
    // inside the current instance (u, v; slot, the instance's object, for any hit
    // its scale) and of the ray (u, v; slot, object, all 32 bits of it, which a stack
    // entry has no room for); the stack proper starts at kStack
    static constexpr int kOxy = 0, kOzT = 1, kDxy = 2, kDzT = 3, kIxy = 4, kIzO = 5, kBestUv = 6, kBest = 7, kHitUv = 8,
                         kHit = 9, kCold = 10;
    // where they lie: `cold` + slot * kColdStride; for any hit `cold` is the start of
    // the local array `mem`, whose stack begins at kStack
    static constexpr int kColdStride = kAnyHit ? 1 : kTraversalThreads, kStack = kAnyHit ? kCold : 0;
    static constexpr int kSlots = kStack + kTraversalStack;
    const WideNode* geom; // the scene's nodes, triangle and instance records
    f3 o, d, inv;         // the current ray (d is read only inside an instance)
    float tmin, tlim;     // tlim: the closest hit so far, in the current ray's units
    uint32_t oct, node, guard;
    int sp;

    __device__ __forceinline__ static uint2 pk(float a, float b) {
        return make_uint2(__float_as_uint(a), __float_as_uint(b));
    }
    __device__ __forceinline__ void set_ray(f3 no, f3 nd, float nt) {
        const RayPre r = precompute(nd);
        o = no;
        inv = r.inv;
        oct = r.oct;
        tmin = nt;
    }

    // False when the scene is empty (the ray misses).
    __device__ __forceinline__ bool start(const DevScene* s, const Ray& r, uint2* cold) {
        geom = s->nodes;
        set_ray(r.o, r.d, r.tmin);
        tlim = r.tmax;
        cold[kOxy * kColdStride] = pk(r.o.x, r.o.y);
        cold[kOzT * kColdStride] = pk(r.o.z, r.tmin);
        cold[kDxy * kColdStride] = pk(r.d.x, r.d.y);
        cold[kDzT * kColdStride] = pk(r.d.z, r.tmax);
        cold[kIxy * kColdStride] = pk(inv.x, inv.y);
        cold[kIzO * kColdStride] = make_uint2(__float_as_uint(inv.z), oct);
        cold[kHit * kColdStride] = make_uint2(kInvalid, kInvalid);
        node = s->tlas_root;
        sp = 0;
        guard = 0;
        return node != kInvalid;
    }

    // The finished ray's hit (t is the ray's t_max when it missed).
    __device__ __forceinline__ HitRec result(const uint2* cold) const {
        HitRec h;
        h.t = tlim;
        h.u = h.v = 0.f;
        h.slot = cold[kHit * kColdStride].x;
        h.inst = kInvalid;
        if (!kAnyHit && h.slot != kInvalid) {
            h.inst = cold[kHit * kColdStride].y;
            h.u = __uint_as_float(cold[kHitUv * kColdStride].x);
            h.v = __uint_as_float(cold[kHitUv * kColdStride].y);
        }
        return h;
    }

    // The record that a node's tri_base names: its distance from `geom` in
    // records, triangles for BLAS nodes, instances for TLAS nodes.
    template <class Record>
    __device__ __forceinline__ const Record* record(uint32_t k) const {
        return reinterpret_cast<const Record*>(geom) + k;
    }
    __device__ __forceinline__ bool push(uint2 e, int* err, uint2* mem) {
        if (sp >= kTraversalStack) { atomicExch(err, 1); return false; }
        mem[kStack + sp++] = e;
        return true;
    }

    // One step = one node visit (with its leaf tests) followed by the stack
    // work that leads to the next node to visit, so every active lane of a
    // warp intersects a node in every step.  Returns true when the ray is
    // finished (or failed: *err set).
    __device__ __forceinline__ bool step(int* err, uint2* mem, uint2* cold) {
        if (++guard > (1u << 22)) { atomicExch(err, 3); return true; }
        uint4 links;  // child_base, tri_base, child_mask, tri_mask
        const uint32_t met = intersect_node(geom + node, o, inv, oct, tmin, tlim, links);
        uint2 group = make_uint2(links.x, to_traversal_order(met & links.z, oct) | (links.z << 1) | kNodeGroup);
        uint32_t tbits = (met * 15u) & links.w;
        if (tbits) {
            if (oct & kInBlas) {
                while (tbits) {
                    const uint32_t b = __ffs(tbits) - 1;
                    tbits &= tbits - 1;
                    const TriRecord tr = load_tri(record<TriRecord>(links.y + __popc(links.w & ((1u << b) - 1u))));
                    float t, u, v;
                    if (tri_test(tr, o, d, tmin, tlim, t, u, v) && t < tlim) {
                        if (kAnyHit) {
                            if (__fdiv_rn(t, __uint_as_float(cold[kBest * kColdStride].y)) < __uint_as_float(cold[kDzT * kColdStride].y)) {
                                cold[kHit * kColdStride].x = tr.slot;
                                return true;
                            }
                        } else {
                            tlim = t;
                            cold[kBestUv * kColdStride] = pk(u, v);
                            cold[kBest * kColdStride].x = tr.slot;
                        }
                    }
                }
            } else {
                // TLAS leaves: resume the node group after the instances.
                if ((group.y & kSlotBits) && !push(group, err, mem)) return true;
                group = make_uint2(0, 0);
                if (!push(make_uint2(links.y, tbits | (links.w << 1)), err, mem)) return true;
            }
        }
        // Find the next node: the nearest child of the current group, else
        // pop (node groups, instance exits and entries) until one is found.
        // Every pass pops one entry, so the loop ends within sp passes.
        for (;;) {
            if (group.y & kSlotBits) {  // a node group with children left (only those stay in `group`)
                const uint32_t i = __ffs(group.y & kSlotBits) - 1;
                const uint32_t s = i ^ (4u * (oct & 7u));
                node = group.x + __popc(group.y & (kSlotBits << 1) & ((1u << s) - 1u));
                group.y &= ~(1u << i);
                return (group.y & kSlotBits) && !push(group, err, mem);
            }
            if (sp == 0) return true;
            const uint2 e = mem[kStack + --sp];
            if (e.y & kNodeGroup) {
                group = e;
                continue;
            }
            if (e.y & kMarker) {
                // Leave the instance: convert the local best back to world t.
                float best = __uint_as_float(cold[kDzT * kColdStride].y);
                if (!kAnyHit) {
                    const uint2 hit = cold[kBest * kColdStride];
                    if (hit.x != kInvalid) {
                        const float tw = __fdiv_rn(tlim, __uint_as_float(e.x));
                        if (tw < best) {
                            best = tw;
                            cold[kHit * kColdStride] = hit;
                            cold[kHitUv * kColdStride] = cold[kBestUv * kColdStride];
                        }
                    }
                }
                tlim = best;
                const uint2 a = cold[kOxy * kColdStride], b = cold[kOzT * kColdStride], c = cold[kIxy * kColdStride], f = cold[kIzO * kColdStride];
                o = mk(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(b.x));
                tmin = __uint_as_float(b.y);
                inv = mk(__uint_as_float(c.x), __uint_as_float(c.y), __uint_as_float(f.x));
                oct = f.y;
                continue;
            }
            // Instance leaf group: enter the next instance.
            const uint32_t b = __ffs(e.y & kSlotBits) - 1;
            const uint32_t rest = e.y & ~(1u << b);
            if (rest & kSlotBits) mem[kStack + sp++] = make_uint2(e.x, rest);
            const float4* ip = reinterpret_cast<const float4*>(
                record<InstanceRecord>(e.x + __popc(e.y & (kSlotBits << 1) & ((1u << b) - 1u))));
            const float4 m0 = __ldg(ip), m1 = __ldg(ip + 1), m2 = __ldg(ip + 2);
            const uint4 m3 = __ldg(reinterpret_cast<const uint4*>(ip + 3));
            if (!m3.z) continue;  // mesh without triangles
            const f3 c0 = mk(m0.x, m0.y, m0.z), c1 = mk(m0.w, m1.x, m1.y), c2 = mk(m1.z, m1.w, m2.x),
                     c3 = mk(m2.y, m2.z, m2.w);
            const uint2 wxy = cold[kDxy * kColdStride], wzt = cold[kDzT * kColdStride];
            const float wx = __uint_as_float(wxy.x), wy = __uint_as_float(wxy.y), wz = __uint_as_float(wzt.x);
            // glam transform_point3a / transform_vector3a: ((c0*x + c1*y) + c2*z) + c3
            const f3 ldu = add_rn(add_rn(scale_rn(c0, wx), scale_rn(c1, wy)), scale_rn(c2, wz));
            const float scale = __fsqrt_rn(dot_rn(ldu, ldu));
            if (scale < FLT_EPSILON) continue;
            if (!push(make_uint2(__float_as_uint(scale), kMarker), err, mem)) return true;
            const f3 lo = add_rn(c3, add_rn(add_rn(scale_rn(c0, o.x), scale_rn(c1, o.y)), scale_rn(c2, o.z)));
            d = normalize_rn(ldu);
            if (kAnyHit) {
                cold[kBest * kColdStride].y = __float_as_uint(scale);
            } else {
                cold[kBest * kColdStride] = make_uint2(kInvalid, m3.y);
                cold[kDzT * kColdStride].y = __float_as_uint(tlim);
            }
            tlim = __fmul_rn(tlim, scale);
            set_ray(lo, d, __fmul_rn(tmin, scale));
            oct |= kInBlas;
            node = m3.x;
            return false;
        }
    }
};

// Percent of an SM's shared memory that eight blocks' cold state takes, reserve included.
constexpr int kColdCarveout = 40;

// Declares `cold`, this thread's cold state: in shared memory, or at the start of
// its local array.
#define AR_COLD_STATE(any, mem, cold)                                                   \
    __shared__ uint2 cold_state_[(any) ? 1 : Traverser<any>::kCold * kTraversalThreads]; \
    uint2* const cold = (any) ? (mem) : cold_state_ + threadIdx.x

// Persistent traversal with dynamic ray fetch.  Every lane of the warp calls
// this (warp-uniform loop).  `counter` hands out ray indices in [0, n) (reset
// to 0 before the launch); load(i, scene, ray) fetches ray i and its scene;
// store(i, hit) writes the result.
template <bool kAnyHit, class Load, class Store>
__device__ __forceinline__ void run_traversal(uint32_t* counter, uint32_t n, int* err, Load load, Store store) {
    Traverser<kAnyHit> tr;
    uint2 mem[Traverser<kAnyHit>::kSlots];
    AR_COLD_STATE(kAnyHit, mem, cold);
    int cur = -1;
    const uint32_t lane = threadIdx.x & 31u;
    // A warp runs every path that any of its rays needs, so few rays are spread
    // over the grid's warps, about 1.5 lanes' worth of each warp's share taking
    // part.  The line lies at 5 rays a warp (kernel time, closest / any hit in an
    // instanced room, packed against spread: 64 rays 58 / 47 -> 34 / 27 us, 4096
    // rays 76 / 83 -> 51 / 67, 20000 rays 85 / 84 -> 78 / 80, 40000 rays 95 / 88
    // -> 93 / 96, 80000 rays 103 / 97 -> 112 / 106: from there on the schedulers
    // have no free issue slots left).
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    bool more = lane < (n < 5u * warps ? (n + n / 2u + warps - 1u) / warps : 32u);
    for (;;) {
        const bool need = more && cur < 0;
        const uint32_t mask = __ballot_sync(0xffffffffu, need);
        if (mask) {
            const int leader = __ffs(mask) - 1;
            uint32_t base = 0;
            if (int(lane) == leader) base = atomicAdd(counter, uint32_t(__popc(mask)));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (need) {
                const uint32_t idx = base + __popc(mask & ((1u << lane) - 1u));
                if (idx < n) {
                    const DevScene* s;
                    Ray r;
                    load(idx, s, r);
                    if (tr.start(s, r, cold)) cur = int(idx);
                    else store(idx, tr.result(cold));
                } else {
                    more = false;
                }
            }
        }
        if (!__any_sync(0xffffffffu, more || cur >= 0)) break;
        if (cur >= 0) {
#pragma unroll 1
            for (int k = 0; k < (kAnyHit ? kStepsAny : kStepsClosest); ++k) {
                if (tr.step(err, mem, cold)) {
                    store(uint32_t(cur), tr.result(cold));
                    cur = -1;
                    break;
                }
            }
        }
    }
}

}  // namespace ar

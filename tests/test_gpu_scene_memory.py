"""Shading records: which meshes have them, and what a scene keeps on the device."""
import numpy as np
import pytest

import agentray
import agentray.scenes as S
import oracle as O
from agentray import _abi as A
from agentray.scene_data import Camera, Light, Material, Mesh, Object, SceneData, integrator_cfg

pytestmark = pytest.mark.gpu


def test_a_plain_mesh_keeps_its_geometry_only(ctx):
    # No normals, no uv, one material: nodes (80 B), triangles (48 B) and instances
    # (64 B), and small tables of the scene.
    g = agentray.Scene(ctx, S.triangle_soup(50_000, seed=3))
    st = g.stats()
    geometry = 80 * (st["num_blas_nodes"] + st["num_tlas_nodes"]) + 48 * st["num_triangles"] + 64 * st["num_instances"]
    assert geometry <= st["device_bytes"] <= geometry + 4096


def _patchwork():
    """Six spheres with every combination of attributes and material tables."""
    rng = np.random.default_rng(5)
    sc = SceneData(A.LIGHT_DIST_POWER)
    tex = sc.add_texture(rng.integers(0, 256, (16, 16, 3)).astype(np.uint8))
    mats = [sc.add_material(Material(albedo=tuple(rng.uniform(0.2, 0.9, 3)))) for _ in range(4)]
    mats.append(sc.add_material(Material(albedo_texture=tex)))
    base = S.icosphere(2)
    n, v = base.num_triangles, len(base.positions)
    uv = rng.uniform(0, 1, (v, 2)).astype(np.float32)
    slots = (np.arange(n) % 5).astype(np.uint32)
    two = np.array([2], np.uint32)
    kinds = [(None, None, None, [mats[0]]), (base.positions, uv, None, [mats[4]]), (None, None, slots, mats),
             (None, None, slots, [mats[1]]), (None, uv, two, mats[1:]), (base.positions, None, slots, mats[:2])]
    for k, (nrm, uvs, sl, table) in enumerate(kinds):
        m = sc.add_mesh(Mesh(base.positions, base.indices, nrm, sl, uvs))
        xf, inv = S.trs((2.2 * (k % 3) - 2.2, 2.2 * (k // 3) - 1.1, 0.0), None, (1.0, 1.0, 1.0))
        sc.add_object(Object(m, table, xf, inv))
    sc.add_light(Light(A.LIGHT_POINT, (1.0, 2.0, 8.0), (60.0, 60.0, 60.0)))
    return sc, Camera((0.0, 0.0, 9.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 45.0, 1.5)


def test_meshes_with_and_without_records_shade_alike(ctx):
    # Same stream as the oracle, before and after rebuilds that reorder the
    # triangles; pixels at edges of two surfaces apart, at the image tests' bar.
    sc, cam = _patchwork()
    cfg = integrator_cfg(A.INTEGRATOR_PT, spp=2, max_depth=3, seed=4)
    ref = O.OracleScene(sc).render(cam, cfg, 96, 64, sampler=O.SAMPLER_COUNTER)
    g = agentray.Scene(ctx, sc)
    pt = agentray.PathTracer(agentray.PathTracerConfig(spp=2, max_depth=3, rr_depth=cfg.rr_depth, seed=4))
    for rebuild in (None, dict(max_leaf_size=1, bvh_width=4), dict(max_leaf_size=4, bvh_width=8)):
        if rebuild:
            g.rebuild(**rebuild)
        img = pt.render(g, cam, 96, 64).rgb.astype(np.float64)
        close = np.abs(img - ref) <= 1e-3 * np.maximum(1.0, np.abs(ref))
        assert ref.max() > 0 and close.all(axis=2).mean() >= 0.995

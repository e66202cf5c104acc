"""Scheduling edges of the kernels: ray counts around the line below which rays
are spread over the grid's warps, renders refilled from a small path pool,
BDPT tiles and batch forms, regions and row runs of the Poisson solvers, the
chained SOR under capture, 8-bit output at odd sizes and alignments.  Each must
give what any other split of the same work gives."""
import numpy as np
import pytest

import agentray
import agentray.scenes as S
from agentray import _abi as A

pytestmark = pytest.mark.gpu


def test_ray_counts_around_the_spreading_line(ctx):
    # Every prefix of a batch gives the batch's own hits, bit for bit: one ray,
    # part of a warp, the largest spread batch and the smallest packed one
    # (5 rays a warp of the persistent grid), and one above it.
    import torch
    sc, _ = S.room(seed=4, sphere_levels=(3, 3, 2, 2), n_boxes=60)
    g = agentray.Scene(ctx, sc)
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 4
    n = 5 * warps + 1
    rng = np.random.default_rng(3)
    ot = np.zeros((n, 4), np.float32)
    dt = np.zeros((n, 4), np.float32)
    ot[:, :3] = rng.uniform((0.1, 0.1, 0.1), (9.9, 4.9, 9.9), (n, 3))
    ot[:, 3] = 1e-4
    d = rng.normal(size=(n, 3))
    dt[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    dt[:, 3] = 4.0
    hits, inst = g.trace_closest(ot, dt)
    occ = g.trace_any(ot, dt)
    assert 0.05 < occ.mean() < 0.95
    np.testing.assert_array_equal(occ != 0, inst != 0xFFFFFFFF)
    for k in (1, 3, 31, 33, 4097, warps, n - 2, n - 1):
        h, i = g.trace_closest(ot[:k], dt[:k])
        np.testing.assert_array_equal(h.view(np.uint32), hits[:k].view(np.uint32))
        np.testing.assert_array_equal(i, inst[:k])
        np.testing.assert_array_equal(g.trace_any(ot[:k], dt[:k]), occ[:k])


@pytest.mark.parametrize("depth", [0, 1, 2, 7])
def test_render_does_not_depend_on_the_path_pool(depth):
    # 40x30x4 = 4800 samples: one tick's worth in the default pool (the render
    # then ends after depth + 1 ticks), refilled over several ticks in a pool of
    # 4096.  FP64 films: only the order of the additions differs.
    sc, cam = S.cornell_box(1)
    images = []
    for capacity in (1 << 22, 4096):
        ctx = agentray.Context(0)
        ctx.set_tuning(path_capacity=capacity)
        g = agentray.Scene(ctx, sc)
        pt = agentray.PathTracer(agentray.PathTracerConfig(spp=4, max_depth=depth, rr_depth=3, seed=5,
                                                           film_precision=A.FILM_F64))
        images.append([pt.render(g, cam, 40, 30).rgb.copy() for _ in range(3)])
        g.close()
        ctx.close()
    assert images[0][0].max() > 0
    for pair in images:
        for img in pair:
            np.testing.assert_allclose(img, images[0][0], rtol=1e-6, atol=1e-9)


@pytest.mark.parametrize("depth,mode,beta", [(1, A.MIS_POWER, 2.0), (10, A.MIS_POWER, 2.0), (11, A.MIS_POWER, 2.0),
                                             (22, A.MIS_POWER, 2.0), (45, A.MIS_POWER, 2.0), (7, A.MIS_UNIFORM, 2.0),
                                             (7, A.MIS_POWER, 1.0)])
def test_bdpt_connection_tiles_match_oracle(ctx, depth, mode, beta):
    # Every size of the connection stage's tile (32, 16, 8 and 4 samples,
    # chosen by the depth), ragged last tiles (9 x 7 x 3 samples), full-length
    # subpaths in a closed room (no roulette), the MIS prefix sums up to 16
    # vertices and the walk beyond them, and the weights that always walk.
    # The walk and the connections round in another order than the oracle, at
    # about 1e-7 of a contribution each; the bar is the image tests' 1e-3.
    from agentray.scene_data import integrator_cfg
    import oracle as O
    sc, cam = S.room(seed=6, sphere_levels=(2, 2, 2, 1), n_boxes=8)
    cfg = integrator_cfg(A.INTEGRATOR_BDPT, spp=3, max_depth=depth, rr_depth=depth + 1, seed=8, mis_mode=mode,
                         mis_beta=beta)
    w, h = 9, 7
    out = np.empty(w * h * 3, np.float32)
    import ctypes as C
    agentray.check(agentray.lib().ar_render(ctx.handle, agentray.Scene(ctx, sc).handle, C.byref(cam.desc()),
                                            C.byref(cfg), w, h, out.ctypes.data, 0))
    ref = O.OracleScene(sc).render(cam, cfg, w, h, sampler=O.SAMPLER_COUNTER)
    gpu = out.reshape(h, w, 3).astype(np.float64)
    assert np.isfinite(gpu).all() and gpu.max() > 0
    np.testing.assert_allclose(gpu, ref, rtol=1e-3, atol=1e-3 * ref.mean())


@pytest.mark.parametrize("h,w,iters", [(1, 1, 200), (1, 70, 7), (65, 1, 5), (16, 16, 12), (193, 193, 13), (300, 500, 1),
                                       (517, 519, 11), (700, 640, 0)])
def test_sor_regions_are_bit_exact(ctx, h, w, iters):
    # Images of one region and of many, ragged against every overlap the solver
    # chooses (24 rings for small images down to 10), odd launch counts and a
    # last launch of fewer sweeps, against the oracle's sequential red-black SOR.
    import oracle as O
    rng = np.random.default_rng(h * 1000 + w)
    primal = rng.uniform(0.0, 2.0, (h, w, 3)).astype(np.float32)
    gx = (rng.normal(size=(h, w, 3)) * 0.2).astype(np.float32)
    gy = (rng.normal(size=(h, w, 3)) * 0.2).astype(np.float32)
    ref = O.poisson_sor_f32(primal, gx, gy, 0.2, iters, 1.6)
    out, _ = agentray.poisson_reconstruct(ctx, primal, gx, gy, 0.2, A.POISSON_SOR, iters, 1.6)
    np.testing.assert_array_equal(out, ref)


def test_chained_sor_under_capture(ctx):
    # The sweeps are launched as a chain; recorded into a graph and replayed
    # twice (the second replay starts on the first one's output buffer) they give
    # the plain call's image, bit for bit.
    import ctypes as C

    import torch
    from agentray.scene_data import integrator_cfg
    h, w = 200, 300
    torch.manual_seed(5)
    films = [torch.rand(h, w, 3, device="cuda") for _ in range(3)]
    cfg = integrator_cfg(A.INTEGRATOR_GDPT, alpha=0.2, poisson_iterations=100, sor_omega=1.6,
                         poisson_solver=A.POISSON_SOR)

    def solve(out, stream):
        agentray.check(agentray.lib().ar_poisson_sor_static(
            C.byref(cfg), w, h, *(f.data_ptr() for f in films), out.data_ptr(), C.c_void_p(stream.cuda_stream)))

    plain, replayed = torch.zeros(h, w, 3, device="cuda"), torch.zeros(h, w, 3, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    solve(plain, stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        solve(replayed, torch.cuda.current_stream())
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(plain, replayed)


@pytest.mark.parametrize("h,w", [(1, 1), (1, 130), (70, 1), (33, 64), (64, 65), (259, 200)])
def test_cg_sizes_reach_the_exact_solution(ctx, h, w):
    # Images narrower than a block of columns, ragged last blocks and row runs of
    # every length the solver chooses.  |x - x*| <= |b - A x| / lambda_min, with
    # lambda_min = alpha = 0.2 and |b - A x| <= 1e-6 |b|; plus the f32 output.
    import oracle as O
    rng = np.random.default_rng(h * 1000 + w)
    primal = rng.uniform(0.0, 2.0, (h, w, 3)).astype(np.float32)
    gx = (rng.normal(size=(h, w, 3)) * 0.2).astype(np.float32)
    gy = (rng.normal(size=(h, w, 3)) * 0.2).astype(np.float32)
    gx[:, -1] = 0
    gy[-1, :] = 0
    exact, _ = O.poisson_exact_f64(primal, gx, gy, 0.2)
    out, res = agentray.poisson_reconstruct(ctx, primal, gx, gy, 0.2, A.POISSON_CG, 2000, 1.6, 1e-6)
    assert 0 <= res <= 1e-6
    div = gx.astype(np.float64) + gy
    div[:, 1:] -= gx[:, :-1]
    div[1:] -= gy[:-1]
    b = np.linalg.norm((0.2 * primal.astype(np.float64) + div).reshape(-1, 3), axis=0)
    want = np.maximum(exact, 0)
    assert np.all(np.abs(out - want) <= 5e-6 * b + 2e-7 * np.abs(want))


@pytest.mark.parametrize("h,w", [(1, 1), (1, 3), (1, 4), (7, 5), (33, 31)])
@pytest.mark.parametrize("tm,gamma", [(A.TONEMAP_CLAMP, 2.2), (A.TONEMAP_REINHARD, 1.0),
                                      (A.TONEMAP_REINHARD_EXTENDED, 0.5)])
def test_rgb8_does_not_depend_on_size_or_alignment(ctx, h, w, tm, gamma):
    # Whole quads, their tails, and images whose address is not 16-byte aligned
    # (one pixel a thread) give the same bytes, at most 1 LSB from the oracle's
    # libm powf on the few values next to a rounding boundary.
    import torch
    import oracle as O
    rng = np.random.default_rng(h * 100 + w)
    hdr = rng.lognormal(-1.0, 1.5, (h, w, 3)).astype(np.float32)
    flat = hdr.reshape(-1)
    flat[:3] = [0.0, -1.0, 1.0]
    dev = torch.from_numpy(hdr).cuda()
    want = agentray.film_to_rgb8(ctx, dev, tm, gamma, 1.5, 4.0).cpu().numpy()
    shifted = torch.zeros(h * w * 3 + 1, device="cuda")[1:].view(h, w, 3)
    shifted.copy_(dev)
    np.testing.assert_array_equal(agentray.film_to_rgb8(ctx, shifted, tm, gamma, 1.5, 4.0).cpu().numpy(), want)
    d = np.abs(want.astype(int) - O.film_to_rgb8(hdr, tm, 4.0, gamma, 1.5).astype(int))
    assert d.max() <= 1 and (d > 0).sum() <= max(1, 1e-3 * d.size)


@pytest.mark.parametrize("depth", [0, 1, 9])
def test_bdpt_small_batches_match_large_ones(ctx, depth):
    # A batch of few samples traces each subpath through all its bounces in one
    # launch, a large one bounce by bounce: a 4-spp render above the line against
    # the sum of its four one-sample shards below it (FP64 films), and the number
    # of rays they trace.
    from agentray import distributed as D
    import torch
    sc, cam = S.room(seed=4, sphere_levels=(3, 3, 2, 2), n_boxes=40)
    g = agentray.Scene(ctx, sc)
    line = torch.cuda.get_device_properties(0).multi_processor_count * 5 * 128 * 3 // 2
    w, h = 331, line // 331 // 2 + 3  # one sample a pixel below the line, four above it
    assert w * h < line < 4 * w * h
    bd = agentray.BidirectionalPathTracer(agentray.BdptConfig(spp=4, max_depth=depth, rr_depth=3, seed=12,
                                                              film_precision=A.FILM_F64))
    full = bd.render(g, cam, w, h).rgb.astype(np.float64)
    stats = ctx.render_stats()
    parts, rays = [], 0
    for k in range(4):
        parts.append(D.render_shard(bd, g, cam, w, h, k, k + 1, np.zeros(w * h * 3, np.float32)).astype(np.float64))
        rays += ctx.render_stats()["extend_rays"]
    assert rays == stats["extend_rays"]
    np.testing.assert_allclose(np.sum(parts, axis=0).reshape(h, w, 3), full, rtol=1e-5, atol=1e-6)

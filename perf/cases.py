"""The calls that users of this library make, as cases to be measured.

Every case goes through the public entry points (agentray.Scene, the three
integrators, agentray.Server, the film and Poisson calls) with its data on the
GPU, over the range of sizes that the benchmark and the tests use: ray batches
of a few thousand to 16 million, images of 128^2 to 1024^2, 4 to 16 samples
per pixel, scenes of 34 to 1,000,000 triangles.

  rays     Scene.trace_closest / trace_any on torch CUDA ray arrays
  render   Integrator.render (PT, BDPT, GDPT) into a CUDA image
  serve    Server.submit / wait for a handful of jobs of the served stream
  poisson  ar_poisson_reconstruct on device films (red-black SOR or CG)
  rgb8     film_to_rgb8 on a CUDA image
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "agent-ray_b200"))

import agentray  # noqa: E402
import agentray.scenes as scenes  # noqa: E402
from agentray import _abi as abi  # noqa: E402

_CONTEXT = None


def _context():
    """One library context for the process, as a renderer keeps it."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = agentray.Context(0)
    return _CONTEXT


def listed():
    return [
        # A picking / probe query batch in an instanced scene: a few thousand rays, latency.
        {"name": "rays_probe", "kind": "rays", "query": "closest", "scene": "room", "count": 4096},
        # Visibility between random point pairs of the same scene, an odd batch of a million.
        {"name": "rays_any", "kind": "rays", "query": "any", "scene": "room", "count": 1000003},
        # The BVH benchmark: 16 million incoherent rays on a soup of a million triangles.
        {"name": "rays_soup", "kind": "rays", "query": "closest", "scene": "soup", "triangles": 1000000,
         "count": 16000000},
        # The smallest job of the served stream, alone: a thumbnail.
        {"name": "pt_thumb", "kind": "render", "integrator": "pt", "scene": "served", "index": 0, "width": 128,
         "height": 128, "spp": 4, "depth": 8, "film64": False},
        # The Cornell box with glass and textures, a ragged size, double-precision film.
        {"name": "pt_cornell", "kind": "render", "integrator": "pt", "scene": "cornell", "width": 321, "height": 243,
         "spp": 9, "depth": 8, "film64": True},
        # An ordinary path-traced job: served scene 4 (139k triangles, 335 instances).
        {"name": "pt_served", "kind": "render", "integrator": "pt", "scene": "served", "index": 4, "width": 512,
         "height": 512, "spp": 16, "depth": 8, "film64": False},
        # The smallest bidirectional job of the served stream.
        {"name": "bdpt_thumb", "kind": "render", "integrator": "bdpt", "scene": "served", "index": 1, "width": 128,
         "height": 128, "spp": 4, "depth": 8, "film64": False},
        # The bidirectional benchmark scene: path length 10, double-precision film, more than one batch.
        {"name": "bdpt_room", "kind": "render", "integrator": "bdpt", "scene": "room", "width": 512, "height": 512,
         "spp": 16, "depth": 10, "film64": True},
        # A gradient-domain render with its default reconstruction (200 SOR iterations).
        {"name": "gdpt_room", "kind": "render", "integrator": "gdpt", "scene": "room", "width": 512, "height": 512,
         "spp": 8, "depth": 8, "film64": False},
        # The reconstruction alone, at the benchmark's size and tolerance (CG with FP64 refinement).
        {"name": "poisson_cg", "kind": "poisson", "solver": "cg", "width": 1024, "height": 1024},
        # Continuous batching: a backlog of mixed jobs of the served stream.
        {"name": "serve_mix", "kind": "serve", "jobs": 12},
        # Film output: tone mapping and gamma of a finished frame.
        {"name": "rgb8_frame", "kind": "rgb8", "tone_mapper": "reinhard_extended", "width": 1921, "height": 1081},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "render", "render", "render", "render", "render", "poisson", "serve",
                       "rgb8"])
    if kind == "rays":
        case = {"kind": kind, "query": rng.choice(["closest", "any"]), "scene": rng.choice(["room", "soup"]),
                "count": _log_int(rng, 1000, 12_000_000) | 1}
        if case["scene"] == "soup":
            case["triangles"] = _log_int(rng, 10_000, 1_000_000)
        return case
    if kind == "render":
        case = {"kind": kind, "integrator": rng.choice(["pt", "pt", "bdpt", "gdpt"]),
                "scene": rng.choice(["cornell", "served", "served", "room"])}
        if case["scene"] == "served":
            case["index"] = rng.randrange(7)
        case["width"] = _log_int(rng, 100, 600)
        case["height"] = _log_int(rng, 100, 500)
        most = 1_000_000 if case["integrator"] == "bdpt" else 3_000_000
        case["spp"] = _log_int(rng, 2, max(3, min(16, most // (case["width"] * case["height"]))))
        case["depth"] = rng.choice([6, 8, 10])
        case["film64"] = rng.random() < 0.3
        return case
    if kind == "poisson":
        return {"kind": kind, "solver": rng.choice(["sor", "cg"]), "width": _log_int(rng, 40, 1024),
                "height": _log_int(rng, 40, 1024)}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randrange(4, 11)}
    return {"kind": kind, "tone_mapper": rng.choice(["clamp", "reinhard", "reinhard_extended"]),
            "width": _log_int(rng, 100, 2200), "height": _log_int(rng, 100, 1300)}


# ------------------------------------------------------------------ inputs --
def _scene_data(case, seed):
    """(scene, camera) of the case; the camera is None for the soup."""
    if case["scene"] == "soup":
        return scenes.triangle_soup(case["triangles"], seed=seed), None
    if case["scene"] == "room":
        return scenes.room(seed=seed)
    if case["scene"] == "cornell":
        return scenes.cornell_box(seed, glass=True, textured=True)
    return scenes.served_scene(case["index"], seed=seed)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform_directions(n, gen):
    d = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float32)
    return d / d.norm(dim=1, keepdim=True)


def _rays(case, seed):
    """(org_tmin, dir_tmax) float32 CUDA arrays."""
    n, gen = case["count"], _generator(seed)
    room = case["scene"] == "room"
    lo = torch.tensor([0.1, 0.1, 0.1] if room else [0.0, 0.0, 0.0], device="cuda")
    hi = torch.tensor([9.9, 4.9, 9.9] if room else [1.0, 1.0, 1.0], device="cuda")
    o = lo + (hi - lo) * torch.rand((n, 3), generator=gen, device="cuda")
    if case["query"] == "any" and room:
        d = lo + (hi - lo) * torch.rand((n, 3), generator=gen, device="cuda") - o
        t_max = d.norm(dim=1, keepdim=True)
        d = d / t_max
    else:
        d = _uniform_directions(n, gen)
        t_max = torch.full((n, 1), 0.25 if case["query"] == "any" else math.inf, device="cuda")
    t_min = torch.full((n, 1), 1e-4, device="cuda")
    return torch.cat([o, t_min], 1).contiguous(), torch.cat([d, t_max], 1).contiguous()


def _integrator(name, spp, depth, seed, film64=False):
    film = abi.FILM_F64 if film64 else abi.FILM_F32
    cls, cfg = {"pt": (agentray.PathTracer, agentray.PathTracerConfig),
                "bdpt": (agentray.BidirectionalPathTracer, agentray.BdptConfig),
                "gdpt": (agentray.GradientDomainPathTracer, agentray.GdptConfig)}[name]
    return cls(cfg(spp=spp, max_depth=depth, rr_depth=3, seed=seed, film_precision=film))


def _films(case, seed):
    """Primal and gradient films as a gradient-domain render leaves them: a
    noisy image and less noisy finite differences of the same picture."""
    h, w, gen = case["height"], case["width"], _generator(seed)
    y, x = torch.meshgrid(torch.linspace(0, 6, h, device="cuda"), torch.linspace(0, 6, w, device="cuda"),
                          indexing="ij")
    phase = torch.rand(3, generator=gen, device="cuda") * 6.0
    clean = 0.6 + 0.3 * torch.sin(x[..., None] * 2 + phase) * torch.cos(y[..., None] * 3 - phase)
    primal = clean * (1 + 0.3 * torch.randn((h, w, 3), generator=gen, device="cuda"))
    gx, gy = torch.zeros_like(clean), torch.zeros_like(clean)
    gx[:, :-1] = clean[:, 1:] - clean[:, :-1]
    gy[:-1] = clean[1:] - clean[:-1]
    gx[:, :-1] += 0.05 * torch.randn((h, w - 1, 3), generator=gen, device="cuda")
    gy[:-1] += 0.05 * torch.randn((h - 1, w, 3), generator=gen, device="cuda")
    return [t.to(torch.float32).contiguous() for t in (primal, gx, gy)]


def _poisson_cfg(case):
    return agentray.integrator_cfg(abi.INTEGRATOR_GDPT, alpha=0.2,
                                   poisson_iterations=200 if case["solver"] == "sor" else 2000, sor_omega=1.6,
                                   poisson_solver=abi.POISSON_SOR if case["solver"] == "sor" else abi.POISSON_CG,
                                   poisson_tolerance=1e-6, gdpt_flags=abi.GDPT_CONSISTENT_DIVERGENCE)


_TONE = {"clamp": abi.TONEMAP_CLAMP, "reinhard": abi.TONEMAP_REINHARD,
         "reinhard_extended": abi.TONEMAP_REINHARD_EXTENDED}


def _hdr(case, seed):
    gen = _generator(seed)
    g = torch.randn((case["height"], case["width"], 3), generator=gen, device="cuda")
    return torch.exp(-1.0 + 1.2 * g).to(torch.float32).contiguous()


def _serve_jobs(case, seed):
    """Jobs of the served stream's distribution at its smaller sizes, on three scenes."""
    rng = np.random.default_rng(seed)
    return [{"scene": i % 3, "res": (128, 256, 512)[i % 3] if i % 4 else 128, "spp": (4, 16)[i % 2],
             "integrator": "bdpt" if i % 10 in (2, 5, 8) else "pt", "seed": int(rng.integers(1 << 30))}
            for i in range(case["jobs"])]


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    state = {"case": case, "ctx": ctx}
    if kind == "rays":
        data, _ = _scene_data(case, seed)
        state["scene"] = agentray.Scene(ctx, data)
        state["rays"] = _rays(case, seed)
    elif kind == "render":
        data, state["camera"] = _scene_data(case, seed)
        state["scene"] = agentray.Scene(ctx, data)
        state["integrator"] = _integrator(case["integrator"], case["spp"], case["depth"], seed, case["film64"])
        state["image"] = torch.empty(case["width"] * case["height"] * 3, dtype=torch.float32, device="cuda")
    elif kind == "serve":
        state["server"] = agentray.Server(ctx, film_budget_bytes=1 << 30, bdpt_batch_samples=1 << 19)
        state["jobs"] = _serve_jobs(case, seed)
        views = [scenes.served_scene(k, seed=seed) for k in (0, 2, 4)]
        state["views"] = [(agentray.Scene(ctx, data), cam) for data, cam in views]
        state["integrators"] = [_integrator(j["integrator"], j["spp"], 8, j["seed"]) for j in state["jobs"]]
        state["images"] = [torch.empty(j["res"] ** 2 * 3, dtype=torch.float32, device="cuda") for j in state["jobs"]]
    elif kind == "poisson":
        state["films"] = _films(case, seed)
        state["cfg"] = _poisson_cfg(case)
        state["image"] = torch.empty_like(state["films"][0])
    else:
        state["hdr"] = _hdr(case, seed)
    torch.cuda.synchronize()
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "rays":
        org, direction = state["rays"]
        if case["query"] == "any":
            return state["scene"].trace_any(org, direction)
        hits, instance = state["scene"].trace_closest(org, direction)
        return {"tuv": hits[:, :3], "prim": hits[:, 3].view(torch.int32), "instance": instance}
    if kind == "render":
        return state["integrator"].render(state["scene"], state["camera"], case["width"], case["height"],
                                          out=state["image"])
    if kind == "serve":
        server, ids = state["server"], []
        for job, integrator, image in zip(state["jobs"], state["integrators"], state["images"]):
            scene, camera = state["views"][job["scene"]]
            ids.append(server.submit(scene, camera, integrator, job["res"], job["res"], out=image))
        for job_id in ids:
            info = server.wait(job_id)
            if info["status"] != "done":
                raise RuntimeError(f"job {job_id}: {info}")
            server.forget(job_id)
        return state["images"]
    if kind == "poisson":
        primal, gx, gy = state["films"]
        h, w, _ = primal.shape
        with ctx.on_torch_stream(primal):
            agentray._lib.check(agentray.lib().ar_poisson_reconstruct(
                ctx.handle, ctypes.byref(state["cfg"]), w, h, primal.data_ptr(), gx.data_ptr(), gy.data_ptr(),
                state["image"].data_ptr(), 1, None))
        return state["image"]
    return agentray.film_to_rgb8(ctx, state["hdr"], _TONE[case["tone_mapper"]], 2.2, 1.5, 4.0)


# -------------------------------------------------------------------- work --
_TRI_BYTES, _TRI_FLOPS, _LEVEL_FLOPS = 48, 40, 24


def _triangles(case):
    if case["scene"] == "served":
        return scenes.SERVED_TRIANGLES[case["index"]]
    return {"room": 195_452, "cornell": 1_316}.get(case["scene"]) or case["triangles"]


def _ray_flops(triangles):
    # a ray descends the tree once (two box tests of 12 operations a level) and tests one triangle
    return _LEVEL_FLOPS * math.log2(triangles) + _TRI_FLOPS


def _render_work(integrator, triangles, width, height, spp):
    # per sample about 3 bounces of an extension and a shadow ray; BDPT joins two such subpaths by
    # about 12 connections; GDPT traces three paths.  Bytes: the scene once, the image once.
    rays = width * height * spp * {"pt": 6, "gdpt": 18, "bdpt": 20}[integrator]
    return triangles * _TRI_BYTES + width * height * 12, rays * (_ray_flops(triangles) + 100)


def work(case):
    kind = case["kind"]
    if kind == "rays":
        triangles = _triangles(case)
        out = 1 if case["query"] == "any" else 20
        return {"bytes": case["count"] * (32 + out) + triangles * _TRI_BYTES,
                "flops": case["count"] * _ray_flops(triangles)}
    if kind == "render":
        nbytes, flops = _render_work(case["integrator"], _triangles(case), case["width"], case["height"], case["spp"])
        return {"bytes": nbytes, "flops": flops}
    if kind == "serve":
        parts = [_render_work(j["integrator"], scenes.SERVED_TRIANGLES[(0, 2, 4)[j["scene"]]], j["res"], j["res"],
                              j["spp"]) for j in _serve_jobs(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    n = case["width"] * case["height"] * 3
    if kind == "poisson":  # three films in, one out; about 10 operations a value and iteration
        return {"bytes": 16 * n, "flops": n * 10 * (200 if case["solver"] == "sor" else 64)}
    return {"bytes": 5 * n, "flops": 20 * n}


# ------------------------------------------------------------------- exact --
def _world_triangles(data):
    """(T, 3, 3) float64 vertices of every instance's triangles, in the world."""
    parts = []
    for obj in data.objects:
        mesh = data.meshes[obj.mesh]
        # the instance is placed by the inverse transform it is traversed with
        inv = obj.inv_transform if obj.inv_transform is not None else np.linalg.inv(np.asarray(obj.transform, np.float64))
        m = np.linalg.inv(np.asarray(inv, np.float64))
        p = mesh.positions.astype(np.float64) @ m[:3, :3].T + m[:3, 3]
        parts.append(p[mesh.indices])
    return torch.from_numpy(np.concatenate(parts)).cuda()


def _exact_hits(case, seed):
    data, _ = _scene_data(case, seed)
    tri = _world_triangles(data)
    org, direction = (r.double() for r in _rays(case, seed))
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    tuv = torch.zeros((org.shape[0], 3), dtype=torch.float64, device="cuda")
    step = max(1, 24_000_000 // tri.shape[0])
    for a in range(0, org.shape[0], step):
        o, d = org[a:a + step, None, :3], direction[a:a + step, None, :3]
        d = d / d.norm(dim=2, keepdim=True)
        h = torch.cross(d.expand(-1, tri.shape[0], 3), e2[None].expand(d.shape[0], -1, 3), dim=2)
        f = 1.0 / (e1 * h).sum(2)
        s = o - v0
        u = f * (s * h).sum(2)
        q = torch.cross(s, e1[None].expand_as(s), dim=2)
        v = f * (d * q).sum(2)
        t = f * (e2 * q).sum(2)
        miss = ~((u >= 0) & (v >= 0) & (u + v <= 1) & (t >= org[a:a + step, 3:4]) & (t <= direction[a:a + step, 3:4]))
        t = torch.where(miss, math.inf, t)
        best, at = t.min(1)
        got = torch.stack([best, u.gather(1, at[:, None])[:, 0], v.gather(1, at[:, None])[:, 0]], 1)
        got[~torch.isfinite(best), 1:] = 0.0
        tuv[a:a + step] = got
    return {"tuv": tuv, "prim": None, "instance": None}


def _divergence(gx, gy):
    div = gx + gy
    div[:, 1:] -= gx[:, :-1]
    div[1:] -= gy[:-1]
    return div


def _dct_matrix(n):
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    m = torch.cos(math.pi / n * (k[None] + 0.5) * k[:, None]) * math.sqrt(2.0 / n)
    m[0] /= math.sqrt(2.0)
    return m, 2.0 - 2.0 * torch.cos(math.pi * k / n)


def _exact_poisson(case, seed):
    cfg = _poisson_cfg(case)
    alpha, omega = float(cfg.alpha), float(cfg.sor_omega)
    primal, gx, gy = (t.double() for t in _films(case, seed))
    rhs = alpha * primal - _divergence(gx, gy)
    h, w, _ = primal.shape
    if case["solver"] == "cg":  # the Neumann stencil is diagonal under the cosine transform
        (cy, ly), (cx, lx) = _dct_matrix(h), _dct_matrix(w)
        spectrum = torch.einsum("ab,bxc,dx->adc", cy, rhs, cx) / (alpha + ly[:, None, None] + lx[None, :, None])
        return torch.einsum("ab,adc,dx->bxc", cy, spectrum, cx).clamp_min(0.0)
    image = primal.clone()
    count = torch.full((h, w, 1), 4.0, dtype=torch.float64, device="cuda")
    count[0] -= 1
    count[-1] -= 1
    count[:, 0] -= 1
    count[:, -1] -= 1
    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    red = ((x + y) % 2 == 0)[..., None]
    for _ in range(int(cfg.poisson_iterations)):
        for colour in (red, ~red):
            around = torch.zeros_like(image)
            around[:, 1:] += image[:, :-1]
            around[:, :-1] += image[:, 1:]
            around[1:] += image[:-1]
            around[:-1] += image[1:]
            swept = (1.0 - omega) * image + omega * (rhs + around) / (alpha + count)
            image = torch.where(colour, swept, image)
    return image.clamp_min(0.0)


def _exact_rgb8(case, seed):
    c = _hdr(case, seed).double() * 1.5
    lum = 0.2126 * c[..., :1] + 0.7152 * c[..., 1:2] + 0.0722 * c[..., 2:]
    if case["tone_mapper"] == "reinhard":
        c = c / (1.0 + lum)
    elif case["tone_mapper"] == "reinhard_extended":
        c = c * (1.0 + lum / 16.0) / (1.0 + lum)
    return torch.clamp(c.clamp(0.0, 1.0) ** (1.0 / 2.2) * 255.0 + 0.5, max=255.0).to(torch.uint8)


def exact(case, seed):
    """What run() returns for these inputs, in 64 bits; None for the images of
    whole renders, whose paths have no closed form, and for large ray batches."""
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    if case["kind"] == "rgb8":
        return _exact_rgb8(case, seed)
    if case["kind"] == "rays" and case["query"] == "closest" and case["count"] * _triangles(case) <= 2_000_000_000:
        return _exact_hits(case, seed)
    return None

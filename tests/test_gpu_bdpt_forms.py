"""The bidirectional tracer against the oracle where the image tests are blind:
the connection's arithmetic to the last bits, and the form that traces large
batches bounce by bounce."""
import numpy as np
import pytest

import agentray
import agentray.scenes as S
import oracle as O
from agentray import _abi as A

pytestmark = pytest.mark.gpu


def _render(ctx, sc, cam, w, h, **cfg):
    bd = agentray.BidirectionalPathTracer(agentray.BdptConfig(film_precision=A.FILM_F64, **cfg))
    img = bd.render(agentray.Scene(ctx, sc), cam, w, h).rgb.astype(np.float64)
    return img, O.OracleScene(sc).render(cam, bd.cfg(), w, h, sampler=O.SAMPLER_COUNTER)


@pytest.mark.parametrize("depth", [1, 2])
def test_connections_to_smooth_conductors_keep_their_bits(ctx, depth):
    # Near its peak the GGX lobe of alpha = 0.1 turns one rounding of the half
    # vector into 1e-5 of the value, also in bright s = 1 splats, so a connection
    # must round as the oracle does.  One sample a pixel and short paths: a pixel
    # is a sum of at most 16 non-negative terms, equal but for the last bit of
    # their weights (FP64 sums rounded to f32) and added in f32 by the oracle, so
    # it agrees to (16 + 4) 2^-24 = 1.2e-6.  Up to 1 pixel in 5000 may differ by
    # a tie between two surfaces.
    sc, cam = S.room(seed=6, sphere_levels=(3, 3, 2, 2), n_boxes=40)
    smooth = [m for k, m in enumerate(sc.materials) if k % 2 and m.emitter_light < 0]
    for m in smooth:
        m.kind, m.roughness, m.f0 = A.MATERIAL_CONDUCTOR, 0.1, (0.9, 0.8, 0.7)
    assert len(smooth) > 3
    img, ref = _render(ctx, sc, cam, 320, 240, spp=1, max_depth=depth, rr_depth=depth + 1, seed=3)
    assert ref.max() > 0
    off = (np.abs(img - ref) > 1.2e-6 * ref).any(axis=2)
    assert off.mean() <= 1 / 5000, (off.sum(), off.mean())


@pytest.mark.parametrize("point_light", [False, True])
def test_large_batches_match_oracle(ctx, point_light):
    # More samples than one launch walks through all bounces (1.5 a lane of its
    # grid), so extension and vertices run bounce by bounce: glass and textures,
    # quad and point light, at the image tests' bars.
    import torch
    line = torch.cuda.get_device_properties(0).multi_processor_count * 5 * 128 * 3 // 2
    sc, cam = S.cornell_box(2, point_light=point_light, glass=True, textured=True)
    w, h = 211, line // 4 // 211 + 2
    assert w * h * 4 > line
    img, ref = _render(ctx, sc, cam, w, h, spp=4, max_depth=6, rr_depth=3, seed=9)
    assert np.isfinite(img).all()
    assert abs(img.mean() - ref.mean()) / ref.mean() < 1e-4
    close = np.abs(img - ref) <= 1e-3 * np.maximum(1.0, np.abs(ref))
    assert close.all(axis=2).mean() >= 0.995, close.all(axis=2).mean()


@pytest.mark.parametrize("depth", [0, 1, 5])
def test_extend_launches_are_counted_as_launched(ctx, depth):
    # A batch of few samples traces all its bounces in one launch, a large one
    # each in its own.
    import torch
    line = torch.cuda.get_device_properties(0).multi_processor_count * 5 * 128 * 3 // 2
    sc, cam = S.cornell_box(1)
    g = agentray.Scene(ctx, sc)
    w, h = 97, line // 97 // 2
    assert w * h < line < 4 * w * h
    for spp, launches in ((1, min(depth, 1)), (4, depth)):
        agentray.BidirectionalPathTracer(agentray.BdptConfig(spp=spp, max_depth=depth, seed=2)).render(g, cam, w, h)
        stats = ctx.render_stats()
        assert stats["extend_launches"] == launches and stats["shadow_launches"] == 1, (spp, stats)


@pytest.mark.parametrize("depth,w,h,spp", [(0, 127, 1, 1), (1, 43, 3, 1), (1, 301, 211, 3), (2, 65, 1, 1),
                                           (3, 97, 5, 2), (4, 301, 211, 3), (5, 33, 31, 1)])
def test_tiles_of_every_width_match_oracle(ctx, depth, w, h, spp):
    # The connection's tiles hold the more samples the shallower the render: 128
    # up to depth 1, 64 up to 4, 32 from 5, the last one ragged, in both forms of
    # the batch.  Image tests' bars, of the pixels that see anything.
    sc, cam = S.cornell_box(2, glass=True, textured=True)
    img, ref = _render(ctx, sc, cam, w, h, spp=spp, max_depth=depth, rr_depth=3, seed=4)
    assert (w * h * spp) % 32 and np.isfinite(img).all()
    assert abs(img.sum() - ref.sum()) <= 1e-4 * ref.sum()
    close = np.abs(img - ref) <= 1e-3 * np.maximum(1.0, np.abs(ref))
    assert close.all(axis=2).mean() >= 0.995, close.all(axis=2).mean()

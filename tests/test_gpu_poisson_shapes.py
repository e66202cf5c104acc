"""Poisson solvers over the shapes that choose their launches: thin images, and
every overlap and run length that the sizes of images lead to."""
import numpy as np
import pytest

import agentray
import oracle as O
from agentray import _abi as A

pytestmark = pytest.mark.gpu


def _films(h, w):
    rng = np.random.default_rng(h * 1000 + w)
    primal = rng.uniform(0.0, 2.0, (h, w, 3)).astype(np.float32)
    gx, gy = ((rng.normal(size=(h, w, 3)) * 0.2).astype(np.float32) for _ in range(2))
    gx[:, -1] = 0
    gy[-1, :] = 0
    return primal, gx, gy


@pytest.mark.parametrize("h,w,iters", [(1, 120001, 3), (50001, 1, 4), (8, 262144, 1), (1, 20000, 5), (1, 30001, 2),
                                       (3, 90000, 2)])
def test_sor_of_thin_images_is_bit_exact(ctx, h, w, iters):
    # Whole-image half sweeps and regions, on both sides of the line between them
    # (regions of 44 pixels a side: 2728, 1137, 5958, 455, 682 and 2046 against 500 +
    # pixels / 600), against the oracle's sequential sweeps.
    films = _films(h, w)
    out, _ = agentray.poisson_reconstruct(ctx, *films, 0.2, A.POISSON_SOR, iters, 1.6)
    np.testing.assert_array_equal(out, O.poisson_sor_f32(*films, 0.2, iters, 1.6))


def _halo(h, w, sms):
    for halo in (24, 20, 16, 12):
        inner = 64 - 2 * halo
        if -(-w // inner) * -(-h // inner) <= sms:
            return halo
    return 10


_SOR = [(40, 40), (250, 250), (300, 400), (430, 430), (517, 519)]


@pytest.mark.parametrize("h,w", _SOR)
def test_sor_of_every_overlap_is_bit_exact(ctx, h, w):
    # One image for each overlap of the regions (on 148 SMs), ragged against it, a
    # last launch of fewer sweeps.
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert [_halo(*s, sms) for s in _SOR] == [24, 20, 16, 12, 10]
    films = _films(h, w)
    out, _ = agentray.poisson_reconstruct(ctx, *films, 0.2, A.POISSON_SOR, 13, 1.6)
    np.testing.assert_array_equal(out, O.poisson_sor_f32(*films, 0.2, 13, 1.6))


def _rows(h, w, sms):
    """Rows that a thread of the conjugate gradient walks down."""
    h, w = (1, h) if w == 1 else (h, w)
    width = 1
    while width < 64 and width < w:
        width *= 2
    rows = 8 if width <= 16 else 16
    while rows > 1 and -(-w // width) * -(-(-(-h // rows)) // (64 // width)) < 5 * sms:
        rows //= 2
    return rows


_CG = [(259, 200), (301, 400), (511, 513), (701, 700), (1023, 1021)]
_CG_THIN = [(1, 150001), (150001, 1), (60011, 2), (40009, 5), (3, 30001), (30001, 17), (2, 3)]


@pytest.mark.parametrize("h,w", _CG + _CG_THIN)
def test_cg_of_every_shape_reaches_the_exact_solution(ctx, h, w):
    # Every number of rows that a thread walks, ragged last runs and columns, and
    # thin images, whose blocks take several runs and whose threads several columns.
    # The Neumann stencil is diagonal under the cosine transform, which gives the
    # exact solution x*; |x - x*| <= |b - A x| / lambda_min with lambda_min = alpha
    # = 0.2 and |b - A x| <= 1e-6 |b|, plus the f32 output.
    import torch
    from scipy.fft import dctn, idctn
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert [_rows(*s, sms) for s in _CG] == [1, 2, 4, 8, 16]
    primal, gx, gy = _films(h, w)
    out, res = agentray.poisson_reconstruct(ctx, primal, gx, gy, 0.2, A.POISSON_CG, 2000, 1.6, 1e-6)
    assert 0 <= res <= 1e-6
    div = gx.astype(np.float64) + gy
    div[:, 1:] -= gx[:, :-1]
    div[1:] -= gy[:-1]
    b = float(np.float32(0.2)) * primal.astype(np.float64) + div
    ly, lx = (2 - 2 * np.cos(np.pi * np.arange(n) / n) for n in (h, w))
    spectrum = float(np.float32(0.2)) + ly[:, None, None] + lx[None, :, None]
    want = np.maximum(idctn(dctn(b, axes=(0, 1), norm="ortho") / spectrum, axes=(0, 1), norm="ortho"), 0)
    norm = np.linalg.norm(b.reshape(-1, 3), axis=0)
    assert np.all(np.abs(out - want) <= 5e-6 * norm + 2e-7 * np.abs(want))

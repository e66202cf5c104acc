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

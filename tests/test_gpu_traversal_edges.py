"""Traversal at the edges of its box tests: rays that start exactly on a node's
low face, where the slab distances are zeros of either sign."""
import numpy as np
import pytest

import agentray
import oracle as O
from agentray.scene_data import Material, Mesh, Object, SceneData

pytestmark = pytest.mark.gpu


def _grid_box(n):
    """The surface of the unit box, each face n x n quads (12 n^2 triangles)."""
    pos, idx = [], []
    for axis in range(3):
        for side in (0.0, 1.0):
            for i in range(n):
                for j in range(n):
                    q = np.empty((4, 3), np.float32)
                    q[:, axis] = side
                    q[:, (axis + 1) % 3] = np.array([i, i + 1, i + 1, i], np.float32) / n
                    q[:, (axis + 2) % 3] = np.array([j, j, j + 1, j + 1], np.float32) / n
                    k = len(pos) * 4
                    pos.append(q)
                    idx += [[k, k + 1, k + 2], [k, k + 2, k + 3]]
    return Mesh(np.concatenate(pos), np.array(idx, np.uint32))


def _low_face_rays(rng, n):
    """Rays on the box's low faces, t_min = 0: the direction leaves through the
    face, or lies in a second low face (-0.0 on its axis) and leaves through the
    first.  Coordinates are multiples of 1/4096, exact under the translations;
    none on a quad's edges or diagonal."""
    o = (rng.integers(0, 512, (n, 3)) * 8 + [1, 2, 4]).astype(np.float32) / 4096
    d = rng.normal(size=(n, 3)).astype(np.float32)
    rows, axis = np.arange(n), rng.integers(0, 3, n)
    o[rows, axis] = 0.0
    d[rows, axis] = -np.abs(d[rows, axis]) - np.float32(0.05)
    second = rows < n // 4
    other = (axis + 1) % 3
    o[rows[second], other[second]] = 0.0
    d[rows[second], other[second]] = -0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    assert np.signbit(d[rows[second], other[second]]).all()
    return o, d


@pytest.mark.parametrize("shift", [(0.0, 0.0, 0.0), (2.0, -4.0, 8.0)])
def test_rays_that_start_on_a_low_face(ctx, shift):
    # The hit at t = 0 is the triangle under the origin (t >= t_min), found by the
    # oracle too where no direction component is zero (there its slab test, as the
    # reference's, multiplies 0 by an infinite reciprocal), so the traversal must
    # find it, in closest and any hit: a far plane at -0 against a near limit of
    # +0 is a hit.
    sc = SceneData()
    mesh = sc.add_mesh(_grid_box(8))
    mat = sc.add_material(Material())
    m = np.eye(4, dtype=np.float32)
    m[:3, 3] = shift
    sc.add_object(Object(mesh, [mat], m))
    far = np.eye(4, dtype=np.float32)
    far[:3, 3] = (64.0, 64.0, 64.0)
    sc.add_object(Object(mesh, [mat], far))
    o, d = _low_face_rays(np.random.default_rng(7), 4000)
    ot = np.concatenate([o + np.asarray(shift, np.float32), np.zeros((len(o), 1), np.float32)], 1)
    dt = np.concatenate([d, np.full((len(o), 1), 1e-3, np.float32)], 1)
    one = slice(len(o) // 4, None)  # rays on one low face
    osc = O.OracleScene(sc)
    ref = osc.trace_closest(ot[one], dt[one])
    assert (ref["inst"] == 0).all() and (ref["t"] == 0).all() and osc.trace_any(ot[one], dt[one]).all()
    g = agentray.Scene(ctx, sc)
    hits, inst = g.trace_closest(ot, dt)
    np.testing.assert_array_equal(inst, 0)
    np.testing.assert_array_equal(hits[:, 0], 0.0)
    np.testing.assert_array_equal(hits[one, 3].view(np.uint32), ref["prim"])
    assert g.trace_any(ot, dt).all()

"""calc_deltas at the edges of its forms, against the oracle bit for bit: one launch a
step (a block's share of one to four vertices, one round of blocks and several) and
three (from 16,385 vertices), on folded sheets, with vertices on and off the mesh, few
rows against many triangles and the other way round."""

import numpy as np
import pytest

from oracle import deltas as od

pytestmark = pytest.mark.gpu

RESIDENT = 152 * 8


def _rows(m, rings, seed):
    from mplicits_gb300 import synthetic
    rng = np.random.default_rng(seed)
    pos, nrm, faces = synthetic.surface_mesh(rings, 2 * rings)
    pos = (pos + rng.normal(0, 0.3 * np.pi * 0.6 / rings, pos.shape)).astype(np.float32)
    i = rng.integers(0, pos.shape[0], m)
    V = np.concatenate([pos[i], nrm[i]], 1).astype(np.float32)
    V[::3, :3] += rng.normal(0, 0.01, V[::3, :3].shape).astype(np.float32)
    V[1::5, 3:] = rng.normal(size=V[1::5, 3:].shape)
    V[7::97, 3:] = 0.0  # no normal
    return V, pos, faces


@pytest.mark.parametrize("m", [1, 2, 3, 5, RESIDENT - 1, RESIDENT, RESIDENT + 1, 2 * RESIDENT + 1,
                               3 * RESIDENT + 2, 4 * RESIDENT, 4 * RESIDENT + 3, 16383, 16384,
                               16385])
@pytest.mark.parametrize("rings,eps", [(8, 2e-4), (24, 2e-2)])
def test_vertex_counts(m, rings, eps):
    from mplicits_gb300.scene import RaycastingScene, calc_deltas
    V, pos, faces = _rows(m, rings, m)
    out, it = calc_deltas(V, RaycastingScene(pos, faces), max_delta=0.3, n_iters=40, eps=eps,
                          return_iterations=True)
    want, it_ref = od.calc_deltas(V, pos, faces, 0.3, 40, eps=eps)
    assert it == it_ref
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("m", [1, 300, 5000, 20000])
def test_few_rows_of_a_dense_mesh(m):
    from mplicits_gb300.scene import RaycastingScene, calc_deltas
    V, pos, faces = _rows(m, 160, 1)
    out, it = calc_deltas(V, RaycastingScene(pos, faces), return_iterations=True)
    want, it_ref = od.calc_deltas(V, pos, faces, cell=0.02, fast=True)
    assert it == it_ref
    np.testing.assert_array_equal(out.cpu().numpy(), want)

"""A scene's grid has at most 1024 cells along an axis, whatever cell side is asked
for: distances and calc_deltas of a thin tube with cells far too small for it, against
the oracle bit for bit."""

import numpy as np
import pytest

from oracle import deltas as od

pytestmark = pytest.mark.gpu


def _tube(n=240, m=6, length=1.4, r=5e-4):
    u, v = np.meshgrid(np.linspace(-0.5, 0.5, n) * length, np.arange(m) * 2 * np.pi / m,
                       indexing="ij")
    nrm = np.stack([0 * u, np.cos(v), np.sin(v)], -1)
    pos = np.stack([u, r * nrm[..., 1], r * nrm[..., 2]], -1)
    i, j = np.meshgrid(np.arange(n - 1), np.arange(m), indexing="ij")
    a, b = i * m + j, i * m + (j + 1) % m
    faces = np.concatenate([np.stack([a, a + m, b], -1).reshape(-1, 3),
                            np.stack([a + m, b + m, b], -1).reshape(-1, 3)])
    return (pos.reshape(-1, 3).astype(np.float32), nrm.reshape(-1, 3).astype(np.float32),
            faces.astype(np.int32))


@pytest.mark.parametrize("cell", [0.0, 1e-3, 2e-10, 1e-12, 1e-30])
def test_any_cell_side(cell):
    from mplicits_gb300.scene import RaycastingScene, calc_deltas
    pos, nrm, faces = _tube()
    scene = RaycastingScene(pos, faces, cell=cell)
    assert max(scene.info()["dims"]) <= 1024
    rng = np.random.default_rng(0)
    pts = (pos[rng.integers(0, len(pos), 500)] + rng.normal(0, 0.01, (500, 3))).astype(np.float32)
    np.testing.assert_array_equal(scene.compute_distance(pts).cpu().numpy(),
                                  od.compute_distance(pos, faces, pts))
    for sign in (1, -1):
        V = np.concatenate([pos, sign * nrm], 1)
        out, it = calc_deltas(V, scene, max_delta=0.05, n_iters=60, return_iterations=True)
        want, it_ref = od.calc_deltas(V, pos, faces, 0.05, 60)
        assert it == it_ref
        np.testing.assert_array_equal(out.cpu().numpy(), want)

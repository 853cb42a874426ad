"""calc_deltas where a block's search finds a few triangles many times: triangles that
lie in hundreds of cells each, so that the warps' lists fill up with entries of the
same ones before they are merged into the vertex's list.  Against the oracle bit for
bit, by searches of a block for every vertex and, with the vertices repeated, by warps
first.  (Of the seeds tried these gave the most wrong rows, 6 to 15, when the merge lost
triangles without ending the certified stretch.)"""

import numpy as np
import pytest

from oracle import deltas as od

pytestmark = pytest.mark.gpu


def _case(seed):
    rng = np.random.default_rng(100000 + seed)
    nt = int(rng.integers(6, 60))
    size = float(rng.choice([0.03, 0.06, 0.1, 0.15, 0.3]))
    cell = size * float(rng.choice([0.1, 0.15, 0.2, 0.3, 0.5]))
    spread = float(rng.choice([0.1, 0.2, 0.5]))
    assert int(rng.integers(0, 3)) == 2  # triangles across one axis
    max_delta = float(rng.choice([0.2, 0.4, 0.8]))
    eps = float(rng.choice([2e-4, 2e-3, 1e-2]))
    iters = int(rng.choice([20, 60, 100]))
    c = rng.uniform(-spread, spread, (nt, 1, 3))
    pos = c + rng.normal(0, size, (nt, 3, 3))
    pos[:, :, 2] = c[:, :, 2]
    pos = pos.reshape(-1, 3).astype(np.float32)
    faces = np.arange(3 * nt, dtype=np.int32).reshape(-1, 3)
    m = 16000
    t, w = rng.integers(0, nt, m), rng.dirichlet([1, 1, 1], m)
    p = (pos.reshape(nt, 3, 3)[t] * w[:, :, None]).sum(1)
    n = rng.normal(size=(m, 3))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    V = np.concatenate([p, n], 1).astype(np.float32)
    return V, pos, faces, cell, dict(max_delta=max_delta, n_iters=iters, eps=eps)


@pytest.mark.parametrize("copies", [1, 3])
@pytest.mark.parametrize("seed", [4217, 1714, 3155, 1329, 3622, 7177, 6220, 4922, 7106, 6972])
def test_merged_lists(seed, copies):
    from mplicits_gb300.scene import RaycastingScene, calc_deltas
    V, pos, faces, cell, args = _case(seed)
    scene = RaycastingScene(pos, faces, cell=cell)
    got = calc_deltas(np.tile(V, (copies, 1)), scene, **args).cpu().numpy()
    want, _ = od.calc_deltas(V, pos, faces, args["max_delta"], args["n_iters"], eps=args["eps"])
    np.testing.assert_array_equal(got, np.tile(want, (copies, 1)))

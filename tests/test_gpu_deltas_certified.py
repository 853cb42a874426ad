"""calc_deltas' certified stretches against the oracle's search at every step,
bit for bit, on meshes where the certificate is tight, void or long: folded
surfaces, slivers and degenerate triangles, eps from 0 to larger than a step,
random normals, normals that do not normalise to unit length, vertices off the
mesh, and vertex counts around the block size."""

import numpy as np
import pytest
import torch

from oracle import deltas as od

pytestmark = pytest.mark.gpu


def _case(name):
    from mplicits_gb300 import synthetic
    rng = np.random.default_rng(5)
    pos, nrm, faces = synthetic.surface_mesh(20, 37)
    edge = np.pi * 0.6 / 20
    if name == "folded":
        pos = pos + rng.normal(0, 0.4 * edge, pos.shape)
    elif name == "slivers":
        pos = pos * np.array([1.0, 1.0, 2e-3])
        pos[:, 1] += 0.3 * pos[:, 0]
    elif name == "degenerate":
        faces = np.concatenate([faces, faces[:50][:, [0, 0, 1]], faces[50:90][:, [2, 2, 2]]])
    elif name == "random_normals":
        nrm = rng.normal(size=nrm.shape)
    elif name == "odd_normals":
        nrm = nrm * np.float32(1.0)
        nrm[::3] *= 3e-23   # squares are subnormal: not of unit length afterwards
        nrm[1::7] = 0.0     # 0 / 0
        nrm[2::11] *= 1e25  # squares overflow
    V = np.concatenate([pos, nrm], 1).astype(np.float32)
    if name == "off_mesh":
        V[::2, :3] += rng.normal(0, 0.3 * edge, V[::2, :3].shape).astype(np.float32)
    return V, pos.astype(np.float32), faces.astype(np.int32)


@pytest.mark.parametrize("name", ["plain", "folded", "slivers", "degenerate", "random_normals",
                                  "odd_normals", "off_mesh"])
@pytest.mark.parametrize("eps,max_delta", [(2e-4, 0.3), (0.0, 0.1), (2e-2, 0.5), (1e-6, 0.05)])
def test_equals_oracle(name, eps, max_delta):
    from mplicits_gb300.scene import RaycastingScene, calc_deltas
    V, pos, faces = _case(name)
    for m in (1, 255, 256, 257, V.shape[0]):
        out, it = calc_deltas(V[:m], RaycastingScene(pos, faces), max_delta=max_delta, n_iters=60,
                              eps=eps, return_iterations=True)
        want, it_ref = od.calc_deltas(V[:m], pos, faces, max_delta, 60, eps=eps)
        assert it == it_ref
        np.testing.assert_array_equal(out.cpu().numpy(), want)


def test_repeated_calls_and_cells():
    """A call leaves nothing behind: a second one on other vertices and grids
    of other cell sizes equals the oracle too."""
    from mplicits_gb300.scene import RaycastingScene, calc_deltas
    V, pos, faces = _case("folded")
    want = {s: od.calc_deltas(V[::s].copy(), pos, faces, 0.2, 40)[0] for s in (1, 2)}
    for cell in (0.0, 0.02, 0.5):
        scene = RaycastingScene(pos, faces, cell=cell)
        for s in (1, 2, 1):
            got = calc_deltas(torch.from_numpy(V[::s].copy()), scene, max_delta=0.2, n_iters=40)
            np.testing.assert_array_equal(got.cpu().numpy(), want[s])

"""GPU marching cubes on the smallest grids: one partial strip of the counting
kernel's four rows, one full strip, and a strip with one or two rows left over, on
noise with exact iso values, bit for bit the CPU restatement (oracle/mc.c)."""

import numpy as np
import pytest

from test_gpu_mc import _assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("seed", [0, 1, 2, 3])
def test_noise(lib, N, seed):
    rng = np.random.default_rng(100 * N + seed)
    S = rng.standard_normal((N, N, N)).astype(np.float32)
    S[rng.random(S.shape) < 0.1] = 0.0
    _assert_same(S)

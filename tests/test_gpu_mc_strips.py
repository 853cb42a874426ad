"""GPU marching cubes at the edges of the counting kernel's eight-row strips and
of the 128- and 512-point steps along a line, on noise (every case, dense lines)
and on noise between wide one-signed stretches: bit for bit the CPU restatement
(oracle/mc.c)."""

import numpy as np
import pytest

from test_gpu_mc import _assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [7, 8, 9, 15, 16, 17, 31, 32, 33, 124, 127, 128, 129, 132])
def test_noise(lib, N):
    rng = np.random.default_rng(N)
    S = rng.standard_normal((N, N, N)).astype(np.float32)
    S[rng.random(S.shape) < 0.05] = 0.0  # exact iso values
    _assert_same(S)


@pytest.mark.parametrize("N", [65, 128, 130, 257, 260])
@pytest.mark.parametrize("sign", [-1.0, 1.0])
def test_one_signed_stretches(lib, N, sign):
    rng = np.random.default_rng(N)
    S = np.full((N, N, N), sign, np.float32)
    for _ in range(40):
        i, j, k = rng.integers(0, N - 3, 3)
        S[i:i + 3, j:j + 3, k:k + 3] = rng.standard_normal((3, 3, 3)).astype(np.float32)
    S[-1, -1, -1], S[0, 0, -1], S[-1, 0, 0] = -sign, -sign, -sign
    _assert_same(S)

"""Rows of hidden weights far below their layer's largest keep their own relative
precision in the FP32 level kernel.

Layer 1 has a few rows of the usual size and the others 2^-s of it, without a
bias; layer 2 takes their activations 2^s times, so that the output depends on
them as much for every s.  The scales are powers of two, which change no relative
rounding: the 16-bit parts of the scaled rows are those of s = 0, and the sines of
their phases (below 2^-4 at s = 0, where the sine is nearly linear) are rounded to
the same relative size.  So the error against float64, in the 2-norm over 20,000
points, is that of s = 0; twice that is allowed, for the roundings that differ."""

import functools

import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(m, x):
    x = x.double()
    for blk, w in zip(m.net[:-1], m.omegas()):
        x = torch.sin(w * (x @ blk[0].weight.double().T + blk[0].bias.double()))
    last = m.net[-1][0]
    return (x @ last.weight.double().T + last.bias.double())[:, 0]


@functools.lru_cache(maxsize=None)
@torch.no_grad()
def _error(width, s):
    from mplicits_gb300.model import SIREN, level_forward
    torch.manual_seed(width)
    m = SIREN(3, 1, [width] * 3, w0=30).cuda()
    big = torch.zeros(width, dtype=torch.bool, device="cuda")
    big[::37] = True
    scale = torch.where(big, 1.0, 2.0 ** -s)
    one, two = m.net[1][0], m.net[2][0]
    one.weight.mul_(torch.where(big, 1.0, 2.0 ** -6)[:, None] * scale[:, None])
    one.bias.mul_(big)
    two.weight.mul_(torch.where(big, 2.0 ** -6, 16.0)[None] / scale[None])
    x = torch.rand(20000, 3, device="cuda") * 2 - 1
    return float((level_forward(m, x, precision="fp32").double() - _exact(m, x)).norm())


@pytest.mark.parametrize("s", [8, 13, 14, 15, 16, 20, 25, 32, 50])
@pytest.mark.parametrize("width", [64, 100, 256])
def test_small_rows(width, s):
    assert _error(width, s) <= 2 * _error(width, 0)

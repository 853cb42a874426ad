"""Layers whose activations are small: the FP32 level kernel is as close to float64
as the FP32 FMA kernel, which the value of level_gradient comes from.

Layer 1's phases are t of the usual (without a bias; a few rows keep theirs), all of
it times 2^-s, and layer 2 takes its activations as many times larger.  Both kernels
round operands and sums by 2^-24 of values of one size, in another order: half as
much again is allowed, in the 2-norm over 20,000 points."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(m, x):
    x = x.double()
    for blk, w in zip(m.net[:-1], m.omegas()):
        x = torch.sin(w * (x @ blk[0].weight.double().T + blk[0].bias.double()))
    last = m.net[-1][0]
    return (x @ last.weight.double().T + last.bias.double())[:, 0]


@pytest.mark.parametrize("s", [0, 10, 30])
@pytest.mark.parametrize("t", [0, -2, -4, -6])
@pytest.mark.parametrize("width", [64, 100, 128, 200, 256])
@torch.no_grad()
def test_as_close_as_the_fma_kernel(width, t, s):
    from mplicits_gb300.grad import level_gradient
    from mplicits_gb300.model import SIREN, level_forward
    torch.manual_seed(width + t)
    m = SIREN(3, 1, [width] * 3, w0=30).cuda()
    big = torch.zeros(width, dtype=torch.bool, device="cuda")
    big[::37] = True
    one, two = m.net[1][0], m.net[2][0]
    scale = torch.where(big, 1.0, 2.0 ** (t - s))
    one.weight.mul_(scale[:, None])
    one.bias.mul_(big)
    two.weight.mul_(torch.where(big, 2.0 ** t, min(16.0, 2.0 ** -t) * 2.0 ** s)[None])
    x = torch.rand(20000, 3, device="cuda") * 2 - 1
    want = _exact(m, x)
    fma = (level_gradient(m, x, precision="fp32")[0].double() - want).norm()
    got = (level_forward(m, x, precision="fp32").double() - want).norm()
    assert got <= 1.5 * fma


def test_large_activations_of_small_rows():
    """Rows whose weights all pull one way reach their bound, 16 times the usual
    activation of such a row: inputs that saturate the first layer."""
    from mplicits_gb300.grad import level_gradient
    from mplicits_gb300.model import SIREN, level_forward
    torch.manual_seed(1)
    m = SIREN(3, 1, [256] * 3, w0=30).cuda()
    with torch.no_grad():
        m.net[0][0].weight.mul_(1e-3)
        m.net[0][0].bias.fill_(torch.pi / 60)       # sin(30 b) = 1
        m.net[1][0].weight.fill_(2.0 ** -15)        # equal weights: the bound is 16 norms
        m.net[1][0].weight.mul_(1 + 0.1 * torch.rand(256, 1, device="cuda"))
        m.net[1][0].bias.zero_()
        m.net[2][0].weight.mul_(4.0)
        x = torch.rand(20000, 3, device="cuda") * 2 - 1
        want = _exact(m, x)
        fma = (level_gradient(m, x, precision="fp32")[0].double() - want).norm()
        got = (level_forward(m, x, precision="fp32").double() - want).norm()
        assert got <= 1.5 * fma

"""Bias, first-layer and output-layer gradients of the tensor-core training step
against float64 sums of the very tiles and seeds the step wrote, at the edges of
32-point tiles, of 64-row blocks and of the sums of 16 blocks.

Tolerance: a sum passes through fewer than 256 FP32 additions in a row (a
lane's or thread's own, the shuffles, one atomic per CTA), so it is within
256 * 2^-24 of the sum of its terms' magnitudes."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 16 * 76, 16 * 76 * 16 + 1, 32 * 152 * 9 + 5])
@pytest.mark.parametrize("widths", [(256,) * 3, (128,) * 3, (256,) * 2, (100,) * 2])
def test_sums(widths, n):
    from mplicits_gb300 import capi
    from mplicits_gb300.model import SIREN
    from mplicits_gb300.train import ResidualTrainer
    torch.manual_seed(n)
    m = SIREN(3, 1, list(widths), w0=30, precision="bf16").cuda()
    x = torch.rand(n, 3, device="cuda") * 2 - 1
    normals = torch.nn.functional.normalize(x, dim=1)
    sdf = torch.rand(n, 1, device="cuda") * 0.04 - 0.02
    tr = ResidualTrainer(m, [], precision="bf16")
    _, grads = tr.loss_and_grads(x, normals, sdf)
    torch.cuda.synchronize()
    assert capi.device_status() == capi.MPL_OK
    grads = [g.double() for g in grads]
    nh, wp, w = len(widths) - 1, 256 if widths[0] > 128 else 128, widths[0]
    rows = (n + 31) // 32 * 128
    off = (-tr._tc_buf.data_ptr()) % 256
    tiles = tr._tc_buf[off:off + 2 * (nh + 1) * rows * wp * 2].view(torch.bfloat16)
    tiles = tiles.view(2, nh + 1, rows // 64, wp // 8, 64, 8).permute(0, 1, 2, 4, 3, 5)
    s, dz = tiles.reshape(2, nh + 1, rows // 4, 4, wp)[:, :, :n, :, :w].double()
    seeds = tr._tc_seeds[:n].double()

    def close(got, terms, scale=1.0):
        want, bound = scale * terms.sum(0), scale * terms.abs().sum(0)
        err = (got.reshape(want.shape) - want).abs()
        assert bool((err <= 256 * 2.0 ** -24 * bound).all()), float((err / bound).max())

    om = 30.0
    for l in range(nh + 1):
        close(grads[2 * l + 1], dz[l][:, 0], om)
    for c in range(3):
        terms = torch.cat([dz[0][:, 0] * x[:, c:c + 1].double(), dz[0][:, 1 + c]])
        close(grads[0][:, c], terms, om)
    close(grads[-2], (seeds[:, :, None] * s[nh]).reshape(4 * n, w))
    close(grads[-1].reshape(1), seeds[:, :1])

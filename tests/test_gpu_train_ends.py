"""FP32 first- and output-layer gradients against float64: all points are the same
one with a seed on its value only, so that every term of a sum is the same number
and its rounding errors add up.  Sixteen points follow each other in a sum (more
beyond 38,912 points), then four groups, then one atomic add per 64 points; each
addition rounds by 2^-24 of the sum, the term itself by 2^-22 (a product and
CUDA's sinf, 2 ulp)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 129, 1000, 5000, 15000, 196608, 300001])
@pytest.mark.parametrize("width", [64, 128, 256])
def test_first_and_output_layer(width, n):
    from mplicits_gb300 import train
    from mplicits_gb300.model import SIREN
    torch.manual_seed(4)
    m = SIREN(3, 1, [width] * 2, w0=30).cuda()
    x = torch.tensor([[0.31, -0.47, 0.12]], device="cuda").expand(n, 3).contiguous()
    grads = [g.double() for g in train.param_grads(m, x, df=torch.full((n,), 0.7, device="cuda"))]
    sc = train._scratch(m, n, x.device)
    pre, da = (t[:2 * n * 4 * width].view(2, n, 4, width) for t in (sc.pre, sc.da))
    blocks = min(-(-n // 64), 4 * 152)
    tol = (-(-n // (4 * blocks)) + 4 + blocks) * 2.0 ** -24 + 2.0 ** -22
    dv = da[0, 0, 0].double()
    last = torch.sin((30.0 * pre[1, 0, 0]).double())  # the phase as the kernel rounds it
    seed = float(torch.tensor(0.7))
    for got, term in ((grads[0], dv[:, None] * x[:1].double()), (grads[1], dv),
                      (grads[-2], seed * last[None])):
        want = n * term
        assert bool(((got - want).abs() <= tol * want.abs()).all())
    assert abs(float(grads[-1]) - n * seed) <= 2.0 ** -23 * n * seed

"""FP32 hidden weight and bias gradients of many points: the serial FP32 sums of
the kernel end after 4096 points, whatever the batch, so the error against
float64 has a bound that does not grow with it.

All points are the same one, with a seed on its value only: every term of a sum
is the same number, whose rounding errors add up instead of averaging out, and
the exact gradient is that number times n.  At most 4096 of them follow each
other in a sum and at most n / 4096 + 152 partial sums in the atomic adds, each
addition rounding by 2^-24 of the sum; the term itself is within 2^-22 (a product
and CUDA's sinf, 2 ulp)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,hidden,n", [(256, 7, 1 << 18), (256, 3, 1 << 20), (64, 3, 1 << 21)])
def test_error_does_not_grow_with_the_batch(width, hidden, n):
    from mplicits_gb300 import train
    from mplicits_gb300.model import SIREN
    torch.manual_seed(3)
    m = SIREN(3, 1, [width] * hidden, w0=30).cuda()
    x = torch.tensor([[0.31, -0.47, 0.12]], device="cuda").expand(n, 3).contiguous()
    df = torch.full((n,), 0.7, device="cuda")
    grads = train.param_grads(m, x, df=df)
    sc = train._scratch(m, n, x.device)
    L, nh = hidden + 1, hidden - 1
    pre = sc.pre[:(nh + 1) * n * 4 * width].view(nh + 1, n, 4, width)[:, 0, 0].clone()
    da = sc.da[:(nh + 1) * n * 4 * width].view(nh + 1, n, 4, width)[:, 0, 0].double()
    tol = (4096 + n / 4096 + 152) * 2.0 ** -24 + 2.0 ** -22
    for l in range(1, L - 1):
        s = torch.sin((30.0 * pre[l - 1]).double())  # the phase as the kernel rounds it
        want = n * da[l][:, None] * s[None, :]
        assert bool(((grads[2 * l].double() - want).abs() <= tol * want.abs()).all()), l
        want = n * da[l]
        assert bool(((grads[2 * l + 1].double() - want).abs() <= tol * want.abs()).all()), l
    del sc
    m._train_scratch = None

"""Half tiles of the FP32 gradient and backward kernels (half_tiles in level.cuh)
against full ones, at the edges of tiles and of the rule: every row's sums run
in the same order in both, so values, gradients, band lists and adjoints are
equal bit for bit (tolerance 0)."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

SMS = 152
NS = [1, 15, 16, 17, 500, 16 * SMS, 16 * SMS + 1, 32 * SMS + 1, 32 * SMS + 8 * SMS,
      32 * SMS + 8 * SMS + 1, 6 * 32 * SMS + 77]


def _net(dims):
    from mplicits_gb300.model import SIREN
    torch.manual_seed(5)
    return SIREN(3, 1, list(dims), w0=30.0).cuda()


def _points(n):
    g = torch.Generator("cuda").manual_seed(7)
    return torch.rand(n, 3, device="cuda", generator=g) * 2 - 1


@pytest.mark.parametrize("n", NS)
@pytest.mark.parametrize("dims", [(64, 64), (128, 128), (100,) * 3, (256,) * 3])
def test_gradient(dims, n):
    """A device-side count takes full tiles."""
    from mplicits_gb300.grad import level_gradient
    m, x = _net(dims), _points(n)
    count = torch.tensor([n], dtype=torch.int32, device="cuda")
    with torch.no_grad():
        S, G = level_gradient(m, x, precision="fp32")
        Sf, Gf = level_gradient(m, x, precision="fp32", n_dev=count, n=n)
    assert torch.equal(S, Sf) and torch.equal(G, Gf)


@pytest.mark.parametrize("n", [1, 17, 500, 6000])
def test_band_and_accumulate(n):
    from mplicits_gb300 import capi
    m, x = _net((128, 128)), _points(n)
    net, packed = m.packed()
    pts = capi.MplPoints(kind=capi.MPL_POINTS_XYZ, xyz=x.data_ptr())
    runs = []
    for count in (None, torch.tensor([n], dtype=torch.int32, device="cuda")):
        S = torch.linspace(-0.1, 0.1, n, device="cuda")
        G = torch.ones(n, 3, device="cuda")
        out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        n_out = torch.zeros(1, dtype=torch.int32, device="cuda")
        band = capi.MplBand(delta=0.05, out_index=out.data_ptr(), count_dev=n_out.data_ptr(),
                            capacity=n)
        capi.check(capi.load().mpl_level_gradient(
            ctypes.byref(net), capi.ptr(packed), ctypes.byref(pts), None, capi.ptr(count), n,
            capi.ptr(S), capi.ptr(G), capi.MPL_ACCUMULATE, ctypes.byref(band), capi.MPL_FP32,
            capi.stream_ptr()), "mpl_level_gradient")
        k = int(n_out)
        runs.append((S, G, out[:k].sort().values))
    (S, G, b), (Sf, Gf, bf) = runs
    assert torch.equal(S, Sf) and torch.equal(G, Gf) and torch.equal(b, bf)
    assert torch.equal(b, torch.nonzero(S.abs() < 0.05).flatten().int())


@pytest.mark.parametrize("width", [64, 128, 256])
@pytest.mark.parametrize("n", [1, 17, 16 * SMS, 32 * SMS + 136, 32 * SMS + 8 * SMS])
def test_backward(width, n):
    """Adjoint rows of n points against those of the first n of 32 * 152 * 7
    points, seven full waves of full tiles."""
    from mplicits_gb300 import train
    m = _net((width,) * 3)
    full = 7 * 32 * SMS
    x, df, dg = _points(full), _points(full)[:, 0].contiguous(), _points(full)
    rows = []
    for k in (full, n):
        train.param_grads(m, x[:k], df=df[:k], dg=dg[:k])
        sc = train._scratch(m, k, x.device)
        rows.append(sc.da[:3 * k * 4 * width].view(3, k, 4, width)[:, :n].clone())
    assert torch.equal(rows[0], rows[1])

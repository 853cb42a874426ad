"""The FP32 level kernel on split FP16 operands (level_split.cuh) at the sizes,
shapes and values where it can go wrong: tile and wave edges, every padded
width and depth, rows of very different magnitude, zero rows, phases beyond its
unwrapped range, infinities and NaN, index lists with bands.

Tolerances: a level of the reference's initialisation is within 1e-5 of float64
(the bound the plain FP32 form has against the reference); with u the float32
unit roundoff 2^-24, phases of size z carry about z u of rounding, which the
scaled cases below multiply by their scale."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(dims, seed, w0=30.0):
    from mplicits_gb300.model import SIREN
    torch.manual_seed(seed)
    return SIREN(3, 1, list(dims), w0=w0).cuda().eval()


@torch.no_grad()
def _bound(m):
    return float(m.net[-1][0].weight.abs().sum() + m.net[-1][0].bias.abs().sum())


@torch.no_grad()
def _exact(m, x):
    x = x.double()
    for blk, w in zip(m.net[:-1], m.omegas()):
        x = torch.sin(w * torch.nn.functional.linear(x, blk[0].weight.double(),
                                                     blk[0].bias.double()))
    last = m.net[-1][0]
    return torch.nn.functional.linear(x, last.weight.double(), last.bias.double())[:, 0]


def _run(m, x, **kw):
    from mplicits_gb300.model import level_forward
    with torch.no_grad():
        return level_forward(m, x, precision="fp32", **kw)


def _points(n, seed=0, scale=1.0):
    g = torch.Generator("cuda").manual_seed(seed)
    return (torch.rand(n, 3, device="cuda", generator=g) * 2 - 1) * scale


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 152 * 128 - 1, 152 * 128, 152 * 128 + 1,
                               2 * 152 * 128 + 77])
@pytest.mark.parametrize("width", [64, 128, 256])
def test_tile_edges(n, width):
    m = _net([width] * 3, 1)
    x = _points(n)
    assert (_run(m, x).double() - _exact(m, x)).abs().max() <= 1e-5


@pytest.mark.parametrize("dims", [[256, 256], [256] * 4, [256] * 5, [256] * 6, [256] * 7,
                                  [64, 64], [64] * 7, [128] * 5, [1, 1], [5, 3, 7], [65, 33],
                                  [200, 100, 256], [129, 255, 250]])
def test_widths_and_depths(dims):
    m = _net(dims, 2)
    x = _points(1000)
    assert (_run(m, x).double() - _exact(m, x)).abs().max() <= 1e-5


def test_rows_of_different_magnitude():
    """Rows scaled by 2^0 .. 2^-15 keep their own relative precision, a zero row
    and a zero layer are exact."""
    m = _net([256, 256, 256], 3)
    with torch.no_grad():
        w = m.net[1][0].weight
        w.mul_(2.0 ** -(torch.arange(256, device="cuda") % 16)[:, None].float())
        w[7] = 0.0
        m.net[1][0].bias.mul_(2.0 ** -(torch.arange(256, device="cuda") % 16).float())
        # the small rows count as much as the others in the next layer
        m.net[2][0].weight.mul_(2.0 ** (torch.arange(256, device="cuda") % 16)[None].float())
    x = _points(5000)
    assert (_run(m, x).double() - _exact(m, x)).abs().max() <= 1e-4  # weights x 2^15, phases x ~10
    with torch.no_grad():
        m.net[1][0].weight.zero_()
    assert (_run(m, x).double() - _exact(m, x)).abs().max() <= 1e-4


@pytest.mark.parametrize("scale", [1e-30, 1e-3, 50.0])
def test_weight_scales(scale):
    m = _net([128, 128, 128], 4)
    with torch.no_grad():
        m.net[1][0].weight.mul_(scale)
        m.net[2][0].weight.mul_(scale)
    x = _points(3000)
    tol = 1e-5 * max(1.0, scale * scale)
    assert (_run(m, x).double() - _exact(m, x)).abs().max() <= tol


def test_far_points_do_not_touch_their_neighbours():
    """Phases beyond the unwrapped range, infinities and NaN: finite points far
    out stay within the output's bound, non-finite ones give NaN, and every
    other point keeps the bits it has alone."""
    m = _net([256, 256, 256], 5)
    x = _points(640)
    alone = _run(m, x)
    y = x.clone()
    far = torch.tensor([3e3, 1e5, 7e6, 1e9, 1e30], device="cuda")
    at = torch.arange(0, 640, 37, device="cuda")
    y[at, 0] = far[torch.arange(at.numel(), device="cuda") % 5]
    y[5] = float("inf")
    y[6, 1] = float("nan")
    got = _run(m, y)
    same = torch.ones(640, dtype=torch.bool, device="cuda")
    same[at] = False
    same[5:7] = False
    assert torch.equal(got[same], alone[same])
    bound = _bound(m)
    assert (got[at].abs() <= bound * 1.0001).all()
    assert torch.isnan(got[5:7]).all()
    # 3000 units out the phase is about 3e4: 3e4 * 2^-24 * a few roundings
    near = at[torch.arange(at.numel(), device="cuda") % 5 == 0]
    assert (got[near].double() - _exact(m, y[near])).abs().max() <= 2e-2 * bound


def test_large_hidden_phases():
    """A hidden layer whose phases exceed the unwrapped range."""
    m = _net([64, 64, 64], 6)
    with torch.no_grad():
        m.net[1][0].weight.mul_(1e7)
    x = _points(300)
    got = _run(m, x)
    bound = _bound(m)
    assert torch.isfinite(got).all() and (got.abs() <= bound * 1.0001).all()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", [0, 1, 2])
def test_non_finite_weights_give_nan(value, where):
    m = _net([64, 64, 64], 7)
    with torch.no_grad():
        m.net[where][0].weight[3, 2] = value
    assert torch.isnan(_run(m, _points(200))).all()


def test_index_list_accumulate_and_band(lib):
    """An index list with a device count, accumulation and a band list equal the
    plain evaluation of the same points."""
    from mplicits_gb300 import capi
    m = _net([256, 256, 256], 8)
    x = _points(3001, 9)
    f = _run(m, x)
    perm = torch.randperm(3001, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    idx = perm[:777].to(torch.int32).contiguous()
    cnt = torch.tensor([700], dtype=torch.int32, device="cuda")
    S = torch.linspace(-0.1, 0.1, 3001, device="cuda")
    want = S.clone()
    sel = idx[:700].long()
    want[sel] = want[sel] + f[sel]
    out = torch.full((3001,), -1, dtype=torch.int32, device="cuda")
    n_out = torch.zeros(1, dtype=torch.int32, device="cuda")
    net, packed = m.packed()
    pts = capi.MplPoints(kind=capi.MPL_POINTS_XYZ, xyz=x.data_ptr())
    band = capi.MplBand(delta=0.05, out_index=out.data_ptr(), count_dev=n_out.data_ptr(),
                        capacity=3001)
    capi.check(capi.load().mpl_level_forward(
        ctypes.byref(net), capi.ptr(packed), ctypes.byref(pts), capi.ptr(idx), capi.ptr(cnt), 777,
        capi.ptr(S), capi.MPL_ACCUMULATE, ctypes.byref(band), capi.MPL_FP32, capi.stream_ptr()),
        "mpl_level_forward")
    assert torch.equal(S, want)
    kept = np.sort(out[:int(n_out)].cpu().numpy())
    ref = sel[want[sel].abs() < np.float32(0.05)].sort().values.cpu().numpy()
    np.testing.assert_array_equal(kept, ref)

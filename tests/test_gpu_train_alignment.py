"""mpl_train_backward adds into the caller's buffers wherever they lie: hidden
weight gradients at every float offset of a 16-byte line, packed back to back
after odd-sized parts.  Up to 64 points are one partial sum per value, added to
zero, so the results are equal bit for bit (tolerance 0)."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _backward(m, x, seeds, at):
    """Gradients with every buffer at a multiple of 64 floats plus ``at``."""
    from mplicits_gb300 import capi
    lib, (net, packed) = capi.load(), m.packed()
    n, wp, L = x.shape[0], m.linears()[0].out_features, len(m.linears())
    fl = ctypes.c_int64()
    capi.check(lib.mpl_train_scratch_floats(ctypes.byref(net), n, ctypes.byref(fl)), "scratch")
    pre, da = (torch.empty(fl.value, device="cuda") for _ in range(2))
    S, G = torch.empty(n, device="cuda"), torch.empty(n, 3, device="cuda")
    capi.check(lib.mpl_train_forward(ctypes.byref(net), capi.ptr(packed), capi.ptr(x), n,
                                     capi.ptr(S), capi.ptr(G), capi.ptr(pre),
                                     capi.stream_ptr()), "forward")
    sizes = [3 * wp] + [wp * wp] * (L - 2) + [wp] + [wp] * (L - 1) + [1]
    parts = []
    for s in sizes:
        t = torch.zeros(s + 64, device="cuda")
        assert t.data_ptr() % 256 == 0
        parts.append(t[at:at + s])
    P = ctypes.c_void_p
    dW = (P * L)(*[t.data_ptr() for t in parts[:L]])
    db = (P * L)(*[t.data_ptr() for t in parts[L:]])
    capi.check(lib.mpl_train_backward(ctypes.byref(net), capi.ptr(packed), capi.ptr(x), n,
                                      capi.ptr(pre), capi.ptr(seeds), capi.ptr(da), dW, db,
                                      capi.stream_ptr()), "backward")
    torch.cuda.synchronize()
    return parts


@pytest.mark.parametrize("at", [1, 2, 3, 4])
@pytest.mark.parametrize("width", [64, 128, 256])
def test_any_float_offset(width, at):
    from mplicits_gb300.model import SIREN
    torch.manual_seed(width)
    m = SIREN(3, 1, [width] * 3, w0=30).cuda()
    x = torch.rand(53, 3, device="cuda") * 2 - 1
    seeds = torch.randn(53, 4, device="cuda")
    for a, b in zip(_backward(m, x, seeds, 0), _backward(m, x, seeds, at)):
        assert torch.equal(a, b) and bool((a != 0).any())

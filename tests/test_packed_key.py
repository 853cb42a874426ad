"""When a level's packed image is made anew: with the C library replaced by a
counter, on the CPU.  A changed parameter always repacks, also where a layer's
weight is computed from parameters; an unchanged level never does."""

import ctypes

import pytest
import torch
from torch.nn.utils import parametrizations, parametrize

from mplicits_gb300 import capi
from mplicits_gb300.model import SIREN


class _Counter:
    def __init__(self):
        self.packs = 0
        self.weights = None

    def mpl_net_packed_bytes(self, net, nbytes):
        ctypes.cast(nbytes, ctypes.POINTER(ctypes.c_int64))[0] = 256
        return 0

    def mpl_net_pack(self, net, weights, biases, packed, stream):
        self.packs += 1
        n = 8 * 8
        self.weights = torch.tensor(
            (ctypes.c_float * n).from_address(weights[1])[:]).reshape(8, 8)
        return 0


@pytest.fixture
def lib(monkeypatch):
    c = _Counter()
    monkeypatch.setattr(capi, "load", lambda *a: c)
    monkeypatch.setattr(capi, "stream_ptr", lambda *a: None)
    return c


def _siren(dtype=torch.float32):
    torch.manual_seed(0)
    return SIREN(3, 1, [8, 8, 8], w0=30).to(dtype)


class _Transposed(torch.nn.Module):
    def forward(self, w):
        return w.t().contiguous().t()


class _Buffered(torch.nn.Module):
    def __init__(self):
        super().__init__()
        self.register_buffer("scale", torch.ones(()))

    def forward(self, w):
        return w * self.scale


class _Shared(torch.nn.Module):
    """The computed weight also follows a parameter of the whole model."""

    def __init__(self, owner):
        super().__init__()
        self.owner = [owner]

    def forward(self, w):
        return w * self.owner[0].gain


def _weight_norm(m):
    parametrizations.weight_norm(m.net[1][0])
    return m.net[1][0].parametrizations.weight.original0


def _transposed(m):
    parametrize.register_parametrization(m.net[1][0], "weight", _Transposed())
    return m.net[1][0].parametrizations.weight.original


def _bias(m):
    parametrize.register_parametrization(m.net[1][0], "bias", _Buffered())
    return m.net[1][0].weight


def _buffered(m):
    p = _Buffered()
    parametrize.register_parametrization(m.net[1][0], "weight", p)
    return p.scale


def _shared(m):
    m.gain = torch.nn.Parameter(torch.ones(()))
    parametrize.register_parametrization(m.net[1][0], "weight", _Shared(m))
    return m.gain


def _plain(m):
    return m.net[1][0].weight


def _attribute(m):
    """The weight as a plain attribute (as the older weight norm leaves it)."""
    w = m.net[1][0].weight.detach().clone()
    del m.net[1][0].weight
    m.net[1][0].weight = w
    return w


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("make", [_plain, _weight_norm, _transposed, _bias, _buffered, _shared,
                                  _attribute])
def test_repacked_when_changed_and_only_then(lib, make, dtype):
    m = _siren(dtype)
    source = make(m)
    with torch.no_grad():
        m.packed()
        for i in range(20):
            source.mul_(1.25)
            m.packed()
            assert lib.packs == i + 2
            assert torch.equal(lib.weights, m.net[1][0].weight.float())
            m.packed()
            m.packed()
            assert lib.packs == i + 2


def test_a_layer_of_any_name(lib):
    """Blocks are indexed, whatever their children are called."""
    from collections import OrderedDict
    m = _siren()
    lin, act = m.net[1][0], m.net[1][1]
    m.net[1] = torch.nn.Sequential(OrderedDict(linear=lin, act=act))
    assert m.linears()[1] is lin
    m.packed()
    assert lib.packs == 1

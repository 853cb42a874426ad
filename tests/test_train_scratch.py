"""The training scratch follows the level's layers: with the C library replaced
by the scratch size's formula, on the CPU."""

import ctypes

import pytest
import torch

from mplicits_gb300 import capi, train
from mplicits_gb300.model import SIREN


class _Sizes:
    def mpl_train_scratch_floats(self, net, n, floats):
        net = ctypes.cast(net, ctypes.POINTER(capi.MplNet))[0]
        w = max(net.dims[i] for i in range(1, net.n_layers))
        wp = 64 if w <= 64 else (128 if w <= 128 else 256)
        ctypes.cast(floats, ctypes.POINTER(ctypes.c_int64))[0] = (net.n_layers - 1) * n * 4 * wp
        return 0


def _widen(m, i, width):
    """Layer i of another width (and the layer after it)."""
    a, b = m.net[i][0], m.net[i + 1][0]
    m.net[i][0] = torch.nn.Linear(a.in_features, width)
    m.net[i + 1][0] = torch.nn.Linear(width, b.out_features)


@pytest.mark.parametrize("first,then", [((64, 64, 64), 50), ((64, 50, 64), 64),
                                        ((64, 64, 64), 100), ((128, 128, 128), 200),
                                        ((100, 64, 60), 128)])
def test_follows_replaced_layers(monkeypatch, first, then):
    monkeypatch.setattr(capi, "load", lambda *a: _Sizes())
    torch.manual_seed(0)
    m = SIREN(3, 1, list(first), w0=30)
    for change in (False, True):
        if change:
            _widen(m, 1, then)
        sc = train._scratch(m, 100, torch.device("cpu"))
        wp = train._padded_width(m)
        for own in (True, False):
            grads = train._unpad(m, sc, own)
            assert [g.shape for g in grads] == [p.shape for p in m.parameters()]
        # the kernels' buffers have the padded shapes
        assert [t.numel() for t in sc.dW] == [3 * wp, wp * wp, wp * wp, wp]
        assert [t.numel() for t in sc.db] == [wp, wp, wp, 1]
        assert sc.pre.numel() >= 3 * 100 * 4 * wp and sc.da.numel() >= 3 * 100 * 4 * wp


def test_another_depth(monkeypatch):
    monkeypatch.setattr(capi, "load", lambda *a: _Sizes())
    m = SIREN(3, 1, [64, 64], w0=30)
    train._scratch(m, 100, torch.device("cpu"))
    deep = SIREN(3, 1, [64, 64, 64, 64], w0=30)
    m.net = deep.net
    sc = train._scratch(m, 50, torch.device("cpu"))
    assert len(sc.dW) == 5 and sc.pre.numel() >= 4 * 50 * 4 * 64


def test_kept_while_nothing_changes(monkeypatch):
    monkeypatch.setattr(capi, "load", lambda *a: _Sizes())
    m = SIREN(3, 1, [64, 64, 64], w0=30)
    sc = train._scratch(m, 100, torch.device("cpu"))
    flat, pre = sc.flat, sc.pre
    for n in (100, 1, 60):
        assert train._scratch(m, n, torch.device("cpu")) is sc
        assert sc.flat is flat and sc.pre is pre

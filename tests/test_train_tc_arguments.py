"""mpl_train_tc_step refuses hidden gradient buffers that its 16-byte adds cannot
take, on the host: nothing is launched, so any address will do here."""

import ctypes

import pytest

from mplicits_gb300 import capi


@pytest.fixture(scope="module")
def lib():
    return capi.load()


@pytest.mark.parametrize("layer,offset,ok", [(1, 0, True), (1, 4, False), (2, 8, False),
                                             (2, 12, False), (0, 4, True), (3, 4, True)])
def test_alignment_of_hidden_gradients(lib, layer, offset, ok):
    P = ctypes.c_void_p
    net = capi.MplNet()
    net.n_layers = 4
    for i, d in enumerate((3, 128, 128, 128, 1)):
        net.dims[i] = d
    for i in range(4):
        net.omega[i] = 30.0
    base = 1 << 20
    dW = (P * 4)(*[base + (offset if l == layer else 0) for l in range(4)])
    db = (P * 4)(*[base + 4] * 4)
    loss = capi.MplLoss(kind=capi.MPL_LOSS_RESIDUAL)
    fake = P(base)
    # no scratch: an accepted call ends at the next check
    st = lib.mpl_train_tc_step(ctypes.byref(net), fake, fake, 100, None, None, fake, fake,
                               ctypes.byref(loss), fake, 0, fake, fake, dW, db, None)
    assert st == (capi.MPL_ERR_CAPACITY if ok else capi.MPL_ERR_INVALID_ARG)

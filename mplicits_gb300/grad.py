"""Analytic input gradients of a level (normals, eikonal term).

``level_gradient`` returns f(x) and df/dx in one launch of the fused
forward-mode kernel (``mpl_level_gradient``).  It is what
``torch.autograd.grad(model_out, model_in)`` on a ``mplicits_gb300.SIREN``
evaluates (the reference obtains it from autograd, i3d/diff_operators.py:
259-265), and what the sphere tracer and marching cubes use for normals.
"""

from __future__ import annotations

import ctypes

import torch

from . import capi


def level_gradient(model, x, S=None, G=None, accumulate=False, precision=None, index=None,
                   n_dev=None, n=None):
    """(S, G): f(x) [P] and df/dx [P, 3] of one level.  With ``index`` the
    points are x[index[q]] and the results land at S[index[q]], G[index[q]].

    In "fp32" the value comes from the FMA kernel, that of ``SIREN.forward``
    from the split-operand kernel: both a few 1e-7 (2-norm) from float64, with
    sums in another order, so a value next to a threshold can fall on either
    side."""
    if not x.is_cuda:
        raise RuntimeError("mplicits_gb300 evaluates levels on a CUDA device only")
    x = x.detach().float().contiguous()
    P = x.shape[0]
    n = P if n is None else n
    if S is None:
        S = torch.empty(P, dtype=torch.float32, device=x.device)
    if G is None:
        G = torch.empty(P, 3, dtype=torch.float32, device=x.device)
    net, packed = model.packed()
    pts = capi.MplPoints(kind=capi.MPL_POINTS_XYZ, xyz=x.data_ptr())
    prec = capi.PRECISIONS[precision or model.precision]
    capi.check(capi.load().mpl_level_gradient(
        ctypes.byref(net), capi.ptr(packed), ctypes.byref(pts), capi.ptr(index),
        capi.ptr(n_dev), n, capi.ptr(S), capi.ptr(G),
        capi.MPL_ACCUMULATE if accumulate else capi.MPL_STORE, None, prec, capi.stream_ptr()),
        "mpl_level_gradient")
    return S, G


def level_backward(model, x, gy):
    """d(model_in) of model_out = f(x) for ``_LevelForward``: gy * df/dx.

    It comes from the fused gradient kernel; under ``create_graph=True``
    (i3d/diff_operators.py:259-265) df/dx is the differentiable op of
    ``mplicits_gb300.train.level_input_grad``, whose own backward is the double
    backward of the eikonal and normal losses.
    """
    from . import train as _train
    shape = x.shape
    if torch.is_grad_enabled():
        G = _train.level_input_grad(model, x.reshape(-1, shape[-1]))
        return (gy.reshape(-1, 1) * G).reshape(shape)
    _, G = level_gradient(model, x.detach().reshape(-1, shape[-1]), precision="fp32")
    return (gy.reshape(-1, 1).to(G.dtype) * G).reshape(shape)

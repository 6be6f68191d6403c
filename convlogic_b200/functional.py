"""Autograd Functions with the reference's names and argument lists.

``FullConvLogicFunction``, ``ConvLogicFunction`` (src/convlogic/convlogic_layer.py:16-82),
``TreeLogicFunction`` (src/convlogic/treelogic_layer.py:15-30), ``LogicLayerCudaFunction``
(src/difflogic/difflogic.py:214-230) and ``GradFactor`` (src/difflogic/functional.py:131-139).

As in the reference the gate argument is a MIXTURE over the 16 gates (soft-max already taken,
or one-hot) and the returned gradient is w.r.t. that mixture.  Each Function accepts one extra,
optional trailing argument ``wmode``; the layer modules pass W_SOFTMAX / W_ARGMAX together with
the raw logits so that the soft-max (and its Jacobian in backward) runs inside the kernels.

Unlike the reference, nothing but the input and an 8-bit arg-max per pooled output is saved for
backward: the gate tree is recomputed at the arg-max position.

``FullConvLogicFunction`` and ``LogicLayerCudaFunction`` are the calling convention (``apply``) over autograd nodes written in
C++ (csrc/torch_bind.cpp): a Python autograd Function over ctypes cost more host time per layer than its kernels take on
small inputs.  The split layers' Functions stay in Python.
"""

import torch
from torch.autograd import Function

from . import ops
from ._lib import W_ARGMAX, W_PROB, W_SOFTMAX, native  # noqa: F401


def _grad_sink(w):
    """(slice, ready-callback) when a gradient bucket (``dp.GradBucket.direct``) wants this parameter's gradient written
    straight into its slice of the flat buffer, else None.  Backward passes then hand the slice to the kernel as its
    output, call ``ready()`` and return no gradient for the parameter: no ``.grad`` accumulation kernel runs."""
    return getattr(w, "_clb_grad_sink", None)


class GradFactor(Function):
    @staticmethod
    def forward(ctx, x, f):
        ctx.f = f
        return x

    @staticmethod
    def backward(ctx, grad_y):
        return grad_y * ctx.f, None


class FullConvLogicFunction:
    """y, or (y[, x2, x3][, indices]) with ``return_intermediate`` / ``return_indices``."""

    @staticmethod
    def apply(x, w_prob, selection, stride_h, stride_w, pad_h, pad_w, kernel_h, kernel_w, return_intermediate=False,
              return_indices=False, wmode=W_PROB, y_feature_major=False):
        return native().block(x, w_prob, selection, stride_h, stride_w, pad_h, pad_w, kernel_h, kernel_w, return_intermediate,
                              return_indices, wmode, y_feature_major)


class ConvLogicFunction(Function):
    @staticmethod
    def forward(ctx, x, w_prob, selection, stride_h, stride_w, pad_h, pad_w, kernel_h, kernel_w, wmode=W_PROB):
        x = x.contiguous()
        w_prob = w_prob.contiguous()
        geom = (stride_h, stride_w, pad_h, pad_w, kernel_h, kernel_w)
        y = ops.conv_fwd(x, w_prob, selection, geom, wmode)
        ctx.save_for_backward(x, w_prob, selection)
        ctx.geom, ctx.wmode = geom, wmode
        return y

    @staticmethod
    def backward(ctx, grad_y):
        x, w, sel = ctx.saved_tensors
        grad_y = grad_y.contiguous()
        gx = gw = None
        if ctx.needs_input_grad[0]:
            gx = ops.conv_bwd_x(grad_y, x, w, sel, ctx.geom, ctx.wmode)
        if ctx.needs_input_grad[1] and ctx.wmode != W_ARGMAX:
            gw = ops.conv_bwd_w(grad_y, x, w, sel, ctx.geom, ctx.wmode)
        return (gx, gw) + (None,) * 8


class TreeLogicFunction(Function):
    @staticmethod
    def forward(ctx, x, w_prob, wmode=W_PROB):
        x = x.contiguous()
        w_prob = w_prob.contiguous()
        y = ops.tree_fwd(x, w_prob, wmode)
        ctx.save_for_backward(x, w_prob)
        ctx.wmode = wmode
        return y

    @staticmethod
    def backward(ctx, grad_y):
        x, w = ctx.saved_tensors
        grad_y = grad_y.contiguous()
        gx = gw = None
        if ctx.needs_input_grad[0]:
            gx = ops.tree_bwd_x(grad_y, x, w, ctx.wmode)
        if ctx.needs_input_grad[1] and ctx.wmode != W_ARGMAX:
            gw = ops.tree_bwd_w(grad_y, x, w, ctx.wmode)
        return gx, gw, None


class LogicLayerCudaFunction:
    """x is feature-major [in_dim, batch]; returns [out_dim, batch]."""

    @staticmethod
    def apply(x, a, b, w, given_x_indices_of_y_start, given_x_indices_of_y, wmode=W_PROB):
        return native().logic(x, a, b, w, given_x_indices_of_y_start, given_x_indices_of_y, wmode, True)


def to_feature_major(x):
    """Feature-major copy of a 2-D activation (its own storage when x is the transposed view a flat layer returned)."""
    xt = x.transpose(0, 1)
    if xt.is_contiguous() or x.requires_grad or not (x.is_cuda and x.dtype == torch.float32 and x.is_contiguous() and x.numel()):
        return xt.contiguous()
    return ops.transpose2d(x)

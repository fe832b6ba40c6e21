"""Operator + pointwise stage + batch normalisation as one native call each (no counterpart in the reference, whose
modules run operator -> torch.matmul -> + bias -> ReLU -> BatchNorm1d as separate kernels, picasso/mesh/layers.py:109-120,
166-175).  Forward: one fused tensor-core kernel makes the operator's rows, multiplies, adds bias, applies ReLU and takes
the statistics of the result; a second pass normalises (in inference the normalisation is part of the first kernel).
Backward: one reduction over (gradient, activation); one tensor-core kernel that takes the gradient back through
normalisation and mask while it loads and multiplies with depth_weights^T (pb200_gradient_rows_matmul); the weight and bias
gradients as a tensor-core contraction over the rows; the operator's own backward kernel.  The operator's output is kept
from the forward pass as a by-product.  The nodes are in csrc/torch_ops.cpp.
"""
from __future__ import annotations

import torch

from ... import _lib
from ...topology import for_backward, ptr, stream_ptr, vertex_csr
from . import conv3d

_precision = _lib.PREC_FP32


def set_pointwise_precision(name: str) -> None:
    """'fp32' (default: bf16 hi+lo operands, about 1e-5 relative) or 'bf16'."""
    global _precision
    if name not in ("fp32", "bf16"):
        raise ValueError(name)
    _precision = _lib.PRECISIONS[name]


def eligible(x: torch.Tensor, channels: int, multiplier: int, activation_fn) -> bool:
    """The fused kernels take depth multiplier 1, channels that are a multiple of 8, and ReLU or no
    activation."""
    return (x.is_cuda and x.dtype == torch.float32 and multiplier == 1 and channels % 8 == 0 and
            (activation_fn is None or isinstance(activation_fn, torch.nn.ReLU)))


def rows_contract(a, b):
    """(a^T @ b, column sums of b as a (1, N) row) with the contraction over rows on the tensor cores
    (pb200_rows_contract); torch for widths that are no multiple of 4."""
    Nrows, M = a.shape
    N = b.shape[1]
    if M % 4 != 0 or N % 4 != 0 or Nrows == 0:
        return a.t() @ b, b.sum(0, keepdim=True)
    dev = a.device
    a, b = conv3d._aligned16(a), conv3d._aligned16(b)
    with torch.cuda.device(dev):
        out = torch.empty(M, N, dtype=a.dtype, device=dev)
        colsum = torch.empty(1, N, dtype=a.dtype, device=dev)
        nb = _lib.query("pb200_rows_contract_workspace_bytes", Nrows, M, N)
        ws = torch.empty(max(nb, 1), dtype=torch.uint8, device=dev)
        _lib.call("pb200_rows_contract", Nrows, M, N, ptr(a), ptr(b), ptr(out), ptr(colsum), _precision, ptr(ws), nb,
                  stream_ptr(dev))
    return out, colsum


_NO_NORM = (0, None, None, None, None, None, 0.0, 0.0)


def vertex2facet_layer(input, face, corners, spatial_weights, depth_weights, biases, tail):
    """tail = (relu, norm mode, gamma, beta, running mean, running var, batches, momentum, eps)."""
    face.requires_grad = False
    rowptr = entries = None
    if torch.is_grad_enabled():
        conv3d._check(input, "input", 2, torch.float32)
        conv3d._check(face, "face", 2, torch.int32)
        csr = for_backward(vertex_csr, face, None, input.shape[0], input.shape[0])
        if csr is not None:
            rowptr, entries = csr.rowptr, csr.entries
    return _lib.ops.v2f_layer(input, face, rowptr, entries, corners, spatial_weights, depth_weights, biases, *tail, _precision)


def facet2vertex_layer(input, filter, coeff, face, nf_count, vt_map, depth_weights, biases, tail):
    for t in (coeff, face, nf_count, vt_map):
        t.requires_grad = False
    conv3d._check(face, "face", 2, torch.int32)
    conv3d._check(vt_map, "vt_map", 1, torch.int32)
    csr = vertex_csr(face, vt_map, vt_map.shape[0], nf_count.shape[0])
    return _lib.ops.f2v_layer(input, face, nf_count, vt_map, csr.rowptr, csr.entries, coeff, filter, depth_weights, biases, *tail,
                              _precision)


def rows_layer(rows, weights, biases, tail):
    return _lib.ops.rows_layer(rows, weights, biases, *tail, _precision)


def _tail(outputs, biases, relu):
    outputs = outputs if biases is None else outputs + biases
    return torch.relu(outputs) if relu else outputs


def rows_pointwise(rows, weights, biases, relu):
    """out = act(rows @ weights + biases): the pointwise layer (the reference's PerItemConv3d, picasso/mesh/layers.py:198-240)
    without normalisation."""
    if not _lib.native_calls():
        return _tail(rows @ weights, biases, relu)
    return rows_layer(rows, weights, biases, (relu, *_NO_NORM))


def vertex2facet_pointwise(input, filter, face, depth_weights, biases, relu):
    if tuple(filter.shape) != (3, input.shape[1], 1):
        raise RuntimeError("filter must have shape (3, C, 1) and depth_weights (C, out_channels)")
    if not _lib.native_calls():
        return _tail(conv3d.vertex2facet(input, filter, face) @ depth_weights, biases, relu)
    eye = torch.eye(3, device=input.device)       # the filter itself stands for the product of basis and weights
    return vertex2facet_layer(input, face, eye, filter.reshape(3, -1), depth_weights, biases, (relu, *_NO_NORM))


def facet2vertex_pointwise(input, filter, coeff, face, nf_count, vt_map, depth_weights, biases, relu):
    if not _lib.native_calls():
        return _tail(conv3d.facet2vertex(input, filter, coeff, face, nf_count, vt_map) @ depth_weights, biases, relu)
    return facet2vertex_layer(input, filter, coeff, face, nf_count, vt_map, depth_weights, biases, (relu, *_NO_NORM))

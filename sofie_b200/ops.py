"""Operator-level calls into libSOFIE_cuda on torch CUDA tensors.

torch is used for device memory and streams only; every computation below is one call through
the C ABI (include/sofie_cuda.h). Names follow the ONNX / SOFIE operators they implement
(reference: src/SOFIE_core/inc/SOFIE/ROperator_{Gemm,Conv,Relu,Pool,Softmax}.hxx).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _build, capi
from .capi import LAYOUT_NCHW, LAYOUT_NHWC


def _stream() -> C.c_void_p:
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _p(t) -> C.c_void_p:
    if t is None:
        return C.c_void_p(0)
    assert t.is_cuda and t.is_contiguous(), "tensors passed to libSOFIE_cuda must be contiguous CUDA tensors"
    return C.c_void_p(t.data_ptr())


_module = None


def _native():
    """The extension module with the calls that are made often (csrc_py/ops_native.cpp); the others below go through ctypes."""
    global _module
    if _module is None:
        capi.load()
        _module = _build.load_ops()
    return _module


def set_engine(engine: int) -> None:
    capi.call("sofie_cuda_set_engine", engine)


def last_engine() -> int:
    return capi.load().sofie_cuda_last_engine()


def gemm_f32(A, B, C_=None, *, transA=0, transB=0, alpha=1.0, beta=1.0, relu=False, out=None, workspace=True):
    """ONNX Gemm / MatMul: Y = alpha*op(A)*op(B) + beta*broadcast(C), optional Relu.

    Where it makes the product faster, six bytes per value of A and B (1 GiB at most) are taken from torch's pool for the duration of the call; when torch
    has no memory for them the product does without. With workspace=False nothing but the result is allocated. The two forms round differently within
    the same error bound."""
    return _native().gemm_f32(A, B, C_, transA, transB, alpha, beta, relu, out, workspace)


def conv_out_hw(H, W, kH, kW, pad, stride, dil=(1, 1)):
    oH = (H + 2 * pad[0] - (dil[0] * (kH - 1) + 1)) // stride[0] + 1
    oW = (W + 2 * pad[1] - (dil[1] * (kW - 1) + 1)) // stride[1] + 1
    return oH, oW


def conv2d_f32(X, W, bias=None, *, shape=None, pad=(0, 0), stride=(1, 1), dil=(1, 1), group=1, relu=False, pool=0,
               x_layout=LAYOUT_NCHW, y_layout=LAYOUT_NCHW, w_packed=False, kernel=None, out=None):
    """ONNX Conv (+Relu, +MaxPool 2x2). `shape` = (N, C, H, W) of the logical input."""
    return _native().conv2d_f32(X, W, bias, shape, pad, stride, dil, group, relu, pool, x_layout, y_layout, w_packed, kernel, out)


def conv2d_pack_f32(W):
    Cout, Cin, kH, kW = W.shape
    P = torch.empty((Cout, kH, kW, Cin), dtype=torch.float32, device=W.device)
    d = capi.Conv2dDesc(0, Cin, 1, 1, Cout, kH, kW, 0, 0, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0)
    capi.call("sofie_cuda_conv2d_pack_f32", _stream(), C.byref(d), _p(W), _p(P))
    return P


def relu_f32(X, out=None):
    return _native().relu_f32(X, out)


def pool2d_f32(X, *, mode=0, kernel=(2, 2), stride=(2, 2), pads=(0, 0, 0, 0), count_include_pad=0,
               layout=LAYOUT_NCHW, shape=None):
    return _native().pool2d_f32(X, mode, kernel, stride, pads, count_include_pad, layout, shape)


def pool3d_f32(X, *, mode=0, kernel=(2, 2, 2), stride=(2, 2, 2), pads=(0, 0, 0, 0, 0, 0), count_include_pad=0):
    """MaxPool (mode 0) / AveragePool (mode 1) of [N, C, D, H, W]; pads = (d, h, w begin, d, h, w end)."""
    N, Cc, D, H, W = X.shape
    o = [-(-(e + pads[i] + pads[i + 3] - kernel[i] + 1) // stride[i]) for i, e in enumerate((D, H, W))]
    Y = torch.empty((N, Cc, *o), dtype=torch.float32, device=X.device)
    d = capi.Pool3dDesc(mode, N, Cc, D, H, W, *kernel, *stride, (capi.i32 * 6)(*pads), count_include_pad)
    capi.call("sofie_cuda_pool3d_f32", _stream(), C.byref(d), _p(X), _p(Y))
    return Y


def conv3d_f32(X, W, bias=None, *, pad=(0, 0, 0), stride=(1, 1, 1), dil=(1, 1, 1), group=1, relu=False):
    """X [N, C, D, H, W], W [Cout, C/group, kD, kH, kW] -> [N, Cout, oD, oH, oW]."""
    N, Cin, D, H, Wd = X.shape
    Cout, _, kD, kH, kW = W.shape
    o = [(e + 2 * pad[i] - (dil[i] * (k - 1) + 1)) // stride[i] + 1 for i, (e, k) in enumerate(((D, kD), (H, kH), (Wd, kW)))]
    Y = torch.empty((N, Cout, *[max(v, 0) for v in o]), dtype=torch.float32, device=X.device)
    d = capi.Conv3dDesc(N, Cin, D, H, Wd, Cout, kD, kH, kW, *pad, *stride, *dil, group, int(relu))
    capi.call("sofie_cuda_conv3d_f32", _stream(), C.byref(d), _p(X), _p(W), _p(bias) if bias is not None else None, _p(Y))
    return Y


def softmax_f32(X, axis=-1):
    return _native().softmax_f32(X, axis)


def conv_transpose2d_f32(X, W, bias=None, pad=(0, 0), stride=(1, 1), dil=(1, 1), out_pad=(0, 0), relu=False, product_form=False):
    """ONNX ConvTranspose, group 1: X [N, C, H, W], W [C, Cout, kH, kW] -> [N, Cout, oH, oW]. product_form: the entry
    point that lowers to one tensor-core GEMM plus a gather (shapes with at least 16 input channels, a multiple of 4)."""
    N, Cin, H, Wd = X.shape
    _, Cout, kH, kW = W.shape
    oH = stride[0] * (H - 1) + dil[0] * (kH - 1) + 1 + out_pad[0] - 2 * pad[0]
    oW = stride[1] * (Wd - 1) + dil[1] * (kW - 1) + 1 + out_pad[1] - 2 * pad[1]
    Y = torch.empty((N, Cout, max(oH, 0), max(oW, 0)), dtype=torch.float32, device=X.device)
    d = capi.ConvTranspose2dDesc(N, Cin, H, Wd, Cout, kH, kW, pad[0], pad[1], stride[0], stride[1], dil[0], dil[1], out_pad[0],
                                 out_pad[1], int(relu))
    b = _p(bias) if bias is not None else None
    if product_form:
        nbytes = capi.load().sofie_cuda_conv_transpose2d_f32_gemm_scratch(C.byref(d))
        scratch = torch.empty(max(nbytes, 256), dtype=torch.uint8, device=X.device)
        capi.call("sofie_cuda_conv_transpose2d_f32_gemm", _stream(), C.byref(d), _p(X), _p(W), b, _p(Y), _p(scratch), nbytes)
    else:
        capi.call("sofie_cuda_conv_transpose2d_f32", _stream(), C.byref(d), _p(X), _p(W), b, _p(Y))
    return Y


def einsum_plan(equation, shape_a, shape_b):
    """Two-operand Einsum without ellipsis -> (output shape, n_out, n_sum, extents, strides in A, strides in B):
    the output labels first, in output order, then every other label in order of first appearance."""
    eq = equation.replace(" ", "")
    lhs, out = eq.split("->") if "->" in eq else (eq, None)
    la, lb = lhs.split(",")
    if "." in eq or len(la) != len(shape_a) or len(lb) != len(shape_b):
        raise ValueError(f"Einsum {equation}: two operands, one label per axis, no ellipsis")
    if out is None:   # implicit form: the labels that appear once, sorted
        out = "".join(sorted(c for c in set(la + lb) if (la + lb).count(c) == 1))
    size = {}
    for labels, shape in ((la, shape_a), (lb, shape_b)):
        for c, n in zip(labels, shape):
            if size.setdefault(c, int(n)) != int(n):
                raise ValueError(f"Einsum {equation}: label {c} has two extents")
    if len(set(la)) != len(la) or len(set(lb)) != len(lb) or len(set(out)) != len(out) or any(c not in size for c in out):
        raise ValueError(f"Einsum {equation}: repeated labels within one operand are not supported")
    summed = [c for c in dict.fromkeys(la + lb) if c not in out]
    labels = list(out) + summed
    if len(labels) > 8:
        raise ValueError("Einsum: at most 8 labels")

    def strides(lab, shape):
        st, dense = {}, 1
        for c, n in zip(reversed(lab), reversed(shape)):
            st[c] = dense
            dense *= int(n)
        return [st.get(c, 0) for c in labels]
    return tuple(size[c] for c in out), len(out), len(summed), [size[c] for c in labels], strides(la, shape_a), strides(lb, shape_b)


def einsum_f32(equation, A, B):
    out_shape, n_out, n_sum, extent, sa, sb = einsum_plan(equation, tuple(A.shape), tuple(B.shape))
    Y = torch.empty(out_shape, dtype=torch.float32, device=A.device)
    pad = lambda v: (C.c_int64 * 8)(*(list(v) + [0] * (8 - len(v))))
    d = capi.EinsumDesc(n_out, n_sum, pad(extent), pad(sa), pad(sb))
    capi.call("sofie_cuda_einsum_f32", _stream(), C.byref(d), _p(A), _p(B), _p(Y))
    return Y


def mlp_desc(M, dims, relu, w_is_nk):
    L = len(dims) - 1
    return capi.MlpDesc(M, L, (capi.i32 * 9)(*(list(dims) + [0] * (8 - L))), (capi.i32 * 8)(*([int(r) for r in relu] + [0] * (8 - L))),
                        (capi.i32 * 8)(*([int(n) for n in w_is_nk] + [0] * (8 - L))))


def mlp_fits(dims):
    """Whether a chain of layers with these widths is within what the fused MLP kernel takes (host arithmetic)."""
    if not 2 <= len(dims) <= capi.MLP_MAX_LAYERS + 1 or max(dims) > capi.MLP_MAX_WIDTH or min(dims) < 1:
        return False
    d = mlp_desc(0, dims, [0] * (len(dims) - 1), [0] * (len(dims) - 1))
    return capi.load().sofie_cuda_mlp_f32_smem(C.byref(d)) <= capi.MLP_MAX_SMEM


def mlp_f32(X, weights, biases, relu, w_is_nk):
    """Fused chain of Gemm (+ Relu) layers; weights[l] is [N, K] when w_is_nk[l] else [K, N]."""
    L = len(weights)
    dims = [X.shape[1]] + [(W.shape[0] if nk else W.shape[1]) for W, nk in zip(weights, w_is_nk)]
    Y = torch.empty((X.shape[0], dims[-1]), dtype=torch.float32, device=X.device)
    d = mlp_desc(X.shape[0], dims, relu, w_is_nk)
    Wp = (C.c_void_p * L)(*[_p(W) for W in weights])
    Bp = (C.c_void_p * L)(*[(_p(b) if b is not None else None) for b in biases])
    capi.call("sofie_cuda_mlp_f32", _stream(), C.byref(d), _p(X), Wp, Bp, _p(Y))
    return Y


UNARY_OPS = {"Sigmoid": 0, "Tanh": 1, "LeakyRelu": 2, "Selu": 3, "Elu": 4, "Neg": 5, "Exp": 6, "Log": 7, "Sqrt": 8,
             "Reciprocal": 9, "Abs": 10, "Erf": 11, "Swish": 12, "Cos": 13, "Sin": 14}
BINARY_OPS = {"Add": 0, "Sub": 1, "Mul": 2, "Div": 3}


def unary_f32(X, op, alpha=0.0):
    return _native().unary_f32(X, UNARY_OPS[op], alpha)


def binary_strides(a_shape, b_shape):
    """Output shape and the rank-4 shape / element strides (0 along broadcast dimensions) of A op B: the descriptor binary_f32 passes."""
    out = tuple(torch.broadcast_shapes(tuple(a_shape), tuple(b_shape)))
    if len(out) > 4:
        raise ValueError("binary operators are built for rank <= 4")

    def strides(shape):
        shape = (1,) * (4 - len(shape)) + tuple(shape)
        return [0 if n == 1 else int(np.prod(shape[i + 1:], dtype=np.int64)) for i, n in enumerate(shape)]

    return out, [1] * (4 - len(out)) + list(out), strides(a_shape), strides(b_shape)


def binary_f32(A, B, op):
    return _native().binary_f32(A, B, BINARY_OPS[op])


def batchnorm_f32(X, scale, bias, mean, N, Cc, HW, layout=LAYOUT_NCHW, relu=False):
    """scale is the folded gamma / sqrt(var + eps)."""
    return _native().batchnorm_f32(X, scale, bias, mean, N, Cc, HW, layout, relu)


def nchw_to_nhwc(X):
    return _native().change_layout(X, True)


def nhwc_to_nchw(X):
    return _native().change_layout(X, False)


def transpose2d(X):
    rows, cols = X.shape
    Y = torch.empty((cols, rows), dtype=X.dtype, device=X.device)
    fn = "sofie_cuda_transpose_f32" if X.dtype == torch.float32 else "sofie_cuda_transpose_i8"
    capi.call(fn, _stream(), _p(X), _p(Y), rows, cols)
    return Y


# ---------------------------------------------------------------- int8 -------------------------
def quantize_u8(X, scale, zp):
    return _native().quantize_u8(X, scale, zp)


def dequantize_u8(X, scale, zp):
    return _native().dequantize_u8(X, scale, zp)


def qlinear_prepare(W_host: np.ndarray, w_is_nk: bool, a_scale, a_zp, w_scale_host: np.ndarray, y_scale,
                    bias_host: np.ndarray | None, device, n_out=None, rows_per_n=None):
    """Per-output-channel requantisation multiplier and int32 correction, computed on the host."""
    W_host = np.ascontiguousarray(W_host, dtype=np.int8)
    w_scale_host = np.ascontiguousarray(w_scale_host, dtype=np.float32)
    if n_out is None:
        n_out = W_host.shape[0] if w_is_nk else W_host.shape[1]
    if rows_per_n is None:
        rows_per_n = W_host.size // n_out
    mult = torch.empty(n_out, dtype=torch.float32, device=device)
    corr = torch.empty(n_out, dtype=torch.int32, device=device)
    bias_p = C.c_void_p(0)
    if bias_host is not None:
        bias_host = np.ascontiguousarray(bias_host, dtype=np.int32)
        bias_p = bias_host.ctypes.data_as(C.c_void_p)
    capi.call("sofie_cuda_qlinear_prepare", _stream(), n_out, rows_per_n, W_host.ctypes.data_as(C.c_void_p),
              int(w_is_nk), float(a_scale), int(a_zp), w_scale_host.ctypes.data_as(C.c_void_p), float(y_scale),
              bias_p, _p(mult), _p(corr))
    return mult, corr


def qlinear_matmul(A, W, mult, corr, *, w_is_nk=True, y_zp=0, relu=False):
    return _native().qlinear_matmul(A, W, mult, corr, w_is_nk, y_zp, relu, None)


def qlinear_matmul_f32(A, W, mult, corr, y_scale, *, w_is_nk=True, y_zp=0, relu=False):
    """QLinearMatMul + DequantizeLinear (same zero point) in one pass: float32 (q - y_zp) * y_scale."""
    return _native().qlinear_matmul(A, W, mult, corr, w_is_nk, y_zp, relu, float(y_scale))


def qlinear_conv2d(X, W, mult, bias=None, *, shape=None, pad=(0, 0), stride=(1, 1), x_zp=0, y_zp=0, relu=False,
                   pool=0, x_layout=LAYOUT_NCHW, y_layout=LAYOUT_NCHW, w_packed=False, kernel=None):
    return _native().qlinear_conv2d(X, W, mult, bias, shape, pad, stride, x_zp, y_zp, relu, pool, x_layout, y_layout, w_packed, kernel)


def qconv2d_pack_i8(W):
    Cout, Cin, kH, kW = W.shape
    P = torch.empty((Cout, kH, kW, Cin), dtype=torch.int8, device=W.device)
    d = capi.QConv2dDesc(0, Cin, 1, 1, Cout, kH, kW, 0, 0, 1, 1, 0, 0, 0, 0, 0, 0, 0)
    capi.call("sofie_cuda_qconv2d_pack_i8", _stream(), C.byref(d), _p(W), _p(P))
    return P


def maxpool2d_u8(X, *, kernel=(2, 2), stride=(2, 2), layout=LAYOUT_NCHW, shape=None):
    return _native().maxpool2d_u8(X, kernel, stride, layout, shape)


# ---------------------------------------------------------------- FP8 --------------------------
def quantize_e4m3(X, scale):
    return _native().quantize_e4m3(X, scale)


def cast_bf16_f32(X):
    Y = torch.empty(X.shape, dtype=torch.float32, device=X.device)
    capi.call("sofie_cuda_cast_bf16_f32", _stream(), _p(X), _p(Y), X.numel())
    return Y


def cast_f32_bf16(X):
    Y = torch.empty(X.shape, dtype=torch.bfloat16, device=X.device)
    capi.call("sofie_cuda_cast_f32_bf16", _stream(), _p(X), _p(Y), X.numel())
    return Y


def amax_f32(X):
    out = torch.empty(1, dtype=torch.float32, device=X.device)
    capi.call("sofie_cuda_amax_f32", _stream(), _p(X), X.numel(), _p(out))
    return out


def gemm_e4m3(A, W, bias=None, *, a_scale=1.0, w_scale=1.0, relu=False, q_scale=0.0, want_bf16=True):
    """A [M,K] and W [N,K] are uint8 tensors holding E4M3 codes. Returns (bf16 Y or None, E4M3 Yq or None)."""
    return _native().gemm_e4m3(A, W, bias, a_scale, w_scale, relu, q_scale, want_bf16, False)


def gemm_e4m3_f32(A, W, bias=None, *, a_scale=1.0, w_scale=1.0, relu=False):
    """The FP8 product with the bf16-rounded result written as float32 (Fp8Gemm + Cast in one pass)."""
    return _native().gemm_e4m3(A, W, bias, a_scale, w_scale, relu, 0.0, True, True)
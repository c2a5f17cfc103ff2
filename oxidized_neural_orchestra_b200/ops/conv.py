"""Python entries to the convolution / pooling gather-scatter kernels (``csrc/kernels/conv.cu``).

Image activations are pixel-major 2-D tensors ``[B*H*W, ld]`` (channels contiguous). The convolution
itself is ``cols @ K^T`` on the tcgen05 GEMM; these kernels build ``cols`` (im2col), fold the column
gradient back (col2im), pool, and convert to and from the flattened NCHW rows dense layers use.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from .gemm import ACT


class OnoConvGeom(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("B", "C", "H", "W", "K", "S", "P", "OH", "OW")]


class OnoConvDgrad(C.Structure):
    _fields_ = [("g", OnoConvGeom), ("F", C.c_int), ("dtype", C.c_int), ("dy", C.c_void_p), ("kt", C.c_void_p), ("aux", C.c_void_p),
                ("dx", C.c_void_p), ("ld_dy", C.c_int), ("ld_kt", C.c_int), ("ld_aux", C.c_int), ("ld_dx", C.c_int), ("dact", C.c_int),
                ("dact_param", C.c_float), ("relu_quirk", C.c_int), ("status", C.c_void_p), ("timeout_ns", C.c_ulonglong)]


class OnoConvFprop(C.Structure):
    _fields_ = [("g", OnoConvGeom), ("F", C.c_int), ("dtype", C.c_int), ("x", C.c_void_p), ("kop", C.c_void_p), ("bias", C.c_void_p),
                ("cols", C.c_void_p), ("y", C.c_void_p), ("ldx", C.c_int), ("ld_kop", C.c_int), ("ld_cols", C.c_int), ("ld_y", C.c_int),
                ("act", C.c_int), ("act_param", C.c_float), ("status", C.c_void_p), ("timeout_ns", C.c_ulonglong)]


_declared = False


def _fn():
    global _declared
    lib = _lib.load()
    if not _declared:
        vp, ci, cf = C.c_void_p, C.c_int, C.c_float
        G = C.POINTER(OnoConvGeom)
        lib.ono_im2col.argtypes = [G, ci, vp, ci, vp, ci, vp, ci, vp]
        lib.ono_col2im.argtypes = [G, ci, vp, ci, vp, ci, ci, cf, ci, vp, ci, vp, ci, vp]
        lib.ono_pool_fwd.argtypes = [G, ci, vp, ci, vp, ci, vp, ci, vp, ci, cf, vp]
        lib.ono_pool_bwd.argtypes = [G, ci, vp, ci, vp, ci, vp, ci, cf, ci, vp, ci, ci, cf, vp, ci, vp, ci, vp]
        lib.ono_nchw_flat.argtypes = [ci, ci, ci, ci, ci, vp, ci, vp, ci, vp, ci, vp, ci, ci, cf, ci, vp]
        lib.ono_conv1_fwd.argtypes = [G, ci, ci, vp, ci, vp, vp, ci, cf, vp, ci, vp]
        lib.ono_conv1_wgrad.argtypes = [G, ci, ci, vp, ci, vp, ci, vp, vp, cf, vp]
        lib.ono_conv1_fwd.restype = lib.ono_conv1_wgrad.restype = ci
        lib.ono_conv_kperm.argtypes = [ci, ci, ci, ci, ci, vp, ci, vp, ci, vp, ci, cf, vp]
        lib.ono_conv_kperm.restype = ci
        lib.ono_conv_dgrad_fits.argtypes = [C.POINTER(OnoConvDgrad)]
        lib.ono_conv_dgrad.argtypes = [C.POINTER(OnoConvDgrad), vp]
        lib.ono_conv_dgrad_fits.restype = lib.ono_conv_dgrad.restype = ci
        lib.ono_conv_fprop_fits.argtypes = [C.POINTER(OnoConvFprop)]
        lib.ono_conv_fprop.argtypes = [C.POINTER(OnoConvFprop), vp]
        lib.ono_conv_fprop_fits.restype = lib.ono_conv_fprop.restype = ci
        lib.ono_conv_dgrad_pays.argtypes = lib.ono_conv_fprop_pays.argtypes = [G, ci, ci]
        lib.ono_conv_dgrad_pays.restype = lib.ono_conv_fprop_pays.restype = ci
        for i, st in ((12, OnoConvDgrad), (13, OnoConvFprop)):
            if lib.ono_sizeof(i) != C.sizeof(st):
                raise RuntimeError(f"ABI mismatch for {st.__name__}")
        lib.ono_pool_flat_fits.argtypes = [G, ci]
        lib.ono_pool_flat_fwd.argtypes = [G, ci, vp, ci, vp, ci, vp, ci, cf, vp, ci, vp]
        lib.ono_pool_flat_bwd.argtypes = [G, ci, vp, ci, vp, ci, vp, ci, cf, ci, vp, ci, ci, cf, vp, ci, vp]
        for f in (lib.ono_im2col, lib.ono_col2im, lib.ono_pool_fwd, lib.ono_pool_bwd, lib.ono_nchw_flat, lib.ono_pool_flat_fits, lib.ono_pool_flat_fwd,
                  lib.ono_pool_flat_bwd):
            f.restype = ci
        _declared = True
    return lib


def geom(B, C_, H, W, K, S, P) -> OnoConvGeom:
    g = OnoConvGeom()
    g.B, g.C, g.H, g.W, g.K, g.S, g.P = B, C_, H, W, K, S, P
    g.OH = (H + 2 * P - K) // S + 1
    g.OW = (W + 2 * P - K) // S + 1
    return g


def _dt(t: torch.Tensor) -> int:
    return 0 if t.dtype == torch.float32 else 1


def _p(t):
    return None if t is None else t.data_ptr()


def _ld(t):
    return 0 if t is None else t.stride(0)


def im2col(g, x, cols, cols_t=None, stream=None):
    lib = _fn()
    _lib.check(lib.ono_im2col(C.byref(g), _dt(x), x.data_ptr(), x.stride(0), cols.data_ptr(), cols.stride(0), _p(cols_t),
                              _ld(cols_t), _lib.stream_ptr(stream)), "ono_im2col")


def col2im(g, dcols, dx, dx_t=None, aux=None, dact=None, dact_param=0.0, relu_quirk=False, stream=None):
    lib = _fn()
    _lib.check(lib.ono_col2im(C.byref(g), _dt(dcols), dcols.data_ptr(), dcols.stride(0), _p(aux), _ld(aux), ACT[dact],
                              dact_param, int(relu_quirk), dx.data_ptr(), dx.stride(0), _p(dx_t), _ld(dx_t),
                              _lib.stream_ptr(stream)), "ono_col2im")


def _fprop(g, F, x, kop, y, cols, bias, act, act_param, status) -> OnoConvFprop:
    s = OnoConvFprop()
    s.g, s.F, s.dtype = g, F, _dt(x)
    s.x, s.kop, s.y, s.cols, s.bias = x.data_ptr(), kop.data_ptr(), y.data_ptr(), _p(cols), _p(bias)
    s.ldx, s.ld_kop, s.ld_y, s.ld_cols = x.stride(0), kop.stride(0), y.stride(0), _ld(cols)
    s.act, s.act_param, s.status = ACT[act], act_param, _p(status)
    return s


def fprop_fits(g, F, x, kop, y, cols=None) -> bool:
    """Whether ``fprop`` takes these sizes, rows and addresses."""
    return bool(_fn().ono_conv_fprop_fits(C.byref(_fprop(g, F, x, kop, y, cols, None, None, 0.0, None))))


def fprop_pays(g, F, dtype) -> bool:
    """Whether ``fprop``, where it fits, is no slower than ``im2col`` and a product."""
    return bool(_fn().ono_conv_fprop_pays(C.byref(g), F, 0 if dtype == torch.float32 else 1))


def fprop(g, F, x, kop, y, cols=None, bias=None, act=None, act_param=0.0, status=None, stream=None):
    """``y = act(im2col(x) @ kop^T + bias)`` in one kernel; ``cols``: also leaves the column matrix there. ``kop``: the kernel tensor as
    ``[F][(ky, kx, c)]`` in the type of ``x``; ``bias`` f32."""
    s = _fprop(g, F, x, kop, y, cols, bias, act, act_param, status)
    _lib.check(_fn().ono_conv_fprop(C.byref(s), _lib.stream_ptr(stream)), "ono_conv_fprop")


def _dgrad(g, F, dy, kt, dx, aux, dact, dact_param, relu_quirk, status) -> OnoConvDgrad:
    s = OnoConvDgrad()
    s.g, s.F, s.dtype = g, F, _dt(dy)
    s.dy, s.kt, s.dx, s.aux = dy.data_ptr(), kt.data_ptr(), dx.data_ptr(), _p(aux)
    s.ld_dy, s.ld_kt, s.ld_dx, s.ld_aux = dy.stride(0), kt.stride(0), dx.stride(0), _ld(aux)
    s.dact, s.dact_param, s.relu_quirk, s.status = ACT[dact], dact_param, int(relu_quirk), _p(status)
    return s


def dgrad_fits(g, F, dy, kt, dx, aux=None, dact=None) -> bool:
    """Whether ``dgrad`` takes these sizes, rows and addresses."""
    return bool(_fn().ono_conv_dgrad_fits(C.byref(_dgrad(g, F, dy, kt, dx, aux, dact, 0.0, False, None))))


def dgrad_pays(g, F, dtype) -> bool:
    """Whether ``dgrad``, where it fits, is no slower than a product and ``col2im``."""
    return bool(_fn().ono_conv_dgrad_pays(C.byref(g), F, 0 if dtype == torch.float32 else 1))


def dgrad(g, F, dy, kt, dx, aux=None, dact=None, dact_param=0.0, relu_quirk=False, status=None, stream=None):
    """Input gradient of a convolution: ``dy [pixels, F] @ K^T`` folded back onto the input's pixels and taken through the derivative ``dact`` of the
    layer below on ``aux``, in one kernel. ``kt``: the kernel tensor as ``[(ky, kx, c)][F]`` in the type of ``dy``. Rows of ``dx`` hold whole
    16-byte pieces, and what lies between the last channel and the end of its piece is written too."""
    s = _dgrad(g, F, dy, kt, dx, aux, dact, dact_param, relu_quirk, status)
    _lib.check(_fn().ono_conv_dgrad(C.byref(s), _lib.stream_ptr(stream)), "ono_conv_dgrad")


def pool_fwd(g, x, y, arg, y_t=None, act=None, act_param=0.0, stream=None):
    lib = _fn()
    _lib.check(lib.ono_pool_fwd(C.byref(g), _dt(x), x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), _p(y_t), _ld(y_t),
                                arg.data_ptr(), ACT[act], act_param, _lib.stream_ptr(stream)), "ono_pool_fwd")


def pool_bwd(g, d, y, arg, dx, dx_t=None, act=None, act_param=0.0, aux=None, dact=None, dact_param=0.0, relu_quirk=False, stream=None):
    """Gradient w.r.t. the pooling layer's input, taken through the derivative ``dact`` of the layer below on ``aux``."""
    lib = _fn()
    _lib.check(lib.ono_pool_bwd(C.byref(g), _dt(d), d.data_ptr(), d.stride(0), y.data_ptr(), y.stride(0), arg.data_ptr(),
                                ACT[act], act_param, int(relu_quirk), _p(aux), _ld(aux), ACT[dact], dact_param, dx.data_ptr(),
                                dx.stride(0), _p(dx_t), _ld(dx_t), _lib.stream_ptr(stream)), "ono_pool_bwd")


def pool_flat_fits(g, dtype) -> bool:
    """Whether the pooling layer and the change to flattened rows run as one kernel."""
    return bool(_fn().ono_pool_flat_fits(C.byref(g), 0 if dtype == torch.float32 else 1))


def pool_flat_fwd(g, x, y, arg, flat, act=None, act_param=0.0, stream=None):
    """``pool_fwd`` and ``nchw_flat`` to rows."""
    _lib.check(_fn().ono_pool_flat_fwd(C.byref(g), _dt(x), x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), arg.data_ptr(), ACT[act],
                                       act_param, flat.data_ptr(), flat.stride(0), _lib.stream_ptr(stream)), "ono_pool_flat_fwd")


def pool_flat_bwd(g, flat, y, arg, dx, act=None, act_param=0.0, aux=None, dact=None, dact_param=0.0, relu_quirk=False, stream=None):
    """``nchw_flat`` from rows and ``pool_bwd``."""
    _lib.check(_fn().ono_pool_flat_bwd(C.byref(g), _dt(flat), flat.data_ptr(), flat.stride(0), y.data_ptr(), y.stride(0), arg.data_ptr(),
                                       ACT[act], act_param, int(relu_quirk), _p(aux), _ld(aux), ACT[dact], dact_param, dx.data_ptr(),
                                       dx.stride(0), _lib.stream_ptr(stream)), "ono_pool_flat_bwd")


def nchw_flat(B, C_, HW, to_flat, img, flat, out_t=None, aux=None, dact=None, dact_param=0.0, relu_quirk=False, stream=None):
    lib = _fn()
    _lib.check(lib.ono_nchw_flat(_dt(img), B, C_, HW, int(to_flat), img.data_ptr(), img.stride(0), flat.data_ptr(),
                                 flat.stride(0), _p(out_t), _ld(out_t), _p(aux), _ld(aux), ACT[dact], dact_param,
                                 int(relu_quirk), _lib.stream_ptr(stream)), "ono_nchw_flat")


def kernel_to_operand(F, C_, K, params_f32, dst, dst_t=None, stream=None):
    """K[F][C][k][k] (flat f32 parameters) -> GEMM operand rows in (ky, kx, c) order, plus its transpose."""
    lib = _fn()
    _lib.check(lib.ono_conv_kperm(F, C_, K, 0, _dt(dst), params_f32.data_ptr(), 0, dst.data_ptr(), dst.stride(0), _p(dst_t),
                                  _ld(dst_t), 0.0, _lib.stream_ptr(stream)), "ono_conv_kperm")


def operand_grad_to_kernel(F, C_, K, src_f32, grads_f32, beta=0.0, stream=None):
    """f32 weight gradient in operand order [F][(ky, kx, c)] -> parameter order K[F][C][k][k], dst = beta*dst + src."""
    lib = _fn()
    _lib.check(lib.ono_conv_kperm(F, C_, K, 1, 0, src_f32.data_ptr(), src_f32.stride(0), grads_f32.data_ptr(), 0, None, 0,
                                  float(beta), _lib.stream_ptr(stream)), "ono_conv_kperm")


def conv1_fwd(g, F, x, kparams_f32, bias_f32, y, act=None, act_param=0.0, stream=None):
    """Direct forward of a convolution with one input channel: y = act(conv(x, K) + b), K given in parameter order."""
    lib = _fn()
    _lib.check(lib.ono_conv1_fwd(C.byref(g), F, _dt(x), x.data_ptr(), x.stride(0), kparams_f32.data_ptr(), _p(bias_f32), ACT[act],
                                 act_param, y.data_ptr(), y.stride(0), _lib.stream_ptr(stream)), "ono_conv1_fwd")


def conv1_wgrad(g, F, x, dy, gk_f32, gb_f32, beta=0.0, stream=None):
    """Weight and bias gradient of a one-input-channel convolution, written in parameter order (g = beta*g + d)."""
    lib = _fn()
    _lib.check(lib.ono_conv1_wgrad(C.byref(g), F, _dt(x), x.data_ptr(), x.stride(0), dy.data_ptr(), dy.stride(0), gk_f32.data_ptr(),
                                   gb_f32.data_ptr(), float(beta), _lib.stream_ptr(stream)), "ono_conv1_wgrad")

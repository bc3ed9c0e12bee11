"""Tensor-level entry to the contraction path: torch tensors in (they only supply device memory
and the stream), the C ABI underneath.  The per-call work (shape checks, allocation of the result, descriptor,
workspace, stream) is done in ``csrc/nml_torch.cpp``.

Each function corresponds to one host op of the reference:

=============================  ================================================================
here                           reference
=============================  ================================================================
conv_forward                   nectar::conv2d / nectar::conv_transpose2d
                               (nectarml/csrc/ops/tensor/conv/conv2d.cpp:401-497)
conv_backward_data             conv2d_backward_input / conv_transpose2d_backward_input
                               (conv2d.cpp:499-542)
conv_backward_weight           conv2d_backward_weight / conv_transpose2d_backward_weight
                               (conv2d.cpp:544-583) + ``out_grad.sum(dim=(0,2,3))``
                               (nectarml/cuda/tensor/conv.py:175-176)
linear_forward / _backward_*   ``x @ W.T + b`` and its gradients
                               (nectarml/nn/linear.py:44-47,
                               nectarml/core/_tensor/numerical.py:864-907)
=============================  ================================================================
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from typing import Optional, Tuple

import torch

from . import _lib
from ._lib import (NML_F16, NML_F32, NML_MATH_3XTF32, NML_MATH_F16, NML_MATH_TF32, NML_NCHW,
                   NML_NHWC, ConvDesc, check)

_MATH = {"f16": NML_MATH_F16, "3xtf32": NML_MATH_3XTF32, "tf32": NML_MATH_TF32}
_LAYOUT = {"nchw": NML_NCHW, "nhwc": NML_NHWC}


class _LazyNative:
    """Stands in for the native module until its first use, so that this file can be imported before the build."""

    def __getattr__(self, name):
        global _native
        _lib.load()
        try:
            from . import _native as module
        except ImportError as e:
            raise _lib.NectarB200Error(f"nectarml_b200/_native.so: {e}; build it with `python -m nectarml_b200.build`") from e
        _native = module
        return getattr(module, name)


_native = _LazyNative()
_DTYPE = {torch.float32: NML_F32, torch.float16: NML_F16, None: -1}


def _dt(t: torch.dtype) -> int:
    if t == torch.float32:
        return NML_F32
    if t == torch.float16:
        return NML_F16
    raise _lib.NectarB200Error(f"only float32 and float16 tensors are supported, got {t}")


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    if t is None:
        return None
    if not t.is_cuda:
        raise _lib.NectarB200Error("tensors must live on a CUDA device (there is no CPU path)")
    if not t.is_contiguous():
        raise _lib.NectarB200Error("tensors must be contiguous")
    return t.data_ptr()


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _out_dtype(t: Optional[torch.dtype]) -> int:
    """Code of a result dtype; -1: that of the call's first tensor."""
    code = _DTYPE.get(t)
    return _dt(t) if code is None else code


@dataclass(frozen=True)
class ConvGeometry:
    """Shape of one Conv2d (``transposed=False``) or ConvTranspose2d layer, input side first."""
    batch: int
    c_in: int
    h: int
    w: int
    c_out: int
    kh: int
    kw: int
    stride: Tuple[int, int] = (1, 1)
    padding: Tuple[int, int] = (0, 0)
    dilation: Tuple[int, int] = (1, 1)
    output_padding: Tuple[int, int] = (0, 0)
    transposed: bool = False

    def native(self):
        """The geometry as the native host path takes it; parsed once per object."""
        h = self.__dict__.get("_native")
        if h is None:
            h = _native.geometry(self.batch, self.c_in, self.h, self.w, self.c_out, self.kh, self.kw, *self.stride, *self.padding,
                                 *self.dilation, *self.output_padding, int(self.transposed))
            self.__dict__["_native"] = h  # (a frozen dataclass: fields, equality and hash are not touched)
        return h

    def __getstate__(self):  # copies and pickles carry the fields alone
        return {k: v for k, v in self.__dict__.items() if k != "_native"}

    def out_hw(self) -> Tuple[int, int]:
        d = self.desc(NML_F32, "nchw", NML_F32, "nchw", NML_F32, "f16", False)
        ho, wo = C.c_int(), C.c_int()
        check(_lib.load().nml_conv_output_size(C.byref(d), C.byref(ho), C.byref(wo)))
        return ho.value, wo.value

    def desc(self, in_dtype, in_layout, out_dtype, out_layout, w_dtype, math, round_out_f16) -> ConvDesc:
        d = ConvDesc()
        d.batch, d.c_in, d.h, d.w = self.batch, self.c_in, self.h, self.w
        d.c_out, d.kh, d.kw = self.c_out, self.kh, self.kw
        d.stride_h, d.stride_w = self.stride
        d.pad_h, d.pad_w = self.padding
        d.dil_h, d.dil_w = self.dilation
        d.outpad_h, d.outpad_w = self.output_padding
        d.transposed = int(self.transposed)
        d.in_dtype, d.in_layout = in_dtype, _LAYOUT[in_layout]
        d.out_dtype, d.out_layout = out_dtype, _LAYOUT[out_layout]
        d.w_dtype = w_dtype
        d.math = _MATH[math]
        d.round_out_f16 = int(bool(round_out_f16))
        return d

    def act_shape(self, which: str, layout: str) -> Tuple[int, int, int, int]:
        """Shape of the layer input (``which='in'``) or output (``'out'``) in the given layout."""
        if which == "in":
            c, h, w = self.c_in, self.h, self.w
        else:
            c = self.c_out
            h, w = self.out_hw()
        return (self.batch, c, h, w) if layout == "nchw" else (self.batch, h, w, c)

    def weight_shape(self) -> Tuple[int, int, int, int]:
        if self.transposed:
            return (self.c_in, self.c_out, self.kh, self.kw)
        return (self.c_out, self.c_in, self.kh, self.kw)


class Workspace:
    """Grow-only device scratch buffer handed to the C ABI (which itself never allocates)."""

    def __init__(self) -> None:
        self.buf: Optional[torch.Tensor] = None

    def get(self, nbytes: int, device) -> Tuple[Optional[int], int]:
        if nbytes == 0:
            return None, 0
        if self.buf is None or self.buf.numel() < nbytes or self.buf.device != torch.device(device):
            self.buf = torch.empty(int(nbytes * 1.25) + 256, dtype=torch.uint8, device=device)
        return self.buf.data_ptr(), self.buf.numel()


_default_ws = Workspace()


def conv_forward(g: ConvGeometry, x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, *,
                 layout: str = "nchw", out_layout: Optional[str] = None, math: str = "f16",
                 out_dtype: Optional[torch.dtype] = None, round_out_f16: bool = False,
                 out: Optional[torch.Tensor] = None, ws: Optional[Workspace] = None) -> torch.Tensor:
    lay = _LAYOUT[layout]
    return _native.conv_forward(g.native(), x, w, bias, out, lay, _LAYOUT[out_layout] if out_layout else lay, _MATH[math],
                                _out_dtype(out_dtype), 1 if round_out_f16 else 0, ws or _default_ws)


def conv_backward_data(g: ConvGeometry, dy: torch.Tensor, w: torch.Tensor, *, layout: str = "nchw",
                       out_layout: Optional[str] = None, math: str = "f16",
                       out_dtype: Optional[torch.dtype] = None, out: Optional[torch.Tensor] = None,
                       ws: Optional[Workspace] = None) -> torch.Tensor:
    lay = _LAYOUT[layout]
    return _native.conv_backward_data(g.native(), dy, w, out, lay, _LAYOUT[out_layout] if out_layout else lay, _MATH[math],
                                      _out_dtype(out_dtype), ws or _default_ws)


def conv_backward_weight(g: ConvGeometry, x: torch.Tensor, dy: torch.Tensor, *, layout: str = "nchw",
                         math: str = "f16", want_bias_grad: bool = True, dw: Optional[torch.Tensor] = None,
                         db: Optional[torch.Tensor] = None,
                         ws: Optional[Workspace] = None) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """dw (fp32, weight-shaped) and db (fp32, c_out); pass ``dw`` / ``db`` to have them written in place, e.g.
    into the views of a flat gradient bucket."""
    return _native.conv_backward_weight(g.native(), x, dy, dw, db, _LAYOUT[layout], _MATH[math], 1 if want_bias_grad else 0,
                                        ws or _default_ws)


def linear_forward(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, *, math: str = "f16",
                   out_dtype: Optional[torch.dtype] = None, round_out_f16: bool = False,
                   out: Optional[torch.Tensor] = None, ws: Optional[Workspace] = None) -> torch.Tensor:
    """y[rows, out] = x[rows, in] @ w[out, in].T + bias."""
    return _native.linear_forward(x, w, bias, out, _MATH[math], _out_dtype(out_dtype), 1 if round_out_f16 else 0, ws or _default_ws)


def linear_backward_data(dy: torch.Tensor, w: torch.Tensor, *, math: str = "f16",
                         out_dtype: Optional[torch.dtype] = None, out: Optional[torch.Tensor] = None,
                         ws: Optional[Workspace] = None) -> torch.Tensor:
    """dx[rows, in] = dy[rows, out] @ w[out, in]."""
    return _native.linear_backward_data(dy, w, out, _MATH[math], _out_dtype(out_dtype), ws or _default_ws)


def linear_backward_weight(x: torch.Tensor, dy: torch.Tensor, *, math: str = "f16", want_bias_grad: bool = True,
                           dw: Optional[torch.Tensor] = None, db: Optional[torch.Tensor] = None,
                           ws: Optional[Workspace] = None) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """dw[out, in] = dy.T @ x (fp32), db[out] = dy.sum(0) (fp32)."""
    return _native.linear_backward_weight(x, dy, dw, db, _MATH[math], 1 if want_bias_grad else 0, ws or _default_ws)


def device_status() -> int:
    """Synchronises and raises if a kernel abandoned a bounded wait since the last call."""
    code = C.c_int(0)
    st = _lib.load().nml_device_status(C.byref(code))
    if st != 0:
        raise _lib.NectarB200Error(f"device-side failure, code {code.value}: "
                                   f"{_lib.load().nml_status_string(st).decode()}")
    return 0


def set_sm_limit(sms: int) -> None:
    """Caps the SMs later launches occupy (0: all); used while a collective shares the GPU."""
    check(_lib.load().nml_set_sm_limit(int(sms)))


def launch_count() -> int:
    return int(_lib.load().nml_launch_count())


def profile_begin(max_records: int) -> None:
    """Start bracketing the next ``max_records`` contraction-kernel launches with CUDA events."""
    check(_lib.load().nml_profile_begin(int(max_records)))


def profile_end(max_records: int):
    """Synchronise and return the recorded per-launch durations (ms) in launch order."""
    buf = (C.c_float * max_records)()
    n = C.c_int(0)
    check(_lib.load().nml_profile_end(buf, max_records, C.byref(n)))
    return [float(buf[i]) for i in range(n.value)]


def tma_box(t: torch.Tensor, box, elem_strides, coords) -> torch.Tensor:
    """Test support: returns one TMA box of a 4-D tensor (``t.shape`` slowest-first, as torch
    prints it; ``box``/``elem_strides``/``coords`` fastest-first, as TMA takes them)."""
    assert t.dim() == 4 and t.is_contiguous()
    dims = list(reversed(t.shape))
    n = 1
    for b, s in zip(box, elem_strides):
        n *= (b + s - 1) // s
    out = torch.zeros(n, dtype=t.dtype, device=t.device)
    arr = lambda v: (C.c_int * 4)(*v)
    check(_lib.load().nml_debug_tma_box(_ptr(t), t.element_size(), arr(dims), arr(box), arr(elem_strides),
                                        arr(coords), _ptr(out), out.numel() * out.element_size(), _stream()))
    return out

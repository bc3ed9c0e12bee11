"""Drop-in for the part of the reference's pybind module ``_nectarml`` that this path covers.

The reference's Python wrappers call ``_nectarml.tensor.conv.conv2d(...)`` and friends with
device pointers as integers plus shape ints and get a device pointer back
(nectarml/cuda/tensor/conv.py:138-146, 157-171, 211-220, 232-247;
nectarml/cuda/tensor/matmul.py:9-10; registration in nectarml/csrc/python/bindings.cpp:41-51,
prototypes in nectarml/csrc/python/ops/tensor/conv.h:71-150 and matmul.h:10-16).  The same
names, argument order and error type (``RuntimeError``) are kept here and forwarded to the
``nml_ref_*`` entry points of the C ABI (by ``csrc/nml_dropin.cpp``).  ``DType`` mirrors the reference's enum
(nectarml/csrc/include/common/dtype.h:15-21); only Float32 and Float16 are valid on this path.
"""
from __future__ import annotations

import enum
from typing import Sequence

from . import _lib


class DType(enum.IntEnum):
    Float32 = 0
    Float16 = 1
    UInt8 = 2
    Int32 = 3
    Bool = 4


class _LazyNative:
    """Stands in for the native module until its first use, so that this file can be imported before the build."""

    def __getattr__(self, name):
        global _native
        _lib.load()
        try:
            from . import _dropin as module
        except ImportError as e:
            raise _lib.NectarB200Error(f"nectarml_b200/_dropin.so: {e}; build it with `python -m nectarml_b200.build`") from e
        _native = module
        return getattr(module, name)


_native = _LazyNative()


def _dtype(dtype) -> int:
    v = int(dtype)
    if v != 0 and v != 1:
        raise RuntimeError("conv / matmul only support float32 and float16")
    return v


class _Conv:
    """``_nectarml.tensor.conv``"""

    @staticmethod
    def conv2d(input_ptr, input_size, weight_ptr, weight_size, bias_ptr, bias_size, output_size, B, C_in, H, W,
               C_out, KH, KW, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w, groups, dtype,
               half_precision) -> int:
        return _native.conv2d(input_ptr, input_size, weight_ptr, weight_size, bias_ptr or 0,
                              bias_size, output_size, B, C_in, H, W, C_out, KH, KW, stride_h, stride_w, padding_h, padding_w,
                              dilation_h, dilation_w, groups, _dtype(dtype), int(bool(half_precision)))

    @staticmethod
    def conv_transpose2d(input_ptr, input_size, weight_ptr, weight_size, bias_ptr, bias_size, output_size, B, C_in,
                         H, W, C_out, KH, KW, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w,
                         output_padding_h, output_padding_w, groups, dtype, half_precision) -> int:
        return _native.conv_transpose2d(input_ptr, input_size, weight_ptr, weight_size,
                                        bias_ptr or 0, bias_size, output_size, B, C_in, H, W, C_out, KH, KW, stride_h, stride_w,
                                        padding_h, padding_w, dilation_h, dilation_w, output_padding_h, output_padding_w, groups,
                                        _dtype(dtype), int(bool(half_precision)))

    @staticmethod
    def conv2d_backward_input(out_grad_ptr, weight_ptr, B, C_in, H, W, C_out, KH, KW, H_out, W_out, stride_h,
                              stride_w, padding_h, padding_w, dilation_h, dilation_w, groups, dtype) -> int:
        return _native.conv2d_backward_input(out_grad_ptr, weight_ptr, B, C_in, H, W, C_out, KH,
                                             KW, H_out, W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w, groups,
                                             _dtype(dtype))

    @staticmethod
    def conv_transpose2d_backward_input(out_grad_ptr, weight_ptr, B, C_in, H, W, C_out, KH, KW, H_out, W_out,
                                        stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w, groups,
                                        dtype) -> int:
        return _native.conv_transpose2d_backward_input(out_grad_ptr, weight_ptr, B, C_in, H, W,
                                                       C_out, KH, KW, H_out, W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w,
                                                       groups, _dtype(dtype))

    @staticmethod
    def conv2d_backward_weight(out_grad_ptr, input_ptr, B, C_in, H, W, C_out, KH, KW, H_out, W_out, stride_h,
                               stride_w, padding_h, padding_w, dilation_h, dilation_w, dtype) -> int:
        return _native.conv2d_backward_weight(out_grad_ptr, input_ptr, B, C_in, H, W, C_out, KH,
                                              KW, H_out, W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w,
                                              _dtype(dtype))

    @staticmethod
    def conv_transpose2d_backward_weight(out_grad_ptr, input_ptr, B, C_in, H, W, C_out, KH, KW, H_out, W_out,
                                         stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w,
                                         dtype) -> int:
        return _native.conv_transpose2d_backward_weight(out_grad_ptr, input_ptr, B, C_in, H, W,
                                                        C_out, KH, KW, H_out, W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w,
                                                        _dtype(dtype))


    # 1-D convolutions (nectarml/csrc/python/ops/tensor/conv.h:11-68; callers nectarml/cuda/tensor/conv.py:12-106)
    @staticmethod
    def conv1d(input_ptr, weight_ptr, bias_ptr, B, C_in, L, C_out, K, stride, padding, dilation, groups, dtype) -> int:
        return _native.conv1d(input_ptr, weight_ptr, bias_ptr or 0, B, C_in, L, C_out, K, stride,
                              padding, dilation, groups, _dtype(dtype))

    @staticmethod
    def conv_transpose1d(input_ptr, weight_ptr, bias_ptr, B, C_in, L, C_out, K, stride, padding, dilation,
                         output_padding, groups, dtype) -> int:
        return _native.conv_transpose1d(input_ptr, weight_ptr, bias_ptr or 0, B, C_in, L, C_out, K,
                                        stride, padding, dilation, output_padding, groups, _dtype(dtype))

    @staticmethod
    def conv1d_backward_input(out_grad_ptr, weight_ptr, B, C_in, L, C_out, K, L_out, stride, padding, dilation,
                              groups, dtype) -> int:
        return _native.conv1d_backward_input(out_grad_ptr, weight_ptr, B, C_in, L, C_out, K, L_out,
                                             stride, padding, dilation, groups, _dtype(dtype))

    @staticmethod
    def conv_transpose1d_backward_input(out_grad_ptr, weight_ptr, B, C_in, L, C_out, K, L_out, stride, padding,
                                        dilation, groups, dtype) -> int:
        return _native.conv_transpose1d_backward_input(out_grad_ptr, weight_ptr, B, C_in, L, C_out,
                                                       K, L_out, stride, padding, dilation, groups, _dtype(dtype))

    @staticmethod
    def conv1d_backward_weight(out_grad_ptr, input_ptr, B, C_in, L, C_out, K, L_out, stride, padding, dilation,
                               dtype) -> int:
        return _native.conv1d_backward_weight(out_grad_ptr, input_ptr, B, C_in, L, C_out, K, L_out,
                                              stride, padding, dilation, _dtype(dtype))

    @staticmethod
    def conv_transpose1d_backward_weight(out_grad_ptr, input_ptr, B, C_in, L, C_out, K, L_out, stride, padding,
                                         dilation, dtype) -> int:
        return _native.conv_transpose1d_backward_weight(out_grad_ptr, input_ptr, B, C_in, L, C_out,
                                                        K, L_out, stride, padding, dilation, _dtype(dtype))


class _Tensor:
    """``_nectarml.tensor``"""
    conv = _Conv()

    @staticmethod
    def matmul(a_ptr, b_ptr, a_shape: Sequence[int], b_shape: Sequence[int], dtype) -> int:
        return _native.matmul(a_ptr, b_ptr, a_shape, b_shape, _dtype(dtype))


tensor = _Tensor()


def free_cuda(ptr: int, n_elements: int = 0, dtype=None) -> None:
    """Releases a result pointer (the reference's ``_nectarml.free_cuda(ptr, n_elements, dtype)``)."""
    _native.free(ptr)

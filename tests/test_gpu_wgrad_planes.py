"""Small weight gradients of many pixels: the sums over the K slices' planes, several threads to an element."""
import pytest
import torch

from gpu_util import assert_f32
from nectarml_b200 import _lib, ops
from nectarml_b200.ops import ConvGeometry

pytestmark = pytest.mark.gpu


# rows of float4s (1x1), taps side by side (several taps, whole groups of four channels), the general form (broken ones, a transposed layer), few
# and many planes, one tap on both sides of 37888 elements, dW that does not start on 16 bytes
# (several: whether that many planes get several threads an element, in fp16, in fp32, in fp32 with dW that does not start on 16 bytes)
@pytest.mark.parametrize("n,c_in,hw,c_out,k,s,transposed,several", [
    (51, 40, 13, 16, 1, 1, False, (1, 1, 1)), (6, 32, 83, 17, 1, 1, False, (1, 1, 1)), (3, 24, 9, 33, 1, 1, False, (0, 1, 0)), (66, 24, 11, 80, 3, 1, False, (1, 1, 1)),
    (40, 136, 20, 9, 3, 1, False, (0, 0, 0)), (6, 182, 73, 33, 3, 1, True, (1, 0, 0)), (20, 25, 24, 30, 5, 1, False, (0, 1, 1)), (12, 102, 17, 33, 3, 2, False, (0, 0, 0)),
    (2, 30, 6, 31, 3, 1, False, (0, 0, 0)), (10, 177, 27, 214, 1, 1, False, (1, 1, 1)), (10, 177, 27, 215, 1, 1, False, (0, 0, 0))])
@pytest.mark.parametrize("math,dtype", [("f16", torch.float16), ("3xtf32", torch.float32)])
@pytest.mark.parametrize("shift", [0, 1])
def test_sums_over_planes(n, c_in, hw, c_out, k, s, transposed, several, math, dtype, shift):
    gen = torch.Generator(device="cuda").manual_seed(n + c_in + c_out)
    g = ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), (k // 2, k // 2), transposed=transposed)
    x = torch.randn(g.act_shape("in", "nhwc"), device="cuda", generator=gen).to(dtype)
    dy = torch.randn(g.act_shape("out", "nhwc"), device="cuda", generator=gen).to(dtype)
    shape = g.weight_shape()
    count = shape[0] * shape[1] * shape[2] * shape[3]
    dw = torch.full((count + shift,), float("nan"), device="cuda")[shift:].view(shape)
    before = _lib.load().nml_debug_launch_count(7)
    ops.conv_backward_weight(g, x, dy, layout="nhwc", math=math, want_bias_grad=False, dw=dw)
    assert _lib.load().nml_debug_launch_count(7) - before == several[0 if math == "f16" else 1 + shift]
    wd = torch.zeros(shape, device="cuda", dtype=torch.double, requires_grad=True)
    f = torch.nn.functional.conv_transpose2d if transposed else torch.nn.functional.conv2d
    y = f(x.permute(0, 3, 1, 2).double(), wd, stride=s, padding=k // 2)
    (want,) = torch.autograd.grad(y, wd, dy.permute(0, 3, 1, 2).double())
    assert_f32(dw.cpu(), want.cpu(), "dw")
    ops.device_status()

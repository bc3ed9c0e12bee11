"""Channel-major fp32 tensors on their way into the two planes of the 3xTF32 split: channel counts around the groups of four and eight that a
thread stores, images of whole and of broken quads of pixels."""
import pytest
import torch

from gpu_util import assert_f32
from nectarml_b200 import ops
from nectarml_b200.ops import ConvGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c_in,c_out", [(1, 5), (4, 12), (12, 8), (60, 67), (67, 60), (68, 130), (132, 3)])
@pytest.mark.parametrize("h,w", [(7, 9), (12, 10)])
def test_channel_groups(c_in, c_out, h, w):
    gen = torch.Generator(device="cuda").manual_seed(c_in * 1000 + c_out + h)
    g = ConvGeometry(3, c_in, h, w, c_out, 3, 3, (1, 1), (1, 1))
    x = torch.randn(3, c_in, h, w, device="cuda", generator=gen)
    wt = torch.randn(c_out, c_in, 3, 3, device="cuda", generator=gen)
    dy = torch.randn(3, c_out, h, w, device="cuda", generator=gen)
    xd, wd = x.double().requires_grad_(), wt.double().requires_grad_()
    y = torch.nn.functional.conv2d(xd, wd, padding=1)
    dx, dw = torch.autograd.grad(y, (xd, wd), dy.double())
    assert_f32(ops.conv_forward(g, x, wt, math="3xtf32").cpu(), y.detach().cpu(), "y")
    assert_f32(ops.conv_backward_data(g, dy, wt, math="3xtf32").cpu(), dx.cpu(), "dx")
    got, db = ops.conv_backward_weight(g, x, dy, math="3xtf32")
    assert_f32(got.cpu(), dw.cpu(), "dw")
    assert_f32(db.cpu(), dy.double().sum((0, 2, 3)).cpu(), "db")
    ops.device_status()

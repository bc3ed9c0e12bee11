"""The patch walk whose weights do not stay in shared memory: the taps of a channel block read one patch, their weights come through a ring, a
few taps to a stage."""
import pytest
import torch

from gpu_util import assert_f32
from nectarml_b200 import _lib, ops
from nectarml_b200.ops import ConvGeometry

pytestmark = pytest.mark.gpu
STREAMED = 4  # kind of nml_debug_launch_count


def streamed():
    return _lib.load().nml_debug_launch_count(STREAMED)


def conv(x, w, g):
    f = torch.nn.functional.conv_transpose2d if g.transposed else torch.nn.functional.conv2d
    return f(x, w, stride=g.stride, padding=g.padding)


# one channel block and a broken one, taps in whole stages and not (9 of 9, 25 and 49 of fewer; 4 a phase in fp32), one column tile of 16 ... 192 columns,
# tiles hanging over the image, several tiles per CTA, the phases of a strided gather: nine taps each, and 9, 12, 12 and 16
@pytest.mark.parametrize("n,c_in,hw,c_out,k,s,transposed", [
    (9, 256, 32, 64, 3, 1, False), (9, 200, 31, 24, 5, 1, False), (87, 64, 31, 144, 3, 1, False), (4, 136, 48, 192, 3, 1, False), (40, 520, 16, 9, 3, 1, True),
    (3, 256, 61, 40, 7, 1, False), (9, 640, 47, 16, 3, 1, False),
    (4, 200, 47, 40, 6, 2, True), (3, 136, 61, 24, 7, 2, True)])
def test_fp16(n, c_in, hw, c_out, k, s, transposed):
    gen = torch.Generator(device="cuda").manual_seed(c_in + c_out)
    g = ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), (k // 2 if s == 1 else 1,) * 2, transposed=transposed)
    x = torch.randn(g.act_shape("in", "nhwc"), device="cuda", generator=gen).half()
    w = (torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.05).half()
    b = torch.randn(c_out, device="cuda", generator=gen).half()
    before = streamed()
    y = ops.conv_forward(g, x, w, b, layout="nhwc", math="f16")
    assert streamed() == before + 1
    want = (conv(x.permute(0, 3, 1, 2).double(), w.double(), g) + b.double().view(-1, 1, 1)).permute(0, 2, 3, 1)
    # one rounding to fp16 (two where a ragged row's bias is added to the rounded sum), fp32 sums well below it
    bound = (want.abs() + b.double().abs() + want.abs().amax() / 64) * 2.0 ** -10
    assert ((y.double() - want).abs() <= bound).all()
    ops.device_status()


@pytest.mark.parametrize("n,c_in,hw,c_out,k,s,transposed", [
    (9, 128, 33, 32, 3, 1, False), (14, 3, 73, 100, 3, 1, False), (33, 70, 31, 64, 3, 1, False), (3, 128, 64, 24, 5, 1, False), (8, 232, 30, 24, 4, 2, True)])
def test_split_of_fp32(n, c_in, hw, c_out, k, s, transposed):
    """Forward, or for an image's few channels the input gradient."""
    gen = torch.Generator(device="cuda").manual_seed(c_in + c_out)
    g = ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), (k // 2 if s == 1 else 1,) * 2, transposed=transposed)
    w = torch.randn(g.weight_shape(), device="cuda", generator=gen)
    x = torch.randn(g.act_shape("in", "nchw"), device="cuda", generator=gen)
    before = streamed()
    if c_in > 3:
        got, want = ops.conv_forward(g, x, w, math="3xtf32"), conv(x.double(), w.double(), g)
    else:
        dy = torch.randn(g.act_shape("out", "nchw"), device="cuda", generator=gen)
        got = ops.conv_backward_data(g, dy, w, math="3xtf32")
        want = torch.nn.functional.conv_transpose2d(dy.double(), w.double(), padding=k // 2)
    assert streamed() == before + 1
    assert_f32(got.cpu(), want.cpu(), "fp32")
    again = ops.conv_forward(g, x, w, math="3xtf32") if c_in > 3 else ops.conv_backward_data(g, dy, w, math="3xtf32")
    assert torch.equal(got, again)
    ops.device_status()


@pytest.mark.parametrize("n,c_in,h,w,c_out,k,by_patches", [
    (82, 50, 3, 3, 184, 5, False), (31, 103, 2, 23, 208, 3, False), (80, 97, 9, 5, 220, 3, False), (41, 49, 7, 14, 211, 5, False),
    (34, 67, 69, 7, 152, 3, True), (14, 111, 23, 35, 131, 5, True), (114, 152, 14, 13, 178, 5, True), (6, 90, 53, 4, 133, 3, True), (3, 24, 10, 22, 151, 3, True)])
def test_wide_tiles_are_weighed_against_the_width_of_boxes(n, c_in, h, w, c_out, k, by_patches):
    """More than 128 columns are one tile, two or several of 64, whichever walk and width are estimated to be the faster: the ones named here
    measured 0.68 to 0.9 of the time of the other walk."""
    gen = torch.Generator(device="cuda").manual_seed(n + c_out)
    g = ConvGeometry(n, c_in, h, w, c_out, k, k, (1, 1), (k // 2, k // 2))
    x = torch.randn(g.act_shape("in", "nhwc"), device="cuda", generator=gen).half()
    wt = (torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.05).half()
    before = streamed()
    y = ops.conv_forward(g, x, wt, None, layout="nhwc", math="f16")
    assert streamed() - before == int(by_patches)
    want = conv(x.permute(0, 3, 1, 2).double(), wt.double(), g).permute(0, 2, 3, 1)
    assert ((y.double() - want).abs() <= (want.abs() + want.abs().amax() / 64) * 2.0 ** -10).all()
    ops.device_status()

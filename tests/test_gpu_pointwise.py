"""1x1 convolutions of unit stride: fp16 rows of pixels go through the Linear layer's rules, channel-major images become images of one row."""
import pytest
import torch

from gpu_util import assert_f32
from nectarml_b200 import _lib, ops
from nectarml_b200.ops import ConvGeometry

pytestmark = pytest.mark.gpu


def as_linear():
    """Passes of 1x1 layers that went through the Linear layer's rules so far."""
    return _lib.load().nml_debug_launch_count(8)


def tensors(g, layout, dtype, seed, shift=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x, dy = (torch.randn(g.act_shape(k, layout), device="cuda", generator=gen).to(dtype) for k in ("in", "out"))
    n = g.c_in * g.c_out
    w = (torch.randn(n + shift, device="cuda", generator=gen) * 0.1).to(dtype)[shift:].view(g.weight_shape())
    return x, w, torch.randn(g.c_out, device="cuda", generator=gen).to(dtype), dy


# weights that start on 16 bytes (read in place) and not (repacked), whole vectors of channels and not, inputs of whole groups of 64 (the input
# gradient reads its weights in place), a K loop of one or two slices on few rows, one pixel per image
@pytest.mark.parametrize("n,c_in,h,w,c_out", [(3, 64, 9, 11, 192), (2, 520, 5, 5, 128), (5, 100, 7, 6, 77), (300, 128, 1, 1, 40), (40, 256, 17, 17, 1000), (2, 8, 3, 3, 8)])
@pytest.mark.parametrize("shift", [0, 1])
def test_fp16_rows(n, c_in, h, w, c_out, shift):
    g = ConvGeometry(n, c_in, h, w, c_out, 1, 1)
    x, wt, b, dy = tensors(g, "nhwc", torch.float16, c_in + c_out, shift)
    assert (wt.data_ptr() & 15) == 2 * shift
    wd, rows = wt.double().view(c_out, c_in), n * h * w
    xd, dyd = x.double().view(rows, c_in), dy.double().view(rows, c_out)
    want = xd @ wd.t() + b.double()
    before = as_linear()
    y = ops.conv_forward(g, x, wt, b, layout="nhwc").double().view(rows, c_out)
    # one rounding to fp16, or two where a ragged row's bias is added to the rounded sum
    assert ((y - want).abs() <= 2.0 ** -10 * (want.abs() + b.double().abs() + want.abs().amax() / 64)).all()
    want = dyd @ wd
    dx = ops.conv_backward_data(g, dy, wt, layout="nhwc").double().view(rows, c_in)
    assert ((dx - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -13 * want.abs().amax()).all()
    dw, db = ops.conv_backward_weight(g, x, dy, layout="nhwc")
    assert_f32(dw.view(c_out, c_in).cpu(), (dyd.t() @ xd).cpu(), "dw")
    assert_f32(db.cpu(), dyd.sum(0).cpu(), "db")
    assert as_linear() == before + 3
    ops.device_status()


# images below and above the size from which results are flat, rows of whole vectors and not, results below and above the size from which one
# row of whole vectors leaves by TMA
@pytest.mark.parametrize("n,c_in,h,w,c_out", [(3, 40, 22, 23, 72), (2, 70, 23, 23, 33), (5, 16, 30, 31, 200), (2, 96, 54, 54, 40), (13, 16, 54, 54, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_channel_major(n, c_in, h, w, c_out, dtype):
    g, math = ConvGeometry(n, c_in, h, w, c_out, 1, 1), "3xtf32" if dtype == torch.float32 else "f16"
    x, wt, b, dy = tensors(g, "nchw", dtype, c_in + c_out)
    wd, xd, dyd = wt.double().view(c_out, c_in), x.double().flatten(2), dy.double().flatten(2)
    y = ops.conv_forward(g, x, wt, b, math=math).double().flatten(2)
    dx = ops.conv_backward_data(g, dy, wt, math=math).double().flatten(2)
    dw, db = ops.conv_backward_weight(g, x, dy, math=math)
    if dtype == torch.float32:
        assert_f32(y.cpu(), (wd @ xd + b.double().view(-1, 1)).cpu(), "y")
        assert_f32(dx.cpu(), (wd.t() @ dyd).cpu(), "dx")
    else:
        for got, want in ((y, wd @ xd + b.double().view(-1, 1)), (dx, wd.t() @ dyd)):
            assert ((got - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -13 * want.abs().amax()).all()
    assert_f32(dw.view(c_out, c_in).cpu(), torch.einsum("nop,nip->oi", dyd, xd).cpu(), "dw")
    assert_f32(db.cpu(), dyd.sum((0, 2)).cpu(), "db")
    ops.device_status()


@pytest.mark.parametrize("n,c_in,h,w,c_out,layout", [(2, 126, 104, 3, 248, "nhwc"), (1, 6, 10, 33, 16, "nchw"), (3, 64, 26, 14, 96, "nchw"), (40, 48, 5, 5, 160, "nhwc")])
def test_weight_gradients_keep_the_sums_of_their_images(n, c_in, h, w, c_out, layout):
    """Pixels of all images in one row make fewer K blocks, which must not become longer sums: the tensor core truncates as it accumulates,
    up to 2^-23 of the running sum per instruction of 16 products.  A block is four of them; here a slice has one or two blocks, whose
    sums then grow to the result as the root of their number: at most 8 * 2^-23 / sqrt(slices), 3.2e-7 for the shortest."""
    g = ConvGeometry(n, c_in, h, w, c_out, 1, 1)
    x, _, _, dy = tensors(g, layout, torch.float16, n + h)
    dw = ops.conv_backward_weight(g, x, dy, layout=layout, want_bias_grad=False)[0].double().view(c_out, c_in)
    flat = (lambda t: t.double().flatten(0, 2)) if layout == "nhwc" else (lambda t: t.double().flatten(2).transpose(1, 2).flatten(0, 1))
    want = flat(dy).t() @ flat(x)
    assert float((dw - want).norm() / want.norm()) <= 3.2e-7
    ops.device_status()


@pytest.mark.parametrize("n,c_in,h,w,c_out,copied", [(66, 104, 62, 29, 24, True), (60, 72, 31, 23, 200, True), (31, 248, 128, 16, 24, True), (2, 208, 1, 2, 1920, True), (16, 480, 64, 43, 1, True), (4, 480, 64, 43, 1, False), (30, 56, 21, 20, 576, False),
                                                    (8, 456, 46, 46, 16, False)])
def test_input_gradients_of_broken_groups(n, c_in, h, w, c_out, copied):
    """Weights whose last group of 64 inputs is far from whole are transposed first (a launch more) where many tiles or a long K loop read it."""
    g = ConvGeometry(n, c_in, h, w, c_out, 1, 1)
    _, wt, _, dy = tensors(g, "nhwc", torch.float16, c_in)
    launches = ops.launch_count()
    dx = ops.conv_backward_data(g, dy, wt, layout="nhwc")
    launches = ops.launch_count() - launches
    want = dy.double() @ wt.double().view(c_out, c_in)
    assert ((dx.double() - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -13 * want.abs().amax()).all()
    ops.device_status()
    assert launches == 1 + int(copied) + int(c_out % 8 != 0)  # (output gradients of broken vectors are converted)


@pytest.mark.parametrize("n,c_in,h,w,c_out,copied", [(64, 8, 21, 16, 200, True), (41, 104, 47, 41, 24, True), (41, 40, 47, 41, 24, True), (41, 64, 47, 41, 24, False),
                                                    (20, 104, 47, 41, 24, False), (30, 8, 25, 24, 24, False)])
def test_short_rows_of_weights(n, c_in, h, w, c_out, copied):
    """Weights of few input channels are copied into rows of whole slices (a launch more) where many tiles read them."""
    g = ConvGeometry(n, c_in, h, w, c_out, 1, 1)
    x, wt, _, _ = tensors(g, "nhwc", torch.float16, c_in)
    launches = ops.launch_count()
    y = ops.conv_forward(g, x, wt, None, layout="nhwc")
    launches = ops.launch_count() - launches
    want = x.double() @ wt.double().view(c_out, c_in).t()
    assert ((y.double() - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -13 * want.abs().amax()).all()
    ops.device_status()
    assert launches == 1 + int(copied)

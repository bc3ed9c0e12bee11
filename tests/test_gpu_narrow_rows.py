"""Row-major results whose width is no multiple of a 128-byte piece of columns: they leave by TMA stores whose last piece hangs over the
end of the row and is clipped there.  Widths around the pieces and the tiles, against float64, with guards around the result."""
import pytest
import torch

from nectarml_b200 import ops
from nectarml_b200.ops import ConvGeometry

pytestmark = pytest.mark.gpu


def guarded(*shape, dtype=torch.float16):
    """A tensor inside a larger one of NaNs; check() says whether they are all still there."""
    n = 1
    for s in shape:
        n *= s
    whole = torch.full((n + 2048,), float("nan"), device="cuda", dtype=dtype)
    return whole[1024:1024 + n].view(shape), lambda: bool(whole[:1024].isnan().all() and whole[1024 + n:].isnan().all())


def assert_rounded(got, want):
    """fp16 results of fp32 sums: one rounding (2^-11), the sums' own error below 2^-13 of the largest term."""
    bound = want.abs() * 2.0 ** -11 + 2.0 ** -13 * want.abs().amax()
    assert ((got.double() - want).abs() <= bound).all()


# one tile of 16 ... 224 columns, tiles whose width is rounded up to a piece (320: two of 192), few and many tiles per CTA
@pytest.mark.parametrize("rows", [3, 129, 40001])
@pytest.mark.parametrize("fout", [16, 24, 32, 40, 72, 96, 104, 160, 192, 224, 320, 328])
def test_linear_rows(rows, fout):
    gen = torch.Generator(device="cuda").manual_seed(rows + fout)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=gen).half()  # noqa: E731
    x, w, b, dy = rnd(rows, 200), rnd(fout, 200), rnd(fout), rnd(rows, 200)
    y, clean = guarded(rows, fout)
    ops.linear_forward(x, w, b, out=y)
    assert_rounded(y, x.double() @ w.double().t() + b.double())
    assert clean()
    dx, clean = guarded(rows, fout)  # the input gradient of a layer of `fout` inputs
    ops.linear_backward_data(dy, w.t().contiguous(), out=dx)
    assert_rounded(dx, dy.double() @ w.double().t())
    assert clean()
    ops.device_status()


# patch walk with 16- and 32-column tiles (four accumulators behind one another), its phases, and fp32 rows of 16 columns
@pytest.mark.parametrize("n,c_in,hw,c_out,k,s,transposed", [
    (3, 64, 19, 16, 3, 1, False), (40, 64, 28, 24, 3, 1, False), (40, 32, 33, 96, 5, 1, False), (5, 64, 17, 48, 4, 2, True), (3, 40, 15, 80, 3, 2, False)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_convolution_rows(n, c_in, hw, c_out, k, s, transposed, dtype):
    gen = torch.Generator(device="cuda").manual_seed(c_in + c_out)
    g = ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), (1, 1), transposed=transposed)
    x = torch.randn(g.act_shape("in", "nhwc"), device="cuda", generator=gen).half()
    w = (torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.1).half()
    y, clean = guarded(*g.act_shape("out", "nhwc"), dtype=dtype)
    ops.conv_forward(g, x, w, None, layout="nhwc", math="f16", out=y)
    conv = torch.nn.functional.conv_transpose2d if transposed else torch.nn.functional.conv2d
    assert_rounded(y, conv(x.permute(0, 3, 1, 2).double(), w.double(), stride=s, padding=1).permute(0, 2, 3, 1))
    assert clean()
    ops.device_status()


# four and eight fp32 columns: by TMA from 148 * 128 rows of eight columns on, below so only with an fp16 bias, of which the short epilogue
# takes a widened copy (a launch more); a few K slices, phases, and resident weights (tiles of 16
# columns, always the short epilogue)
@pytest.mark.parametrize("c_out", [4, 8])
@pytest.mark.parametrize("n,c_in,h,w,k,s,transposed,by_tma", [
    (1, 160, 148, 256, 1, 1, False, True), (1, 160, 147, 128, 1, 1, False, True), (3, 100, 151, 171, 1, 1, False, True), (2, 256, 75, 70, 1, 2, True, True),
    (2, 40, 149, 167, 3, 1, False, False)])
def test_four_and_eight_fp32_columns(c_out, n, c_in, h, w, k, s, transposed, by_tma):
    gen = torch.Generator(device="cuda").manual_seed(c_in + c_out)
    g = ConvGeometry(n, c_in, h, w, c_out, k, k, (s, s), (k // 2, k // 2), transposed=transposed)
    x = torch.randn(g.act_shape("in", "nhwc"), device="cuda", generator=gen).half()
    wt = (torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.1).half()
    b = torch.randn(c_out, device="cuda", generator=gen).half()
    y, clean = guarded(*g.act_shape("out", "nhwc"), dtype=torch.float32)
    launches = [ops.launch_count()]
    conv = torch.nn.functional.conv_transpose2d if transposed else torch.nn.functional.conv2d
    want = conv(x.permute(0, 3, 1, 2).double(), wt.double(), stride=s, padding=k // 2).permute(0, 2, 3, 1)
    for bias in (None, b):
        ops.conv_forward(g, x, wt, bias, layout="nhwc", math="f16", out=y)
        launches.append(ops.launch_count())
        ref = want if bias is None else want + bias.double()
        assert (y.double() - ref).abs().max() <= 1e-5 * ref.abs().max()
        assert clean()
    ops.device_status()
    assert (launches[2] - launches[1]) - (launches[1] - launches[0]) == (0 if by_tma else 1)


@pytest.mark.parametrize("n,c_in,h,w,c_out,k,whole_pieces", [(114, 300, 8, 9, 152, 5, False), (9, 88, 90, 5, 144, 5, False), (5, 64, 9, 14, 192, 3, True)])
def test_long_k_loops_are_worth_tiles_that_are_no_whole_pieces(n, c_in, h, w, c_out, k, whole_pieces):
    """Two tiles of 96 columns leave by the plain epilogue, with a widened copy of the bias (a launch), three of 64 by TMA."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = ConvGeometry(n, c_in, h, w, c_out, k, k, (1, 1), (k // 2, k // 2))
    x = torch.randn(g.act_shape("in", "nhwc"), device="cuda", generator=gen).half()
    wt = (torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.05).half()
    b = torch.randn(c_out, device="cuda", generator=gen).half()
    y, clean = guarded(*g.act_shape("out", "nhwc"))
    launches = [ops.launch_count()]
    for bias in (None, b):
        ops.conv_forward(g, x, wt, bias, layout="nhwc", math="f16", out=y)
        launches.append(ops.launch_count())
    want = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), wt.double(), b.double(), padding=k // 2).permute(0, 2, 3, 1)
    # (the bias of the plain epilogue is added to the rounded sum)
    assert ((y.double() - want).abs() <= (want.abs() + b.double().abs()) * 2.0 ** -10 + 2.0 ** -13 * want.abs().amax()).all()
    assert clean()
    ops.device_status()
    assert (launches[2] - launches[1]) - (launches[1] - launches[0]) == (0 if whole_pieces else 1)

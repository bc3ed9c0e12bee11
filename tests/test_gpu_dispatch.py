"""Sizes at the edges of the dispatch rules: batched products in one launch, rows that do not start on 16 bytes, K
split over CTAs for few-tile layers.  fp16 results are compared with the oracle on fp16-rounded inputs (1e-2 rel / 1e-3
abs), fp32 ones with 1e-5 of max|ref|, as everywhere in this suite."""
import numpy as np
import pytest
import torch

from gpu_util import F16, F32, assert_f16, assert_f32, dev, fetch, host
from nectarml_b200 import _lib, _nectarml, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,m,k,n", [
    (3, 1, 8, 1), (5, 127, 64, 63), (2, 128, 64, 64), (4, 129, 96, 65), (3, 333, 64, 333), (2, 40, 130, 257), (7, 130, 72, 264),
    (2, 300, 200, 512)])
def test_batched_matmul_entries_share_a_launch(batch, m, k, n, oracle):
    rng = np.random.default_rng(m * n + k)
    a = rng.standard_normal((batch, m, k), dtype=np.float32)
    b = rng.standard_normal((batch, k, n), dtype=np.float32)
    a32, b32 = dev(a), dev(b)
    launches = ops.launch_count()
    ptr = _nectarml.tensor.matmul(a32.data_ptr(), b32.data_ptr(), a.shape, b.shape, F32)
    assert ops.launch_count() - launches <= 4  # conversion of A and of B, the product, at most one more
    assert_f32(fetch(ptr, (batch, m, n)), oracle.matmul(a, b), "fp32")
    a16, b16 = dev(a, torch.float16), dev(b, torch.float16)
    ptr = _nectarml.tensor.matmul(a16.data_ptr(), b16.data_ptr(), a.shape, b.shape, F16)
    r = oracle.round_f16
    assert_f16(fetch(ptr, (batch, m, n), np.float16), oracle.matmul(r(a), r(b)), "fp16")
    ops.device_status()


# tall and narrow, short and wide: what the conversions cost decides whether the operands are read in place (one launch, else
# three)
@pytest.mark.parametrize("batch,m,k,n,launches32,launches16", [
    (40, 15001, 6, 1, 3, 3), (9, 3000, 16, 8, None, None), (30, 12000, 40, 9, 3, None), (17, 1367, 72, 40, None, None), (70, 12, 284, 1199, 1, None),
    (90, 4, 129, 602, 1, 1), (24, 190, 471, 33, None, None), (64, 45, 64, 1001, 1, None), (300, 1, 40, 77, 1, 1)])
def test_batched_matmul_tall_and_wide(batch, m, k, n, launches32, launches16):
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(batch, m, k, device="cuda", generator=gen)
    b = torch.randn(batch, k, n, device="cuda", generator=gen)
    for dt, code, want_launches in ((torch.float32, F32, launches32), (torch.float16, F16, launches16)):
        ad, bd = a.to(dt), b.to(dt)
        torch.cuda.synchronize()
        before = ops.launch_count()
        ptr = _nectarml.tensor.matmul(ad.data_ptr(), bd.data_ptr(), a.shape, b.shape, code)
        launched = ops.launch_count() - before
        want = (ad.double() @ bd.double()).cpu().numpy()
        if dt == torch.float32:
            assert_f32(fetch(ptr, (batch, m, n)), want, "fp32")
        else:  # (an absolute bound of the results' size)
            assert_f16(fetch(ptr, (batch, m, n), np.float16), want, "fp16", atol=1e-3 * max(1.0, k ** 0.5))
        assert want_launches is None or launched == want_launches, (dt, launched)
    ops.device_status()


@pytest.mark.parametrize("fout", [1, 2, 9, 31, 33, 63, 65, 127, 257, 333])
@pytest.mark.parametrize("rows", [1, 130])
def test_rows_that_do_not_start_on_16_bytes(rows, fout, oracle):
    rng = np.random.default_rng(rows * 1000 + fout)
    x = rng.standard_normal((rows, 72), dtype=np.float32)
    w = (rng.standard_normal((fout, 72), dtype=np.float32) * 0.2).astype(np.float32)
    b = rng.standard_normal(fout, dtype=np.float32)
    assert_f32(host(ops.linear_forward(dev(x), dev(w), dev(b), math="3xtf32")), oracle.linear_forward(x, w, b), "fp32")
    r, h = oracle.round_f16, torch.float16
    want = oracle.linear_forward(r(x), r(w), r(b))
    assert_f16(host(ops.linear_forward(dev(x, h), dev(w, h), dev(b, h))), want, "fp16")
    assert_f16(host(ops.linear_forward(dev(x, h), dev(w, h))), oracle.linear_forward(r(x), r(w), None), "fp16, no bias")
    got = host(ops.linear_forward(dev(x), dev(w), dev(b), math="f16", round_out_f16=True))
    assert_f16(got, want, "fp32 tensors, fp16 arithmetic")
    assert np.array_equal(got, r(got)), "rounded through fp16"
    ops.device_status()


# pixel boxes of channel-major results: the fewest boxes are 2 x 1 x 64 and 1 x 1 x 128 pixels, taken only where the K loop outlasts
# their stores; images narrower than eight pixels; both groups of epilogue warps (more tiles than SMs)
@pytest.mark.parametrize("n,c_in,h,w,c_out,k,s", [
    (64, 8, 62, 62, 24, 1, 1), (64, 8, 30, 62, 24, 3, 1), (128, 40, 5, 21, 24, 5, 1), (70, 16, 9, 5, 40, 3, 1), (128, 8, 7, 7, 72, 1, 1), (130, 16, 31, 3, 33, 3, 2), (9, 8, 131, 61, 40, 3, 2)])
def test_channel_major_results_of_any_width(n, c_in, h, w, c_out, k, s):
    gen = torch.Generator(device="cuda").manual_seed(n + w)
    g = ops.ConvGeometry(n, c_in, h, w, c_out, k, k, (s, s), (k // 2, k // 2))
    x = torch.randn(n, c_in, h, w, device="cuda", generator=gen)
    wt = torch.randn(c_out, c_in, k, k, device="cuda", generator=gen) * 0.1
    dy = torch.randn(n, c_out, *g.out_hw(), device="cuda", generator=gen)
    for dt, math, check in ((torch.float32, "3xtf32", assert_f32), (torch.float16, "f16", assert_f16)):
        xd, wd, dyd = x.to(dt), wt.to(dt), dy.to(dt)
        x64 = xd.double().requires_grad_()
        y64 = torch.nn.functional.conv2d(x64, wd.double(), stride=s, padding=k // 2)
        (dx64,) = torch.autograd.grad(y64, (x64,), dyd.double())
        check(host(ops.conv_forward(g, xd, wd, math=math)), y64.detach().cpu().numpy(), f"y {dt}")
        check(host(ops.conv_backward_data(g, dyd, wd, math=math)), dx64.cpu().numpy(), f"dx {dt}")
    ops.device_status()


# few columns, whose slices cost as much as those of 64; boxes of a K split; boxes of several phases
@pytest.mark.parametrize("n,c_in,h,w,c_out,k,s", [(64, 14, 64, 19, 3, 4, 2), (16, 200, 50, 11, 64, 4, 1), (40, 3, 76, 28, 320, 7, 3)])
def test_channel_major_boxes_by_time(n, c_in, h, w, c_out, k, s):
    test_channel_major_results_of_any_width(n, c_in, h, w, c_out, k, s)


# operands read in place: one row, one column, K of one value and of no whole slice, rows that start anywhere, K loops shared by the
# blocks of a cluster (the last of them with nothing to do)
@pytest.mark.parametrize("rows,fin,fout", [(1, 1, 1), (1, 70, 33), (129, 33, 130), (64, 513, 127), (33, 288, 65), (5, 2049, 3), (300, 36, 1025), (40, 96, 130)])
@pytest.mark.parametrize("shift", [0, 1])
def test_products_in_place(rows, fin, fout, shift, oracle):
    rng = np.random.default_rng(rows + fin)
    sizes = {"x": (rows, fin), "w": (fout, fin), "dy": (rows, fout), "b": (fout,)}
    host_of = {k: rng.standard_normal(s, dtype=np.float32) for k, s in sizes.items()}
    x, w, dy, b = (torch.cat([torch.zeros(shift, device="cuda"), dev(v).flatten()])[shift:].view(v.shape) for v in host_of.values())
    xh, wh, dyh, bh = host_of.values()
    launches, in_place = ops.launch_count(), launches_of(IN_PLACE)
    y = ops.linear_forward(x, w, b, math="3xtf32")
    dx = ops.linear_backward_data(dy, w, math="3xtf32")
    assert ops.launch_count() - launches == 2 and launches_of(IN_PLACE) - in_place == 2
    assert_f32(host(y), oracle.linear_forward(xh, wh, bh), "y")
    assert_f32(host(dx), dyh.astype(np.float64) @ wh.astype(np.float64), "dx")
    dw, db = ops.linear_backward_weight(x, dy, math="3xtf32")
    assert_f32(host(dw), dyh.T.astype(np.float64) @ xh.astype(np.float64), "dw")
    assert_f32(host(db), dyh.astype(np.float64).sum(0), "db")
    r = oracle.round_f16
    atol = 1e-3 * max(1.0, fin ** 0.5)  # (of the results' size)
    if shift == 0 or fin % 8:  # (rows that TMA would read have to start on 16 bytes)
        x16, w16, b16 = (torch.cat([torch.zeros(shift, device="cuda"), dev(v).flatten()]).half()[shift:].view(v.shape) for v in (xh, wh, bh))
        assert_f16(host(ops.linear_forward(x16, w16, b16)), oracle.linear_forward(r(xh), r(wh), r(bh)), "fp16 operands", atol=atol)
    half = host(ops.linear_forward(x, w, b, math="3xtf32", out_dtype=torch.float16))
    assert_f16(half, oracle.linear_forward(xh, wh, bh), "fp16 result", atol=atol)
    rounded = host(ops.linear_forward(x, w, b, math="3xtf32", round_out_f16=True))
    assert np.array_equal(rounded, half)
    assert torch.equal(y, ops.linear_forward(x, w, b, math="3xtf32"))
    ops.set_sm_limit(140)  # (contraction kernel: these blocks do not keep to a limit)
    try:
        assert_f32(host(ops.linear_forward(x, w, b, math="3xtf32")), oracle.linear_forward(xh, wh, bh), "y, limited")
    finally:
        ops.set_sm_limit(0)
    ops.device_status()


# long fp32 K loops of few tiles are the contraction kernel's: both sides of the limit, by the launches (one in place); in place with two
# waves of blocks (570 of 296 at a time), and with clusters of two on SMs that hold two blocks (224 on 148)
@pytest.mark.parametrize("rows,fin,fout,forward,in_place", [
    (1, 2000, 6, True, True), (1, 3456, 6, True, False), (60, 3456, 100, True, False), (2, 3, 1800, False, True), (2, 3, 3877, False, False), (85, 1, 3328, False, False),
    (12160, 5, 336, True, True), (1003, 249, 824, True, True)])
def test_long_products_of_few_tiles(rows, fin, fout, forward, in_place, oracle):
    rng = np.random.default_rng(fin + fout)
    xh, wh = rng.standard_normal((rows, fin if forward else fout), dtype=np.float32), rng.standard_normal((fout, fin), dtype=np.float32)
    launches = ops.launch_count()
    got = ops.linear_forward(dev(xh), dev(wh), math="3xtf32") if forward else ops.linear_backward_data(dev(xh), dev(wh), math="3xtf32")
    assert (ops.launch_count() - launches == 1) == in_place
    assert_f32(host(got), oracle.linear_forward(xh, wh, None) if forward else xh.astype(np.float64) @ wh.astype(np.float64), "result")
    ops.device_status()


# fp16 rows that TMA reads have to start on 16 bytes.  Where they do not, the call says so by the map that was refused, also at
# sizes that are read in place and have no scratch.
@pytest.mark.parametrize("rows,fin,fout", [(32, 56, 8), (11, 8, 22), (535, 128, 16), (300, 512, 256)])
@pytest.mark.parametrize("which", ["x", "w"])
def test_unaligned_rows_are_refused_by_name(rows, fin, fout, which):
    t = {"x": (rows, fin), "w": (fout, fin)}
    x, w = (torch.zeros(a * b + 1, device="cuda", dtype=torch.float16)[int(k == which):][:a * b].view(a, b) for k, (a, b) in t.items())
    for bias in (None, torch.zeros(fout, device="cuda", dtype=torch.float16)):
        with pytest.raises(_lib.NectarB200Error, match="cuTensorMapEncodeTiled"):
            ops.linear_forward(x, w, bias)
    ops.device_status()


@pytest.mark.parametrize("batch,m,k,n", [(2, 4, 64, 7), (5, 300, 64, 301), (3, 700, 512, 264)])
def test_unaligned_batched_rows_are_refused_by_name(batch, m, k, n):
    a = torch.zeros(batch * m * k + 1, device="cuda", dtype=torch.float16)[1:]
    b = torch.zeros(batch, k, n, device="cuda", dtype=torch.float16)
    with pytest.raises(RuntimeError, match="cuTensorMapEncodeTiled"):
        _nectarml.tensor.matmul(a.data_ptr(), b.data_ptr(), (batch, m, k), (batch, k, n), F16)
    ops.device_status()


# column sums in one launch up to 1024 rows: fewer rows than blocks of a cluster, a share that is no multiple of eight, the last
# vector of the last column block, both sides of the limit
@pytest.mark.parametrize("rows", [1, 7, 9, 64, 65, 519, 1024, 1025])
@pytest.mark.parametrize("fout", [8, 264, 520])
def test_bias_gradient_sums(rows, fout):
    gen = torch.Generator(device="cuda").manual_seed(rows + fout)
    for dt, math in ((torch.float16, "f16"), (torch.float32, "3xtf32")):
        x = torch.randn(rows, 64, device="cuda", generator=gen).to(dt)
        dy = (torch.randn(rows, fout, device="cuda", generator=gen) + 0.5).to(dt)
        _, db = ops.linear_backward_weight(x, dy, math=math)
        assert_f32(host(db), dy.double().sum(0).cpu().numpy(), f"db {dt}", tol=1e-6)
        assert torch.equal(db, ops.linear_backward_weight(x, dy, math=math)[1])
    ops.device_status()


# between conversions and contraction, fp32 rows of more than 256 columns up to 512 of them; beside a product in place up to 1024 (the
# launches of a weight gradient that are its sums')
@pytest.mark.parametrize("fin,fout,sums", [(1024, 256, [1, 1, 1, 2]), (1024, 772, [1, 2, 2, 2]), (16, 260, [1, 1, 1, 2])])
def test_wide_bias_gradient_sums(fin, fout, sums):
    gen = torch.Generator(device="cuda").manual_seed(fout)
    launches = []
    for rows in (512, 513, 1024, 1025):
        x, dy = torch.randn(rows, fin, device="cuda", generator=gen), torch.randn(rows, fout, device="cuda", generator=gen) + 0.5
        before = ops.launch_count()
        _, db = ops.linear_backward_weight(x, dy, math="3xtf32")
        with_sums = ops.launch_count() - before
        assert_f32(host(db), dy.double().sum(0).cpu().numpy(), "db", tol=1e-6)
        before = ops.launch_count()
        ops.linear_backward_weight(x, dy, math="3xtf32", want_bias_grad=False)
        launches.append(with_sums - (ops.launch_count() - before))
    assert launches == sums
    ops.device_status()


DOUBLE_TILES, IN_PLACE, TURNED, STRIPS = 0, 2, 3, 5  # kinds of nml_debug_launch_count


def launches_of(kind):
    return _lib.load().nml_debug_launch_count(kind)


# turned round, in fp16 and where the sizes say so in fp32: one row tile and several, columns of one pixel tile and of three, K of no whole
# vector and of whole ones (read in place), entries of one column tile and of more, two K slices on both sides of eight groups of rows an SM, one
# slice above it with strips that make 2.2 waves and one; up to there, and above by estimate, strips read in place take fp16 products (`strips`)
@pytest.mark.parametrize("batch,m,k,n,fp32_too,strips", [
    (100, 129, 96, 65, False, True), (300, 127, 64, 63, False, True), (64, 333, 64, 333, False, True), (40, 257, 130, 257, True, False),
    (103, 3010, 2, 39, True, False), (64, 130, 72, 261, False, True), (40, 257, 136, 257, False, False), (20, 333, 192, 333, False, False),
    (74, 512, 96, 255, False, True), (74, 513, 96, 255, False, False), (148, 520, 72, 65, False, False),
    (44, 80, 11, 1819, False, False), (74, 600, 48, 255, False, True)])
def test_batched_matmul_turned_round(batch, m, k, n, fp32_too, strips):
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    a, b = torch.randn(batch, m, k, device="cuda", generator=gen), torch.randn(batch, k, n, device="cuda", generator=gen)
    for dt, code in ((torch.float16, F16),) + (((torch.float32, F32),) if fp32_too else ()):
        ad, bd = a.to(dt), b.to(dt)
        torch.cuda.synchronize()
        before = launches_of(TURNED), launches_of(STRIPS)
        ptr = _nectarml.tensor.matmul(ad.data_ptr(), bd.data_ptr(), a.shape, b.shape, code)
        assert (launches_of(TURNED) - before[0], launches_of(STRIPS) - before[1]) == ((0, 1) if strips and dt == torch.float16 else (1, 0))
        want = (ad.double() @ bd.double()).cpu().numpy()
        if dt == torch.float32:
            assert_f32(fetch(ptr, (batch, m, n)), want, "fp32")
        else:  # (an absolute bound of the results' size)
            assert_f16(fetch(ptr, (batch, m, n), np.float16), want, "fp16", atol=1e-3 * k ** 0.5)
    ops.device_status()


@pytest.fixture
def four_pairs():
    """Plans for eight SMs, on which small layers have as many rounds of tiles as large ones on all; some launch of the test
    has to have had double tiles."""
    ops.set_sm_limit(8)
    before = launches_of(DOUBLE_TILES)
    yield
    ops.set_sm_limit(0)
    assert launches_of(DOUBLE_TILES) > before


# pair tiles are 256 x 256 and four run at a time: five to eight of them in one round of double tiles (the last row tile missing
# from 1100 rows, the last columns from 1000), and nine rows as four double tiles with a single one behind them.  K is summed
# in fp32 (errors of sqrt(K) * 2^-24 of the terms' size), the result rounded to fp16: 1e-2 rel holds that many times over, and
# the absolute bound is 1e-3 of the results' size, sqrt(K) * 0.2.
@pytest.mark.parametrize("rows,fin,fout", [(1100, 1600, 256), (1280, 1984, 248), (512, 2048, 1000), (2300, 3200, 256), (2304, 3136, 232)])
def test_double_tiles_linear(rows, fin, fout, oracle, four_pairs):
    rng = np.random.default_rng(rows + fin)
    h, r = torch.float16, oracle.round_f16
    x = rng.standard_normal((rows, fin), dtype=np.float32)
    w = (rng.standard_normal((fout, fin), dtype=np.float32) * 0.2).astype(np.float32)
    b = rng.standard_normal(fout, dtype=np.float32)
    want = oracle.linear_forward(r(x), r(w), r(b))
    atol = 1e-3 * 0.2 * fin ** 0.5
    assert_f16(host(ops.linear_forward(dev(x, h), dev(w, h), dev(b, h))), want, "bias", atol=atol)
    assert_f16(host(ops.linear_forward(dev(x, h), dev(w, h))), oracle.linear_forward(r(x), r(w), None), "no bias", atol=atol)
    # the same product as an input gradient (W read in place, columns inner) of the layer fout <- fin
    assert_f16(host(ops.linear_backward_data(dev(x, h), dev(w.T, h))), oracle.linear_forward(r(x), r(w), None), "dx", atol=atol)
    ops.device_status()


# the transposed copy of the weights: widths of no whole groups on both sides of its limit, and very wide layers of many rows
@pytest.mark.parametrize("rows,fin,fout", [(3000, 1000, 1000), (2900, 1000, 1000), (5003, 776, 1000), (8192, 3072, 128), (8200, 3080, 136)])
def test_linear_input_gradient_with_transposed_weights(rows, fin, fout):
    gen = torch.Generator(device="cuda").manual_seed(rows + fin)
    dy = torch.randn(rows, fout, device="cuda", generator=gen).half()
    w = (torch.randn(fout, fin, device="cuda", generator=gen) * 0.2).half()
    want = dy.double() @ w.double()
    assert_f16(host(ops.linear_backward_data(dy, w)), want.cpu().numpy(), "dx", atol=1e-3 * 0.2 * fout ** 0.5)
    ops.device_status()


# both sides of each of its limits, by the launches (the copy is one more)
@pytest.mark.parametrize("rows,fin,fout,copied", [
    (8192, 8, 128, 1), (8191, 8, 128, 0), (8192, 8, 120, 0), (8192, 40, 1960, 1), (8192, 40, 1944, 0), (2200, 1000, 1000, 1), (2199, 1000, 1000, 0),
    (8192, 3072, 1024, 1), (8192, 3072, 1016, 0), (8184, 3072, 1024, 0)])
def test_where_the_weights_are_transposed(rows, fin, fout, copied):
    dy, w = torch.zeros(rows, fout, device="cuda", dtype=torch.float16), torch.zeros(fout, fin, device="cuda", dtype=torch.float16)
    launches = ops.launch_count()
    ops.linear_backward_data(dy, w)
    assert ops.launch_count() - launches == 1 + copied
    test_linear_input_gradient_with_transposed_weights(rows, fin, fout)


# weights that do not start on 16 bytes: through the copy from 8192 rows on with whole groups of 64 outputs, whether or not aligned ones
# would take it, and refused elsewhere
@pytest.mark.parametrize("rows,fin,fout,taken", [(8192, 512, 128, True), (8195, 520, 64, True), (8192, 3072, 64, True), (8192, 512, 136, False), (4096, 512, 128, False), (3000, 1000, 1000, False)])
def test_linear_input_gradient_with_unaligned_weights(rows, fin, fout, taken):
    gen = torch.Generator(device="cuda").manual_seed(rows + fin)
    dy = torch.randn(rows, fout, device="cuda", generator=gen).half()
    w = (torch.randn(fout * fin + 1, device="cuda", generator=gen) * 0.2).half()[1:].view(fout, fin)
    if not taken:
        with pytest.raises(_lib.NectarB200Error, match="cuTensorMapEncodeTiled"):
            ops.linear_backward_data(dy, w)
    else:
        assert torch.equal(ops.linear_backward_data(dy, w), ops.linear_backward_data(dy, w.clone()))
        want = dy.double() @ w.double()
        assert_f16(host(ops.linear_backward_data(dy, w)), want.cpu().numpy(), "dx", atol=1e-3 * 0.2 * fout ** 0.5)
    ops.device_status()


@pytest.mark.parametrize("rows,fin,fout", [(4096, 640, 512), (4096, 1280, 512), (4100, 1280, 448), (2048, 1024, 2304)])
def test_double_tiles_linear_weight_gradient(rows, fin, fout, oracle, four_pairs):
    rng = np.random.default_rng(rows + fin)
    h, r = torch.float16, oracle.round_f16
    x, dy = rng.standard_normal((rows, fin), dtype=np.float32), rng.standard_normal((rows, fout), dtype=np.float32)
    dw, db = ops.linear_backward_weight(dev(x, h), dev(dy, h))
    assert_f32(host(dw), r(dy).T.astype(np.float64) @ r(x).astype(np.float64), "dw")
    assert_f32(host(db), r(dy).astype(np.float64).sum(0), "db")
    ops.device_status()


@pytest.mark.parametrize("n,c_in,hw,c_out,k,s,p,tr", [
    (5, 128, 16, 256, 3, 1, 1, False), (3, 128, 21, 256, 5, 1, 2, False), (5, 256, 18, 512, 4, 2, 1, False), (2, 384, 16, 128, 4, 2, 1, True), (5, 512, 9, 256, 4, 2, 1, True)])
def test_double_tiles_convolutions(n, c_in, hw, c_out, k, s, p, tr, oracle, four_pairs):
    """Boxes of pixels, the phases of a gather, 128-column tiles, and row tiles of a weight gradient that belong to
    different taps."""
    rng = np.random.default_rng(c_in + hw)
    h, r = torch.float16, oracle.round_f16
    g = ops.ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), (p, p), transposed=tr)
    x = rng.standard_normal((n, c_in, hw, hw), dtype=np.float32)
    w = (rng.standard_normal(g.weight_shape(), dtype=np.float32) * 0.05).astype(np.float32)
    dy = rng.standard_normal((n, c_out, *g.out_hw()), dtype=np.float32)
    xd, wd, dyd = dev(x, h, nhwc=True), dev(w, h), dev(dy, h, nhwc=True)
    # (float64 convolutions on the GPU: the oracle's loops would take minutes)
    f = torch.nn.functional
    x64, w64, dy64 = (torch.from_numpy(r(a)).cuda().double() for a in (x, w, dy))
    x64.requires_grad_()
    w64.requires_grad_()
    y64 = (f.conv_transpose2d if tr else f.conv2d)(x64, w64, stride=s, padding=p)
    y64.backward(dy64)
    atol = 1e-3 * 0.05 * (max(c_in, c_out) * k * k) ** 0.5
    assert_f16(host(ops.conv_forward(g, xd, wd, layout="nhwc"), nhwc=True), y64.detach().cpu().numpy(), "y", atol=atol)
    assert_f16(host(ops.conv_backward_data(g, dyd, wd, layout="nhwc"), nhwc=True), x64.grad.cpu().numpy(), "dx", atol=atol)
    dw, db = ops.conv_backward_weight(g, xd, dyd, layout="nhwc")
    assert_f32(host(dw), w64.grad.cpu().numpy(), "dw")
    assert_f32(host(db), dy64.sum((0, 2, 3)).cpu().numpy(), "db")
    ops.device_status()


@pytest.mark.parametrize("rows,c", [(1, 8), (3, 64), (1000, 24), (37, 2048)])
@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("with_res", [False, True])
def test_batch_norm_backward_with_and_without_y(rows, c, act, with_res):
    """The activation's derivative from y, from x, and from the forward's mask: the same bits, zeros and values that
    round to zero included."""
    import ctypes as C
    from nectarml_b200 import _lib
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(rows + c + act)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=gen)  # noqa: E731
    x, dy, res = rnd(rows, c).half(), rnd(rows, c).half(), (rnd(rows, c).half() if with_res else None)
    gamma, beta = rnd(c), rnd(c) * 0.3
    gamma[::3] = 0.0     # y is beta there ...
    beta[::6] = 2.0e-8   # ... and rounds to zero, or is zero
    beta[3::6] = 0.0
    need = C.c_size_t()
    _lib.check(lib.nml_bn_workspace_size(rows, c, C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    p = lambda t: t.data_ptr() if t is not None else None  # noqa: E731
    got = []
    for masked in (False, True):
        y, dx, dres = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
        mask = torch.zeros(rows * c // 8, dtype=torch.uint8, device="cuda") if with_res else None
        mean, rstd, dg, db = (torch.empty(c, device="cuda") for _ in range(4))
        if masked:
            _lib.check(lib.nml_bn_forward_masked(p(x), rows, c, p(gamma), p(beta), p(res), act, 0.2, 1e-5, p(y), 0, None, 0, p(mask),
                                                 p(mean), p(rstd), p(ws), need.value, st))
            _lib.check(lib.nml_bn_backward_masked(p(dy), 0, None, 0, p(mask), p(x), rows, c, p(gamma), p(beta), p(mean), p(rstd), act, 0.2, p(dx),
                                                  p(dres), p(dg), p(db), p(ws), need.value, st))
        else:
            _lib.check(lib.nml_bn_forward(p(x), rows, c, p(gamma), p(beta), p(res), act, 0.2, 1e-5, p(y), p(mean), p(rstd), p(ws),
                                          need.value, st))
            _lib.check(lib.nml_bn_backward(p(dy), p(y), p(x), rows, c, p(gamma), p(mean), p(rstd), act, 0.2, p(dx), p(dres), p(dg), p(db),
                                           p(ws), need.value, st))
        got.append((y, dx, dres, mean, rstd, dg, db))
    ops.device_status()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("c,k,s,p,d,hw,c_out", [
    (3, 7, 2, 3, 1, 37, 64), (3, 7, 2, 3, 1, 64, 64), (3, 3, 1, 1, 1, 16, 48), (7, 5, 1, 2, 1, 32, 64), (4, 4, 2, 1, 1, 34, 64), (1, 5, 2, 2, 1, 33, 128), (3, 3, 2, 1, 1, 16, 192), (2, 2, 2, 0, 1, 32, 64),
    (3, 8, 2, 3, 1, 40, 64), (3, 7, 4, 3, 1, 64, 96), (3, 7, 1, 3, 1, 24, 64), (5, 7, 2, 3, 1, 37, 64)])
def test_few_channel_windows(c, k, s, p, d, hw, c_out, oracle):
    """Image-like layers, four and eight channels per window pixel, through forward and weight gradient; the transposed layer
    that produces such an image, through its weight gradient.  dw is summed over at most 2 * 64 * 64 fp16 products."""
    rng = np.random.default_rng(c * 100 + k * 10 + s)
    h, r = torch.float16, oracle.round_f16
    g = ops.ConvGeometry(2, c, hw, hw, c_out, k, k, (s, s), (p, p), (d, d))
    ho, wo = g.out_hw()
    x = rng.standard_normal((2, c, hw, hw), dtype=np.float32)
    w = (rng.standard_normal((c_out, c, k, k), dtype=np.float32) * 0.1).astype(np.float32)
    b = rng.standard_normal(c_out, dtype=np.float32)
    dy = rng.standard_normal((2, c_out, ho, wo), dtype=np.float32)
    args = ((s, s), (p, p), (d, d))
    y_o, dw_o, db_o = oracle.conv2d(r(x), r(w), r(b), *args), oracle.conv2d_backward_weight(r(dy), r(x), w.shape, *args), oracle.bias_grad(r(dy))
    for layout in ("nhwc", "nchw"):
        nhwc = layout == "nhwc"
        xd, dyd = dev(x, h, nhwc=nhwc), dev(dy, h, nhwc=nhwc)
        assert_f16(host(ops.conv_forward(g, xd, dev(w, h), dev(b, h), layout=layout), nhwc=nhwc), y_o, f"y {layout}")
        dw, db = ops.conv_backward_weight(g, xd, dyd, layout=layout)
        assert_f32(host(dw), dw_o, f"dw {layout}", tol=2e-5)
        assert_f32(host(db), db_o, f"db {layout}", tol=2e-5)
    assert_f16(host(ops.conv_forward(g, dev(x), dev(w), dev(b), math="f16")), y_o, "y, fp32 tensors")
    # the transposed layer c_out -> c whose output gradient is the image
    gt = ops.ConvGeometry(2, c_out, ho, wo, c, k, k, (s, s), (p, p), (d, d), (hw - ((ho - 1) * s - 2 * p + d * (k - 1) + 1),) * 2, True)
    dw, db = ops.conv_backward_weight(gt, dev(dy, h, nhwc=True), dev(x, h, nhwc=True), layout="nhwc")
    assert_f32(host(dw), oracle.conv_transpose2d_backward_weight(r(x), r(dy), (c_out, c, k, k), *args), "dw, transposed", tol=2e-5)
    assert_f32(host(db), oracle.bias_grad(r(x)), "db, transposed", tol=2e-5)
    ops.device_status()


@pytest.mark.parametrize("rows,fin,fout,math", [
    (5541, 1776, 1008, "3xtf32"), (4128, 2064, 1000, "3xtf32"), (4096, 512, 2048, "f16"), (33, 64, 64, "f16"), (700, 200, 72, "f16"),
    (700, 200, 72, "3xtf32"), (9000, 256, 256, "f16")])
def test_weight_gradient_plans(rows, fin, fout, math):
    """Tile width, pairs and K split of the weight gradient, against float64: every element within the rounding of a sum over
    `rows` products (fp32 accumulation: 2.5e-9 of the sum of magnitudes per term and accumulator, 4096 terms at most)."""
    gen = torch.Generator(device="cuda").manual_seed(rows)
    dt = torch.float16 if math == "f16" else torch.float32
    x = torch.randn(rows, fin, device="cuda", generator=gen).to(dt)
    dy = torch.randn(rows, fout, device="cuda", generator=gen).to(dt)
    dw, db = ops.linear_backward_weight(x, dy, math=math)
    ops.device_status()
    want = dy.double().T @ x.double()
    assert float((dw.double() - want).norm() / want.norm()) < 2e-5
    assert float((dw.double() - want).abs().max()) < 1e-4 * rows ** 0.5
    assert float((db.double() - dy.double().sum(0)).abs().max()) < 1e-5 * rows ** 0.5 * 10


@pytest.mark.parametrize("rows,c", [(1, 8), (5, 64), (1000, 24), (37, 2048)])
@pytest.mark.parametrize("norm", [False, True])
def test_outputs_as_channels_of_a_concatenation(rows, c, norm):
    """Two layers whose outputs meet in a concatenation, written and differentiated in place: the values are the separate
    layers' bits, the gradient of an output read twice is the sum of both (fp16 once at the end, and once in each of
    the two parts of the normalisation's dx it is compared with, which may cancel: half an ulp, 2**-11, of all three).  The normalisation's dx is itself a difference of fp32
    terms of at most gamma * rstd * max|dz| * (2 + |xhat|), |xhat| below 6 here: a few roundings of 8 times that (one row:
    the terms cancel to nothing, rstd is 316)."""
    gen = torch.Generator(device="cuda").manual_seed(rows + c)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=gen)  # noqa: E731
    x, z, dy, dcat = rnd(rows, c).half(), rnd(rows, c).half(), rnd(rows, c).half(), rnd(rows, 2 * c).half()
    gamma, beta, ws, n = rnd(c), rnd(c), ops.Workspace(), ops._native
    empty = lambda: (torch.empty(c, device="cuda"), torch.empty(c, device="cuda"))  # noqa: E731
    dsum = (dy.float() + dcat[:, c:].float())
    if norm:
        y0, none, mean, rstd, _ = n.bn_forward(x, None, gamma, beta, 2, 0.2, 1e-5, None, False, ws)
        assert none is None
        y, wide, *_ = n.bn_forward(x, None, gamma, beta, 2, 0.2, 1e-5, None, True, ws)
        (dg, db), (dg2, db2) = empty(), empty()
        dx = n.bn_backward(dy, dcat, False, None, x, gamma, beta, mean, rstd, 2, 0.2, False, dg, db, ws)[0]
        both = [n.bn_backward(d, None, False, None, x, gamma, beta, mean, rstd, 2, 0.2, False, dg2, db2, ws)[0].float()
                for d in (dy, dcat[:, c:].contiguous())]
        want, size = both[0] + both[1], both[0].abs() + both[1].abs()
        terms = gamma.abs() * rstd * dsum.abs().max()
        # the join: z's layer fills the first channels and reads its part of the gradient
        a0, _, m2, r2, _ = n.bn_forward(z, None, gamma, beta, 1, 0.2, 1e-5, None, False, ws)
        cat = n.bn_forward(z, None, gamma, beta, 1, 0.2, 1e-5, wide, False, ws)[0]
        assert cat.data_ptr() == wide.data_ptr() and torch.equal(cat, torch.cat((a0, y0), dim=1))
        got = n.bn_backward(dcat, None, True, None, z, gamma, beta, m2, r2, 1, 0.2, False, dg, db, ws)[0]
        sep = n.bn_backward(dcat[:, :c].contiguous(), None, False, None, z, gamma, beta, m2, r2, 1, 0.2, False, dg2, db2, ws)[0]
        assert torch.equal(got, sep) and torch.equal(dg, dg2) and torch.equal(db, db2)
    else:
        y0, _ = n.act_forward(x, 2, 0.2, False)
        y, wide = n.act_forward(x, 2, 0.2, True)
        assert torch.equal(y0, torch.nn.functional.leaky_relu(x, 0.2))
        dx = n.act_backward(dy, dcat, x, 2, 0.2)
        want = dsum * torch.where(x > 0, 1.0, 0.2)
        size, terms = want.abs(), 0.0
    ops.device_status()
    assert torch.equal(y, y0) and torch.equal(wide[:, c:], y0)
    assert bool(((dx.float() - want).abs() <= 2.0 ** -11 * (want.abs() + size) + 2.0 ** -23 + 64 * 2.0 ** -24 * terms).all())


@pytest.mark.parametrize("n", [1, 2, 511, 4097, 3 * 64 * 64 * 5])
def test_l1_loss(n):
    """Sum in fp32 of n values below 8, in shares: n * 2**-24 relative at the very most."""
    from nectarml_b200 import train
    gen = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(n, device="cuda", generator=gen).half().requires_grad_()
    b = torch.randn(n, device="cuda", generator=gen).half()
    b[::3] = a.detach()[::3]
    loss = train._L1Fn.apply(a, b, 7.0)
    loss.backward(torch.full_like(loss, 16384.0))
    d = a.detach().double() - b.double()
    want = float(d.abs().sum() / 7.0)
    assert abs(float(loss.detach()) - want) <= (n * 2.0 ** -24 + 2.0 ** -22) * want
    assert torch.equal(a.grad, (torch.sign(d).float() * (torch.tensor(16384.0) / 7.0).item()).half())


@pytest.mark.parametrize("rows,c", [(7, 8), (8, 24), (9, 72), (2048, 136), (2049, 1024), (129, 2048), (4096, 512), (4097, 512),
                                    (16384, 8), (16385, 8)])
@pytest.mark.parametrize("with_res", [False, True])
def test_batch_norm_in_one_launch_and_in_three(rows, c, with_res):
    """Both sides of the line between the forms, and their remainders, against float64.  Unit-normal data: a thread and the tree
    above it add at most 100 numbers in fp32, so mean and E[x^2] are off by 100 * 2**-24 = 6e-6, rstd by half as much times
    (1 + mean^2 / var), and y by gamma * (2 + |xhat|) of that, below 1e-4 * gamma; the gradients' sums likewise, relative to
    the sum of the magnitudes (the normalised input's |xhat| is below 6)."""
    gen = torch.Generator(device="cuda").manual_seed(rows + c)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=gen)  # noqa: E731
    x, dy, res = rnd(rows, c).half(), rnd(rows, c).half(), (rnd(rows, c).half() if with_res else None)
    gamma, beta, ws, n = rnd(c).abs() + 0.1, rnd(c), ops.Workspace(), ops._native
    dg, db = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    y, _, mean, rstd, mask = n.bn_forward(x, res, gamma, beta, 2, 0.2, 1e-5, None, False, ws)
    dx, dres = n.bn_backward(dy, None, False, mask, x, gamma, beta, mean, rstd, 2, 0.2, with_res, dg, db, ws)
    ops.device_status()
    x64, dy64 = x.double(), dy.double()
    m, var = x64.mean(0), x64.var(0, unbiased=False)
    r = (var + 1e-5).rsqrt()
    xhat = (x64 - m) * r
    z = xhat * gamma + beta + (res.double() if with_res else 0.0)
    want = torch.where(z > 0, z, 0.2 * z)
    scale = 1.0 + m * m * r * r
    assert bool(((mean - m).abs() <= 1e-5).all()) and bool(((rstd - r).abs() <= 1e-5 * r * scale).all())
    assert bool(((y - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -24 + 1e-4 * gamma * scale).all())
    dz = dy64 * torch.where(y > 0, 1.0, 0.2)  # (the kernel's own signs: a value that rounds to zero may have either)
    wg, wb = (dz * xhat).sum(0), dz.sum(0)
    assert bool(((db - wb).abs() <= 1e-5 * dz.abs().sum(0)).all())
    assert bool(((dg - wg).abs() <= 1e-4 * scale * (dz.abs() * (1 + xhat.abs())).sum(0)).all())
    wdx = gamma * r * (dz - wb / rows - xhat * wg / rows)
    assert bool(((dx - wdx).abs() <= 2.0 ** -11 * wdx.abs() + 2.0 ** -24 + 1e-3 * scale * gamma * r * dz.abs().amax(0)).all())
    if with_res:
        assert torch.equal(dres, dz.half())


@pytest.mark.parametrize("batch,c,hw,s,dtype", [(64, 128, 23, 2, torch.float32), (65, 64, 32, 3, torch.float16), (43, 96, 32, 3, torch.float32),
                                               (64, 64, 33, 2, torch.float16)])
def test_strided_input_gradient_into_nchw_through_a_copy(batch, c, hw, s, dtype):
    """Sizes just above four million values, with planes that are and are not a multiple of four pixels: the bits of the same
    gradient into NHWC; and with no room for the copy in the workspace, the direct stores' (the same sums, rounded once)."""
    import ctypes as C
    from nectarml_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(hw)
    g = ops.ConvGeometry(batch, c, hw, hw, 64, 3, 3, (s, s), (1, 1))
    ho, wo = g.out_hw()
    dy = torch.randn(batch, 64, ho, wo, device="cuda", generator=gen).half()
    w = torch.randn(64, c, 3, 3, device="cuda", generator=gen).half()
    got = ops.conv_backward_data(g, dy, w, layout="nchw", out_dtype=dtype)
    want = ops.conv_backward_data(g, dy.permute(0, 2, 3, 1).contiguous(), w, layout="nhwc", out_dtype=dtype)
    assert torch.equal(got, want.permute(0, 3, 1, 2))
    code = _lib.NML_F16 if dtype == torch.float16 else _lib.NML_F32
    d, need, st = g.desc(_lib.NML_F16, "nchw", code, "nchw", _lib.NML_F16, "f16", False), C.c_size_t(), torch.cuda.current_stream().cuda_stream
    lib = _lib.load()
    _lib.check(lib.nml_conv_workspace_size(C.byref(d), 1, C.byref(need)))
    room = need.value - got.numel() * got.element_size()
    ws, direct = torch.empty(room + 256, dtype=torch.uint8, device="cuda"), torch.empty_like(got)
    _lib.check(lib.nml_conv_backward_data(C.byref(d), dy.data_ptr(), w.data_ptr(), direct.data_ptr(), ws.data_ptr(), ws.numel(), st))
    ops.device_status()
    assert torch.equal(direct, got)

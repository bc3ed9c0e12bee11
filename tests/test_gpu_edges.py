"""Inputs at the far ends of what the entry points accept: very long sums, scratch limits, values and pointers that a fast path
has to hand on."""
import contextlib
import threading
import time

import pytest
import torch

from gpu_util import F32, assert_f32, fetch, host
from nectarml_b200 import _nectarml, ops, train

pytestmark = pytest.mark.gpu


def test_weight_gradient_of_more_rows_than_the_slices_halve():
    """787000 rows in fp32: 24594 K blocks, where 192 slices no longer keep a sum within 4096 terms.  A term costs 2.5e-9 of
    its sum (the tensor core truncates as it accumulates): 1e-5 at 4128 terms, of |dw| where the slices' signs agree; and
    as much again for the fp32 additions."""
    rows, fin, fout = 787000, 160, 64
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, dy = (torch.randn(rows, f, device="cuda", generator=gen) for f in (fin, fout))
    dw, db = ops.linear_backward_weight(x, dy, math="3xtf32")
    ops.device_status()
    assert_f32(host(dw), (dy.double().T @ x.double()).cpu().numpy(), "dw", 2e-5)
    assert_f32(host(db), dy.double().sum(0).cpu().numpy(), "db", 2e-5)


@pytest.mark.parametrize("act,slope", [(1, 0.0), (2, 0.2)])
def test_activation_of_overflowed_values(act, slope):
    """Infinities and NaN through the activation that stands alone, and overflowed gradients through its backward, as torch's
    relu / leaky_relu treat them: nothing passes a ReLU that is shut, not even an infinity times zero."""
    inf, nan = float("inf"), float("nan")
    values = torch.tensor([inf, -inf, nan, 0.0, -0.0, 1.0, -1.0, 65504.0, -65504.0, 6e-8, -6e-8], device="cuda").half()
    x = values.repeat_interleave(len(values)).repeat(8).view(-1, 8).contiguous()
    dy = values.repeat(len(values)).repeat(8).view(-1, 8).contiguous()
    want_x = x.clone().requires_grad_()
    want = torch.relu(want_x) if act == 1 else torch.nn.functional.leaky_relu(want_x, slope)
    want.backward(dy)
    y, wide = ops._native.act_forward(x, act, slope, True)
    dx = ops._native.act_backward(dy, None, x, act, slope)
    ops.device_status()
    for got, ref in ((y, want.detach()), (wide[:, 8:], want.detach()), (dx, want_x.grad)):
        assert torch.allclose(got.float(), ref.float(), rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("device_count", [False, True])
def test_l1_loss_of_views(offset, device_count):
    """A target that starts anywhere in its storage, and a divisor that is a tensor: torch's formula, gradient included."""
    gen = torch.Generator(device="cuda").manual_seed(offset)
    flat = torch.randn(4 + 5 * 7 * 3, device="cuda", generator=gen).half()
    target = flat[offset:offset + 5 * 7 * 3].view(1, 5, 7, 3)
    out = torch.randn(1, 5, 7, 3, device="cuda", generator=gen).half()
    count = torch.tensor(315.0, device="cuda") if device_count else 315
    got_out, want_out = out.clone().requires_grad_(), out.clone().requires_grad_()
    got = train.TrainStep(None, "l1")._loss(got_out, target, count)
    want = (want_out.float() - target.float()).abs().sum() / 315
    got.backward()
    want.backward()
    ops.device_status()
    assert abs(float(got.detach()) - float(want.detach())) <= 1e-6 * float(want.detach())
    assert torch.equal(got_out.grad, want_out.grad)


def test_batched_matmul_of_many_thin_entries_keeps_its_scratch():
    """Entries with one or a few products per value: the converted operands are up to 32 times the operands (K is padded to a
    slice), 2 GB here, and go through the workspace in shares of at most 1 GB (a quarter more is allocated)."""
    batch, m, k, n = 8192, 8, 1, 1024
    gen = torch.Generator(device="cuda").manual_seed(3)
    a, b = torch.randn(batch, m, k, device="cuda", generator=gen), torch.randn(batch, k, n, device="cuda", generator=gen)
    torch.cuda.synchronize()
    before, launches = torch.cuda.mem_get_info()[0], ops.launch_count()
    ptr = _nectarml.tensor.matmul(a.data_ptr(), b.data_ptr(), a.shape, b.shape, F32)
    torch.cuda.synchronize()
    grown, launches = before - torch.cuda.mem_get_info()[0], ops.launch_count() - launches
    got = fetch(ptr, (batch, m, n))
    ops.device_status()
    assert grown <= 1.25 * 2 ** 30 + got.nbytes + (64 << 20), grown
    assert launches <= 16  # (shares, not entries)
    assert_f32(got, (a.double() * b.double()).cpu().numpy(), "products")


@pytest.mark.parametrize("case", [(10, 64, 91, 108, 256, 4, 2, 1, True, "f16", "nchw"), (102, 512, 5, 32, 8, 1, 2, 0, False, "3xtf32", "nchw"),
                                  (1, 512, 26, 17, 256, 7, 2, 3, False, "3xtf32", "nhwc")])
def test_static_entry_point_without_optional_scratch(case):
    """Layers whose full plan (a copy of the result, planes of a K split) does not fit the built-in scratch: the plan without
    gives the result of the call with a workspace.  The fp32 sums differ in order alone: 2.5e-9 of the result per term."""
    import ctypes as C
    from nectarml_b200 import _lib
    b, ci, h, w, co, k, s, p, tr, math, lay = case
    g = ops.ConvGeometry(b, ci, h, w, co, k, k, (s, s), (p, p), transposed=tr)
    gen = torch.Generator(device="cuda").manual_seed(b)
    x = torch.randn(g.act_shape("in", lay), device="cuda", generator=gen)
    wt = torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.1
    bias = torch.randn(co, device="cuda", generator=gen)
    want = ops.conv_forward(g, x, wt, bias, layout=lay, math=math)
    got = torch.empty_like(want)
    d = g.desc(_lib.NML_F32, lay, _lib.NML_F32, lay, _lib.NML_F32, math, False)
    _lib.check(_lib.load().nml_conv_forward_static(C.byref(d), x.data_ptr(), wt.data_ptr(), bias.data_ptr(), got.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream))
    _lib.check(_lib.load().nml_conv_forward_static(None, None, None, None, None, None))
    assert_f32(host(got), host(want), "static", 1e-6 + 2.5e-9 * ci * k * k)


def test_out_of_memory_has_torchs_type():
    """A result that no GPU holds: torch.OutOfMemoryError (what programs catch to try again with a smaller batch)."""
    x = torch.zeros(1, 8, device="cuda").expand(1 << 28, 8)
    with pytest.raises(torch.OutOfMemoryError):
        ops.linear_forward(x, torch.zeros(1 << 20, 8, device="cuda"))
    ops.device_status()


def test_other_threads_run_while_a_call_waits_for_the_queue():
    """The GPU is kept busy for about half a second while more launches are issued than its queue holds: the call that waits
    for room must not keep Python's lock, so another thread's clock has no gap of that length."""
    x, w, out = torch.zeros(8, 64, device="cuda").half(), torch.zeros(64, 64, device="cuda").half(), torch.empty(8, 64, device="cuda").half()
    ops.linear_forward(x, w, out=out)
    torch.cuda.synchronize()
    gaps, stop = [0.0], threading.Event()

    def clock():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            gaps[0] = max(gaps[0], now - last)
            last = now

    t = threading.Thread(target=clock)
    t.start()
    torch.cuda._sleep(1_000_000_000)
    begin = time.perf_counter()
    for _ in range(4000):
        ops.linear_forward(x, w, out=out)
    waited = time.perf_counter() - begin
    stop.set()
    t.join()
    ops.device_status()
    assert waited > 0.2, "the queue never filled"
    assert gaps[0] < 0.5 * waited, (gaps[0], waited)


def test_passes_of_two_threads_on_one_stream_do_not_mix():
    """Both share the default workspace: a pass's kernels are issued together, so each gets its own result, to the bit."""
    gen = torch.Generator(device="cuda").manual_seed(9)
    data = []
    for rows in (96, 352):
        x, dy = (torch.randn(rows, f, device="cuda", generator=gen) for f in (160, 72))
        data.append((x, dy, ops.linear_backward_weight(x, dy, math="3xtf32")))
    wrong = []

    def work(x, dy, want):
        for _ in range(400):
            dw, db = ops.linear_backward_weight(x, dy, math="3xtf32")
            if not (torch.equal(dw, want[0]) and torch.equal(db, want[1])):
                wrong.append(x.shape)

    threads = [threading.Thread(target=work, args=d) for d in data for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ops.device_status()
    assert not wrong, wrong


def test_saved_tensor_hooks_see_what_the_layers_keep():
    """Everything a layer saves for its backward passes through the hooks on saved tensors (which move it to the host here),
    and the gradients are the same bits; a second backward through freed tensors is refused."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    store = train.ParamStore("cuda")
    conv, bn = train.Conv(store, 8, 16, 3, 1, 1), train.BatchNormAct(store, 16)
    store.finalize(1)
    store.p32.copy_(torch.randn(store.n, device="cuda", generator=gen))
    store.sync_half()
    rnd = lambda *s: torch.randn(s, device="cuda", generator=gen).half()  # noqa: E731
    x, res, dy, token = rnd(2, 6, 6, 8), rnd(2, 6, 6, 16), rnd(2, 6, 6, 16), torch.zeros((), device="cuda", requires_grad=True)
    results, packed = [], []

    def pack(t):
        packed.append(tuple(t.shape))
        return t.cpu()

    for hooked in (False, True):
        leaf = x.clone().requires_grad_()
        store.begin_backward(False)
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()) if hooked else contextlib.nullcontext():
            y = bn(conv(leaf, token), token, train.ACT_RELU, residual=res)
        y.backward(dy)
        results.append((leaf.grad, store.grad.clone()))
        with pytest.raises(RuntimeError, match="second time"):
            y.backward(dy)
    ops.device_status()
    assert sorted(packed) == sorted([(2, 6, 6, 8), (2, 6, 6, 16), (16,), (16,), (2 * 6 * 6 * 16 // 8,)])
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_sm_limit_holds_for_the_next_launch_too():
    """Two long products in a stream under a limit of half the SMs: the second must not take the other half while it waits for
    the first, so a small product on another stream (a collective, in earnest) runs at once and not after the first."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x, w = torch.zeros(32768, 8192, device="cuda").half(), torch.zeros(8192, 8192, device="cuda").half()
    out = [torch.empty(32768, 8192, device="cuda").half() for _ in range(2)]
    a, b, ws = torch.zeros(128, 512, device="cuda").half(), torch.zeros(512, 512, device="cuda").half(), ops.Workspace()
    side, event = torch.cuda.Stream(), lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731
    ops.set_sm_limit(sms // 2)
    try:
        for _ in range(2):  # (once to warm up)
            torch.cuda.synchronize()
            begin, first, small = event(), event(), event()
            begin.record()
            ops.linear_forward(x, w, out=out[0])
            first.record()
            torch.cuda.synchronize()
            alone = begin.elapsed_time(first)
            with torch.cuda.stream(side):
                c = torch.empty(128, 512, device="cuda").half()
            torch.cuda.synchronize()
            begin.record()
            for o in out:
                ops.linear_forward(x, w, out=o)
            time.sleep(0.001)
            with torch.cuda.stream(side):
                ops.linear_forward(a, b, out=c, ws=ws)
                small.record()
            torch.cuda.synchronize()
            ended = begin.elapsed_time(small)
    finally:
        ops.set_sm_limit(0)
    ops.device_status()
    assert alone > 3.0, alone
    assert ended < 0.7 * alone, (ended, alone)


def test_profile_counts_the_turn_into_nchw():
    """A strided gradient into NCHW through a copy: the recorded duration holds the copy's turn.  The 205 MB are read and written
    once more, 50 us at 8 TB/s; half of that tells the two apart."""
    g = ops.ConvGeometry(256, 256, 28, 28, 64, 3, 3, (2, 2), (1, 1))
    best = {}
    for layout in ("nchw", "nhwc"):
        dy = torch.zeros(g.act_shape("out", layout), device="cuda").half()
        w = torch.zeros(g.weight_shape(), device="cuda").half()
        out = torch.empty(g.act_shape("in", layout), device="cuda")
        ops.conv_backward_data(g, dy, w, layout=layout, out=out)
        ops.profile_begin(5)
        for _ in range(5):
            ops.conv_backward_data(g, dy, w, layout=layout, out=out)
        times = ops.profile_end(5)
        assert len(times) == 5
        best[layout] = min(times)
    ops.device_status()
    assert best["nchw"] - best["nhwc"] > 0.025, best


# input gradients (or transposed forwards) with a handful of channels at strides above one, into fp32 NHWC: kernels, strides and
# paddings whose images do not suit the patch walk; (batch, channels in, h, w, channels out, kernel, stride, padding,
# output padding, transposed)
PACKED = [
    (5, 4, 1, 45, 1, (1, 3), (2, 1), (0, 1), (0, 0), False), (9, 3, 15, 4, 8, (3, 3), (2, 2), (0, 0), (0, 0), False),
    (18, 1, 7, 13, 192, (3, 1), (2, 2), (2, 0), (0, 0), False), (22, 4, 2, 40, 3, (4, 4), (2, 2), (3, 2), (0, 0), False),
    (4, 2, 14, 28, 8, (3, 1), (2, 2), (2, 0), (0, 0), False), (11, 1, 3, 4, 4, (3, 3), (2, 2), (0, 2), (0, 0), False),
    (11, 1, 12, 32, 3, (7, 7), (2, 2), (5, 4), (1, 1), True), (22, 64, 4, 5, 4, (1, 1), (2, 2), (0, 0), (0, 1), True),
    (2, 8, 12, 17, 4, (1, 3), (1, 2), (0, 1), (0, 0), True), (3, 16, 16, 16, 3, (4, 4), (2, 2), (1, 1), (0, 0), True),
]


@pytest.mark.parametrize("case", PACKED)
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.float16])
def test_phase_packed_columns(case, out_dtype):
    """All output phases in the columns of one walk, each value to its own pixel and nothing beside the result: against float64
    on fp16 operands (fp32 sums of at most 200 * 49 products, 1e-6 of the result's norm; half an ulp of fp16 where it is stored
    so), with a canary on both sides of the output."""
    b, ci, h, w, co, k, s, p, op, tr = case
    g = ops.ConvGeometry(b, ci, h, w, co, *k, s, p, (1, 1), op, tr)
    gen = torch.Generator(device="cuda").manual_seed(h * w)
    wt = (torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.2).half()
    src = torch.randn(g.act_shape("in" if tr else "out", "nhwc"), device="cuda", generator=gen).half()
    shape = g.act_shape("out" if tr else "in", "nhwc")
    n = shape[0] * shape[1] * shape[2] * shape[3]
    flat = torch.full((n + 2 * 4096,), 7.0, device="cuda", dtype=out_dtype)
    out = flat[4096:4096 + n].view(shape)
    if tr:
        ops.conv_forward(g, src, wt, layout="nhwc", out=out)
    else:
        ops.conv_backward_data(g, src, wt, layout="nhwc", out=out)
    ops.device_status()
    x, wd = src.double().permute(0, 3, 1, 2), wt.double()
    pad = op if tr else [(e + 2 * q - kk) % ss for e, q, kk, ss in zip((h, w), p, k, s)]
    want = torch.nn.functional.conv_transpose2d(x, wd, None, s, p, pad).permute(0, 2, 3, 1)
    assert float((out.double() - want).norm() / want.norm()) <= (1e-6 if out_dtype == torch.float32 else 5e-4)
    assert bool((flat[:4096] == 7).all()) and bool((flat[4096 + n:] == 7).all())

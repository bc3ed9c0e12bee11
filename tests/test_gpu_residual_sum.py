"""The gradient of a residual block's input as one pass: the C entry point against its two halves, and the autograd nodes
against the same block with the sum left to the engine."""
import ctypes as C

import pytest
import torch

from nectarml_b200 import _lib, ops, train
from nectarml_b200.ops import ConvGeometry

pytestmark = pytest.mark.gpu


# a tile of one and of several pieces, ragged pixels, the patch walk, the phases of a strided gather, a K loop split over CTAs, widths that
# end within a piece, and eight channels, which no TMA store takes (accepted for the phases of a stride alone)
@pytest.mark.parametrize("n,c_in,hw,c_out,k,s", [
    (4, 256, 28, 64, 1, 1), (3, 64, 13, 128, 3, 1), (2, 128, 15, 64, 3, 2), (2, 512, 4, 512, 3, 1), (3, 24, 9, 40, 3, 1), (2, 72, 11, 16, 1, 1), (5, 320, 7, 64, 1, 2),
    (3, 8, 11, 40, 3, 2), (2, 8, 64, 24, 1, 2)])
@pytest.mark.parametrize("masked", [False, True])
def test_input_gradient_with_an_addend(n, c_in, hw, c_out, k, s, masked):
    gen = torch.Generator(device="cuda").manual_seed(c_in + hw)
    rnd = lambda *shape: torch.randn(shape, device="cuda", generator=gen)  # noqa: E731
    g = ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), (k // 2, k // 2))
    dy = rnd(n, *g.out_hw(), c_out).half()
    w = (rnd(c_out, c_in, k, k) * 0.1).half()
    add = rnd(n, hw, hw, c_in).half()
    keep = torch.rand(add.shape, device="cuda", generator=gen) < 0.5
    bits = (keep.view(-1, 8).int() << torch.arange(8, device="cuda")).sum(1).to(torch.uint8)
    below = 0.2
    d = g.desc(_lib.NML_F16, "nhwc", _lib.NML_F16, "nhwc", _lib.NML_F16, "f16", False)
    lib, need = _lib.load(), C.c_size_t()
    _lib.check(lib.nml_conv_workspace_size(C.byref(d), 1, C.byref(need)))
    ws = torch.empty(max(need.value, 1), dtype=torch.uint8, device="cuda")
    dx = torch.empty_like(add)
    _lib.check(lib.nml_conv_backward_data_add(C.byref(d), dy.data_ptr(), w.data_ptr(), add.data_ptr(), bits.data_ptr() if masked else None,
                                              below, dx.data_ptr(), ws.data_ptr(), need.value, torch.cuda.current_stream().cuda_stream))
    plain = torch.nn.functional.conv_transpose2d(dy.permute(0, 3, 1, 2).double(), w.double(), stride=s, padding=k // 2,
                                                 output_padding=hw - ((g.out_hw()[0] - 1) * s - 2 * (k // 2) + k)).permute(0, 2, 3, 1)
    want = plain + (torch.where(keep, add.double(), add.double() * below) if masked else add.double())
    # one rounding to fp16 of the sum, or two where a second pass adds: 2^-10 of the larger addend
    bound = 2.0 ** -10 * (plain.abs() + add.double().abs()) + 1e-3
    assert ((dx.double() - want).abs() <= bound).all()
    ops.device_status()


# which plan takes the sum, by its kernels (weights' repack, product, pass of the sum): pairs under a long K loop and many values leave
# it to a pass, single CTAs add in the epilogue
@pytest.mark.parametrize("n,c_in,hw,c_out,k,s,kernels", [
    (11, 512, 28, 512, 3, 1, 3), (16, 256, 27, 1024, 3, 1, 3), (16, 128, 56, 512, 3, 1, 3), (3, 256, 56, 256, 3, 1, 2), (16, 512, 28, 128, 1, 1, 2), (13, 512, 27, 256, 4, 2, 2)])
def test_sums_beside_pairs(n, c_in, hw, c_out, k, s, kernels):
    before = ops.launch_count()
    test_input_gradient_with_an_addend(n, c_in, hw, c_out, k, s, True)
    assert ops.launch_count() - before == kernels


@pytest.mark.parametrize("c_in,hw,k,s,in_epilogue", [(24, 9, 3, 1, True), (72, 11, 1, 1, True), (72, 12, 3, 2, True), (8, 11, 3, 2, False), (8, 12, 1, 2, False)])
def test_sums_of_narrow_results(c_in, hw, k, s, in_epilogue):
    before = sums_in_epilogues()
    test_input_gradient_with_an_addend(2, c_in, hw, 40, k, s, True)
    assert sums_in_epilogues() - before == int(in_epilogue)


# the mask's bytes may start anywhere: widths whose pieces are whole groups of eight bytes, and one whose are not
@pytest.mark.parametrize("c_in", [64, 256, 72])
@pytest.mark.parametrize("shift", [1, 4, 7])
def test_mask_at_any_offset(c_in, shift):
    gen = torch.Generator(device="cuda").manual_seed(c_in + shift)
    rnd = lambda *shape: torch.randn(shape, device="cuda", generator=gen)  # noqa: E731
    g = ConvGeometry(3, c_in, 10, 10, 64, 1, 1)
    dy, w, add = rnd(3, 10, 10, 64).half(), (rnd(64, c_in, 1, 1) * 0.1).half(), rnd(3, 10, 10, c_in).half()
    bits = torch.randint(0, 256, (add.numel() // 8,), device="cuda", generator=gen).to(torch.uint8)
    moved = torch.cat([torch.zeros(shift, device="cuda", dtype=torch.uint8), bits])[shift:]
    d = g.desc(_lib.NML_F16, "nhwc", _lib.NML_F16, "nhwc", _lib.NML_F16, "f16", False)
    lib, need = _lib.load(), C.c_size_t()
    _lib.check(lib.nml_conv_workspace_size(C.byref(d), 1, C.byref(need)))
    ws, got = torch.empty(max(need.value, 1), dtype=torch.uint8, device="cuda"), []
    for mask in (bits, moved):
        got.append(torch.empty_like(add))
        _lib.check(lib.nml_conv_backward_data_add(C.byref(d), dy.data_ptr(), w.data_ptr(), add.data_ptr(), mask.data_ptr(), 0.25,
                                                  got[-1].data_ptr(), ws.data_ptr(), need.value, torch.cuda.current_stream().cuda_stream))
    assert moved.data_ptr() % 8 == shift and torch.equal(*got)
    ops.device_status()


# (with all the scratch the call could want, so that nothing but the refusal in question stops it)
def test_input_gradient_with_an_addend_refuses():
    lib = _lib.load()
    dy, w, add, dx = (torch.zeros(8192, device="cuda", dtype=torch.float16) for _ in range(4))
    ws = torch.empty(1 << 24, device="cuda", dtype=torch.uint8)
    INVALID, UNSUPPORTED = 1, 4

    def call(layout="nhwc", channels=16, stride=1, add=add, dx=dx, add_shift=0, dx_shift=0):
        g = ConvGeometry(1, channels, 8, 8, 16, 3, 3, (stride, stride), (1, 1))
        d = g.desc(_lib.NML_F16, layout, _lib.NML_F16, layout, _lib.NML_F16, "f16", False)
        return lib.nml_conv_backward_data_add(C.byref(d), dy.data_ptr(), w.data_ptr(), add.data_ptr() + add_shift, None, 0.0, dx.data_ptr() + dx_shift,
                                              ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)

    assert call(channels=24) == _lib.NML_OK and call(channels=8, stride=2) == _lib.NML_OK
    assert call(channels=12) == UNSUPPORTED and call(channels=24, layout="nchw") == UNSUPPORTED
    assert call(channels=16) == UNSUPPORTED and call(channels=8) == UNSUPPORTED  # (no more than 16 columns over all phases)
    assert call(channels=24, add_shift=8) == INVALID and call(channels=24, dx_shift=2) == INVALID
    for shift in (0, 16, 2 * 8 * 8 * 24 - 16):  # whole and partial overlap
        assert call(channels=24, add=dx, add_shift=shift) == INVALID and call(channels=24, dx=add, dx_shift=shift) == INVALID
    assert call(channels=24, add=dx, add_shift=2 * 8 * 8 * 24) == _lib.NML_OK
    ops.device_status()


def sums_in_epilogues():
    return _lib.load().nml_debug_launch_count(1)


class Block:
    """x -> conv, norm, ReLU, conv, norm + x, ReLU; ``through`` is what the residual passes on its way."""

    def __init__(self, c=64, mid=32, act=train.ACT_RELU):
        self.store = store = train.ParamStore("cuda")
        self.c1, self.b1 = train.Conv(store, c, mid, 1, 1, 0), train.BatchNormAct(store, mid)
        self.c2, self.b2 = train.Conv(store, mid, c, 3, 1, 1), train.BatchNormAct(store, c)
        store.finalize(1)
        gen = torch.Generator(device="cuda").manual_seed(5)
        for i, shape in enumerate(store.shapes):
            store.w32(i).copy_(torch.randn(shape, device="cuda", generator=gen) * 0.1 if len(shape) == 4 else torch.ones(shape, device="cuda"))
        store.sync_half()
        self.act, self.t = act, torch.zeros((), device="cuda", requires_grad=True)

    def __call__(self, x, through=lambda r: r):
        self.store.begin_backward(True)
        y = self.b1(self.c1(x, self.t), self.t, train.ACT_RELU)
        return self.b2(self.c2(y, self.t), self.t, self.act, residual=through(x))


def tensors(c=64):
    gen = torch.Generator(device="cuda").manual_seed(9)
    return torch.randn(4, 14, 14, c, device="cuda", generator=gen).half(), torch.randn(4, 14, 14, c, device="cuda", generator=gen).half()


def close(a, b):
    # (the engine rounds the two gradients and their sum to fp16, the kernel their sum)
    return ((a.double() - b.double()).abs() <= 2.0 ** -9 * (a.double().abs() + b.double().abs()) + 4e-3).all()


@pytest.mark.parametrize("act", [train.ACT_NONE, train.ACT_RELU, train.ACT_LEAKY])
def test_block_input_gradient(act):
    x0, dy = tensors()
    block, x = Block(act=act), x0.clone().requires_grad_()
    sums = sums_in_epilogues()
    (fused,) = torch.autograd.grad(block(x), (x,), dy)
    grads = block.store.grad.clone()
    assert sums_in_epilogues() - sums == 1
    (engine,) = torch.autograd.grad(block(x, lambda r: r.view_as(r)), (x,), dy)  # (another edge: the engine adds)
    assert sums_in_epilogues() - sums == 1
    assert torch.equal(grads, block.store.grad)
    assert close(fused, engine) and not torch.equal(fused, torch.zeros_like(fused))
    # a graph kept for a second pass, with another gradient, and then again the first
    y = block(x)
    first = torch.autograd.grad(y, (x,), dy, retain_graph=True)[0]
    twice = torch.autograd.grad(y, (x,), 2 * dy, retain_graph=True)[0]
    again = torch.autograd.grad(y, (x,), dy)[0]
    assert torch.equal(first, fused) and torch.equal(again, fused) and close(twice, 2 * fused)
    assert sums_in_epilogues() - sums == 4


def test_block_input_gradient_reaches_whoever_asks():
    x0, dy = tensors()
    block, x = Block(), x0.clone().requires_grad_()
    (fused,) = torch.autograd.grad(block(x), (x,), dy)
    # an input that is not a leaf, a hook on it, and .backward()
    leaf = x0.clone().requires_grad_()
    seen = []
    inner = leaf * 1.0
    inner.register_hook(lambda g: seen.append(g.clone()))
    block(inner).backward(dy)
    assert torch.equal(leaf.grad, fused) and len(seen) == 1 and torch.equal(seen[0], fused)
    # two blocks in a row, and a third use of the input beside them
    a, b = Block(), Block()
    y = b(a(x)) + 2 * x
    (got,) = torch.autograd.grad(y, (x,), dy)
    z = b(a(x, lambda r: r.view_as(r)), lambda r: r.view_as(r)) + 2 * x.view_as(x)
    (want,) = torch.autograd.grad(z, (x,), dy)
    assert close(got, want)
    # the residual alone (the branch detached), and the branch alone: nothing is left with a convolution that is not run
    with torch.no_grad():
        h = block.b1(block.c1(x, block.t), block.t, train.ACT_RELU)
    y = block.b2(block.c2(h, block.t), block.t, train.ACT_RELU, residual=x)
    (only,) = torch.autograd.grad(y, (x,), dy)
    assert torch.equal(only, torch.where(y > 0, dy, torch.zeros_like(dy)))
    # gradients of something between the two alone
    h = block.c1(x, block.t)
    y = block.b2(block.c2(block.b1(h, block.t, train.ACT_RELU), block.t), block.t, train.ACT_RELU, residual=x)
    (dh,) = torch.autograd.grad(y, (h,), dy, retain_graph=True)
    (dx,) = torch.autograd.grad(y, (x,), dy)
    assert torch.equal(dx, fused) and dh.abs().max() > 0
    # a hook on the normalisation's node sees the gradient of its residual
    y = block(x)
    got = []
    y.grad_fn.register_hook(lambda gi, go: got.append(gi[1]))
    (dx,) = torch.autograd.grad(y, (x,), dy)
    assert got[0] is not None and close(dx, fused)


# a hook on the first convolution's node is given that convolution's input gradient, and what it puts in its place is all it
# replaces: the residual's share is neither shown to it nor scaled by it
@pytest.mark.parametrize("act", [train.ACT_NONE, train.ACT_RELU])
def test_hook_on_the_first_convolution(act):
    x0, dy = tensors()
    block, x = Block(act=act), x0.clone().requires_grad_()
    (fused,) = torch.autograd.grad(block(x), (x,), dy)

    def first_convolution(node):
        while node.name() != "ConvBackward" or node.next_functions[0][0].name() != "torch::autograd::AccumulateGrad":
            node = node.next_functions[0][0]
        return node

    y = block(x)
    residual = torch.where(y > 0, dy, torch.zeros_like(dy)) if act == train.ACT_RELU else dy
    for scale in (None, 0.0):
        seen = []

        def hook(gi, go):
            seen.append(gi[0].clone())
            return None if scale is None else (gi[0] * scale, gi[1])

        y = block(x)
        first_convolution(y.grad_fn).register_hook(hook)
        sums = sums_in_epilogues()
        (dx,) = torch.autograd.grad(y, (x,), dy)
        assert sums_in_epilogues() == sums
        assert close(seen[0].double() + residual.double(), fused) and not close(seen[0], fused)
        assert close(dx, fused) if scale is None else torch.equal(dx, residual)


def test_block_input_gradient_on_two_streams_and_in_a_graph():
    x0, dy = tensors()
    block, x = Block(), x0.clone().requires_grad_()
    (fused,) = torch.autograd.grad(block(x), (x,), dy)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    block.store.begin_backward(True)
    h = block.c1(x, block.t)  # made on another stream than the rest: the engine adds
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = block.b2(block.c2(block.b1(h, block.t, train.ACT_RELU), block.t), block.t, train.ACT_RELU, residual=x)
    torch.cuda.current_stream().wait_stream(side)
    (dx,) = torch.autograd.grad(y, (x,), dy)
    torch.cuda.synchronize()
    assert close(dx, fused)
    block, x = Block(), x0.clone().requires_grad_()  # (warmed up on a stream of its own, as a capture wants it)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            torch.autograd.grad(block(x), (x,), dy)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with train.capture_into(graph):
        (dx,) = torch.autograd.grad(block(x), (x,), dy)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(dx, fused)

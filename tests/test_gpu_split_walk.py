"""The finishing pass of forward walks whose K loop is cut over many CTAs: few results of many planes, as vectors and value by value, in every
layout, with a bias and without."""
import os
import subprocess
import sys

import pytest
import torch

from gpu_util import assert_f32
from nectarml_b200 import _lib, ops
from nectarml_b200.ops import ConvGeometry

pytestmark = pytest.mark.gpu


def deep_finishes():
    return _lib.load().nml_debug_launch_count(6)


CONVOLUTIONS = [(3, 512, 4, 64, 4, 2), (1, 700, 5, 33, 3, 1), (2, 1024, 3, 40, 3, 1), (1, 256, 8, 3, 5, 1), (16, 512, 2, 512, 4, 2)]


@pytest.mark.parametrize("n,c_in,hw,c_out,k,s", CONVOLUTIONS)
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("math,dtype", [("3xtf32", torch.float32), ("f16", torch.float16)])
def test_convolutions(n, c_in, hw, c_out, k, s, layout, math, dtype):
    before = deep_finishes()
    gen = torch.Generator(device="cuda").manual_seed(c_in + c_out)
    g = ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), ((k - 1) // 2,) * 2)
    x = torch.randn(g.act_shape("in", layout), device="cuda", generator=gen).to(dtype)
    w = (torch.randn(g.weight_shape(), device="cuda", generator=gen) * 0.05).to(dtype)
    b = torch.randn(c_out, device="cuda", generator=gen).to(dtype)
    to_nchw = (lambda t: t.permute(0, 3, 1, 2)) if layout == "nhwc" else (lambda t: t)
    want = torch.nn.functional.conv2d(to_nchw(x).double(), w.double(), stride=s, padding=(k - 1) // 2)
    for bias in (b, None):
        y = to_nchw(ops.conv_forward(g, x, w, bias, layout=layout, math=math))
        ref = want + (bias.double().view(-1, 1, 1) if bias is not None else 0.0)
        if dtype == torch.float32:
            assert_f32(y.cpu(), ref.cpu(), "fp32")
        else:  # one rounding to fp16, or two where a ragged row's bias is added to the rounded sum
            assert ((y.double() - ref).abs() <= 2.0 ** -10 * (ref.abs() + b.double().abs().view(-1, 1, 1) + ref.abs().amax() / 64)).all()
    ops.device_status()
    assert deep_finishes() == before + 2


@pytest.mark.parametrize("rows,fin,fout", [(16, 4096, 512), (22, 5248, 97), (1, 3000, 1000), (129, 6000, 60)])
def test_linear(rows, fin, fout):
    gen = torch.Generator(device="cuda").manual_seed(rows + fout)
    x, w, b = (torch.randn(s, device="cuda", generator=gen) for s in ((rows, fin), (fout, fin), (fout,)))
    before = deep_finishes()
    assert_f32(ops.linear_forward(x, w, b, math="3xtf32").cpu(), (x.double() @ w.double().t() + b.double()).cpu(), "fp32")
    y = ops.linear_forward(x, w, b, math="f16", round_out_f16=True)  # fp32 tensors, fp16 arithmetic
    ref = x.half().double() @ w.half().double().t() + b.half().double()
    assert ((y.double() - ref).abs() <= 2.0 ** -9 * (ref.abs() + ref.abs().amax() / 64)).all()
    assert torch.equal(y, y.half().float())
    ops.device_status()
    assert deep_finishes() > before


_OUTPUTS = """
import sys, torch
sys.path.insert(0, sys.argv[1])
from nectarml_b200 import _lib, ops
from nectarml_b200.ops import ConvGeometry
from test_gpu_split_walk import CONVOLUTIONS
out, gen = [], torch.Generator(device="cuda").manual_seed(5)
for n, c_in, hw, c_out, k, s in CONVOLUTIONS:
    g = ConvGeometry(n, c_in, hw, hw, c_out, k, k, (s, s), ((k - 1) // 2,) * 2)
    for layout in ("nchw", "nhwc"):
        for math, dtype in (("3xtf32", torch.float32), ("f16", torch.float16)):
            x, w, b = (torch.randn(v, device="cuda", generator=gen).to(dtype) for v in (g.act_shape("in", layout), g.weight_shape(), (c_out,)))
            out.append(ops.conv_forward(g, x, w, b, layout=layout, math=math).cpu())
ops.device_status()
torch.save((out, _lib.load().nml_debug_launch_count(6)), sys.argv[2])
"""


def test_both_finishing_passes_add_in_the_same_order(tmp_path):
    """The same planes through either kernel: results of the same bits."""
    here = os.path.dirname(os.path.abspath(__file__))
    results = []
    for deep in ("0", "1"):
        path = str(tmp_path / deep)
        env = dict(os.environ, NML_TUNE_DEEP=deep, PYTHONPATH=os.path.dirname(here))
        res = subprocess.run([sys.executable, "-c", _OUTPUTS, here, path], capture_output=True, text=True, timeout=300, env=env)
        assert res.returncode == 0, res.stderr[-2000:]
        results.append(torch.load(path))
    assert results[0][1] == 0 and results[1][1] == len(results[1][0]) == 4 * len(CONVOLUTIONS)
    assert all(torch.equal(a, b) for a, b in zip(results[0][0], results[1][0]))

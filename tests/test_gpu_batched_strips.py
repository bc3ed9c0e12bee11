"""Batched fp16 products of one or two K slices whose rows are no whole vectors: strips of 128 columns read in place."""
import pytest
import torch

from gpu_util import F16, fetch
from nectarml_b200 import _lib, _nectarml, ops

import numpy as np

pytestmark = pytest.mark.gpu
IN_PLACE, TURNED, STRIPS = 2, 3, 5  # kinds of nml_debug_launch_count


def product(a, b, batch, m, k, n):
    ptr = _nectarml.tensor.matmul(a.data_ptr(), b.data_ptr(), (batch, m, k), (batch, k, n), F16)
    return torch.from_numpy(fetch(ptr, (batch, m, n), np.float16).astype(np.float64))


# K of one value, a part of a slice, a whole one, a value more, two; one strip and a column more; one group of 64 rows, a row more, strips cut over
# blocks (few entries) and not (many)
@pytest.mark.parametrize("k", [1, 8, 63, 64, 65, 100, 128])
@pytest.mark.parametrize("batch,m,n", [(2, 32, 33), (3, 64, 127), (2, 65, 129), (5, 700, 61), (150, 70, 257), (2, 33, 1001)])
@pytest.mark.parametrize("shift", [0, 1])
def test_strips(batch, m, n, k, shift):
    gen = torch.Generator(device="cuda").manual_seed(batch * m + n + k)
    make = lambda count: torch.randn(count + shift, device="cuda", generator=gen).half()[shift:]  # noqa: E731
    # (rows of whole vectors that do not start on 16 bytes are refused, as everywhere)
    a = make(batch * m * k) if k % 8 else torch.randn(batch * m * k, device="cuda", generator=gen).half()
    b = make(batch * k * n)
    lib = _lib.load()
    counts = lambda: [lib.nml_debug_launch_count(kind) for kind in (STRIPS, TURNED, IN_PLACE)] + [ops.launch_count()]  # noqa: E731
    before = counts()
    got = product(a, b, batch, m, k, n)
    assert counts() == [before[0] + 1, before[1], before[2], before[3] + 1]
    ad, bd = a.double().view(batch, m, k), b.double().view(batch, k, n)
    want, terms = (ad @ bd).cpu(), (ad.abs() @ bd.abs()).cpu()
    # one rounding to fp16 (half an ulp, 2^-25 among the smallest), fp32 sums that lose at most 2^-22 of their terms' size a step of 16
    assert ((got - want).abs() <= want.abs() * 2.0 ** -11 + 2.0 ** -25 + terms * 2.0 ** -22 * (k / 16 + 1)).all()
    ops.device_status()


def test_infinities_and_nan():
    a = torch.ones(2, 40, 64, device="cuda", dtype=torch.float16)
    b = torch.ones(2, 64, 35, device="cuda", dtype=torch.float16)
    a[0, 3, 5] = float("inf")
    b[1, 7, 34] = float("nan")
    got = product(a, b, 2, 40, 64, 35)
    want = torch.full((2, 40, 35), 64.0, dtype=torch.float64)
    want[0, 3] = float("inf")
    want[1, :, 34] = float("nan")
    assert torch.equal(got.nan_to_num(-1.0), want.nan_to_num(-1.0))


def test_rows_that_do_not_start_on_16_bytes_stay_refused():
    a = torch.zeros(2 * 40 * 64 + 1, device="cuda", dtype=torch.float16)[1:]
    b = torch.zeros(2 * 64 * 35, device="cuda", dtype=torch.float16)
    with pytest.raises(RuntimeError, match="cuTensorMapEncodeTiled"):
        product(a, b, 2, 40, 64, 35)

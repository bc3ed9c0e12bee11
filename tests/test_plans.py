"""What the planner answers without a GPU: workspace queries run the whole plan in its measuring mode."""
import ctypes as C

import pytest

from nectarml_b200 import _lib, ops
from nectarml_b200._lib import NML_F32, NML_PASS_BACKWARD_WEIGHT


def ceil_div(a, b):
    return (a + b - 1) // b


def test_every_3xtf32_weight_gradient_has_a_plan(lib):
    """K blocks are 32 rows.  A sum has at most 4096 terms while 192 slices allow it, so a long gradient has at least
    min(K / 128, 190) slices (192 rounded down to a count without an empty slice), each with a plane of all row tiles."""
    fin, fout = 160, 64
    row_tiles = ceil_div(ceil_div(fin, 32) * 32, 128)
    need = C.c_size_t()
    missing = []
    for k in range(1, 40001):
        d = ops._linear_desc(32 * k, fin, fout, NML_F32, NML_F32, NML_F32, "3xtf32", False)
        assert lib.nml_linear_workspace_size(C.byref(d), NML_PASS_BACKWARD_WEIGHT, C.byref(need)) == _lib.NML_OK
        slices = min(ceil_div(k, 128), 190)
        planes = slices * fout * row_tiles * 128 * 4 if slices > 1 else 0
        if need.value < 2 * 4 * 32 * k * (fin + fout) + planes:
            missing.append(k)
    assert not missing, (len(missing), missing[:5])

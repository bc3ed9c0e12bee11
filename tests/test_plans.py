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
        d = _lib.LinearDesc(32 * k, fin, fout, NML_F32, NML_F32, NML_F32, _lib.NML_MATH_3XTF32, 0)
        assert lib.nml_linear_workspace_size(C.byref(d), NML_PASS_BACKWARD_WEIGHT, C.byref(need)) == _lib.NML_OK
        slices = min(ceil_div(k, 128), 190)
        planes = slices * fout * row_tiles * 128 * 4 if slices > 1 else 0
        if need.value < 2 * 4 * 32 * k * (fin + fout) + planes:
            missing.append(k)
    assert not missing, (len(missing), missing[:5])


# (batch, c_in, h, w, c_out, kernel, stride, padding, transposed, math, out layout): scratch without the regions that only buy speed
# fits the static entry point's array, with them it does not
STATIC = [
    (10, 64, 91, 108, 256, 4, 2, 1, True, "f16", "nchw"),       # NHWC copy of a ragged strided result
    (108, 64, 19, 7, 512, 7, 2, 3, True, "3xtf32", "nchw"),
    (1, 512, 26, 17, 256, 7, 2, 3, False, "3xtf32", "nhwc"),    # planes of a K split
    (102, 512, 5, 32, 8, 1, 2, 0, False, "3xtf32", "nchw"),
]


@pytest.mark.parametrize("case", STATIC)
def test_static_entry_point_takes_what_fits_without_optional_scratch(lib, case):
    import torch
    if torch.cuda.is_available():
        pytest.skip("stands in for pointers with numbers; the GPU suite runs such a layer")
    b, ci, h, w, co, k, s, p, tr, math, lay = case
    g = ops.ConvGeometry(b, ci, h, w, co, k, k, (s, s), (p, p), transposed=tr)
    d = g.desc(NML_F32, lay, NML_F32, lay, NML_F32, math, False)
    st = lib.nml_conv_forward_static(C.byref(d), 256, 256, None, 256, None)
    assert st == _lib.NML_OK + 3, lib.nml_status_string(st)  # (CUDA: no device here; not "needs N bytes of scratch")


def test_output_copy_is_bounded(lib):
    """Above 1 GB the strided result is stored directly: a workspace is kept by its caller and stays this large."""
    need = C.c_size_t()
    for batch, copied in ((12, True), (55, False)):
        g = ops.ConvGeometry(batch, 8, 87, 113, 512, 4, 4, (2, 2), (1, 1), transposed=True)
        ho, wo = g.out_hw()
        d = g.desc(NML_F32, "nchw", NML_F32, "nchw", NML_F32, "f16", False)
        assert lib.nml_conv_workspace_size(C.byref(d), 0, C.byref(need)) == _lib.NML_OK
        assert (need.value > batch * 512 * ho * wo * 4) == copied


def test_no_read_only_loads_in_the_kernels():
    """Grids become resident before the ones in front have written what they read, so no kernel may use read-only loads: neither
    the intrinsics nor const __restrict__ pointers, which the compiler reads through the same path."""
    import glob
    import os
    import re
    csrc = os.path.join(os.path.dirname(_lib.__file__), "csrc")
    files = glob.glob(os.path.join(csrc, "*.cu")) + glob.glob(os.path.join(csrc, "*.cuh"))
    assert len(files) >= 6
    for path in files:
        code = re.sub(r"//[^\n]*", "", open(path).read())
        found = re.findall(r"__ldg\s*\(|__ldc[gsavl]+\s*\(|__ldlu\s*\(|global\.nc|const\s+\w+\s*\*\s*__restrict__", code)
        assert not found, (os.path.basename(path), found[:3])

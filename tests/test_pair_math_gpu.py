"""The branch-free pair arithmetic of the batched kernels against the IEEE operations it stands
for, through the library's own comparison kernels (every float of the range, counted on the
device): the root of squared distances in box units, the table index by the rounded reciprocal, and
the minimum image on the adder.  The expected count of differences is zero in each."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _mismatches(what, lo, hi, par=0.0):
    from epsr_python_translation_b200 import _lib
    lib = _lib.load(require_device=True)
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    _lib.check(lib.epsr_check_pair_math(what, lo, hi, float(par), C.c_void_p(out.data_ptr()),
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return int(out.item())


def test_root_equals_ieee_for_every_float():
    assert _mismatches(0, 0, 1) == 0                                     # zero
    assert _mismatches(0, (127 - 60) << 23, (127 + 4) << 23) == 0        # 2^-60 .. 2^4, all of them


def test_root_of_the_smallest_distances():
    assert _mismatches(0, (127 - 100) << 23, (127 - 60) << 23) == 0      # 2^-100 .. 2^-60, all of them


@pytest.mark.parametrize("stepcl", [0.03 / 14.42, 0.03 / 31.7, 0.03 / 84.3, 0.01 / 33.3, 0.05 / 500.0])
def test_table_index_equals_the_division(stepcl):
    import numpy as np
    hi = int(np.float32(4000.0 * stepcl).view(np.uint32))
    assert _mismatches(1, 0x20000000, hi, stepcl) == 0
    assert _mismatches(1, 0, 1, stepcl) == 0


@pytest.mark.parametrize("stepcl", [0.002 / 31.7, 0.001 / 84.3, 0.87 / 16384])
def test_table_index_of_fine_grids(stepcl):
    import numpy as np
    assert _mismatches(1, 0x20000000, int(np.float32(16384.0 * stepcl).view(np.uint32)), stepcl) == 0


def test_minimum_image_square():
    import numpy as np
    top = int(np.float32(4.0).view(np.uint32))
    assert _mismatches(2, 0x30000000, top) == 0                          # positive differences up to 4
    assert _mismatches(2, 0xB0000000, top | 0x80000000) == 0             # and negative ones

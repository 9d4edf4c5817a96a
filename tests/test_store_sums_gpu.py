"""The strict sums of the pair store (ftest, ftestb): one float addition after another in store order, on both sides of
the warp's blocks of 512 entries."""

import numpy as np
import pytest

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import BoxArrays

pytestmark = pytest.mark.gpu
f32 = np.float32


def _in_order(x):
    return np.cumsum(np.concatenate([np.zeros(1, f32), x.astype(f32)]), dtype=f32)[-1]


@pytest.mark.parametrize("nmol", [1, 2, 32, 33, 46, 90, 511, 512, 513])
def test_strict_sums_in_store_order(nmol):
    from epsr_python_translation_b200.device import DeviceBox
    s = configs.c1_water(seed=nmol, nmol=nmol)
    box = BoxArrays.from_system(s)
    d = DeviceBox(box)
    d.cell_list(10, box.sepmax)
    e = np.random.default_rng(nmol).normal(size=nmol).astype(f32)
    e[::3] = 0.0
    ft, fb = d.fmolec1(e, strict=True)
    st = d.download_store()
    nintra = np.count_nonzero(e)
    assert np.array_equal(np.sort(st["ergpair"][:nintra]), np.sort(e[e != 0]))
    want = f32(_in_order(st["ergpair"][nintra:]) / f32(nmol)), f32(_in_order(e) / f32(nmol))
    assert np.array_equal(np.array([ft, fb], f32).view(np.uint32), np.array(want, f32).view(np.uint32))

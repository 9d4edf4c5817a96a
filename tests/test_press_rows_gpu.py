"""press on stores a caller laid out itself, with rows of one slot and more, up to as many as the kernel's
shared memory lists.  The two molecules' pair is the only term, so the fast sums are the strict ones."""

import numpy as np
import pytest
import torch

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import BoxArrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 57788])
def test_fast_press_of_one_pair(M):
    from epsr_python_translation_b200.device import DeviceBox
    box = BoxArrays.from_system(configs.c1_water(seed=2, nmol=2))
    d = DeviceBox(box)
    d.cell_list(10, box.sepmax)
    d.fmolec1(np.zeros(2, np.float32), strict=True)
    want = d.press(strict=True)
    assert want[0] != 0.0 and want[1] != 0.0
    mol = np.zeros((2, M), np.int32)
    mol[0, 0] = 1
    d.s_mol, d.nnbrefmax = torch.from_numpy(mol).reshape(-1).cuda(), M
    d.store.nnbrefmax, d.store.molergpair = M, d.s_mol.data_ptr()
    d.s_nergpairm[:2].fill_(1)
    for strict in (True, False):
        assert d.press(strict=strict) == want

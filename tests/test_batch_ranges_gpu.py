"""The ranges a caller gives the batched moves: rint and rfeat_c are distances of centres, and every atom
of a partner within them counts.  A box of one DMSO molecule among water needs partners within the range
plus the two largest extents, DMSO's and water's, which is less than BatchBoxes' twice the largest: the
same moves, features and energy changes under either, and the running energy is the total's."""

import ctypes as C

import numpy as np
import pytest
import torch

from epsr_python_translation_b200 import configs

pytestmark = pytest.mark.gpu


def _sweeps(s, tight):
    from epsr_python_translation_b200.batch import FEAT_IN, BatchBoxes, BoxDesc
    bb = BatchBoxes([s], rot_deg=180.0, trans_A=0.0, seed=9)
    if tight:
        d = bb.descs[0]
        r = np.sqrt(s.xa.astype(np.float64) ** 2 + s.ya.astype(np.float64) ** 2 + s.za.astype(np.float64) ** 2)
        by_mol = np.sort([r[a:a + n].max() for a, n in zip(s.naf, s.nato)])
        less = by_mol[-1] - by_mol[-2] - 4e-6
        assert less > 0.02
        d.rint, d.rfeat_c = d.rint - less, d.rfeat_c - less
        assert bb.box_t.numel() == C.sizeof(BoxDesc)
        bb.box_t.copy_(torch.from_numpy(np.frombuffer(bytes(d), np.uint8).copy()))
    per = bb.steps_per_sweep * bb.nslot
    rec = {"x": torch.zeros(8 * per, FEAT_IN, dtype=torch.bfloat16, device="cuda"),
           "t": torch.zeros(4 * per, dtype=torch.float32, device="cuda"), "n": 0}
    bb.total_energy()
    for _ in range(4):
        bb.sweep("record", record=rec)
    bb.check_status()
    running = float(bb.energy.cpu()[0])
    total = float(bb.total_energy().cpu()[0])
    scale = float(bb.emol.abs().sum().cpu())
    return rec["x"].view(torch.int16).cpu().numpy(), rec["t"].cpu().numpy(), bb.download(), running, total, scale


@pytest.mark.parametrize("seed", [1, 2])
def test_centre_ranges(seed):
    nw = 330
    L = ((10 + 3 * nw) / 0.1) ** (1.0 / 3.0)
    s = configs.build_system("one", [configs.dmso_template(), configs.water_template()], [1, nw], L, seed=seed,
                             min_heavy=2.0)
    a, b = _sweeps(s, False), _sweeps(s, True)
    assert np.array_equal(a[0], b[0])
    ok = np.isfinite(a[1])
    assert np.array_equal(ok, np.isfinite(b[1])) and ok.sum() > nw
    # the sums differ in the order of their doubles alone
    assert np.all(np.abs(a[1][ok] - b[1][ok]) <= np.spacing(np.abs(a[1][ok])))
    assert all(np.array_equal(a[2][k].view(np.uint32), b[2][k].view(np.uint32)) for k in a[2])
    for x in (a, b):
        # float sums of at most 30 terms a pair of molecules, in the changes and in the totals
        assert abs(x[3] - x[4]) <= 64 * 2.0 ** -24 * x[5] * 4

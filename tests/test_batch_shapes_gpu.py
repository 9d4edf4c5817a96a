"""The batched moves in every form of their kernels: with and without the cell-ordered copy of the
molecules (a caller's structure may lack it), few moves (1,024 threads a move), some (512) and many
(256), boxes whose tables fit beside the search in shared memory and a mixture whose tables don't.  The
same sweep gives the same features and moves; the energies are sums of the same doubles in another
order, so the recorded float32 targets may differ in their last place.  And the cells' members in
ascending order for few, many and very many of them."""

import numpy as np
import pytest
import torch

from epsr_python_translation_b200 import configs

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "one_box": lambda: [configs.c1_water(seed=21, nmol=40)],
    "mixture": lambda: [configs.c2_mixture(seed=22, ndmso=60, nwater=120)],
    "boxes_24": lambda: [configs.c1_water(seed=30 + i, nmol=60) for i in range(24)],
    "boxes_48": lambda: [configs.silica(seed=60 + i, natom=240) for i in range(48)],
}


def _sweep(systems, flags):
    from epsr_python_translation_b200.batch import FEAT_IN, BatchBoxes
    bb = BatchBoxes(systems, rot_deg=20.0, trans_A=0.6, seed=9)
    bb.c.threads = flags
    per = bb.steps_per_sweep * bb.nslot
    rec = {"x": torch.zeros(2 * per, FEAT_IN, dtype=torch.bfloat16, device="cuda"),
           "t": torch.zeros(per, dtype=torch.float32, device="cuda"), "n": 0}
    bb.total_energy()
    bb.sweep("record", record=rec)
    bb.sweep("plain")
    bb.check_status()
    return rec["x"].view(torch.int16).cpu().numpy(), rec["t"].cpu().numpy(), bb.download(), bb.counters_host(), bb.nslot


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_forms_agree(name):
    from epsr_python_translation_b200.batch import CELL_MOL
    systems = SYSTEMS[name]()
    x, t, co, cnt, nslot = _sweep(systems, 256 | CELL_MOL)
    for flags in (256, 128, 64 | CELL_MOL):
        x2, t2, co2, cnt2, _ = _sweep(systems, flags)
        assert np.array_equal(x, x2)
        ok = np.isfinite(t)
        assert np.array_equal(ok, np.isfinite(t2)) and ok.any()
        assert np.all(np.abs(t[ok] - t2[ok]) <= np.spacing(np.abs(t[ok])))
        for k in ("xa", "ya", "za", "xadd", "yadd", "zadd"):
            assert np.array_equal(co[k].view(np.uint32), co2[k].view(np.uint32)), (k, flags)
        assert np.array_equal(cnt, cnt2)


@pytest.mark.parametrize("natom", [33, 256, 257])
def test_cell_members_ascend(natom):
    """Every molecule of the box in one cell."""
    from epsr_python_translation_b200.batch import BatchBoxes
    bb = BatchBoxes([configs.silica(seed=5, natom=natom + 243), configs.c1_water(seed=4, nmol=30)], seed=3)
    m0 = bb.systems[0].nmol
    for a in (bb.xadd, bb.yadd, bb.zadd):
        a[:natom] = 0.11
        a[natom:m0] = torch.linspace(-0.49, 0.49, m0 - natom, device="cuda")
    bb.begin_sweep()
    start, mols = bb.cell_start.cpu().numpy(), bb.cell_mols.cpu().numpy()
    nc0 = bb.descs[0].ncell ** 3
    s = start[:nc0 + 1]
    assert s[0] == 0 and s[-1] == m0 and np.max(np.diff(s)) >= natom
    for c in range(nc0):
        assert np.all(np.diff(mols[s[c]:s[c + 1]]) > 0)
    assert np.array_equal(np.sort(mols[:m0]), np.arange(m0))


def test_feature_rows_on_a_two_byte_boundary():
    """Recorded features may lie at any element of the caller's array."""
    from epsr_python_translation_b200.batch import FEAT_IN, BatchBoxes
    out = []
    for off in (0, 1, 3):
        bb = BatchBoxes([configs.c1_water(seed=21, nmol=40)], rot_deg=20.0, trans_A=0.6, seed=9)
        per = bb.steps_per_sweep * bb.nslot
        flat = torch.zeros(2 * per * FEAT_IN + 4, dtype=torch.bfloat16, device="cuda")
        rec = {"x": flat[off:off + 2 * per * FEAT_IN].view(2 * per, FEAT_IN),
               "t": torch.zeros(per, dtype=torch.float32, device="cuda"), "n": 0}
        assert rec["x"].data_ptr() % 4 == 2 * (off % 2)
        bb.sweep("record", record=rec)
        bb.check_status()
        out.append((rec["x"].contiguous().view(torch.int16).cpu().numpy(), rec["t"].cpu().numpy()))
        assert not flat[:off].any() and not flat[off + 2 * per * FEAT_IN:].any()
    for x, t in out[1:]:
        assert np.array_equal(x, out[0][0]) and x.any()
        assert np.array_equal(t.view(np.uint32), out[0][1].view(np.uint32))

"""The cycles whose sums are exact (strict float sums in list order; double sums of a box with
rotational groups in a cycle without rotations) on the walk against the sequential kernel, which a
store without its mirror index selects: the same moves of the same stream.  Strict cycles agree
bit for bit; the double sums add the same doubles in another order, so a change may differ where
their rounding to float does (one unit in the last place)."""

import numpy as np
import pytest
import torch

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import BoxArrays, Ran1State, trsteps

pytestmark = pytest.mark.gpu
f32 = np.float32


def _box(s, groups):
    from epsr_python_translation_b200.device import DeviceBox
    from epsr_python_translation_b200.intra import IntraModel
    box = BoxArrays.from_system(s)
    d = DeviceBox(box)
    d.cell_list(10, box.sepmax)
    d.fmolec1(configs.intra_energies(s), strict=True)
    tmax, tmin = trsteps(box.natomr)
    d.mc_setup(rejrate=0.75, stepr=1.0, stepm=1.0, wholerot=np.full(s.nmoltype, f32(0.05), f32),
               wholetrans=np.full(s.nmoltype, f32(0.3) / s.dmax, f32), ran1=Ran1State(idum=-77), trstepmax=tmax,
               trstepmin=tmin)
    if groups:
        r = configs.rotations(s)
        d.set_rotations(IntraModel(d, **configs.intra_model(s), ngrot=r["ngrot"]), r["nrf"], r["nrl"], r["axis"],
                        r["first"], r["last"], r["atoms"])
        d.m_internrot.copy_(torch.tensor([0.05, 0.02]))
    return d


SYSTEMS = {
    # fewer molecules than the enumerated window, than the warps, one list chunk, several chunks
    "water_4": lambda: configs.c1_water(seed=3, nmol=4), "water_9": lambda: configs.c1_water(seed=4, nmol=9),
    "water_100": lambda: configs.c1_water(seed=5), "water_1200": lambda: configs.c1_water(seed=6, nmol=1200),
    "mixture_45": lambda: configs.c2_mixture(seed=7, ndmso=15, nwater=30),
    "silica_301": lambda: configs.silica(seed=8, natom=301),
}


@pytest.mark.parametrize("name,groups", [(k, False) for k in SYSTEMS] + [("mixture_45", True)])
def test_walk_matches_sequential_kernel(name, groups):
    s = SYSTEMS[name]()
    a, b = _box(s, groups), _box(s, groups)
    b.store.mirror = None            # the sequential kernel
    for _ in range(3):
        for d in (a, b):
            d.molfit(strict=not groups, rotcycle=False)
            d.check_status()
        x, y = a.download_mc(), b.download_mc()
        if groups:
            assert np.all(np.abs(x["den"] - y["den"]) <= np.spacing(np.abs(y["den"])))
        else:
            assert np.array_equal(x["den"].view(np.uint32), y["den"].view(np.uint32))
            assert x["fadds"] == y["fadds"]
        for k in ("acc", "wholerot", "wholetrans", "internrot", "interntrans", "nwhole", "nmovem", "nstepreject"):
            assert np.array_equal(x[k], y[k]), k
        assert np.array_equal(x["ran1"].as_array(), y["ran1"].as_array())
        ca, cb = a.download_coords(), b.download_coords()
        assert all(np.array_equal(ca[k].view(np.uint32), cb[k].view(np.uint32)) for k in ca)
        assert np.array_equal(a.download_store()["ergpair"], b.download_store()["ergpair"])


@pytest.mark.parametrize("name,groups", [("water_100", False), ("mixture_45", False), ("mixture_45", True)])
def test_stale_mirror_goes_to_the_sequential_kernel(name, groups):
    """Rows in another order than the mirror index was built for (a host that rewrote them): the exact
    cycles need no mirror, so they move as without one."""
    s = SYSTEMS[name]()
    a, b = _box(s, groups), _box(s, groups)
    b.store.mirror = None
    rng = np.random.default_rng(11)
    M, nm = a.nnbrefmax, a.s_nergpairm.cpu().numpy()
    mol, ref = (t[:s.nmol * M].cpu().numpy().reshape(-1, M) for t in (a.s_mol, a.s_ref))
    for m in range(s.nmol):
        p = np.concatenate([[0], 1 + rng.permutation(nm[m] - 1)])
        mol[m, :nm[m]], ref[m, :nm[m]] = mol[m, p], ref[m, p]
    for d in (a, b):
        for t, v in ((d.s_mol, mol), (d.s_ref, ref)):
            t[:s.nmol * M].copy_(torch.from_numpy(v.reshape(-1)))
    for _ in range(2):
        for d in (a, b):
            d.molfit(strict=not groups, rotcycle=False)
            d.check_status()
        x, y = a.download_mc(), b.download_mc()
        assert np.array_equal(x["acc"], y["acc"])
        assert np.array_equal(x["den"].view(np.uint32), y["den"].view(np.uint32))
        assert np.array_equal(x["ran1"].as_array(), y["ran1"].as_array())
        ca, cb = a.download_coords(), b.download_coords()
        assert all(np.array_equal(ca[k].view(np.uint32), cb[k].view(np.uint32)) for k in ca)
        assert np.array_equal(a.download_store()["ergpair"], b.download_store()["ergpair"])


@pytest.mark.parametrize("off", [4, 8])
def test_scratch_on_a_four_byte_boundary(off):
    """A scratch that only the sequential kernel can use: the same strict cycles as on any other."""
    s = SYSTEMS["mixture_45"]()
    a, b = _box(s, False), _box(s, False)
    nb = b.lib.epsr_molfit_scratch_bytes(s.nmol, s.natom, b.nnbrefmax)
    buf = torch.zeros(nb + 16, dtype=torch.uint8, device="cuda")
    b.scratch = lambda name, n: buf[off:off + n]
    for _ in range(2):
        for d in (a, b):
            d.molfit(strict=True)
            d.check_status()
        x, y = a.download_mc(), b.download_mc()
        assert np.array_equal(x["acc"], y["acc"]) and np.array_equal(x["den"].view(np.uint32), y["den"].view(np.uint32))
        assert np.array_equal(a.download_store()["ergpair"], b.download_store()["ergpair"])
    assert not buf.any()


def _chains(seed=9):
    """Molecules of 64 atoms (the largest the kernels take), of 46 and of three."""
    grid = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) * 1.6
    big, mid = (configs.MolTemplate(k, ["C"] * n, grid[:n] - grid[:n].mean(axis=0)) for k, n in (("big", 64), ("mid", 46)))
    return configs.build_system("chains", [big, mid, configs.water_template()], [2, 2, 6], 30.0, seed=seed)


def _same(a, b):
    for d in (a, b):
        d.molfit(strict=True)
        d.check_status()
    x, y = a.download_mc(), b.download_mc()
    assert np.array_equal(x["acc"], y["acc"]) and np.array_equal(x["den"].view(np.uint32), y["den"].view(np.uint32))
    assert np.array_equal(x["ran1"].as_array(), y["ran1"].as_array())
    assert np.array_equal(a.download_store()["ergpair"], b.download_store()["ergpair"])


@pytest.mark.parametrize("maxat", [0, 64, 45, 3])
def test_largest_molecules_and_a_box_that_understates_them(maxat):
    """The sequential kernel never read the box's maxat; where it is less than the molecules have, their strict
    cycles go there."""
    s = _chains()
    a, b = _box(s, False), _box(s, False)
    assert np.count_nonzero(a.s_nergpairm.cpu().numpy() > 1) >= 4
    a.cbox.maxat = maxat
    b.store.mirror = None
    for _ in range(2):
        _same(a, b)


@pytest.mark.parametrize("ntype", [190, 240])
def test_strict_cycles_of_boxes_with_many_atom_types(ntype):
    """The type pairs of 240 types do not fit the energy pass's shared memory; the sequential kernel reads them
    where they are."""
    s = SYSTEMS["mixture_45"]()
    a, b = _box(s, False), _box(s, False)
    n = s.ntype
    ref = torch.zeros(ntype, ntype, dtype=torch.int32, device="cuda")
    ref[:n, :n] = a.npairref.reshape(n, n)
    a.cbox.ntype, a.cbox.npairref = ntype, ref.data_ptr()
    for _ in range(2):
        _same(a, b)


@pytest.mark.parametrize("nmol,walks", [(2, 0), (7, 0), (8, 1)])
def test_few_molecules_stay_on_the_sequential_kernel(nmol, walks):
    """One launch against nine: below eight molecules the sequential kernel is the faster one."""
    import ctypes as C
    s = configs.c1_water(seed=3, nmol=nmol)
    a, b = _box(s, False), _box(s, False)
    b.store.mirror = None
    ms, n = C.c_double(), C.c_int64()
    a.lib.epsr_timing_enable(1)
    try:
        a.molfit(strict=True)
        torch.cuda.synchronize()
        a.lib.epsr_timing_read(b"spec_walk_kernel", C.byref(ms), C.byref(n))
    finally:
        a.lib.epsr_timing_enable(0)
    assert n.value == walks
    b.molfit(strict=True)
    x, y = a.download_mc(), b.download_mc()
    assert np.array_equal(x["den"].view(np.uint32), y["den"].view(np.uint32))
    for _ in range(2):
        _same(a, b)

"""The pair store against the C oracle, bit for bit, where its kernels branch: rows beyond the entries that
are ranked (the bitonic network sorts them), partial groups of four partner atoms (molecules of 1, 3 and
10 atoms), a triclinic cell, cells of more than 256 members and regions beyond a thread's 32 remembered
entries, and a store with as many sums as several CTAs take.  The double sums of the fast mode are those of
the same float32 energies in another order: 1e-12 of the summed magnitudes before their rounding to float."""

import numpy as np
import pytest

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import BoxArrays
from oracle import oracle
from tests.goldens import assert_bits_equal

pytestmark = pytest.mark.gpu
f32 = np.float32


def _dense():
    """A box narrower than twice the tables' range: nearly every molecule is a partner."""
    box = BoxArrays.from_system(configs.c1_water(seed=5, nmol=700))
    box.dmax = f32(15.0)
    box.xstar = (box.x / box.dmax).astype(f32)
    return box


def _triclinic():
    box = BoxArrays.from_system(configs.c2_mixture(seed=6, ndmso=12, nwater=24))
    box.cubic = False
    box.lat6 = np.array([1.0, 0.1, 0.05, 0.995, 0.08, 0.99], f32)
    box.lat9 = np.array([1.0, 0.0, 0.0, 0.1, 0.995, 0.0, 0.05, 0.08, 0.99], f32)
    return box


BOXES = {
    "dense_700": (_dense, 10), "triclinic": (_triclinic, 10),
    "silica": (lambda: BoxArrays.from_system(configs.silica(seed=3, natom=303)), 10),
    "mixture": (lambda: BoxArrays.from_system(configs.c2_mixture(seed=4, ndmso=41, nwater=83)), 7),
    "crowded_cells": (lambda: BoxArrays.from_system(configs.c1_water(seed=8, nmol=2300)), 290),
}


@pytest.mark.parametrize("name", list(BOXES))
def test_store_matches_oracle(name):
    from epsr_python_translation_b200.device import DeviceBox
    make, nmolcell = BOXES[name]
    box = make()
    eintra = np.random.default_rng(1).standard_normal(box.nmol).astype(f32)
    eintra[::3] = 0
    oc = oracle.cell_list(box, nmolcell, box.sepmax)
    ost = oracle.fmolec1(box, oc, eintra, capacity=box.nmol * min(box.nmol, 800))
    d = DeviceBox(box)
    d.cell_list(nmolcell, box.sepmax)
    sums = d.fmolec1(eintra, strict=True)
    st = d.download_store()
    assert st["nergpair"] == ost["nergpair"]
    n = st["nergpair"]
    assert_bits_equal(st["ergpair"], ost["ergpair"][:n], "ergpair")
    assert np.array_equal(st["nergpairm"], ost["nergpairm"])
    M = st["nnbrefmax"]
    om, oref = ost["molergpair"].reshape(box.nmol, M), ost["ergpairref"].reshape(box.nmol, M)
    for m in range(box.nmol):
        k = int(st["nergpairm"][m])
        assert np.array_equal(st["molergpair"][m, :k], om[m, :k]) and np.array_equal(st["ergpairref"][m, :k], oref[m, :k])
    if name == "dense_700":
        assert st["nergpairm"].max() > 512
    fast = d.fmolec1(eintra, strict=False)
    e = st["ergpair"][int(np.count_nonzero(eintra)):].astype(np.float64)
    for got, v in ((fast[0], e), (fast[1], eintra.astype(np.float64))):
        ref = v.sum() / box.nmol
        assert abs(float(got) - ref) <= 2.0 ** -24 * abs(ref) + 1e-12 * np.abs(v).sum() / box.nmol
    assert np.isfinite(sums[0])


def test_long_region_matches_fine_cells():
    """A region of 9,000 molecules (past a thread's remembered entries) holds the pairs that fine cells find."""
    from epsr_python_translation_b200.device import DeviceBox
    box = BoxArrays.from_system(configs.c3_water(seed=2, nmol=9000))
    pairs = []
    for nmolcell in (1200, 10):
        d = DeviceBox(box)
        d.cell_list(nmolcell, box.sepmax)
        d.fmolec1(np.zeros(box.nmol, f32), strict=False)
        st = d.download_store()
        rows = np.repeat(np.arange(box.nmol), st["nergpairm"])
        cols = np.concatenate([st["molergpair"][m, :k] for m, k in enumerate(st["nergpairm"])])
        ref = np.concatenate([st["ergpairref"][m, :k] for m, k in enumerate(st["nergpairm"])])
        e = st["ergpair"][ref - 1]
        o = np.lexsort((cols, rows))
        pairs.append((rows[o], cols[o], e[o], st["nnbrefmax"]))
    assert pairs[0][3] == 9000 and pairs[1][3] < 9000
    assert np.array_equal(pairs[0][0], pairs[1][0]) and np.array_equal(pairs[0][1], pairs[1][1])
    assert_bits_equal(pairs[0][2], pairs[1][2], "energies")


@pytest.mark.parametrize("zero", [False, True])
@pytest.mark.parametrize("nmol,nmolcell,rmax", [(1, 10, None), (2, 10, None), (3, 10, None), (4, 10, None), (5, 10, None),
                                                (16, 1, 0.0), (64, 1, 0.0), (200, 1, 0.0), (200, 2, 0.0)])
def test_short_rows_match_oracle(nmol, nmolcell, rmax, zero):
    """Rows of one to five entries, from small boxes and from cells that are their own region (two molecules
    at most in the first three), with and without intramolecular entries; the mirror index pairs each entry
    with the other one of its energy."""
    from epsr_python_translation_b200.device import DeviceBox
    box = BoxArrays.from_system(configs.c1_water(seed=nmol, nmol=nmol))
    rmax = box.sepmax if rmax is None else f32(rmax)
    eintra = np.zeros(nmol, f32) if zero else np.random.default_rng(nmol).standard_normal(nmol).astype(f32)
    oc = oracle.cell_list(box, nmolcell, rmax)
    ost = oracle.fmolec1(box, oc, eintra, capacity=nmol * (oc["nnbrefmax"] + 1))
    d = DeviceBox(box)
    d.cell_list(nmolcell, rmax)
    d.fmolec1(eintra, strict=True)
    st = d.download_store()
    M, n = st["nnbrefmax"], st["nergpair"]
    assert M == oc["nnbrefmax"] and n == ost["nergpair"]
    assert_bits_equal(st["ergpair"], ost["ergpair"][:n], "ergpair")
    assert np.array_equal(st["nergpairm"], ost["nergpairm"])
    om, oref = ost["molergpair"].reshape(nmol, M), ost["ergpairref"].reshape(nmol, M)
    mirror = d.s_mirror[:nmol * M].cpu().numpy()
    for m in range(nmol):
        k = int(st["nergpairm"][m])
        assert np.array_equal(st["molergpair"][m, :k], om[m, :k]) and np.array_equal(st["ergpairref"][m, :k], oref[m, :k])
        for s in range(k):
            p = st["molergpair"][m, s]
            if p != m:
                e = int(mirror[m * M + s])
                assert e // M == p and st["molergpair"][p, e % M] == m
                assert st["ergpairref"][p, e % M] == st["ergpairref"][m, s]


@pytest.mark.parametrize("nmol,nmolcell,rmax,M", [(100, 10, None, 1), (100, 10, None, 90), (200, 1, 0.1, 15),
                                                  (200, 1, 0.1, 21)])
def test_too_few_slots_are_refused(nmol, nmolcell, rmax, M):
    """Regions of more molecules than the store has slots (all of them, some, the largest): refused with the
    capacity error whatever the scratch held, and the box's next store, with the slots it needs, is the
    oracle's."""
    import torch

    from epsr_python_translation_b200 import _lib
    from epsr_python_translation_b200.device import DeviceBox
    box = BoxArrays.from_system(configs.c1_water(seed=5, nmol=nmol))
    rmax = box.sepmax if rmax is None else f32(rmax)
    eintra = np.ones(nmol, f32)
    oc = oracle.cell_list(box, nmolcell, rmax)
    ost = oracle.fmolec1(box, oc, eintra, capacity=nmol * nmol)
    d = DeviceBox(box)
    d.cell_list(nmolcell, rmax)
    need = d.nnbrefmax
    assert need > M
    nb = d.lib.epsr_fmolec1_scratch_bytes(nmol, d.cells.ncell, need)
    d.scratch("fmolec1", nb).fill_(0x7f)
    for name in ("_s_mol", "_s_ref"):
        d._buf(name, nmol * need, torch.int32).fill_(0x7f7f7f7f)
    d.nnbrefmax = M
    with pytest.raises(_lib.EpsrGpuError) as e:
        d.fmolec1(eintra, strict=True)
    assert e.value.code == 3
    d.nnbrefmax = need
    d.fmolec1(eintra, strict=True)
    st = d.download_store()
    n = st["nergpair"]
    assert n == ost["nergpair"] and np.array_equal(st["nergpairm"], ost["nergpairm"])
    assert_bits_equal(st["ergpair"], ost["ergpair"][:n], "ergpair")


@pytest.mark.parametrize("off", [4, 8, 12])
def test_scratch_on_a_four_byte_boundary(off):
    """The store needs four-byte alignment of its scratch, no more."""
    import torch

    from epsr_python_translation_b200.device import DeviceBox
    box = BoxArrays.from_system(configs.c2_mixture(seed=4, ndmso=41, nwater=83))
    eintra = np.random.default_rng(1).standard_normal(box.nmol).astype(f32)
    out = []
    for shift in (0, off):
        d = DeviceBox(box)
        d.cell_list(7, box.sepmax)
        buf = torch.zeros(d.lib.epsr_fmolec1_scratch_bytes(box.nmol, d.cells.ncell, d.nnbrefmax) + 16, dtype=torch.uint8,
                          device="cuda")
        d.scratch = lambda name, nb, buf=buf, shift=shift: buf[shift:shift + nb]
        sums = d.fmolec1(eintra, strict=True), d.fmolec1(eintra, strict=False)
        st = d.download_store()
        out.append((sums, st, d.s_mirror[:box.nmol * d.nnbrefmax].cpu().numpy()))
        assert not buf[:shift].any()
    (s0, a, m0), (s1, b, m1) = out
    assert s0 == s1 and np.array_equal(m0, m1) and a["nergpair"] == b["nergpair"]
    assert all(np.array_equal(a[k], b[k]) for k in ("nergpairm", "molergpair", "ergpairref"))
    assert_bits_equal(a["ergpair"], b["ergpair"], "ergpair")

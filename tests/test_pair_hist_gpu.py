"""The intermolecular histograms against the C oracle, bit for bit (integer counts, exactly normalised),
at the edges of the pair kernel: distances on the bins' halves and at zero, one and several origin
chunks and target tiles, origins all or sampled, a triclinic cell, more atom types than the staged rows
hold, and bins so fine that the index is always divided."""

import numpy as np
import pytest
import torch

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import BoxArrays, Ran1State
from oracle import oracle
from tests.goldens import assert_bits_equal

pytestmark = pytest.mark.gpu
f32 = np.float32


def _grid_box(nmol, ld=None, cellst=None, spread=True):
    """Atoms on a cubic grid of half a bin: many distances are odd multiples of half a bin, some are zero."""
    box = BoxArrays.from_system(configs.c1_water(seed=2, nmol=nmol))
    if cellst is not None:
        box.cellst = f32(cellst)
    if spread:
        h = f32(0.5) * f32(box.cellst) / f32(box.dmax)
        rng = np.random.default_rng(nmol)
        for k in ("xadd", "yadd", "zadd"):
            setattr(box, k, (rng.integers(-60, 60, box.xadd.size).astype(f32) * h).astype(f32))
        for k in ("xa", "ya", "za"):
            setattr(box, k, (rng.integers(-3, 4, box.xa.size).astype(f32) * h).astype(f32))
    return box


def _many_types(nmol, ntype):
    box = BoxArrays.from_system(configs.c1_water(seed=3, nmol=nmol))
    rng = np.random.default_rng(ntype)
    box.itype = rng.integers(0, ntype, box.itype.size).astype(np.int32)
    ref = np.zeros((ntype, ntype), np.int32)
    pairs = [(i, j) for i in range(ntype) for j in range(i, ntype)]
    for k, (i, j) in enumerate(pairs):
        ref[i, j] = ref[j, i] = k
    box.npairref = ref
    box.n1extr = np.array([p[0] for p in pairs], np.int32)
    box.n2extr = np.array([p[1] for p in pairs], np.int32)
    z = np.zeros((len(pairs),) + box.xavs.shape[1:], f32)
    box.xavs, box.xavs1, box.ecoul, box.ecoul1 = z, z.copy(), z.copy(), z.copy()
    box.cfrac = np.full(ntype, f32(1.0 / ntype), f32)
    return box


def _triclinic(nmol):
    box = BoxArrays.from_system(configs.c1_water(seed=4, nmol=nmol))
    box.cubic = False
    box.lat6 = np.array([1.0, 0.2, -0.1, 0.9, 0.15, 0.95], f32)
    return box


BOXES = {
    "halves_8": lambda: _grid_box(8), "halves_43": lambda: _grid_box(43), "halves_86": lambda: _grid_box(86),
    "halves_700": lambda: _grid_box(700), "water_1201": lambda: _grid_box(1201, spread=False),
    "triclinic_150": lambda: _triclinic(150), "types_16": lambda: _many_types(60, 16), "types_17": lambda: _many_types(60, 17),
}


@pytest.mark.parametrize("ngr", [0, 7])
@pytest.mark.parametrize("name", list(BOXES))
def test_pair_histograms_match_oracle(name, ngr):
    from epsr_python_translation_b200.device import DeviceBox
    box = BOXES[name]()
    d = DeviceBox(box)
    st = Ran1State(idum=-5)
    rmx = np.full(box.npairs, f32(-2.0), f32)
    rmx[::2] = f32(3.5)
    t = d.ran1_tensor(st)
    got = d.atogen(ngr, t, rmx)
    wav, potex, ref, after = oracle.atogen(box, ngr, st, rmx)
    assert got == ref
    mine, mp = d.download_wav()
    assert_bits_equal(mine[:, :, 1:box.npt1 + 1], wav[:, :, 1:box.npt1 + 1], "wav")
    assert_bits_equal(mp, potex, "potex")
    assert np.array_equal(t.cpu().numpy(), after.as_array())


def test_index_is_divided_where_bins_are_fine():
    """A step below 0.87/4000 takes the division for every pair: same counts as the oracle's."""
    from epsr_python_translation_b200.device import DeviceBox
    box = _grid_box(90, spread=False)
    box.cellst = f32(box.dmax) * f32(1.0 / 9000.0)
    d = DeviceBox(box)
    st = Ran1State(idum=-6)
    t = d.ran1_tensor(st)
    rmx = np.full(box.npairs, f32(-2.0), f32)
    d.atogen(0, t, rmx)
    wav, potex, _, _ = oracle.atogen(box, 0, st, rmx)
    mine, mp = d.download_wav()
    assert_bits_equal(mine[:, :, 1:box.npt1 + 1], wav[:, :, 1:box.npt1 + 1], "wav")
    assert_bits_equal(mp, potex, "potex")


@pytest.mark.parametrize("nq,npt1", [(1, 2), (63, 17), (64, 18), (65, 513), (300, 514), (257, 1200)])
def test_gensq_sums_match_sequential(nq, npt1):
    """gensq's sums in order over r against the same sums in numpy, one float32 operation at a time, at the
    edges of its groups and chunks and for both strides of the transform table."""
    from epsr_python_translation_b200 import transforms
    rng = np.random.default_rng(nq)
    npairs, ld = 3, npt1 + 1
    wav = rng.standard_normal((2, npairs, ld)).astype(f32)
    wav[0][rng.random((npairs, ld)) < 0.3] = 0
    ycoh = rng.standard_normal(ld).astype(f32)
    F = rng.standard_normal((ld, nq + 1)).astype(f32)
    n2 = np.array([0, 1, 1], np.int32)
    ns = np.array([1.0, 2.5], f32)
    ref = np.zeros((2, npairs, nq + 1), f32)
    for ic in range(npairs):
        s1 = np.zeros(nq + 1, f32)
        s2 = np.zeros(nq + 1, f32)
        s3 = f32(0)
        for j in range(2, npt1 + 1):
            if abs(wav[0, ic, j]) > 0:
                s1 = s1 + wav[0, ic, j] * F[j]
            s2 = s2 + ((wav[1, ic, j] - ycoh[j]) * ns[n2[ic]]) * F[j]
            s3 = s3 + wav[1, ic, j]
        ref[0, ic], ref[1, ic] = s1, s2 if s3 > 0 else np.zeros(nq + 1, f32)
    dev = torch.from_numpy(wav.reshape(-1)).cuda()
    for table, sj, si in ((F, nq + 1, 1), (np.ascontiguousarray(F.T), 1, ld)):
        out = transforms.gensq(nq, npt1, dev, ld, table, sj, si, ycoh, n2, ns, npairs).cpu().numpy()
        assert_bits_equal(out.reshape(2, npairs, nq + 1)[:, :, 1:], ref[:, :, 1:], "sofq")


@pytest.mark.parametrize("nr,nq,npairs", [(1, 4, 1), (7, 256, 3), (9, 257, 32), (64, 600, 33)])
def test_stog_sums_match_sequential(nr, nq, npairs):
    """stog's sums in order over Q against numpy's, one float32 operation at a time, with the sine in double
    rounded once, at the edges of its r points, pairs and chunks, with windows, and at r = 0.  The device's
    double sine may differ from numpy's in its last bit, which moves a float32 sine at most by one unit:
    the bound is 2^-23 of the magnitude of the summed terms."""
    from epsr_python_translation_b200 import transforms
    rng = np.random.default_rng(nr)
    q = np.concatenate([[0], 0.05 * np.arange(1, nq + 1)]).astype(f32)
    r = np.concatenate([[0], 0.03 * np.arange(nr)]).astype(f32)
    s = rng.standard_normal((npairs, nq + 1)).astype(f32)
    lo = rng.integers(-1, 3, npairs).astype(np.int32)
    hi = np.where(np.arange(npairs) % 2, nq, max(nq - 3, 1)).astype(np.int32)
    xwt = rng.standard_normal(npairs).astype(f32)
    out = transforms.stog(0.1, q, s, r, lo, hi, xwt).cpu().numpy()
    pi = f32(np.pi)
    sfac = f32(f32(f32(f32(0.5) * (q[4] - q[3])) / pi) / pi) / f32(0.1)
    for ic in range(npairs):
        qm = pi / q[min(nq, max(1, hi[ic]))]
        x = (qm * q).astype(f32)
        with np.errstate(invalid="ignore", divide="ignore"):
            lw = np.where(x == 0, f32(1), np.where(x < pi, np.sin(x.astype(np.float64)).astype(f32) / x, f32(0))).astype(f32)
        tot = np.zeros(nr + 1, f32)
        mag = np.zeros(nr + 1, np.float64)
        for i in range(max(1, lo[ic]), min(nq, hi[ic]) + 1):
            sn = np.where(r > 0, np.sin((q[i] * r).astype(f32).astype(np.float64)).astype(f32), q[i]).astype(f32)
            term = s[ic, i] * ((q[i] * sn).astype(f32) * lw[i])
            tot = (tot + term).astype(f32)
            mag += np.abs(term.astype(np.float64)) + 2.0 ** -3 * np.abs(tot)
        with np.errstate(invalid="ignore", divide="ignore"):
            v = (sfac * tot).astype(f32)
            ref = xwt[ic] + np.where(r > 0, v / r, v)
            tol = 2.0 ** -21 * (np.abs(xwt[ic]) + sfac * mag / np.where(r > 0, r, 1))
        assert np.all(np.abs(out[ic, 1:] - ref[1:]) <= tol[1:])


def _sheared(box):
    box.cubic = False
    box.lat6 = np.array([1.0, 0.2, -0.1, 0.9, 0.15, 0.95], f32)
    return box


SHEARED = {"one": lambda: _grid_box(1), "halves_43": lambda: _grid_box(43), "halves_86": lambda: _grid_box(86),
           "water_1201": lambda: _grid_box(1201, spread=False), "types_16": lambda: _many_types(60, 16),
           "types_17": lambda: _many_types(60, 17), "mixture": lambda: BoxArrays.from_system(configs.c2_mixture(seed=5, ndmso=60, nwater=90))}


@pytest.mark.parametrize("ngr", [0, 7])
@pytest.mark.parametrize("name", list(SHEARED))
def test_sheared_cells_match_oracle(name, ngr):
    """The general cell's own loop: one and several origin chunks and tiles, origins all or sampled, few and many types."""
    from epsr_python_translation_b200.device import DeviceBox
    box = _sheared(SHEARED[name]())
    d = DeviceBox(box)
    st = Ran1State(idum=-8)
    rmx = np.full(box.npairs, f32(-2.0), f32)
    rmx[::2] = f32(3.5)
    t = d.ran1_tensor(st)
    got = d.atogen(ngr, t, rmx)
    wav, potex, ref, after = oracle.atogen(box, ngr, st, rmx)
    assert got == ref
    mine, mp = d.download_wav()
    assert_bits_equal(mine[:, :, 1:box.npt1 + 1], wav[:, :, 1:box.npt1 + 1], "wav")
    assert_bits_equal(mp, potex, "potex")
    assert np.array_equal(t.cpu().numpy(), after.as_array())

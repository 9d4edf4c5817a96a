"""The intramolecular cycle of a box with rotational groups (molfit.py:124-267) where molecules without
groups stand before molecules with them in index order, and single atoms among them: the kernel's
warps pass from a molecule that is not rotated to one that is, in every order, and the cycle equals the
C oracle's bit for bit (its cosines injected)."""

import numpy as np
import pytest

from epsr_python_translation_b200 import configs
from epsr_python_translation_b200.box import BoxArrays, Ran1State, trsteps
from oracle import oracle
from tests.goldens import assert_bits_equal

pytestmark = pytest.mark.gpu
f32 = np.float32


def _system(seed):
    w, d, o = configs.water_template(), configs.dmso_template(), configs.atom_template("Si")
    parts = [(o, 2), (w, 3), (d, 2), (w, 1), (d, 1), (o, 1), (d, 3), (o, 2), (w, 2), (d, 1)]
    L = (sum(n * len(t.labels) for t, n in parts) / 0.08) ** (1.0 / 3.0)
    return configs.build_system("order", [t for t, _ in parts], [n for _, n in parts], L, seed=seed)


@pytest.mark.parametrize("stepmi", [1.0, 0.0])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_groups_behind_plain_molecules(seed, stepmi):
    import torch

    from epsr_python_translation_b200.device import DeviceBox
    from epsr_python_translation_b200.intra import IntraModel
    s = _system(seed)
    r = configs.rotations(s)
    turns = r["ngrot"] > 0
    assert np.count_nonzero(~turns[:-1] & turns[1:]) >= 3
    m = dict(configs.intra_model(s), ngrot=r["ngrot"])
    ob, d = BoxArrays.from_system(s), DeviceBox(BoxArrays.from_system(s))
    model = IntraModel(d, **m)
    e = oracle.en_mole_intra_all(ob, m)
    oc = oracle.cell_list(ob, 10, ob.sepmax)
    ost = oracle.fmolec1(ob, oc, e, capacity=ob.nmol * ob.nmol)
    M = oc["nnbrefmax"]
    ost = dict(nnbrefmax=M, nergpair=ost["nergpair"], nergpairm=np.ascontiguousarray(ost["nergpairm"], np.int32),
               molergpair=np.ascontiguousarray(ost["molergpair"][:, :M], np.int32).reshape(-1),
               ergpairref=np.ascontiguousarray(ost["ergpairref"][:, :M], np.int32).reshape(-1),
               ergpair=np.array(ost["ergpair"][: ost["nergpair"]], f32))
    d.cell_list(10, ob.sepmax)
    d.fmolec1(e, strict=True)
    nmt = ob.nmoltype
    tmax, tmin = trsteps(ob.natomr)
    steps = dict(wholerot=np.full(nmt, f32(0.05)), wholetrans=np.full(nmt, f32(0.3) / f32(ob.dmax)),
                 internrot=np.full(nmt, f32(0.05)), interntrans=np.full(nmt, f32(0.02) / f32(ob.dmax)))
    d.mc_setup(rejrate=f32(0.75), stepr=f32(1.0), stepm=f32(1.0), ran1=Ran1State(idum=-seed), trstepmax=tmax,
               trstepmin=tmin, fadds=f32(0.5), **steps)
    d.set_rotations(model, r["nrf"], r["nrl"], r["axis"], r["first"], r["last"], r["atoms"])
    mc = dict(rejrate=f32(0.75), ireset=0, ngrot=r["ngrot"], **{k: v.copy() for k, v in steps.items()})
    rot = dict(model=m, nrf=r["nrf"], nrl=r["nrl"], axis=r["axis"].reshape(-1), first=r["first"], last=r["last"],
               atoms=r["atoms"], stepri=f32(1.0))
    fb = torch.tensor([-0.25], dtype=torch.float32, device="cuda")
    ran1, fadds, faddbs = Ran1State(idum=-seed), f32(0.5), f32(-0.25)
    rejected = 0
    for _cycle in range(4):
        fadds, faddbs, nmovei, ninter, _, ran1, cosv = oracle.molfit_shake_rot(ob, ost, mc, rot, stepmi, ran1, fadds,
                                                                                faddbs)
        d.set_cos_override(cosv)
        got = model.molfit_shake(stepmi, fb).cpu().numpy()
        d.check_status()
        assert np.array_equal(got, nmovei)
        rejected += ninter[nmt:].sum()
        assert np.array_equal(d.m_ninter.cpu().numpy(), ninter)
        co, x = d.download_coords(), d.download_mc()
        for k in co:
            assert_bits_equal(co[k], getattr(ob, k), k)
        assert_bits_equal(d.download_store()["ergpair"], ost["ergpair"], "ergpair")
        for k in ("interntrans", "internrot"):
            assert_bits_equal(x[k], mc[k], k)
        assert np.array_equal(x["nstepreject"], mc["nstepreject"])
        assert_bits_equal(np.array([x["fadds"], fb.cpu().numpy()[0]], f32), np.array([fadds, faddbs], f32), "fadds")
        assert np.array_equal(x["ran1"].iv, ran1.iv) and x["ran1"].idum == ran1.idum
    assert rejected > 0

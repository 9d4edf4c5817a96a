"""Timed cases of the pair path: what a program that uses the package has it do, by kind of call.

* ``step``      one EPSR iteration of a box through ``EpsrIteration`` (native driver) with the
                device -> host copy of its results, as a refinement run makes it over and over:
                cell list, pair store, Monte Carlo cycles, g(r), S(Q), the fits, the refined
                potential, the running averages;
* ``cycles``    whole-molecule Monte Carlo cycles alone (``DeviceBox.molfit``), the fast form of
                an equilibration or the strict form whose sums are the reference's bit for bit;
* ``store``     the cell list, the pair-energy store and press of a box whose coordinates moved;
* ``structure`` g(r), S(Q), the data-set difference and g(r) back from S(Q) of one configuration;
* ``fit``       the empirical-potential coefficient fit on given differences;
* ``batch``     one sweep of many uneven boxes (water and SiO2-like) and their all-pairs g(r);
* ``learned``   delayed-acceptance sweeps with the surrogate network over several boxes;
* ``train``     one training step of that network.

The boxes have the compositions, densities, potentials and grids of ``configs`` (rigid water,
DMSO + water, SiO2-like); their molecules are put on a jittered lattice at random orientations
instead of by rejection, which gives a liquid-like start at any size in milliseconds.
"""

from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from epsr_python_translation_b200 import configs, transforms
from epsr_python_translation_b200.batch import BatchBoxes
from epsr_python_translation_b200.box import BoxArrays, Ran1State, trsteps
from epsr_python_translation_b200.device import DeviceBox
from epsr_python_translation_b200.iteration import EpsrIteration
from epsr_python_translation_b200.learned import LearnedMC
from epsr_python_translation_b200.surrogate import H, IN, SurrogateNet

f32 = np.float32


def listed():
    return [
        # the smallest box anyone refines (and the size of a first test run): all latency
        dict(name="step_water_100", kind="step", ndmso=0, nwater=100, sweeps=5, nq=600, ndata=3, intra=0, rotfreq=0),
        # the ordinary refinement: the reference's own example composition, three isotope data sets
        dict(name="step_mixture_600", kind="step", ndmso=200, nwater=400, sweeps=5, nq=600, ndata=3, intra=0,
             rotfreq=0),
        # the same with flexible molecules and rotating methyl groups, as the reference's example runs it
        dict(name="step_flexible_600", kind="step", ndmso=200, nwater=400, sweeps=5, nq=600, ndata=3, intra=5,
             rotfreq=2),
        # the largest refinement: 20,000 water, 100 sweeps between refinements, data to 50 1/A
        dict(name="step_water_20000", kind="step", ndmso=0, nwater=20000, sweeps=100, nq=1000, ndata=1, intra=0,
             rotfreq=0),
        # equilibration of a large mixture: Monte Carlo cycles only
        dict(name="cycles_mixture_8000", kind="cycles", ndmso=2700, nwater=5300, cycles=5, strict=False),
        # cycles whose sums follow the reference's order, for runs that must reproduce it
        dict(name="cycles_strict_777", kind="cycles", ndmso=259, nwater=518, cycles=1, strict=True),
        # a new configuration brought in: neighbour structures, pair energies, pressure
        dict(name="store_mixture_8000", kind="store", ndmso=2700, nwater=5300),
        # analysis of one large configuration over sampled origins
        dict(name="structure_mixture_8000", kind="structure", ndmso=2700, nwater=5300, nq=600, ndata=3),
        # a longer Q range than the example's, the reference's summation order
        dict(name="fit_strict_1000", kind="fit", nq=1000, nterms=97, sets=1, strict=True),
        # many boxes at once: sizes log-uniform in 300-30,000 atoms
        dict(name="batch_64", kind="batch", boxes=64, amin=300, amax=30000),
        # four 8,000-molecule mixtures with the learned first stage
        dict(name="learned_4x8000", kind="learned", boxes=4, ndmso=2700, nwater=5300, sweeps=2),
        # one optimiser step on a batch of move pairs, late in the learning-rate schedule
        dict(name="train_2048", kind="train", rows=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mixture(rng, lo, hi):
    """DMSO and water counts of a drawn box: about one to two, as the listed mixtures."""
    n = _log_int(rng, lo, hi)
    nd = max(2, int(round(n * rng.uniform(0.30, 0.36))))
    return nd, n - nd


def draw(rng):
    kind = rng.choice(["step", "step", "cycles", "cycles", "store", "structure", "fit", "batch", "learned", "train"])
    if kind == "step":
        nq = rng.randint(400, 1000)
        if rng.random() < 0.5:
            n = _log_int(rng, 100, 20000)
            return dict(kind=kind, ndmso=0, nwater=n, sweeps=_log_int(rng, 2, 40), nq=nq, ndata=rng.randint(1, 3),
                        intra=0, rotfreq=0)
        nd, nw = _mixture(rng, 150, 3000)
        flexible = rng.random() < 0.3 and nd + nw <= 900
        return dict(kind=kind, ndmso=nd, nwater=nw, sweeps=rng.randint(3, 12), nq=nq, ndata=rng.randint(1, 3),
                    intra=5 if flexible else 0, rotfreq=2 if flexible else 0)
    if kind == "cycles":
        if rng.random() < 0.25:
            nd, nw = _mixture(rng, 150, 1500)
            return dict(kind=kind, ndmso=nd, nwater=nw, cycles=1, strict=True)
        if rng.random() < 0.5:
            return dict(kind=kind, ndmso=0, nwater=_log_int(rng, 100, 20000), cycles=rng.randint(2, 8), strict=False)
        nd, nw = _mixture(rng, 150, 8000)
        return dict(kind=kind, ndmso=nd, nwater=nw, cycles=rng.randint(2, 8), strict=False)
    if kind in ("store", "structure"):
        nd, nw = (0, _log_int(rng, 100, 20000)) if rng.random() < 0.5 else _mixture(rng, 150, 8000)
        c = dict(kind=kind, ndmso=nd, nwater=nw)
        if kind == "structure":
            c.update(nq=rng.randint(400, 1000), ndata=rng.randint(1, 3))
        return c
    if kind == "fit":
        return dict(kind=kind, nq=rng.randint(300, 1000), nterms=rng.randint(40, 130), sets=rng.randint(1, 3),
                    strict=rng.random() < 0.5)
    if kind == "batch":
        amin = _log_int(rng, 300, 900)
        return dict(kind=kind, boxes=rng.randint(4, 48), amin=amin, amax=_log_int(rng, 4 * amin, 20000))
    if kind == "learned":
        nd, nw = _mixture(rng, 1500, 8000)
        return dict(kind=kind, boxes=rng.randint(1, 4), ndmso=nd, nwater=nw, sweeps=1)
    return dict(kind=kind, rows=128 * rng.randint(4, 32))


# ----------------------------------------------------------------------------- boxes
def _lattice(rng, n, counts):
    """Fractions in [0, 1) of ``counts`` sites a side n: cell corners for the first count, and
    for a second one the cell centres and then face centres (a CsCl-like packing)."""
    g = np.stack(np.meshgrid(*(np.arange(n),) * 3, indexing="ij"), axis=-1).reshape(-1, 3).astype(np.float64)
    out = [g[rng.permutation(n ** 3)[:counts[0]]]]
    if len(counts) > 1:
        centres = (g + 0.5)[rng.permutation(n ** 3)]
        faces = np.concatenate([g + 0.5 * (1 - np.eye(3)[k]) for k in range(3)])
        out.append(np.concatenate([centres, faces[rng.permutation(3 * n ** 3)]])[:counts[1]])
    return np.concatenate(out) / n


def _fill(base, templates, counts, frac, rng):
    """The box ``base`` (its potentials, grids and types) with counts[k] molecules of template k
    at the given fractional centres (small random displacements) and random orientations."""
    nmol = int(sum(counts))
    lab = base.type_labels
    L = base.L
    centres = frac + rng.uniform(-0.15, 0.15, size=(nmol, 3)) / L
    centres = centres - np.round(centres)
    q = rng.normal(size=(nmol, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    a, b, c, d = q.T
    rot = np.stack([a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c),
                    2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b),
                    2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d], axis=-1)
    rot = rot.reshape(nmol, 3, 3)
    offs, itype, m0 = [], [], 0
    for t, n in zip(templates, counts):
        offs.append(np.einsum("mij,aj->mai", rot[m0:m0 + n], t.pos).reshape(-1, 3))
        itype.append(np.tile([lab.index(x) for x in t.labels], n))
        m0 += n
    offs = (np.concatenate(offs) / L).astype(f32)
    centres = centres.astype(f32)
    itype = np.concatenate(itype).astype(np.int32)
    nato = np.concatenate([np.full(n, len(t.labels), np.int32) for t, n in zip(templates, counts)])
    mtype = np.concatenate([np.full(n, k, np.int32) for k, n in enumerate(counts)])
    naf = np.concatenate([[0], np.cumsum(nato)[:-1]]).astype(np.int32)
    natom = itype.shape[0]
    cfrac = np.array([f32(np.count_nonzero(itype == k)) / f32(natom) for k in range(len(lab))], f32)
    return dataclasses.replace(
        base, itype=itype, mtype=mtype, naf=naf, nato=nato, xa=offs[:, 0].copy(), ya=offs[:, 1].copy(),
        za=offs[:, 2].copy(), xadd=centres[:, 0].copy(), yadd=centres[:, 1].copy(), zadd=centres[:, 2].copy(),
        cfrac=cfrac)


def liquid(ndmso, nwater, seed, temperature=298.0, ep_coeffs=30):
    """Rigid water, or DMSO + water, at 0.1 atoms per cubic Angstrom."""
    rng = np.random.default_rng([seed, 17])
    L = ((10 * ndmso + 3 * nwater) / 0.1) ** (1.0 / 3.0)
    if ndmso:
        templates, counts = [configs.dmso_template(), configs.water_template()], [ndmso, nwater]
    else:
        templates, counts = [configs.water_template()], [nwater]
    n = int(math.ceil(counts[0] ** (1.0 / 3.0) - 1e-9))
    base = configs.build_system("liquid", templates, [1] * len(templates), L, temperature=temperature,
                                seed=seed % (1 << 31), min_heavy=1.0, ep_coeffs=ep_coeffs)
    return _fill(base, templates, counts, _lattice(rng, n, counts), rng)


def silica(natom, seed, temperature):
    """Single-atom Si and O molecules at 0.0662 atoms per cubic Angstrom."""
    rng = np.random.default_rng([seed, 19])
    L = (natom / 0.0662) ** (1.0 / 3.0)
    templates = [configs.atom_template("Si"), configs.atom_template("O")]
    counts = [natom // 3, natom - natom // 3]
    n = int(math.ceil(natom ** (1.0 / 3.0) - 1e-9))
    base = configs.build_system("silica", templates, [1, 1], L, temperature=temperature, seed=seed % (1 << 31),
                                min_heavy=1.0)
    return _fill(base, templates, counts, _lattice(rng, n, [natom]), rng)


def bond_energies(s, k_bond=1000.0):
    """Harmonic energy of every molecule's bonds (configs.intra_energies, over all at once)."""
    out = np.zeros(s.nmol)
    pos = np.stack([s.xa, s.ya, s.za], axis=-1).astype(np.float64) * float(s.dmax)
    for t, bonds in enumerate(s.bonds):
        m = np.nonzero(s.mtype == t)[0]
        for i, j, length in bonds:
            d = pos[s.naf[m] + i] - pos[s.naf[m] + j]
            out[m] += k_bond * (np.sqrt((d * d).sum(axis=1)) - abs(length)) ** 2
    return out.astype(f32)


def workload(case, seed):
    """One iteration's inputs on the box of ``case`` (configs.make_workload for any size)."""
    s = liquid(case["ndmso"], case["nwater"], seed)
    rng = np.random.default_rng([seed, 23])
    nq, ndata, nterms = case["nq"], case["ndata"], 116
    q = configs.qgrid(nq, 0.05)
    foqols, ycoh = configs.transform_table(s, q, s.grid["npt1"])
    ep = configs.ep_refinement(s, nterms, seed=seed % (1 << 31))
    expr = configs.pwrexpq_basis(q, nterms, ep.pdmin, ep.pdstep, ep.psigma2)
    w = rng.uniform(0.2, 1.0, size=(ndata, s.npairs))
    w /= w.sum(axis=1, keepdims=True)
    qq = q.astype(np.float64)[1:]
    data = np.zeros((ndata, nq + 1), f32)
    for d in range(ndata):
        data[d, 1:] = (0.05 * np.sin(2.9 * qq + d) * np.exp(-0.05 * qq) + rng.normal(0, 0.005, size=nq)).astype(f32)
    nmt = s.nmoltype
    return configs.Workload(
        name="liquid", system=s, eintra=bond_energies(s), q=q, foqols=foqols, ycoh=ycoh, expr=expr, nterms=nterms,
        data=data, weights=w, wholerot=np.full(nmt, f32(10.0 / 180.0), f32),
        wholetrans=np.full(nmt, f32(0.5) / s.dmax, f32), ntimes=case.get("sweeps", 1),
        xwt=np.linspace(0.5, 1.5, s.npairs).astype(f32), ep=ep, intra=case.get("intra", 0),
        rotfreq=case.get("rotfreq", 0),
        internrot=np.array([f32(0.05) if t.rot_groups else f32(0.0) for t in s.moltemplates], f32))


def _device_box(s, seed):
    """A box on the device with its neighbour structures, pair store and Monte Carlo state."""
    box = BoxArrays.from_system(s)
    d = DeviceBox(box)
    tmax, tmin = trsteps(box.natomr)
    d.mc_setup(rejrate=0.75, stepr=1.0, stepm=1.0, wholerot=np.full(s.nmoltype, f32(10.0 / 180.0), f32),
               wholetrans=np.full(s.nmoltype, f32(0.5) / s.dmax, f32), ran1=Ran1State(idum=-(seed % 100003) - 1),
               trstepmax=tmax, trstepmin=tmin)
    return d


def _screening_net(seed):
    """Network weights that screen overlaps as a trained network does: a few hidden units count
    the contacts below 1.6 A that a move makes and breaks, over a small random background."""
    rng = np.random.default_rng([seed, 29])
    w1 = rng.standard_normal((H, IN)) * (0.3 / math.sqrt(IN))
    w2 = rng.standard_normal((H, H)) * (0.3 / math.sqrt(H))
    w3 = rng.standard_normal(H) * (0.3 / math.sqrt(H))
    bins = np.arange(IN // 2) % 64
    close = np.where(bins < 13, (13.0 - bins) / 6.5, 0.0)       # 0.125 A a bin
    for u in range(4):
        w1[u, :IN // 2] = -close if u % 2 else close
        w1[u, IN // 2:] = close if u % 2 else -close
        w2[u] = 0.0
        w2[u, u] = 1.0
        w3[u] = 2.0 if u % 2 else -2.0
    return dict(w1=w1, b1=np.zeros(H), w2=w2, b2=np.zeros(H), w3=w3, b3=np.zeros(1))


# ----------------------------------------------------------------------------- prepare
def _prepare_step(case, seed):
    it = EpsrIteration(workload(case, seed), ran1_seed=-(seed % 100003) - 1, native=True)
    it.step()                       # sizes the native driver's buffers
    return dict(it=it)


def _prepare_cycles(case, seed):
    s = liquid(case["ndmso"], case["nwater"], seed)
    d = _device_box(s, seed)
    d.cell_list(10, d.host.sepmax)
    d.fmolec1(bond_energies(s), strict=case["strict"])
    return dict(d=d, cycles=case["cycles"], strict=case["strict"])


def _prepare_store(case, seed):
    s = liquid(case["ndmso"], case["nwater"], seed)
    return dict(d=_device_box(s, seed), eintra=torch.from_numpy(bond_energies(s)).cuda())


def _prepare_structure(case, seed):
    wl = workload(case, seed)
    d = _device_box(wl.system, seed)
    b = d.host
    t = lambda a, dt=f32: torch.from_numpy(np.ascontiguousarray(a, dt)).cuda()  # noqa: E731
    return dict(d=d, nq=wl.nq, rho=float(b.natom) / float(wl.system.L) ** 3, ran1=d.m_ran1,
                rminex=torch.full((b.npairs,), -2.0, device="cuda"), ycoh=t(wl.ycoh[:b.npt + 1]),
                foqols=t(wl.foqols), ns=torch.ones(b.ntype, device="cuda"), data=t(wl.data),
                weights=t(wl.weights, np.float64), q=t(wl.q), r=t(b.x[:b.npt1 + 1]),
                lo=torch.full((b.npairs,), 2, dtype=torch.int32, device="cuda"),
                hi=torch.full((b.npairs,), wl.nq, dtype=torch.int32, device="cuda"), xwt=t(wl.xwt))


def _prepare_fit(case, seed):
    rng = np.random.default_rng([seed, 31])
    nq, nterms, sets = case["nq"], case["nterms"], case["sets"]
    expr = configs.pwrexpq_basis(configs.qgrid(nq, 0.05), nterms, 1.0 + 0.1 / 9.0, 0.1, 0.01)
    E = expr[1:].reshape(nq, nterms).astype(np.float64)
    y = np.zeros((sets, nq + 1), f32)
    y[:, 1:] = (rng.uniform(-0.05, 0.05, size=(sets, nterms)) @ E.T + rng.normal(0, 0.005, size=(sets, nq))).astype(f32)
    st = np.zeros(35, np.int32)
    st[0] = -(seed % 100003) - 1
    return dict(y=torch.from_numpy(y).cuda(), expr=torch.from_numpy(expr).cuda(), nq=nq, nterms=nterms,
                wtold=torch.zeros(sets, nterms + 1, device="cuda"), step=np.full(sets, f32(0.01), f32),
                ran1=torch.from_numpy(st).cuda(), strict=case["strict"])


def _prepare_batch(case, seed):
    rng = np.random.default_rng([seed, 37])
    # the sizes are the case's, the same for every seed: evenly spread over the range's logarithm
    sizes = np.exp(np.linspace(math.log(case["amin"]), math.log(case["amax"]), case["boxes"]))
    temps = rng.uniform(298.0, 1500.0, case["boxes"])
    systems = []
    for k, (n, temp) in enumerate(zip(sizes, temps)):
        if k % 2 == 0:
            systems.append(liquid(0, max(4, int(round(n / 3.0))), seed + k, temperature=float(temp), ep_coeffs=0))
        else:
            systems.append(silica(max(12, int(round(n))), seed + k, float(temp)))
    bb = BatchBoxes(systems, seed=seed % 65536)
    bb.total_energy()
    return dict(bb=bb, graph=bb.capture("plain"))


def _prepare_learned(case, seed):
    systems = [liquid(case["ndmso"], case["nwater"], seed + k) for k in range(case["boxes"])]
    lm = LearnedMC(systems, seed=seed % 65536)
    lm.net = SurrogateNet(params=_screening_net(seed))
    lm.bb.capture("da", lm.net)
    return dict(lm=lm, sweeps=case["sweeps"])


def _features(seed, rows):
    """Rows of radial neighbour counts (a quarter each, as the features are scaled) and their
    orders exchanged, with targets of a few kT."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    mean = (torch.arange(IN // 2, device="cuda") % 64 + 0.5) ** 2 / 64.0 ** 2 * 6.0
    a = torch.poisson(mean.expand(rows // 2, -1), generator=g) * 0.25
    b = (a + torch.poisson(mean.expand(rows // 2, -1) * 0.1, generator=g) * 0.25)
    x = torch.stack([torch.cat([a, b], 1), torch.cat([b, a], 1)], 1).reshape(rows, IN).to(torch.bfloat16)
    t = (4.0 * torch.randn(rows // 2, generator=g, device="cuda")).clamp(-12.0, 12.0)
    return x, t


def _training_net(seed):
    """A network in mid-training: random weights and biases of a trained network's size."""
    rng = np.random.default_rng([seed, 41])
    return SurrogateNet(params=dict(w1=rng.standard_normal((H, IN)) / math.sqrt(IN), b1=0.1 * rng.standard_normal(H),
                                    w2=rng.standard_normal((H, H)) / math.sqrt(H), b2=0.1 * rng.standard_normal(H),
                                    w3=rng.standard_normal(H) / math.sqrt(H), b3=0.1 * rng.standard_normal(1)))


def _prepare_train(case, seed):
    x, t = _features(seed, case["rows"])
    net = _training_net(seed)
    return dict(net=net, x=x, xt=x.t().contiguous(), t=t, rows=case["rows"], loss=torch.zeros(1, device="cuda"))


# ----------------------------------------------------------------------------- run
def _run_step(s):
    it = s["it"]
    it.step()
    (co, wav, coeffs), _ = it.download_outputs()
    return dict(co, wav=wav, coeffs=coeffs, sofq=it.sofq, gofr=it.gofr, ftest=it.ftest, energy=it.energy,
                pressure=it.pressc, step=it.stepp, trials=it.fit_trials, pairs=it.pair_updates)


def _run_cycles(s):
    d = s["d"]
    for _ in range(s["cycles"]):
        d.molfit(strict=s["strict"])
    return dict(xa=d.xa, ya=d.ya, za=d.za, xadd=d.xadd, yadd=d.yadd, zadd=d.zadd, den=d.m_den, acc=d.m_acc,
                fadds=d.m_fadds, ran1=d.m_ran1, rot=d.m_wholerot, trans=d.m_wholetrans)


def _run_store(s):
    d = s["d"]
    d.cell_list(10, d.host.sepmax)
    ftest = d.fmolec1(s["eintra"], strict=False)
    press = d.press(strict=False)
    return dict(cells=d.c_mols, counts=d.s_nergpairm, n=d.s_n, ftest=ftest, press=press)


def _run_structure(s):
    d, nq = s["d"], s["nq"]
    b = d.host
    n = d.atogen(0, s["ran1"], s["rminex"], ycoh=s["ycoh"])
    sofq = transforms.gensq(nq, b.npt1, d.a_wav, b.npt + 1, s["foqols"], nq + 1, 1, s["ycoh"], d.n2extr, s["ns"],
                            b.npairs).view(2, b.npairs, nq + 1)
    diff = transforms.ptgnsq_difference(s["data"], s["weights"], sofq[1])
    gofr = transforms.stog(s["rho"], s["q"], sofq[1], s["r"], s["lo"], s["hi"], s["xwt"])
    return dict(wav=d.a_wav, potex=d.a_potex, sofq=sofq, diff=diff, gofr=gofr, n=n, pairs=d.last_pair_updates)


def _run_fit(s):
    r = transforms.fit_expansion_batch(s["y"], s["expr"], s["wtold"], s["step"], 1, s["nq"], 1, s["nterms"], 1000, 10,
                                       s["ran1"], strict=s["strict"])
    return dict(wt=r["wt"], wtold=r["wtold"], yout=r["yout"], stepr=r["stepr"], chisq=r["chisq"], trials=r["trials"],
                ran1=s["ran1"])


def _run_batch(s):
    bb = s["bb"]
    s["graph"].replay()
    bb.histograms()
    return dict(pos=bb.pos.view(-1, 4)[:, :3], xadd=bb.xadd, energy=bb.energy, counters=bb.counters,
                counts=bb.h_counts, wav=bb.h_wav, potex=bb.h_potex, pairs=bb.h_pairs)


def _run_learned(s):
    lm = s["lm"]
    energies, _, counters, _ = lm.run(s["sweeps"], "da")
    return dict(energies=energies, counters=counters, pos=lm.bb.pos.view(-1, 4)[:, :3], xadd=lm.bb.xadd)


def _run_train(s):
    net = s["net"]
    # the learning rate of the last of 24 epochs on a half cosine from 1e-3
    net.train_step(s["x"], s["xt"], 0, s["rows"], s["t"], 4.3e-6, loss=s["loss"])
    return dict(loss=s["loss"], w1=net.w1, b1=net.b1, w2=net.w2, b2=net.b2, w3=net.w3, b3=net.b3, m=net.m1, v=net.v1)


_PREPARE = dict(step=_prepare_step, cycles=_prepare_cycles, store=_prepare_store, structure=_prepare_structure,
                fit=_prepare_fit, batch=_prepare_batch, learned=_prepare_learned, train=_prepare_train)
_RUN = dict(step=_run_step, cycles=_run_cycles, store=_run_store, structure=_run_structure, fit=_run_fit,
            batch=_run_batch, learned=_run_learned, train=_run_train)


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return _RUN[state["kind"]](state)


# ----------------------------------------------------------------------------- work
PAIR_ENERGY = 26.0      # operations of one atom-pair energy
PAIR_UPDATE = 17.0      # operations of one binned distance


def _within(natom, L, rcut):
    """Atom pairs (ordered) closer than rcut, of natom atoms in a cube of side L."""
    return natom * (natom / L ** 3) * 4.0 / 3.0 * math.pi * min(rcut, 0.62 * L) ** 3


def _box_numbers(case):
    natom = 10 * case["ndmso"] + 3 * case["nwater"]
    return natom, case["ndmso"] + case["nwater"], (natom / 0.1) ** (1.0 / 3.0), 21 if case["ndmso"] else 3


def _structure_work(case):
    natom, nmol, L, npairs = _box_numbers(case)
    npt1 = L / 2.0 / 0.03
    origins = min(1000, nmol) / nmol * natom
    pairs = natom * natom / 2.0 if nmol <= 1000 else origins * natom
    flops = PAIR_UPDATE * pairs + 4.0 * npairs * npt1 * case["nq"] + 8.0 * npairs * npt1 * case["nq"]
    bytes_ = 16.0 * natom + 4.0 * (npt1 * case["nq"] + 4 * npairs * npt1 + 6 * npairs * case["nq"])
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind == "fit":
        trials = 1100.0 * case["sets"]
        return dict(bytes=4.0 * case["nq"] * (case["nterms"] + 2.0 * case["sets"]),
                    flops=2.0 * trials * case["nq"] * case["nterms"])
    if kind == "train":
        r = case["rows"]
        par = H * IN + H * H + 3 * H + 1
        return dict(bytes=2.0 * r * IN + 2.0 * r + 4.0 * par * 6, flops=2.0 * r * (2 * H * IN + 3 * H * H))
    if kind == "batch":
        sizes = np.exp(np.linspace(math.log(case["amin"]), math.log(case["amax"]), case["boxes"]))
        flops = bytes_ = 0.0
        for n in sizes:
            L = (n / 0.085) ** (1.0 / 3.0)
            flops += PAIR_UPDATE * n * n / 2.0 + 2.0 * PAIR_ENERGY * _within(n, L, 12.0)
            bytes_ += 64.0 * n + 3 * 8.0 * L / 0.03
        return dict(bytes=float(bytes_), flops=float(flops))
    natom, nmol, L, npairs = _box_numbers(case)
    near = _within(natom, L, 12.0)
    entries = nmol * (nmol / L ** 3) * 4.0 / 3.0 * math.pi * min(14.0, 0.62 * L) ** 3 / 2.0
    cycle = (32.0 * natom + 16.0 * entries, 2.0 * PAIR_ENERGY * near)
    if kind == "cycles":
        return dict(bytes=cycle[0] * case["cycles"], flops=cycle[1] * case["cycles"])
    if kind == "learned":
        feat = 12.0 * 2.0 * _within(natom, L, 8.0) + 2.0 * 2.0 * nmol * (IN * H + H * H)
        k = case["boxes"] * case["sweeps"]
        return dict(bytes=k * (64.0 * natom + 4.0 * nmol * IN), flops=k * (feat + 0.2 * cycle[1]))
    store = (32.0 * natom + 20.0 * entries, PAIR_ENERGY * near)
    if kind == "store":
        return dict(bytes=store[0] + 8.0 * entries, flops=store[1])
    sb, sf = _structure_work(case)
    if kind == "structure":
        return dict(bytes=sb, flops=sf)
    fits = 2.0 * 1100.0 * case["ndata"] * case["nq"] * 116
    return dict(bytes=store[0] + 8.0 * entries + case["sweeps"] * cycle[0] + sb,
                flops=store[1] + case["sweeps"] * cycle[1] + sf + fits)


# ----------------------------------------------------------------------------- exact
def _ran1(idum, n):
    """n values of the reference's ran1 (auxiliary_routines.py:324) from a negative seed."""
    d = max(-idum, 1)
    iv = [0] * 32
    for j in range(40, 0, -1):
        d = 16807 * d % 2147483647
        if j <= 32:
            iv[j - 1] = d
    iy, out = iv[0], np.zeros(n)
    for k in range(n):
        d = 16807 * d % 2147483647
        j = iy >> 26
        iy, iv[j] = iv[j], d
        out[k] = f32(f32(4.656612873077393e-10) * f32(iy))
    return out


def _exact_structure(case, seed):
    wl = workload(case, seed)
    s = wl.system
    nmol, natom, npairs, npt, npt1 = s.nmol, s.natom, s.npairs, s.grid["npt"], s.grid["npt1"]
    ld = npt + 1
    step = float(f32(s.cellst) / f32(s.dmax))
    dev = "cuda"
    T = lambda a, dt=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(dev, dt)  # noqa: E731
    ngr = min(1000, nmol)
    prob = ngr / nmol
    full = prob >= 1.0
    cand = np.arange(nmol - 1 if full else nmol)
    u = _ran1(-(seed % 100003) - 1, len(cand))
    frac = np.bincount(s.mtype, minlength=s.nmoltype) / nmol
    first = np.array([np.nonzero(s.mtype == t)[0][0] for t in range(s.nmoltype)])
    sel = cand[(u < f32(prob)) | (first[s.mtype[cand]] == cand) | (frac[s.mtype[cand]] < prob)]
    mol = np.repeat(np.arange(nmol), s.nato)
    counted = np.isin(mol, sel) | (full & (mol == nmol - 1))
    csam = np.bincount(s.itype[counted], minlength=s.ntype).astype(np.float64)
    pos = np.stack([s.xa, s.ya, s.za], -1).astype(f32)
    centre = np.stack([s.xadd, s.yadd, s.zadd], -1).astype(f32)
    absol = T((pos + centre[mol]).astype(f32))
    molt, typ, ref = T(mol, torch.int64), T(s.itype, torch.int64), T(s.npairref, torch.int64)
    counts = torch.zeros(2, npairs * ld, dtype=torch.float64, device=dev)

    def binned(part, ia, ja, d):
        z = torch.floor(d / step + 0.5).long() + 2
        ok = (z > 1) & (z <= npt1)
        at = ref[typ[ia], typ[ja]] * ld + z
        counts[part] += torch.bincount(at[ok], minlength=npairs * ld).double()

    off = T(pos)
    for t, tm in enumerate(s.moltemplates):
        a0 = T(s.naf[s.mtype == t], torch.int64)
        for i in range(len(tm.labels)):
            for j in range(i + 1, len(tm.labels)):
                x = off[a0 + i] - off[a0 + j]
                x = x - torch.round(x)
                binned(0, a0 + i, a0 + j, torch.sqrt((x * x).sum(-1)))
    origin = T(np.nonzero(np.isin(mol, sel))[0], torch.int64)
    for k in range(0, origin.numel(), 256):
        o = origin[k:k + 256]
        x = absol[o][:, None] - absol[None]
        x = x - torch.round(x)
        d = torch.sqrt((x * x).sum(-1))
        use = molt[None] > molt[o][:, None] if full else molt[None] != molt[o][:, None]
        ia, ja = torch.nonzero(use, as_tuple=True)
        binned(1, o[ia], ja, d[ia, ja])
    counts = counts.view(2, npairs, ld)
    n1, n2 = s.n1extr, s.n2extr
    cf = s.cfrac.astype(np.float64)
    same = n1 == n2
    cp1 = T(cf[n1] * cf[n2] * natom * np.where(same, 1.0, 2.0))
    cp2 = T(csam[n1] * cf[n2] + np.where(same, 0.0, csam[n2] * cf[n1]))
    ycoh = T(wl.ycoh[:ld])
    wav = torch.zeros(2, npairs, ld, dtype=torch.float64, device=dev)
    wav[0, :, 1:npt1 + 1] = 2.0 * counts[0, :, 1:npt1 + 1] / cp1[:, None]
    wav[1, :, 1:npt1 + 1] = (2.0 if full else 1.0) * counts[1, :, 1:npt1 + 1] / cp2[:, None]
    F = T(wl.foqols)[2:npt1 + 1]
    sofq = torch.stack([wav[0, :, 2:npt1 + 1] @ F, (wav[1, :, 2:npt1 + 1] - ycoh[2:npt1 + 1]) @ F])
    sofq[:, :, 0] = 0.0
    diff = T(wl.weights) @ sofq[1] - T(wl.data)
    q, r = T(wl.q), T(s.grid["x"][:npt1 + 1])
    qmax = math.pi / float(wl.q[wl.nq])
    x = qmax * q[2:]
    lorch = torch.where(x < math.pi, torch.sinc(x / math.pi), torch.zeros_like(x))
    sfac = 0.5 * float(f32(wl.q[4]) - f32(wl.q[3])) / math.pi ** 2 / float(f32(natom / s.L ** 3))
    rr = torch.clamp(r, min=1e-30)
    kern = torch.where(r[:, None] > 0, q[None, 2:] * torch.sin(q[None, 2:] * r[:, None]) / rr[:, None],
                       (q[2:] ** 2)[None].expand(r.numel(), -1))
    gofr = T(wl.xwt)[:, None] + sfac * (sofq[1][:, 2:] * lorch) @ kern.t()
    gofr[:, 0] = 0.0
    return dict(wav=wav.reshape(-1), potex=None, sofq=sofq, diff=diff, gofr=gofr, n=None, pairs=None)


def _exact_train(case, seed):
    x, t = _features(seed, case["rows"])
    net = _training_net(seed)
    p = {k: getattr(net, k).double() for k in ("w1", "b1", "w2", "b2", "w3", "b3")}
    half = lambda w: w.to(torch.bfloat16).double()  # noqa: E731
    x, t = x.double(), t.double()
    leaf = {k: (half(v) if k in ("w1", "w2") else v.clone()).requires_grad_() for k, v in p.items()}
    silu = torch.nn.functional.silu
    y = silu(silu(x @ leaf["w1"].t() + leaf["b1"]) @ leaf["w2"].t() + leaf["b2"]) @ leaf["w3"] + leaf["b3"]
    sq = (0.5 * (y[0::2] - y[1::2]) - t) ** 2
    # the step's gradient is that of half the mean squared pair error, counted once per row
    sq.mean().backward()
    out = dict(loss=sq.detach().sum().reshape(1))
    m, v = [], []
    for k in ("w1", "b1", "w2", "b2", "w3", "b3"):
        g = leaf[k].grad
        out[k] = p[k] - 4.3e-6 * g / (g.abs() + 1e-8)
        m.append(0.1 * g.reshape(-1))
        v.append(0.001 * (g * g).reshape(-1))
    return dict(out, m=torch.cat(m), v=torch.cat(v))


def exact(case, seed):
    if case["kind"] == "structure":
        return _exact_structure(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None

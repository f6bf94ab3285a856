"""Result processing's kernels at the sizes where they can go wrong: ordering
with and without NaN energies, RMSDs and clusters over one word of runs and
one more, the largest count that takes the RMSDs of all pairs and the first
that does not, and re-scored energies with and without flexible residues.

The RMSDs and clusters are checked against a plain restatement of
generate_output's greedy clustering (host/src/processresult.cpp:688-746) on
the returned poses."""
import ctypes as C
import math
import threading

import numpy as np
import pytest
import torch

from adgpu_b200 import device, frontend, result, synth

pytestmark = pytest.mark.gpu


def inputs(runs, pop, flex=False, seed=3, calm=False):
    spec = synth.grid_spec(88, synth.MAP_TYPES_5, seed=77)
    maps = synth.quantize_maps(synth.make_maps_fast(spec))
    grid = frontend.Grid.from_maps(maps, synth.MAP_TYPES_5, spec.spacing, spec.origin)
    text = "\n".join(synth.pdbqt_lines(synth.ligand_for(2, 7, 14, 3))[0]) + "\n"
    fr = synth.flexres_text([synth.make_flexres(100, 8, 2, anchor=np.array([-6.5, 4.5, 0.0]))]) if flex else None
    lig = frontend.Ligand(grid, text, fr, run=frontend.default_dockpars(grid.spacing, pop), num_runs=runs)
    rng = np.random.default_rng(seed)
    ng = lig.dockpars.num_of_genes
    base = rng.uniform(-180.0, 180.0, (4, 64)).astype(np.float32)
    base[:, :3] = 44.0 + rng.normal(0.0, 2.0, (4, 3))
    if calm:                                        # torsions near the input conformer's: few clashes
        base[:, 6:] = 0.0
        base[:, :3] = 44.0
    pops = base[np.arange(runs) % 4].repeat(pop, axis=0)
    pops[:, :ng] += rng.normal(0.0, 1.0, (runs * pop, ng)).astype(np.float32) * np.where(np.arange(ng) < 3, 0.8, 15.0)
    pops[:, ng:] = 0.0
    return grid, lig, pops.astype(np.float32), rng.normal(-5.0, 2.0, runs * pop).astype(np.float32)


def stable_order(e):
    """Stable ascending order inside the NaN-free stretches."""
    perm, s, nan = np.arange(len(e)), 0, np.isnan(e)
    while s < len(e):
        t = s
        while t < len(e) and not nan[t]:
            t += 1
        perm[s:t] = s + np.argsort(e[s:t], kind="stable")
        s = max(t, s + 1)
    return perm


def rmsd(x, y, types):
    d2 = ((x[:, None] - y[None]) ** 2).sum(2)
    d2[types[:, None] != types[None]] = 1e9
    return np.sqrt(np.minimum(d2.min(1), 100000.0).mean())


@pytest.mark.parametrize("runs,nans", [(1, False), (2, False), (32, True), (33, False), (100, True), (1024, False), (1025, False)])
def test_order_and_clusters(runs, nans):
    pop = 5
    grid, lig, pops, en = inputs(runs, pop)
    if nans:
        en[[3, pop + 2, 7 * pop]] = np.nan
    en[2] = en[4]
    dev, de = torch.from_numpy(pops).cuda(), torch.from_numpy(en).cuda()
    out = result.process_result(lig, torch.from_numpy(grid.reference_layout()).cuda(), dev, de, runs)
    perm = np.concatenate([r * pop + stable_order(en[r * pop:(r + 1) * pop]) for r in range(runs)])
    np.testing.assert_array_equal(dev.cpu().numpy(), pops[perm])
    np.testing.assert_array_equal(de.cpu().numpy(), en[perm])
    n = lig.dockpars.true_ligand_atoms
    off = 256 * 4                                   # kernelconstant_interintra: charges, then types
    types = np.frombuffer(bytes(lig.tables["interintra"]), np.uint32)[off // 4:off // 4 + n].astype(int)
    key = np.array([r.inter_e + r.interflex_e for r in out.runs], np.float32)
    order = stable_order(key)
    assert [out.runs[r].energy_rank for r in order] == list(range(runs))
    xyz, centres, ids = out.best_xyz[:, :n], [], np.zeros(runs, int)
    for r in order:
        d = [rmsd(xyz[r], xyz[c], types) for c in centres]
        assert not any(abs(v - 2.0) < 1e-9 for v in d)
        hit = next((k for k, v in enumerate(d) if v <= 2.0), None)
        if hit is None:
            centres.append(r)
            hit, d = len(centres) - 1, d + [0.0]
        ids[r] = hit + 1
        assert out.runs[r].rmsd_from_cluster_center == pytest.approx(d[hit], abs=1e-6)
    assert [r.cluster_id for r in out.runs] == ids.tolist()
    assert [c.size for c in out.clusters] == np.bincount(ids)[1:].tolist()
    assert runs < 8 or 1 < len(centres) < runs


@pytest.mark.parametrize("flex", [False, True])
def test_rescored_energies(flex):
    """Every entity's energies against the scorer's terms: the distance tables
    round r to 0.01 A, so a term of r^-12 at 1 A or more is off by at most
    12 * 0.005 = 6 % (vdW energies below 1e6: the pairs' r^-12 coefficients are
    near 1e6 kcal/mol A^12)."""
    runs, pop = 3, 40
    grid, lig, pops, en = inputs(runs, pop, flex, calm=True)
    layout = grid.reference_layout()
    job = device.DeviceJob(lig.tables, lig.dockpars, layout, runs, lig.prng)
    job.activate()
    dev, de = torch.from_numpy(pops).cuda(), torch.from_numpy(en).cuda()
    out = result.process_result(lig, job.grid, dev, de, runs, result.default_params(rescore_entities=1))
    _, t = device.score_terms(dev.cpu().numpy())
    inside = (t[:, 7] == 0) & (t[:, 3] < 1e6)       # all atoms in the box
    assert inside.sum() > 10
    # (the split of the terms into inter and intra follows flexible residues; their sum does not)
    got = out.entities.reshape(-1, 3)[:, :2].sum(1)
    want, size = t[:, :6].sum(1), np.abs(t[:, :6]).sum(1)
    assert (np.abs(got - want) <= 0.06 * size + 0.02)[inside].all()
    best = np.array([[r.inter_e, r.interflex_e, r.intra_e, r.intraflex_e] for r in out.runs])
    np.testing.assert_allclose(best.sum(1), out.entities[:, 0, :2].sum(1), rtol=1e-6)


def test_populations_aligned_to_a_float():
    """Populations anywhere a float may lie: ordered as 16-byte aligned ones."""
    runs, pop = 3, 7
    grid, lig, pops, en = inputs(runs, pop)
    layout = torch.from_numpy(grid.reference_layout()).cuda()
    for off in (0, 1, 2):
        dev = torch.zeros(pops.size + off, device="cuda")[off:].view(pops.shape)
        assert dev.data_ptr() % 16 == 4 * off
        dev.copy_(torch.from_numpy(pops))
        de = torch.zeros(en.size + off, device="cuda")[off:]
        de.copy_(torch.from_numpy(en))
        result.process_result(lig, layout, dev, de, runs)
        perm = np.concatenate([r * pop + stable_order(en[r * pop:(r + 1) * pop]) for r in range(runs)])
        np.testing.assert_array_equal(dev.cpu().numpy(), pops[perm])
        np.testing.assert_array_equal(de.cpu().numpy(), en[perm])


def test_calls_of_several_threads():
    """Calls of different run counts at the same time: the clustering's shared
    memory grows with the runs (66 KB at 720, 128 KB at 1,024)."""
    pop, sizes, errors, labels = 2, (720, 1024), [], {}
    jobs = {}
    for runs in sizes:
        grid, lig, pops, en = inputs(runs, pop)
        jobs[runs] = (lig, torch.from_numpy(grid.reference_layout()).cuda(), torch.from_numpy(pops).cuda(), torch.from_numpy(en).cuda())
        out = result.process_result(*jobs[runs], runs)
        labels[runs] = [r.cluster_id for r in out.runs]
    start = threading.Barrier(4)

    def worker(runs):
        lig, layout, pops, en = jobs[runs][0], *[t.clone() for t in jobs[runs][1:]]
        torch.cuda.synchronize()
        start.wait()
        try:
            for _ in range(25):
                assert [r.cluster_id for r in result.process_result(lig, layout, pops, en, runs).runs] == labels[runs]
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=worker, args=(r,)) for r in sizes * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def pair_sums(xyz, pairs, charges, dp, nlig):
    """calc_intraE_f (host/src/processligand.cpp:2058-2331) for carbon atoms:
    intramolecular and ligand-flexres energy, every operation in the host
    code's type and the float sums in the pairs' order."""
    m = C.CDLL("libm.so.6")
    for f in (m.powf, m.expf):
        f.restype, f.argtypes = C.c_float, [C.c_float] * (2 if f is m.powf else 1)
    f4, ld = np.float32, np.longdouble
    dist, r12, r6, elec, desolv = f4(0), [], [], [], []
    lam, eps0, A, rk = (np.float64(ld(x)) for x in ("0.003627", "78.4", "-8.5525", "7.7839"))
    B, sigma = eps0 - A, f4(3.6)
    for _ in range(2048):
        dist = f4(np.float64(dist) + 0.01)
        r6.append(f4(1) / f4(m.powf(dist, 6)))
        r12.append(f4(1) / f4(m.powf(dist, 12)))
        eps = np.float64(ld(A) + ld(B) / (ld(1) + ld(rk * math.exp(-lam * B * np.float64(dist)))))
        elec.append(f4(np.float64(f4(dp.coeff_elec)) / (np.float64(dist) * eps)))
        desolv.append(f4(dp.coeff_desolv) * f4(m.expf(f4(-1) * dist * dist / (f4(2) * sigma * sigma))))
    eps12 = 0.1662 * math.sqrt(0.150 * 0.150)
    vA, vB, opt, delta = eps12 * 4.0 ** 12, 2 * eps12 * 4.0 ** 6, f4(4.0), f4(0.5) * f4(dp.smooth)
    s = [f4(-0.00143 + np.float64(f4(np.float64(f4(dp.qasp)) * abs(q)))) for q in charges]
    w = f4(33.5103)
    bin_of = lambda d: max(0, int(np.floor(f4(f4(100) * d) + f4(0.5))) - 1)  # noqa: E731
    terms = []                                       # (ligand-flexres, vdW, elec, desolv) in the pairs' order
    for i, j in pairs:
        d = f4(math.sqrt(((xyz[i] - xyz[j]) ** 2).sum()))
        vdw = a = b = f4(0)
        if d < f4(8):
            sd = d + delta if d <= opt - delta else (opt if d < opt + delta else d - delta)
            vdw = f4(vA * np.float64(r12[bin_of(sd)])) - f4(vB * np.float64(r6[bin_of(sd)]))
        if np.float64(d) < 20.48:
            assert d > f4(dp.elec_min_distance)
            a = f4(np.float64(f4(charges[i])) * charges[j]) * elec[bin_of(d)]
            b = (s[i] * w + s[j] * w) * desolv[bin_of(d)]
        terms.append(((i >= nlig) != (j >= nlig), vdw, a, b))

    def sums(order):
        vw = el = ds = inter = f4(0)
        for flex, vdw, a, b in order:
            if flex:
                inter = inter + vdw
                inter = inter + (a + b)
            else:
                vw, el, ds = vw + vdw, el + a, ds + b
        return vw + el + ds, inter

    return sums(terms), sums(terms[::-1])


def test_sums_in_the_pairs_order():
    """The re-scored sums are the host's float sums bit for bit (a ligand and a
    flexible residue of carbon atoms); in another order they would not be."""
    runs, pop = 24, 3
    spec = synth.grid_spec(40, synth.MAP_TYPES_5, seed=77)
    grid = frontend.Grid.from_maps(synth.quantize_maps(synth.make_maps_fast(spec)), synth.MAP_TYPES_5, spec.spacing, spec.origin)

    def carbon(lines):
        return [x[:77] + "C" if x.startswith(("ATOM", "HETATM")) else x for x in lines]

    lig_lines = carbon(synth.pdbqt_lines(synth.ligand_for(2, 5, 24, 5))[0])
    flex_lines = carbon(synth.flexres_text([synth.make_flexres(100, 8, 2, anchor=np.array([-4.0, 3.0, 0.0]))]).splitlines())
    lig = frontend.Ligand(grid, "\n".join(lig_lines) + "\n", "\n".join(flex_lines) + "\n",
                          run=frontend.default_dockpars(grid.spacing, pop), num_runs=runs)
    dp = lig.dockpars
    charges = [float(x[70:76]) for x in lig_lines + flex_lines if x.startswith(("ATOM", "HETATM"))]
    assert len(charges) == dp.num_of_atoms > dp.true_ligand_atoms
    pairs = np.frombuffer(bytes(lig.tables["intracontrib"]), np.uint32)[:2 * dp.num_of_intraE_contributors].reshape(-1, 2).astype(int)
    pops = torch.from_numpy(lig.initpop.copy()).cuda()
    en = torch.zeros(runs * pop, device="cuda")
    out = result.process_result(lig, torch.from_numpy(grid.reference_layout()).cuda(), pops, en, runs)
    other = 0
    for r in range(runs):
        want, reverse = pair_sums(out.best_xyz[r], pairs, charges, dp, dp.true_ligand_atoms)
        # (of the poses' coordinates, best_xyz's rounding is in the last bit of a double)
        assert (out.runs[r].intra_e, out.runs[r].interflex_e) == tuple(float(x) for x in want), r
        other += want != reverse
    assert other > runs // 2
    # the ligand's electrostatic map energy from its atoms' own, in their order (atoms outside the box add none)
    for r in range(runs):
        e = out.peratom[r, :dp.true_ligand_atoms, 1]
        assert out.runs[r].inter_e_elec == np.cumsum(np.where(e == 100000.0, np.float32(0), e), dtype=np.float32)[-1], r

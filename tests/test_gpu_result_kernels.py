"""Result processing's kernels at the sizes where they can go wrong: ordering
with and without NaN energies, RMSDs and clusters over one word of runs and
one more, the largest count that takes the RMSDs of all pairs and the first
that does not, and re-scored energies with and without flexible residues.

The RMSDs and clusters are checked against a plain restatement of
generate_output's greedy clustering (host/src/processresult.cpp:688-746) on
the returned poses."""
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

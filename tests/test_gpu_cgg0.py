"""Ligands with CG-G0 pairs (flexible rings: a bond energy of 50 kcal/mol/A
that holds an opened ring's ends together), which have kernels of their own:
scores against the oracle, and the docking loops and the engine against each
other."""
import numpy as np
import pytest
import torch

from adgpu_b200 import device, dock, engine, frontend, synth
from oracle import oraclepy

pytestmark = pytest.mark.gpu

RUNS, POP = 3, 40


def ring_text(heavy, tors):
    """A synthetic ligand two of whose atoms, in different fragments, are a ring's ends."""
    lines = synth.pdbqt_lines(synth.ligand_for(2, heavy, heavy, tors))[0]
    atoms = [k for k, x in enumerate(lines) if x.startswith(("ATOM", "HETATM"))]
    carbons = [k for k in atoms if lines[k][77:].strip() in ("C", "A")]
    for k, t in ((carbons[0], "CG0"), (carbons[-1], "G0")):
        lines[k] = lines[k][:77] + t
    return "\n".join(lines) + "\n"


@pytest.fixture(scope="module")
def grid():
    spec = synth.grid_spec(40, synth.MAP_TYPES_5, seed=41)
    maps = synth.quantize_maps(synth.make_maps_fast(spec))
    maps["CG0"] = maps["C"]
    return frontend.Grid.from_maps(maps, synth.MAP_TYPES_5 + ["CG0"], spec.spacing, spec.origin)


def prepared(grid, heavy, tors):
    return frontend.Ligand(grid, ring_text(heavy, tors), run=frontend.default_dockpars(grid.spacing, POP), num_runs=RUNS)


def job(grid, lig):
    j = device.DeviceJob(lig.tables, lig.dockpars, grid.reference_layout(), RUNS, lig.prng)
    j.activate()
    return j


# one warp of atoms, and more than the 64 of which 128 threads split a pose
@pytest.mark.parametrize("heavy,tors", [(16, 4), (64, 12)])
@pytest.mark.parametrize("tpp", [0, 32, 64, 128])
def test_scores(grid, heavy, tors, tpp, monkeypatch):
    monkeypatch.setenv("ADGPU_THREADS_PER_POSE", str(tpp))
    lig = prepared(grid, heavy, tors)
    g = lig.initpop.copy()
    g[:, :3] = 20.0 + 0.3 * (g[:, :3] - 20.0)
    host = oraclepy.HostTables(lig.tables, lig.dockpars, grid.reference_layout())
    e_ref, g_ref = host.score(g, True)
    terms = np.array([host.score_terms(x)[2] for x in g])
    assert (terms[:, 6] > 0).all()
    job(grid, lig)
    e, gr = device.score(g, True)
    t = device.score_terms(g)[1]
    # 1e-4 and, for cancellation, 1e-6 of the summed terms; gradients: one
    # quantum (1/1024, genes >= 3 scaled) a quantised term, which the
    # orientation genes take through a step of 1e-3 rad (tests/helpers.py)
    tol = 1e-4 * np.abs(e_ref) + 1e-6 * (np.abs(terms[:, :7]).sum(1) + 16777216.0 * terms[:, 7])
    assert (np.abs(e - e_ref) <= tol).all() and (np.abs(device.score(g, False) - e_ref) <= tol).all()
    np.testing.assert_allclose(t[:, 6], terms[:, 6], rtol=1e-4)
    dp = lig.dockpars
    bound = np.where(np.arange(64) < 3, 1.0, (grid.spacing / 0.0174533) ** 2) * (dp.num_of_atoms + 2 * dp.num_of_intraE_contributors) / 1024
    bound[3:6] *= 8e3 / 1024
    assert (np.abs(gr - g_ref)[:, :dp.num_of_genes] <= (1e-4 * np.abs(g_ref) + bound)[:, :dp.num_of_genes]).all()


@pytest.mark.parametrize("search", ["sw", "ad", "adam", "fire"])
def test_docking_loops_agree(grid, search, monkeypatch):
    lig, out = prepared(grid, 24, 6), []
    monkeypatch.setenv("ADGPU_THREADS_PER_POSE", "64")
    for arm in (dock.dock, dock.dock_host_loop):
        j = job(grid, lig)
        out.append(arm(j, lig.initpop, search, nev=4000))
    assert dock.last_stats()["pipelined"] == 1       # the first arm's (the host loop has none)
    for k in ("conformations", "energies", "evals_per_run"):
        a, b = (np.asarray(getattr(x, k).cpu() if isinstance(getattr(x, k), torch.Tensor) else getattr(x, k)) for x in out)
        np.testing.assert_array_equal(a, b)
    # AutoStop: the synchronous loop, until the budget
    j = job(grid, lig)
    r = dock.dock(j, lig.initpop, search, 4000, autostop=dock.AutoStopParams(100, 0.01, 1 << 40))
    assert dock.last_stats()["pipelined"] == 0
    np.testing.assert_array_equal(r.energies.cpu().numpy(), out[0].energies.cpu().numpy())


def test_engine_beside_other_ligands(grid):
    """A ring ligand's request makes the tick's kernel the one for CG-G0 pairs:
    the other ligands' results do not change with it."""
    plain = [frontend.Ligand(grid, "\n".join(synth.pdbqt_lines(synth.ligand_for(2, 3, h, t))[0]) + "\n",
                             run=frontend.default_dockpars(grid.spacing, POP), num_runs=RUNS) for h, t in ((12, 2), (30, 7))]
    ring = prepared(grid, 24, 6)

    def dock_all(ligands):
        eng = engine.Engine()
        rec = eng.add_receptor(grid)
        ids = [eng.submit(x, rec, "ad", 4000) for x in ligands]
        eng.run()
        return [eng.result(i) for i in ids]

    mixed, alone, rings = dock_all([ring] + plain), dock_all(plain), dock_all([ring])
    for a, b in zip(mixed, rings + alone):
        np.testing.assert_array_equal(a.best_energies, b.best_energies)
        np.testing.assert_array_equal(a.best_genotypes, b.best_genotypes)
        np.testing.assert_array_equal(a.evals, b.evals)

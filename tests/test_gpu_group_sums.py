"""Paths that deal a pose out differently must give the same bits: 128 threads
per pose with the sums of 64 (small launches with gradients, dockings with
AutoStop), the split of a pose's work among 128 threads, and the pipelined
loop with AutoStop against the synchronous one."""
import numpy as np
import pytest

from adgpu_b200 import device, dock, frontend, lib, synth

pytestmark = pytest.mark.gpu

# (heavy atoms, torsions, flexible residues): rigid and without pairs, one warp
# of atoms, more than one, and more than the 64 that share sums
LIGANDS = [(3, 0, 0), (16, 4, 0), (32, 8, 0), (40, 10, 1), (64, 20, 0)]


@pytest.fixture(scope="module")
def grid():
    spec = synth.grid_spec(40, synth.MAP_TYPES_5, seed=41)
    maps = synth.quantize_maps(synth.make_maps_fast(spec))
    g = frontend.Grid.from_maps(maps, synth.MAP_TYPES_5, spec.spacing, spec.origin)
    return g, g.reference_layout()


def job(grid, heavy, tors, flex, runs, monkeypatch, tpp=0, pipeline=True):
    text = "\n".join(synth.pdbqt_lines(synth.ligand_for(2, heavy, heavy, tors))[0]) + "\n"
    fr = synth.flexres_text([synth.make_flexres(100 + k, 8, 2, anchor=np.array([-4.0, 3.0, 0.0])) for k in range(flex)])
    lig = frontend.Ligand(grid[0], text, fr if flex else None, num_runs=runs)
    monkeypatch.setenv("ADGPU_THREADS_PER_POSE", str(tpp))
    monkeypatch.setenv("ADGPU_DOCK_PIPELINE", "1" if pipeline else "0")
    j = device.DeviceJob(lig.tables, lig.dockpars, grid[1], runs, lig.prng)
    j.activate()
    return j, lig


@pytest.mark.parametrize("heavy,tors,flex", LIGANDS)
@pytest.mark.parametrize("n", [1, 150, 592, 593, 740, 741])
def test_scores_of_small_launches(grid, heavy, tors, flex, n, monkeypatch):
    out = []
    for tpp in (0, 64):
        _, lig = job(grid, heavy, tors, flex, 5, monkeypatch, tpp)
        g = lig.initpop[:n].copy()
        g[:, :3] = 20.0 + 0.3 * (g[:, :3] - 20.0)
        out.append(device.score(g, True))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("entry", ["adgpu_gradient_minad", "adgpu_gradient_minadam", "adgpu_gradient_minfire"])
@pytest.mark.parametrize("heavy,tors,flex", LIGANDS[1:])
def test_searches_of_small_launches(grid, heavy, tors, flex, entry, monkeypatch):
    out = []
    for tpp in (0, 64):
        j, lig = job(grid, heavy, tors, flex, 1, monkeypatch, tpp)
        c, e = j.population(lig.initpop)
        lib.call("adgpu_calc_initpop", 150, 64, c, e)
        lib.call(entry, 150, 64, c, e)
        out.append((c.cpu().numpy(), e.cpu().numpy(), j.evals_new.cpu().numpy(), j.prng.cpu().numpy()))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("search,runs,heavy,tors,flex", [
    ("ad", 1, 16, 4, 0), ("ad", 5, 32, 8, 0), ("ad", 13, 40, 10, 1), ("ad", 26, 16, 4, 0), ("ad", 5, 64, 20, 0),
    ("sw", 5, 16, 4, 0), ("sw", 13, 32, 8, 0), ("adam", 2, 16, 4, 0), ("adam", 21, 16, 4, 0), ("fire", 2, 16, 4, 0)])
def test_autostop_pipelined_matches_synchronous(grid, search, runs, heavy, tors, flex, monkeypatch):
    """A budget that ends the docking, and a tolerance wide enough for AutoStop
    to end it.  The random states and the evaluation counters are part of the
    result: a docking that goes on from them must not depend on what was run
    ahead of the stop."""
    pipelines = search != "fire"                     # (which runs the same loop twice)
    for nev, stopstd in ((60_000, 0.15), (3_000_000, 3.0)):
        out = []
        for pipeline in (True, False):
            j, lig = job(grid, heavy, tors, flex, runs, monkeypatch, 0, pipeline)
            r = dock.dock(j, lig.initpop, search, nev, autostop=dock.AutoStopParams(2, stopstd, 0))
            assert dock.last_stats()["pipelined"] == (pipeline and pipelines)
            out.append((r.generations, r.autostopped, r.evals_per_run, r.energies.cpu().numpy(), r.conformations.cpu().numpy(),
                        j.prng.cpu().numpy(), j.evals_new.cpu().numpy()))
        assert out[0][:2] == out[1][:2]
        assert out[0][1] or nev == 60_000
        for a, b in zip(out[0][2:], out[1][2:]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("heavy,tors,flex", LIGANDS[1:])
def test_128_threads_match_host_loop(grid, heavy, tors, flex, monkeypatch):
    """The early end of discarded searches leaves a docking's results as they
    are, in a docking of few generations."""
    for search in ("sw", "fire"):
        out = []
        for arm in (dock.dock, dock.dock_host_loop):
            j, lig = job(grid, heavy, tors, flex, 3, monkeypatch, 128)
            r = arm(j, lig.initpop, search, 100_000)
            out.append((r.generations, r.evals_per_run, r.energies.cpu().numpy(), r.conformations.cpu().numpy()))
        assert out[0][0] == out[1][0]
        for a, b in zip(out[0][1:], out[1][1:]):
            np.testing.assert_array_equal(a, b)


def test_discarded_evaluations_are_counted(grid, monkeypatch):
    """evals_executed holds every evaluation executed, those of searches that
    end early because their generation is discarded among them.  Kept ADAM
    searches make 300, discarded ones at least the 32 to the first look at the
    stop."""
    runs = 3
    j, lig = job(grid, 32, 8, 0, runs, monkeypatch, 128)
    r = dock.dock(j, lig.initpop, "adam", nev=200_000)
    st = dock.last_stats()
    new = j.evals_new.cpu().numpy()[:runs * lig.dockpars.pop_size]
    early = new[new < 300]
    assert st["generations_discarded"] >= 1 and len(early) > 0
    assert early.min() >= 32
    kept = r.evals_per_run.sum() - runs * lig.dockpars.pop_size
    assert st["evals_executed"] >= kept + early.sum()

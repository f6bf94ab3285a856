"""Poses with a NaN or infinite gene against the oracle: a pair at a NaN
distance makes the energy NaN, and a force component that is NaN is clamped to
8 kcal/mol/A in size like a large one, whatever a warp scores beside it."""
import ctypes as C

import numpy as np
import pytest
import torch

from adgpu_b200 import device, frontend, lib, synth
from oracle import oraclepy

pytestmark = pytest.mark.gpu

NAN, INF = np.nan, np.inf
# (gene, value): translation, orientation, torsion
GENES = [(0, INF), (1, -INF), (2, NAN), (0, 200.0), (4, INF), (5, NAN), (6, NAN), (7, INF)]


def poses(flex):
    """The prepared job, the genotypes (every third with a gene of GENES) and the oracle's scores."""
    spec = synth.grid_spec(40, synth.MAP_TYPES_5, seed=41)
    grid = frontend.Grid.from_maps(synth.quantize_maps(synth.make_maps_fast(spec)), synth.MAP_TYPES_5, spec.spacing, spec.origin)
    text = "\n".join(synth.pdbqt_lines(synth.ligand_for(2, 5, 24, 5))[0]) + "\n"
    fr = synth.flexres_text([synth.make_flexres(100, 8, 2, anchor=np.array([-4.0, 3.0, 0.0]))]) if flex else None
    lig = frontend.Ligand(grid, text, fr, num_runs=2)
    layout, dp = grid.reference_layout(), lig.dockpars
    g = lig.initpop[:3 * len(GENES)].copy()
    g[:, :3] = 20.0 + 0.3 * (g[:, :3] - 20.0)
    for k, (gene, value) in enumerate(GENES):
        g[3 * k, gene] = value                       # between finite poses
    want = oraclepy.HostTables(lig.tables, dp, layout).score(g, True)
    return device.DeviceJob(lig.tables, dp, layout, 2, lig.prng), g, want


def check(job, flex, e, gr, e_only, want_e, want_g):
    nan = np.isnan(want_e)
    assert 0 < nan.sum() < len(GENES)
    np.testing.assert_array_equal(np.isnan(e), nan)
    np.testing.assert_array_equal(np.isnan(e_only), nan)
    # finite poses: 1e-4 of the energy
    assert np.all(np.abs(e - want_e)[~nan] <= 1e-4 * np.abs(want_e[~nan]) + 0.1)
    # Translation genes: 1e-4 and one quantum (1/1024) a quantised term.  (The
    # sign of a NaN component follows which of its pair's atoms is taken first,
    # and a couple takes its shared atom first: torsion genes show that, the
    # total force over the ligand's pairs does not.)
    if not flex:
        bound = 1e-4 * np.abs(want_g[:, :3]) + (job.dp.num_of_atoms + 2 * job.dp.num_of_intraE_contributors) / 1024.0
        assert np.all((np.abs(gr - want_g)[:, :3] <= bound)[3 * np.arange(len(GENES))])


@pytest.mark.parametrize("flex", [0, 1])
@pytest.mark.parametrize("tpp", [0, 32, 64, 128])
def test_scores(tpp, flex, monkeypatch):
    job, g, want = poses(flex)
    monkeypatch.setenv("ADGPU_THREADS_PER_POSE", str(tpp))
    job.activate()
    check(job, flex, *device.score(g, True), device.score(g, False), *want)


@pytest.mark.parametrize("flex", [0, 1])
def test_no_allocation_scores(flex):
    """The scorer on the reference's grid layout: a NaN coordinate reads inside the maps."""
    job, g, want = poses(flex)
    x, out = torch.from_numpy(g).cuda(), []
    for grads in (True, False):
        e = torch.zeros(len(g), device="cuda")
        gr = torch.zeros((len(g), 64), device="cuda")
        lib.call("adgpu_score_genotypes_noalloc", C.cast(C.pointer(job.g), C.c_void_p), len(g), x, e, gr if grads else None)
        torch.cuda.synchronize()
        out += [e.cpu().numpy(), gr.cpu().numpy()][:2 if grads else 1]
    check(job, flex, *out, *want)

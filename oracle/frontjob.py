"""Docking inputs for the oracle prepared by this package's own front end, with
the interface of refpy.RefJob: for where the reference's sources, and with
them its front end, are not there to build (refpy.available()).  The tables
of the two front ends are equal (tests/test_frontend.py).

TEST INFRASTRUCTURE ONLY: imported by tests/, by __graft_entry__.smoke() and by
bench.py's CPU-baseline leg; never by the product.
"""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np

from adgpu_b200 import abi, frontend


class FrontJob:
    def __init__(self, fld: str, ligand: str, nrun: int, seed: tuple, pop: int, flexres: str | None = None):
        grid = frontend.Grid.read(fld)
        self.lig = frontend.Ligand(grid, open(ligand).read(), open(flexres).read() if flexres else None,
                                   run=frontend.default_dockpars(grid.spacing, pop), seed=seed, num_runs=nrun)
        dp = self.lig.dockpars
        gr = abi.KcGrads.from_buffer_copy(bytes(self.lig.tables["grads"]))
        self.info = SimpleNamespace(
            num_of_atoms=dp.num_of_atoms, true_ligand_atoms=dp.true_ligand_atoms,
            num_of_rotbonds=sum(n > 0 for n in gr.num_rotating_atoms_per_rotbond), num_of_genes=dp.num_of_genes,
            num_of_intraE_contributors=dp.num_of_intraE_contributors, pop_size=dp.pop_size, num_of_runs=nrun,
            num_of_lsentities=dp.num_of_lsentities, num_of_map_atypes=dp.num_of_map_atypes,
            gridsize=list(grid.dims), spacing=grid.spacing, grid_origin=list(grid.origin))
        self._grid = grid.reference_layout()

    def blob(self, name: str) -> np.ndarray:
        if name == "dockpars":
            return np.frombuffer(bytes(self.lig.dockpars), np.uint8).copy()
        if name == "grid":
            return self._grid.copy()
        if name in ("initpop", "prng"):
            return np.asarray(getattr(self.lig, name)).reshape(-1).copy()
        return np.asarray(self.lig.tables[name]).view(np.uint8).copy()

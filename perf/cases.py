"""The docking work that the performance figures are taken on.

Each case is one call that a user's program makes through this package's
public entry points: scoring genotypes, docking a ligand (plain, with the
device-side AutoStop, or with the generation loop on the host as a program
written against the reference's kernel API runs it), docking a batch through
the engine, and processing the final populations of a docking.

Receptors and ligands are the seeded synthetic ones of adgpu_b200.synth; a
case names the ligand, the seed gives the initial populations and the random
streams.  The receptor and the prepared ligand are kept between states, as a
program that docks into one receptor keeps them.

Results: gradients are fixed-point sums and a run's random decisions come from
its own streams, so a docking repeats bit for bit; a search of hundreds of
steps amplifies any rounding into another path, so dockings and their
processing are compared exactly.  Scores have a tolerance.
"""
import math
import os
import random
import sys
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "autodock-gpu_b200"))

from adgpu_b200 import abi, device, dock, engine, frontend, lib, result, synth  # noqa: E402

DEV = "cuda:0"
POP = 150                     # the reference's default population (--psize)


def listed():
    return [
        # one pose of a fragment-sized ligand, energy and gradient: the smallest call, launch and synchronisation
        dict(name="score_one", call="score", heavy=16, tors=4, npts=40, maps=5, flex=0, n=1, grads=True, ligand=0),
        # a population of 100 runs of the plain workload's ligand, energies and gradients
        dict(name="score_grads", call="score", heavy=40, tors=10, npts=60, maps=5, flex=0, n=15000, grads=True, ligand=0),
        # rescoring many poses of a large flexible ligand, energies only
        dict(name="score_large", call="score", heavy=64, tors=32, npts=80, maps=7, flex=0, n=120000, grads=False, ligand=1),
        # a small docking: fragment-sized ligand, few runs
        dict(name="dock_small", call="dock", heavy=16, tors=4, npts=40, maps=5, flex=0, runs=10, search="ad", nev=250000, ligand=0),
        # one run of a drug-sized ligand, a look at one ligand: nothing to fill the GPU with
        dict(name="dock_one_run", call="dock", heavy=27, tors=7, npts=60, maps=5, flex=0, runs=1, search="ad", nev=250000, ligand=2),
        # the reference's default settings: 20 runs, ADADELTA, stopped by AutoStop
        dict(name="dock_autostop", call="autostop", heavy=32, tors=8, npts=60, maps=5, flex=0, runs=20, search="ad", nev=500000, ligand=3),
        # the plain workload: 100 runs of a 40-atom, 10-torsion ligand
        dict(name="dock_ad", call="dock", heavy=40, tors=10, npts=60, maps=5, flex=0, runs=100, search="ad", nev=250000, ligand=0),
        # the same with Solis-Wets (energies only)
        dict(name="dock_sw", call="dock", heavy=40, tors=10, npts=60, maps=5, flex=0, runs=100, search="sw", nev=250000, ligand=0),
        # two flexible residues, ADAM, a larger box with seven ligand types
        dict(name="dock_flex_adam", call="dock", heavy=40, tors=10, npts=80, maps=7, flex=2, runs=50, search="adam", nev=150000, ligand=4),
        # the generation loop on the host, one call per kernel, as a program of the reference's kernel API runs it
        dict(name="host_loop", call="host", heavy=33, tors=9, npts=60, maps=5, flex=0, runs=20, search="ad", gens=20, ligand=5),
        # a screening batch: uneven ligands admitted together
        dict(name="engine_batch", call="engine", heavy=64, tors=32, npts=60, maps=5, flex=0, runs=20, search="ad", nev=30000, count=24, ligand=6),
        # ordering, re-scoring and clustering the final populations of 100 runs
        dict(name="result_100", call="result", heavy=40, tors=10, npts=60, maps=5, flex=0, runs=100, every=True, ligand=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["score", "score", "dock", "dock", "dock", "dock", "autostop", "autostop", "host", "engine", "result"])
    heavy = _log(rng, 8, 64)
    c = dict(call=call, heavy=heavy, tors=rng.randint(0, min(32, heavy // 2)), npts=2 * rng.randint(18, 45),
             maps=rng.choice([5, 7]), flex=0 if call == "engine" else rng.choice([0, 0, 0, 1, 2]), ligand=rng.randint(100, 999))
    if call == "score":
        c.update(n=_log(rng, 1, 60000), grads=rng.random() < 0.7)
        return c
    c["runs"] = _log(rng, 1, 100)
    if call == "result":
        c["every"] = rng.random() < 0.6
        return c
    c["search"] = rng.choice(["ad", "ad", "ad", "sw", "adam", "fire"])
    # a docking's cost against the largest listed one's: pairs grow with the square of the atoms
    cost = ((heavy + 10 * c["flex"]) / 40.0) ** 2 + 0.2
    if call == "host":
        c["runs"] = min(c["runs"], 40)
        c["gens"] = rng.randint(3, 20)
    elif call == "engine":
        c.update(runs=rng.randint(4, 20), count=rng.randint(3, 24), nev=_log(rng, 15000, 60000))
        c["nev"] = int(min(c["nev"], max(10000, 1.5e7 / (cost * c["runs"] * c["count"]))))
    else:
        c["nev"] = int(min(_log(rng, 40000, 500000), max(40000, 2.5e7 / (cost * c["runs"]))))
        c["runs"] = max(1, min(c["runs"], int(2.5e7 / (cost * c["nev"]))))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

@lru_cache(maxsize=4)
def _receptor(npts, maps):
    types = synth.MAP_TYPES_5 if maps == 5 else synth.MAP_TYPES_7
    spec = synth.grid_spec(npts, types, seed=12345 + npts)
    grid = frontend.Grid.from_maps(synth.quantize_maps(synth.make_maps_fast(spec, DEV)), types, spec.spacing, spec.origin)
    return grid, grid.reference_layout()


@lru_cache(maxsize=64)
def _pdbqt(heavy, tors, ligand):
    return "\n".join(synth.pdbqt_lines(synth.ligand_for(2, ligand, heavy, tors))[0]) + "\n"


@lru_cache(maxsize=8)
def _flexres(count):
    rng = np.random.default_rng(77)
    return synth.flexres_text([synth.make_flexres(100 + k, int(rng.integers(8, 11)), int(rng.integers(2, 5)),
                                                  anchor=np.array([-3.0 + 6.0 * k, 4.0, 0.0])) for k in range(count)])


def _ligand(c, seed, runs):
    """The case's ligand prepared with `runs` initial populations drawn from the seed."""
    grid, _ = _receptor(c["npts"], c["maps"])
    words = np.random.default_rng([seed & 0x7FFFFFFF, 11]).integers(1, 2**31 - 1, 3)
    return frontend.Ligand(grid, _pdbqt(c["heavy"], c["tors"], c["ligand"]), _flexres(c["flex"]) if c["flex"] else None,
                           run=frontend.default_dockpars(grid.spacing, POP), seed=tuple(int(w) for w in words), num_runs=runs)


def _batch(c, seed):
    """The engine case's ligands: sizes uneven, up to the case's."""
    r = random.Random(c["ligand"])
    out = []
    for k in range(c["count"]):
        heavy = max(8, round(c["heavy"] * r.uniform(0.16, 1.0)))
        tors = min(heavy // 2, round(c["tors"] * r.random()))
        out.append(_ligand(dict(c, heavy=heavy, tors=tors, ligand=c["ligand"] + k), seed + 7919 * k, c["runs"]))
    return out


class _Search:
    """One ligand's tables, maps, populations and random streams on the GPU."""

    def __init__(self, c, seed, runs):
        self.case = c
        self.lig = _ligand(c, seed, runs)
        self.job = device.DeviceJob(self.lig.tables, self.lig.dockpars, _receptor(c["npts"], c["maps"])[1], runs, self.lig.prng, DEV)
        self.init = torch.from_numpy(self.lig.initpop[:runs * POP]).to(DEV)
        self.prng = self.job.prng.clone()


def _poses(c, lig):
    """Poses as a search holds them: random orientations and torsions, positions around the middle of the box."""
    g = torch.from_numpy(lig.initpop[:c["n"]]).to(DEV)
    g[:, :3] = c["npts"] / 2 + 0.35 * (g[:, :3] - c["npts"] / 2)
    return g


def prepare(case, seed):
    c = dict(case)
    call = c["call"]
    if call == "score":
        s = _Search(c, seed, -(-c["n"] // POP))
        s.poses = _poses(c, s.lig)
        s.energies = torch.zeros(c["n"], device=DEV)
        s.grads = torch.zeros((c["n"], abi.GENOTYPE_STRIDE), device=DEV) if c["grads"] else None
        # every state of a case has the same ligand and maps, so the active ligand is the one to score
        # whichever state was prepared last
        s.job.activate()
        return s
    if call in ("dock", "autostop", "host"):
        return _Search(c, seed, c["runs"])
    if call == "result":
        # final populations: the initial ones after a short docking
        s = _Search(c, seed, c["runs"])
        s.job.activate()
        r = dock.dock(s.job, s.init, "ad", nev=1 << 40, ngen=2)
        # the runs' entities in the order the GA leaves them
        s.conf, s.en = r.conformations.clone(), r.energies.clone()
        s.conf_out, s.en_out = torch.empty_like(s.conf), torch.empty_like(s.en)
        s.params = result.default_params(rescore_entities=1 if c["every"] else 0)
        return s
    if call == "engine":
        eng = engine.Engine()
        return dict(case=c, engine=eng, receptor=eng.add_receptor(_receptor(c["npts"], c["maps"])[0]), ligands=_batch(c, seed))
    raise ValueError(call)


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

def run(s):
    c = s["case"] if isinstance(s, dict) else s.case
    call = c["call"]
    if call == "score":
        lib.call("adgpu_score_genotypes", c["n"], s.poses, s.energies, s.grads)
        return (s.energies, s.grads) if c["grads"] else s.energies
    if call == "engine":
        eng = s["engine"]
        ids = [eng.submit(lg, s["receptor"], c["search"], c["nev"]) for lg in s["ligands"]]
        eng.run()
        res = [eng.result(i) for i in ids]
        return [np.concatenate([getattr(r, k) for r in res]) for k in ("best_energies", "best_genotypes", "evals", "generations")]
    if call == "result":
        s.conf_out.copy_(s.conf)           # the call orders the populations in place
        s.en_out.copy_(s.en)
        p = result.process_result(s.lig, s.job.grid, s.conf_out, s.en_out, c["runs"], s.params)
        per_run = np.array([(r.inter_e, r.intra_e, r.energy, r.rmsd_from_ref, r.rmsd_from_cluster_center) for r in p.runs], np.float32)
        clusters = np.array([(r.cluster_id, r.cluster_subrank, r.energy_rank) for r in p.runs], np.int32)
        out = [s.conf_out, s.en_out, p.best_xyz, p.peratom, per_run, clusters]
        return out + [p.entities] if c["every"] else out
    # a ligand's docking: its tables made the active ones, then the generations
    s.job.prng.copy_(s.prng)
    s.job.activate()
    if call == "dock":
        r = dock.dock(s.job, s.init, c["search"], nev=c["nev"])
    elif call == "autostop":
        r = dock.dock(s.job, s.init, c["search"], nev=c["nev"], autostop=dock.AutoStopParams())
    else:
        r = dock.dock_host_loop(s.job, s.init, c["search"], nev=1 << 40, ngen=c["gens"])
    return [r.conformations, r.energies, r.evals_per_run, r.generations]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _ignored(lig, n):
    """The atoms that the maps are not asked for."""
    at = abi.KcInterintra.ignore_inter_const.offset
    return np.frombuffer(bytes(lig.tables["interintra"]), np.uint8)[at:at + n] != 0


@lru_cache(maxsize=256)
def _counts(heavy, tors, npts, maps, flex, ligand):
    lig = _ligand(dict(heavy=heavy, tors=tors, npts=npts, maps=maps, flex=flex, ligand=ligand), 0, 0)
    dp = lig.dockpars
    n = dp.num_of_atoms
    scored = int((~_ignored(lig, n)).sum())
    rots = int(((np.frombuffer(bytes(lig.tables["rotlist"]), np.int32)[:dp.rotbondlist_length] & abi.RLIST_DUMMY_MASK) == 0).sum())
    gr = abi.KcGrads.from_buffer_copy(bytes(lig.tables["grads"]))
    turned = int(sum(gr.num_rotating_atoms_per_rotbond[:dp.num_of_genes - 6]))
    return n, scored, dp.num_of_intraE_contributors, rots, turned, dp.num_of_genes


def _per_eval(c):
    """Floating operations of one evaluation (energy and gradient, energy alone) and the atoms scored."""
    n, scored, q, rots, turned, _ = _counts(c["heavy"], c["tors"], c["npts"], c["maps"], c["flex"], c["ligand"])
    return 40 * rots + 200 * scored + 80 * q + 25 * turned + 30 * n, 40 * rots + 100 * scored + 45 * q, scored, n


def work(case):
    c = dict(case)
    points = (c["npts"] + 1) ** 3
    map_bytes = 4 * (c["maps"] + 2) * points
    row = 4 * abi.GENOTYPE_STRIDE
    if c["call"] == "engine":
        r = random.Random(c["ligand"])
        flops = nbytes = 0
        for k in range(c["count"]):
            heavy = max(8, round(c["heavy"] * r.uniform(0.16, 1.0)))
            tors = min(heavy // 2, round(c["tors"] * r.random()))
            grad, energy, _, _ = _per_eval(dict(c, heavy=heavy, tors=tors, ligand=c["ligand"] + k))
            flops += c["runs"] * c["nev"] * (energy if c["search"] == "sw" else grad)
            nbytes += c["runs"] * POP * row * 2 + c["runs"] * row
        return {"bytes": nbytes + map_bytes, "flops": flops}
    grad, energy, scored, n = _per_eval(c)
    if c["call"] == "score":
        return {"bytes": c["n"] * (row * (2 if c["grads"] else 1) + 4) + min(map_bytes, 96 * scored * c["n"]),
                "flops": c["n"] * (grad if c["grads"] else energy)}
    pop = c["runs"] * POP
    if c["call"] == "result":
        poses = pop if c["every"] else c["runs"]
        return {"bytes": pop * row * 2 + poses * 12 + c["runs"] * n * 32, "flops": poses * energy}
    # initial populations and random streams in, final populations out; the maps
    evals = c["runs"] * (c["nev"] if c["call"] != "host" else c["gens"] * POP * 70)
    if c["call"] == "autostop":
        evals = min(evals, c["runs"] * 150000)      # AutoStop ends most dockings well before the limit
    return {"bytes": pop * row * 3 + map_bytes, "flops": evals * (energy if c["search"] == "sw" else grad)}


def tolerance(case):
    if case["call"] != "score":
        return "exact"
    # measured against 64 bits: energies 2e-5 to 5e-5 (clashing pairs' r^-12 in 32 bits); gradients 5e-4 to 3e-3, nearly
    # all of it in the orientation genes, angle differences taken through a step of 1e-3 rad and rounded to 1/1024
    return {"rel": 1e-2, "max": 0.3} if case["grads"] else {"rel": 2e-4, "max": 1e-3}


# ---------------------------------------------------------------------------
# the scorer in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    c = dict(case)
    if c["call"] != "score":
        return None               # a search in 64 bits takes another path after some steps
    lig = _ligand(c, seed, -(-c["n"] // POP))
    layout = _receptor(c["npts"], c["maps"])[1]
    parts = [_score64(lig, layout, x, c["grads"]) for x in torch.split(_poses(c, lig), 4000)]
    e = torch.cat([p[0] for p in parts])
    return (e, torch.cat([p[1] for p in parts])) if c["grads"] else e


def _t64(x):
    return torch.tensor(np.asarray(x, np.float64), device=DEV)


def _quant(v):
    """A gradient term as the scorer defines it: rounded to 1/1024, at most 8 in size (in units of 1/1024)."""
    return torch.round(torch.clamp(v * 1024.0, -8192.0, 8192.0))


def _turn(p, q):
    """Vectors p [B, 3] turned by quaternions q [B, 4] (x, y, z, w)."""
    u, w = q[:, :3], q[:, 3:]
    z = 2.0 * torch.linalg.cross(u, p)
    return p + z * w + torch.linalg.cross(u, z)


def _score64(lig, layout, genotypes, grads):
    dp = lig.dockpars
    n, nl, ng, q = dp.num_of_atoms, dp.true_ligand_atoms, dp.num_of_genes, dp.num_of_intraE_contributors
    t = {k: abi.TABLE_TYPES[k].from_buffer_copy(bytes(lig.tables[k])) for k in abi.TABLE_TYPES}
    ii, ki, cf, gr = t["interintra"], t["intra"], t["conform"], t["grads"]
    rad, pi2 = float(np.float32(0.0174533)), float(np.float32(2 * np.float32(math.pi)))
    sp = float(dp.grid_spacing)
    g = genotypes.double()
    b = g.shape[0]
    # pose
    phi, theta, half = g[:, 3] * rad, g[:, 4] * rad, g[:, 5] * rad * 0.5
    axis = torch.stack([torch.sin(theta) * torch.cos(phi), torch.sin(theta) * torch.sin(phi), torch.cos(theta)], 1)
    rot = torch.cat([torch.sin(half)[:, None] * axis, torch.cos(half)[:, None]], 1)
    nt = ng - 6
    uv = _t64(cf.rotbonds_unit_vectors_const[:]).view(-1, 3)
    mv = _t64(cf.rotbonds_moving_vectors_const[:]).view(-1, 3)
    ht = g[:, 6:ng] * rad * 0.5
    ref = _t64(cf.ref_coords_const[:]).view(-1, 3)
    xyz = [ref[a].expand(b, 3) for a in range(n)]
    for el in np.frombuffer(bytes(lig.tables["rotlist"]), np.int32)[:dp.rotbondlist_length].tolist():
        if el & abi.RLIST_DUMMY_MASK:
            continue
        a = el & abi.RLIST_ATOMID_MASK
        if el & abi.RLIST_GENROT_MASK:
            if a < nl:
                xyz[a] = _turn(xyz[a], rot) + g[:, :3]
        else:
            k = (el & abi.RLIST_RBONDID_MASK) >> abi.RLIST_RBONDID_SHIFT
            qk = torch.cat([torch.sin(ht[:, k:k + 1]) * uv[k], torch.cos(ht[:, k:k + 1])], 1)
            xyz[a] = _turn(xyz[a] - mv[k], qk) + mv[k]
    p = torch.stack(xyz, 1)                                            # [B, N, 3]
    # intermolecular terms
    gx, gy, gz, m = dp.gridsize_x, dp.gridsize_y, dp.gridsize_z, dp.num_of_map_atypes
    maps = _t64(layout[::4]).view(m + 2, gz, gy, gx)
    charge = _t64(ii.atom_charges_const[:n])
    scored = torch.from_numpy(~_ignored(lig, n)).to(DEV)
    mtype = torch.tensor([min(ii.atom_types_map_const[a], m - 1) for a in range(n)], device=DEV)
    top = _t64([gx - 1, gy - 1, gz - 1])
    out = ((p < 0) | (p >= top)).any(2) & scored
    use = scored & ~out
    lo = torch.minimum(torch.clamp(torch.floor(p), min=0), top - 1)
    d = p - lo
    x0, y0, z0 = (lo[..., k].long() for k in range(3))
    v = {}
    for i in (0, 1):
        for j in (0, 1):
            for k in (0, 1):
                at = (z0 + k, y0 + j, x0 + i)
                v[i, j, k] = maps[(mtype.expand_as(z0),) + at] + charge * maps[(m,) + at] + charge.abs() * maps[(m + 1,) + at]
    w = [(1 - d[..., k], d[..., k]) for k in range(3)]
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    inter = sum(v[i, j, k] * w[0][i] * w[1][j] * w[2][k] for (i, j, k) in v)
    e = torch.where(use, inter, zero).sum(1) + 16777216.0 * out.sum(1)
    force = None
    if grads:
        dx = sum((2 * i - 1) * v[i, j, k] * w[1][j] * w[2][k] for (i, j, k) in v)
        dy = sum((2 * j - 1) * v[i, j, k] * w[0][i] * w[2][k] for (i, j, k) in v)
        dz = sum((2 * k - 1) * v[i, j, k] * w[0][i] * w[1][j] for (i, j, k) in v)
        force = torch.where(use[..., None], _quant(torch.stack([dx, dy, dz], 2) / sp), zero)
        force = torch.where(out[..., None], zero + 16777216.0, force)
    # intramolecular pairs
    if q:
        pairs = torch.from_numpy(np.frombuffer(bytes(lig.tables["intracontrib"]), np.uint32)[:2 * q].astype(np.int64)).to(DEV).view(q, 2)
        a1, a2 = pairs[:, 0], pairs[:, 1]
        nat = dp.num_of_atypes
        ty = torch.tensor(list(ii.atom_types_const[:n]), device=DEV)
        t1, t2 = ty[a1], ty[a2]
        tp = t1 * nat + t2
        ex = torch.tensor(list(ki.VWpars_exp_const[:nat * nat]), device=DEV)[tp]
        em, en = ((ex >> 8) & 0xFF).double(), (ex & 0xFF).double()
        ac, bd, req = (_t64(x[:nat * nat])[tp] for x in (ki.VWpars_AC_const, ki.VWpars_BD_const, ki.reqm_AB_const))
        ds, dv = _t64(ki.dspars_S_const[:]), _t64(ki.dspars_V_const[:])
        q1, q2 = charge[a1], charge[a2]
        sol = dp.coeff_desolv * ((ds[t1] + dp.qasp * q1.abs()) * dv[t2] + (ds[t2] + dp.qasp * q2.abs()) * dv[t1])
        qq = dp.coeff_elec * q1 * q2
        s = p[:, a1] - p[:, a2]
        dist = torch.linalg.norm(s, dim=2)
        r = dist * sp
        hs = 0.5 * dp.smooth
        sd = torch.minimum(torch.maximum(req, r - hs), r + hs)
        tm, tn = ac * sd ** -em, bd * sd ** -en
        near = r < 8.0
        pg = torch.where(near, (en * tn - em * tm) / sd, zero)
        rr = torch.clamp(r, min=dp.elec_min_distance)
        d2 = rr * rr
        num = -0.1063 * d2 * (1.0 - 0.001947 * d2) + 12.96
        den = d2 * (d2 * (0.000112 * d2 + 0.00357) + 0.4137) + 12.96
        dsv = sol * num / den
        rs = 1.0 / (rr + 1.26366)
        diel = 1.10859 * rs * rs + 0.010358
        es = qq / rr
        far = r < 20.48
        e = e + (torch.where(near, tm - tn, zero) + torch.where(far, diel * es + dsv, zero)).sum(1)
        if grads:
            pg = pg - torch.where(far, es * (diel / rr + 2.21718 * rs ** 3) + 0.0771605 * rr * dsv, zero)
            fp = _quant(-s * (pg / torch.clamp(dist, min=1e-15))[..., None])
            force.index_add_(1, a1, -fp)
            force.index_add_(1, a2, fp)
    if not grads:
        return e, None
    force = force / 1024.0
    # genes
    gg = torch.zeros((b, abi.GENOTYPE_STRIDE), dtype=torch.float64, device=DEV)
    lf, lp = force[:, :nl], (p[:, :nl] - g[:, None, :3]) * sp
    gg[:, :3] = _quant(lf.sum(1) * sp)
    tq = torch.linalg.cross(lp, lf).sum(1)
    tl = torch.linalg.norm(tq, dim=1)
    small = tl < 1e-3
    scale = torch.where(small, 0.5 - tl * tl / 48.0, math.sin(0.0005) / tl)
    qt = torch.cat([tq * scale[:, None], torch.where(small, 1.0 - tl * tl * 0.125, zero + math.cos(0.0005))[:, None]], 1)
    ax, ay, az, aw = qt.unbind(1)
    bx, by, bz, bw = rot.unbind(1)
    tx = aw * bx + ax * bw + ay * bz - az * by
    ty_ = aw * by - ax * bz + ay * bw + az * bx
    tz = aw * bz + ax * by - ay * bx + az * bw
    tw = aw * bw - ax * bx - ay * by - az * bz
    sign = torch.where(torch.sin(theta) < 0, -1.0, 1.0).double()
    wrap = lambda x: x - torch.trunc(x / pi2) * pi2  # noqa: E731
    target = [wrap(torch.atan2(sign * ty_, sign * tx) + pi2), pi2 + sign * _acos(tz / torch.sqrt(1.0 - tw * tw)), 2.0 * _acos(tw)]
    over = torch.where(small, zero + 1.0, tl * 1000.0)
    corr = 4.0 * torch.sin(half) ** 2
    for j in range(3):
        x = over * (wrap(target[j] - wrap(pi2 + g[:, 3 + j] * rad) + pi2 / 2) - pi2 / 2)
        if j == 0:
            x = x * torch.sin(theta) ** 2
        if j < 2:
            x = x * corr
        gg[:, 3 + j] = _quant(x * rad)
    for k in range(nt):
        o, end = gr.rotbonds[2 * k], gr.rotbonds[2 * k + 1]
        at = list(gr.rotbonds_atoms[abi.MAX_ATOMS * k:abi.MAX_ATOMS * k + gr.num_rotating_atoms_per_rotbond[k]])
        u = p[:, end] - p[:, o]
        u = u / torch.linalg.norm(u, dim=1, keepdim=True)
        arm = torch.linalg.cross(p[:, at] - p[:, o:o + 1], force[:, at])
        gg[:, 6 + k] = _quant((arm * u[:, None]).sum(2) * sp * rad).sum(1)
    gg = gg / 1024.0
    gg[:, 3:] *= sp * sp / (rad * rad)
    return e, gg


def _acos(x):
    """The fit of the arc cosine that the orientation genes are defined through."""
    a, b, c, d = 9.78056e-05, -0.00104588, 0.00418716, -0.00314347
    o, y = -(a + b + c + d), x.abs()
    ac = (((o * y ** 4 + a) * y ** 3 + b) * y * y + c) * y + d
    ac = ac + 2.74084 * torch.sqrt(torch.clamp(2.0 - torch.sqrt(2.0 + 2.0 * y), min=0)) - 0.370388 * torch.sqrt(torch.clamp(2.0 - 2.0 * y, min=0))
    return torch.copysign(ac, x) + torch.where(x < 0, math.pi, 0.0).double()

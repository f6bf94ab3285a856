"""AutoStop's statistics against a plain restatement of the reference's class
(host/inc/autostop.hpp:83-222), float operation for float operation and the
sums in its order: the tolerance at which the docking's stop moves from one
check to another is found to the last bit on the host, and the device has to
stop where the host does on both sides of it."""
import numpy as np
import pytest

from adgpu_b200 import device, dock, frontend, synth

pytestmark = pytest.mark.gpu
f4 = np.float32


def average(a):
    return f4(0) if a[2] < 1 else a[0] / a[2]


def stddev(a):
    if a[2] < 1:
        return f4(0)
    sq = a[1] * a[2] - a[0] * a[0]
    return f4(0) if abs(float(sq)) <= 0.000001 or sq < 0 else np.sqrt(sq) / a[2]


def running(e):
    """Sum, sum of squares and number of energies, added one after another."""
    if not len(e):
        return [f4(0)] * 3
    return [np.cumsum(e, dtype=f4)[-1], np.cumsum(e * e, dtype=f4)[-1], f4(len(e))]


class AutoStop:
    def __init__(self, pop, stopstd, freq):
        self.ntop, self.ncream, self.stopstd, self.freq = pop, pop // 10, f4(stopstd), freq
        self.first, self.threshold, self.width = True, f4(1 << 24), f4(1 << 24)
        self.avg, self.std, self.best_n = f4(-(1 << 24)), f4(1 << 24), 1
        self.delta = f4(2.0 * float(self.width) / self.ntop)
        self.rolling, self.rc = np.zeros((4, 4), f4), 0

    def tabulate(self, e):
        self.best = min(f4(1 << 24), e.min())
        below = e[e < self.threshold]
        ends = float(self.threshold) - 2.0 * float(self.width) + (np.arange(self.ntop, dtype=f4) * self.delta).astype(np.float64)
        bins = np.searchsorted(ends, below.astype(np.float64), side="right")     # the first end above the energy
        return running(below), [running(below[bins == m]) for m in range(self.ntop)]

    def check(self, generation, energies):
        for _ in range(9 if generation == 0 else 1):
            if not abs(float(self.avg)) > 0.00001:
                break
            a, bins = self.tabulate(energies)
            self.avg, self.std, self.best_n = average(a), stddev(a), int(a[2])
            if self.first:
                self.width, self.first = self.std, False
                self.threshold = self.avg + self.width
            else:
                a, low = [f4(0)] * 3, 0
                for b in bins:
                    if b[2] >= 1 and low < self.ncream and (
                            a[2] < 4 or abs(float(average(a) - average(b))) < 2.0 * float(self.stopstd)):
                        a, low = [x + y for x, y in zip(a, b)], low + 1
                if low:
                    self.avg, self.std, self.best_n = average(a), stddev(a), int(a[2])
                self.width = self.stopstd if self.std < f4(0.5) * self.stopstd else self.std
                self.threshold = self.avg + f4(self.ncream) * self.width / f4(self.best_n)
            self.delta = f4(2.0 * float(self.width) / (self.ntop - 1))
        n = f4(self.best_n)
        self.rolling[self.rc] = self.avg * n, (self.std * self.std + self.avg * self.avg) * n, n, self.best
        self.rc = (self.rc + 1) % 4
        r = self.rolling
        a = [((r[0, k] + r[1, k]) + r[2, k]) + r[3, k] for k in range(3)]
        best = (((r[0, 3] + r[1, 3]) + r[2, 3]) + r[3, 3]) / f4(4)
        sq = [r[k, 3] * r[k, 3] for k in range(4)]
        var = (((sq[0] + sq[1]) + sq[2]) + sq[3]) / f4(4) - best * best
        return bool(stddev(a) < self.stopstd and generation >= 4 * self.freq and var <= f4(0.00002))


def stop_of(checks, pop, stopstd, freq):
    """The generation of the first satisfied check, or None."""
    s = AutoStop(pop, stopstd, freq)
    with np.errstate(all="ignore"):
        return next((g for g, e in checks if s.check(g, e)), None)


@pytest.mark.parametrize("search,runs,pipeline", [("ad", 4, 1), ("ad", 4, 0), ("ad", 26, 1), ("sw", 6, 1), ("adam", 3, 1), ("fire", 3, 0)])
def test_stop_to_the_last_bit_of_the_tolerance(search, runs, pipeline, monkeypatch):
    spec = synth.grid_spec(40, synth.MAP_TYPES_5, seed=41)
    grid = frontend.Grid.from_maps(synth.quantize_maps(synth.make_maps_fast(spec)), synth.MAP_TYPES_5, spec.spacing, spec.origin)
    text = "\n".join(synth.pdbqt_lines(synth.ligand_for(2, 16, 16, 4))[0]) + "\n"
    lig, freq, ngen = frontend.Ligand(grid, text, num_runs=runs), 2, 40
    monkeypatch.setenv("ADGPU_DOCK_PIPELINE", str(pipeline))

    def job():
        j = device.DeviceJob(lig.tables, lig.dockpars, grid.reference_layout(), runs, lig.prng)
        j.activate()
        return j

    checks = []
    dock.dock_host_loop(job(), lig.initpop, search, nev=1 << 40, ngen=ngen,
                        autostop=(freq, 0, lambda g, e, total: checks.append((g, e.copy())) or False))
    pop, lo, hi = lig.dockpars.pop_size, f4(1e-3), f4(8.0)
    late = lambda s: stop_of(checks, pop, s, freq) or ngen  # noqa: E731  (None: the generations run out)
    first, last = late(hi), late(lo)
    assert first < last
    while np.nextafter(lo, hi) < hi:                  # two neighbouring tolerances on either side of a change
        mid = ((lo.view(np.int32) + hi.view(np.int32)) // 2).astype(np.int32).view(f4)
        lo, hi = (lo, mid) if late(mid) == first else (mid, hi)
    assert late(lo) != late(hi)
    for s in (lo, hi):
        r = dock.dock(job(), lig.initpop, search, nev=1 << 40, ngen=ngen, autostop=dock.AutoStopParams(freq, float(s), 0))
        assert dock.last_stats()["pipelined"] == pipeline
        assert r.generations == late(s)
        assert r.autostopped == (late(s) < ngen)

"""The autotuner on both kernel families: on the list kernels every trial's launch shape gives
the same bits; on the row kernels its steps are plain steps, and nothing is chosen or kept."""
import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu


def _pair():
    params = capi.params(capi.PROFILE_BASELINE, 0.1)
    parts, cfg = scenes.dam_break((24, 16, 24), (2.4, 2.4, 2.4), seed=61)
    return SphSolver(params=params), SphSolver(params=params), parts, cfg


def _same(a, b):
    got, want = a.download(0), b.download(0)
    for f in ("id", "position", "velocity"):
        assert got[f].tobytes() == want[f].tobytes(), f


def test_shapes_of_the_list_kernels_give_the_same_bits(monkeypatch):
    monkeypatch.setenv("FGB_LIST_CAP", "96")  # asks for the list kernels and fixes no tuned value
    tuned_solver, plain_solver, parts, cfg = _pair()
    a = Batch(tuned_solver, [(scenes.copy_particles(parts), cfg)])
    assert not a.row_kernels()
    r = a.autotune(2)
    assert r.trials == 14 and r.steps == 28
    b = Batch(plain_solver, [(scenes.copy_particles(parts), cfg)])
    b.step(r.steps)
    c = Batch(tuned_solver, [(scenes.copy_particles(parts), cfg)])  # of the tuned shape
    c.step(r.steps)
    _same(a, b)
    _same(c, b)
    for x in (a, b, c):
        x.close()
    tuned_solver.close()
    plain_solver.close()


def test_the_row_kernels_choose_nothing(monkeypatch):
    tuned_solver, plain_solver, parts, cfg = _pair()
    a = Batch(tuned_solver, [(scenes.copy_particles(parts), cfg)])
    assert a.row_kernels()
    results = [a.autotune(3) for _ in range(4)]
    for r in results:
        assert (r.trials, r.steps, r.persistent, r.particles_per_thread, r.verlet) == (14, 42, 0, 1, 0)
        assert (r.block, r.skin) == (results[0].block, results[0].skin) and r.ms_per_step > 0
    b = Batch(plain_solver, [(scenes.copy_particles(parts), cfg)])
    b.step(4 * 42)
    _same(a, b)
    a.close()
    b.close()
    # what a list batch of the solver starts with is the untuned shape
    monkeypatch.setenv("FGB_LIST_CAP", "96")
    stages = []
    for s in (tuned_solver, plain_solver):
        x = Batch(s, [(scenes.copy_particles(parts), cfg)])
        x.step(2)
        x.sync()
        stages.append((x.launches, x.probe(capi.PROBE_LIST_COUNT, np.uint16).tobytes()))
        x.close()
    assert stages[0] == stages[1]
    tuned_solver.close()
    plain_solver.close()

"""Rows of neighbours that grow while a server steps their scene stay within its budget: they
take what admission leaves, and the rest of their particles walk their cells, with the same
results."""
import ctypes

import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.serve import Server
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu

N, STEPS = 3000, 16


def _crowd(seed):
    rng = np.random.default_rng(seed)
    parts = scenes.block((N, 1, 1), (0.0, 0.0, 0.0), seed)
    parts["position"] = (rng.random(3 * N) * 0.2).astype(np.float32)
    return parts, scenes.config((0.0, 0.0, 0.0), (0.3, 0.2, 0.2))


def _footprint(solver, cfg, n=N):
    out = ctypes.c_uint64()
    capi.check(solver.lib.fgb_scene_footprint(solver.handle, ctypes.byref(cfg), n, 0, ctypes.byref(out)))
    return out.value


def _serve(requests, room):
    """Results, and the longest row that the footprint of a scene has grown to, in a server whose
    budget has room for `requests` scenes and `room` more entries in the rows of one."""
    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    made = [_crowd(11 + k) for k in range(requests)]
    sv = Server(solver, budget_bytes=2 * (requests * _footprint(solver, made[0][1]) + 4 * N * room),
                max_steps_per_tick=1)
    tickets = [sv.submit(cfg, parts, STEPS) for parts, cfg in made]
    sv.drain(100)
    got = [sv.fetch(t)[0] for t in tickets]
    stats = sv.stats()
    assert stats.completed == requests
    sv.close()
    cfg = made[0][1]
    words = max((_footprint(solver, cfg, n + 1) - _footprint(solver, cfg, n)) // 4 for n in (2100, 5000))
    solver.close()
    return made, got, words


@pytest.mark.parametrize("requests", [1, 2])
def test_rows_grow_within_the_budget(requests):
    # a footprint counts 144 entries a row; 100 more fit for one scene's particles
    made, got, small = _serve(requests, 100)
    _, free, large = _serve(requests, 4096)
    rest = (178 + 64) // 4 + 16
    assert small - rest <= 144 + 100 // requests < large - rest
    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    for (parts, cfg), a, b in zip(made, got, free):
        alone = Batch(solver, [(scenes.copy_particles(parts), cfg)])
        alone.step(STEPS)
        want = alone.download(0)
        for f in ("id", "position", "velocity", "colour"):
            assert a[f].tobytes() == want[f].tobytes() and b[f].tobytes() == want[f].tobytes(), f
        alone.close()
    solver.close()

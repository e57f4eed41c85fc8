"""Hit rows that cannot grow stay as they are: a refused allocation costs no step and no
result, and later batches do not inherit the length that was refused.  Rows that do grow give
the same bits however many steps a call takes."""
import os

import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu

FIELDS = ("id", "type", "mass", "position", "velocity", "colour")
PROFILES = [capi.PROFILE_BASELINE, capi.PROFILE_REF]
CALLS = (1, 1, 3, 2, 2)  # steps of each call; rows may grow between them


@pytest.fixture()
def limit():
    lib = capi.load()

    def set_to(nbytes):
        capi.check(lib.fgb_test_alloc_limit(nbytes))

    yield set_to
    set_to(0)


def _crowd(n, seed=1):
    """n particles in a cube of two cells a side: all rows overflow at first."""
    rng = np.random.default_rng(seed)
    parts = scenes.block((n, 1, 1), (0.0, 0.0, 0.0), seed)
    parts["position"] = (rng.random(3 * n) * 0.2).astype(np.float32)
    parts["velocity"] = (rng.random(3 * n) - 0.5).astype(np.float32)
    return parts, scenes.config((0.0, 0.0, 0.0), (0.3, 0.2, 0.2))


def _steps(batch):
    for steps in CALLS:
        batch.step(steps)
        batch.sync()  # what overflowed is known at the next call
    got = batch.download(0)
    assert batch.error_flags() == 0
    return got


def _batch(solver, made, env=None):
    os.environ.update(env or {})
    try:
        return Batch(solver, [(scenes.copy_particles(made[0]), made[1])])
    finally:
        for k in env or {}:
            del os.environ[k]


def _walked(profile, made):
    solver = SphSolver(h=0.1, profile=profile)
    batch = _batch(solver, made, {"FGB_VERLET": "0"})
    got = _steps(batch)
    batch.close()
    solver.close()
    return got


def _same(got, want):
    for f in FIELDS:
        assert got[f].tobytes() == want[f].tobytes(), f


# (limit in entries of a row, settings): growth refused, the first rows refused as well, and the list kernels'
@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("entries,env", [
    (0, {}), (60, {}), (17, {}), (0, {"FGB_HIT_CAP": "8", "FGB_LIST_CAP": "8"}),
])
def test_refused_rows_cost_no_result(limit, profile, entries, env):
    made, n = _crowd(3000), 3000
    want = _walked(profile, made)
    solver = SphSolver(h=0.1, profile=profile)
    if entries:
        limit(4 * entries * (n + 31))
    batch = _batch(solver, made, env)
    # nothing larger than the rows that the batch has
    first = entries or int(env.get("FGB_HIT_CAP", 256 if profile == capi.PROFILE_REF else 96))
    limit(4 * first * (n + 31))
    _same(_steps(batch), want)
    again = _batch(solver, made, env)  # not of the length that was refused
    _same(_steps(again), want)
    limit(0)
    after = _batch(solver, made, env)
    _same(_steps(after), want)
    for b in (batch, again, after):
        b.close()
    solver.close()


@pytest.mark.parametrize("profile", PROFILES)
def test_frames_go_on_after_a_refusal(limit, profile):
    made, n = _crowd(3000, 2), 3000
    solver, plain = SphSolver(h=0.1, profile=profile), SphSolver(h=0.1, profile=profile)
    got, want = scenes.copy_particles(made[0]), scenes.copy_particles(made[0])
    for frame in range(6):
        limit(0 if frame == 0 or frame > 3 else 4 * 96 * (n + 31))
        solver.advance(made[1], got)
        limit(0)
        plain.advance(made[1], want)
        _same(got, want)
    solver.close()
    plain.close()

"""An error of an early step of a long call is known while the call's later steps run."""
import time

import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu


def test_a_long_call_reports_on_the_way():
    lib = capi.load()
    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    parts, cfg = scenes.cube_scene(4096, 3)
    # tile 0 of every sort never publishes; the next tile gives up after a few thousand polls
    capi.check(lib.fgb_test_lookback_fault(0, 4096))
    try:
        batch = Batch(solver, [(parts, cfg)])
        capi.check(lib.fgb_batch_prepare(batch.handle))
    finally:
        capi.check(lib.fgb_test_lookback_fault(0xFFFFFFFF, 0))
    t0 = time.perf_counter()
    batch.step(400)
    while True:  # a call that takes no step tells what is known
        try:
            batch.step(0)
        except capi.FluidError as e:
            assert e.code == capi.FGB_ERR_TIMEOUT
            break
        assert time.perf_counter() - t0 < 60
    t1 = time.perf_counter()
    assert batch.error_flags() & 1  # waits for the call's last step
    t2 = time.perf_counter()
    batch.close()
    solver.close()
    # known after 16 of 400 steps and what it takes to queue them
    assert t1 - t0 < 0.5 * (t2 - t0)

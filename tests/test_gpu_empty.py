"""A batch without particles takes every call that one with particles does, before it is filled
and after it was drained."""
import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu


def _calls(batch):
    capi.check(batch.lib.fgb_batch_prepare(batch.handle))
    assert batch.autotune(2).steps == 0  # no step to time
    batch.set_timing(True)
    capi.check(batch.lib.fgb_batch_prepare(batch.handle))
    batch.set_timing(False)
    batch.step(3)
    assert len(batch.download(0)["mass"]) == 0 and len(batch.surface(0)) == 0
    assert len(batch.probe(capi.PROBE_DISPLACEMENT, np.float32)) == 0
    batch.sync()
    assert batch.error_flags() == 0


@pytest.mark.parametrize("profile", [capi.PROFILE_BASELINE, capi.PROFILE_REF])
def test_empty_batches_take_every_call(profile):
    solver = SphSolver(params=capi.params(profile, 0.1))
    cfg = scenes.config((0.0, 0.0, 0.0), (2.0, 2.0, 2.0), surface=1)
    batch = Batch(solver, [(scenes.block((0, 1, 1), (0.0, 0.0, 0.0), 1), cfg)])
    _calls(batch)
    source = [((1.0, 1.0, 1.0), (0.0, 0.0, 0.0), 400, 7, 0xFF00FF00)]
    for _ in range(2):  # filled, and drained again
        assert batch.sources_drains(0, source, []) == 400
        batch.step(2)
        fresh = Batch(solver, [(batch.download(0), cfg)])
        batch.step(2)
        fresh.step(2)
        got, want = batch.download(0), fresh.download(0)
        for f in ("type", "mass", "position", "velocity", "colour"):
            assert got[f].tobytes() == want[f].tobytes(), f
        fresh.close()
        assert batch.sources_drains(0, [], [((1.0, 1.0, 1.0), 100.0)]) == 0
        _calls(batch)
    batch.close()
    solver.close()

"""An edit that needs larger arrays than the device has memory for leaves the batch as it was:
its state, its next steps and the next edit.  Without memory even for its own step arrays a
batch refuses to step, and its state can still be read."""
import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu

FIELDS = ("id", "type", "mass", "position", "velocity", "colour")
N = 13824  # 96 entries a row: 5.3 MB, 16 (the least): 885 kB; a position array 221 kB


@pytest.fixture()
def limit():
    lib = capi.load()

    def set_to(nbytes):
        capi.check(lib.fgb_test_alloc_limit(nbytes))

    yield set_to
    set_to(0)


def _source(rate):
    return [((0.6, 0.9, 0.6), (0.0, 0.0, 0.0), rate, 9, 0xFFFFFFFF)]


def _same(a, b):
    for f in FIELDS:
        assert a[f].tobytes() == b[f].tobytes(), f


def _batch(solver, count):
    made = [scenes.cube_scene(N, 51 + k) for k in range(count)]
    batch = Batch(solver, [(scenes.copy_particles(p), c) for p, c in made])
    batch.step(2)
    return batch, [c for _, c in made]


def _steps_as_fresh(solver, batch, cfgs):
    fresh = Batch(solver, [(batch.download(k), c) for k, c in enumerate(cfgs)])
    batch.step(2)
    fresh.step(2)
    for k in range(len(cfgs)):
        got, want = batch.download(k), fresh.download(k)
        for f in ("type", "mass", "position", "velocity", "colour"):
            assert got[f].tobytes() == want[f].tobytes(), f
    assert batch.error_flags() == 0
    fresh.close()


# (limit, emitted): the state arrays are refused; the step arrays are, once the state has moved
@pytest.mark.parametrize("count", [1, 3])
@pytest.mark.parametrize("nbytes,rate", [(1 << 20, 90000), (1 << 20, 20000)])
def test_a_refused_edit_leaves_the_batch_as_it_was(limit, count, nbytes, rate):
    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    batch, cfgs = _batch(solver, count)
    before = [batch.download(k) for k in range(count)]
    limit(nbytes * count)
    with pytest.raises(capi.FluidError) as e:
        batch.sources_drains(count - 1, _source(rate * count), [])
    assert e.value.code == capi.FGB_ERR_OOM
    for k in range(count):
        _same(batch.download(k), before[k])
    limit(0)
    _steps_as_fresh(solver, batch, cfgs)
    assert batch.sources_drains(count - 1, _source(rate * count), []) > N
    _steps_as_fresh(solver, batch, cfgs)
    batch.close()
    solver.close()


def test_a_batch_without_step_arrays_refuses_to_step(limit):
    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    batch, _ = _batch(solver, 1)
    before = batch.download(0)
    limit(600000)  # below the least rows of the present particles
    with pytest.raises(capi.FluidError):
        batch.sources_drains(0, _source(20000), [])
    limit(0)
    for call in (lambda: batch.step(1), lambda: batch.surface(0), lambda: batch.sources_drains(0, _source(16), []),
                 lambda: capi.check(batch.lib.fgb_batch_prepare(batch.handle))):
        with pytest.raises(capi.FluidError) as e:
            call()
        assert e.value.code == capi.FGB_ERR_OOM
    _same(batch.download(0), before)
    batch.upload(0, before)
    batch.close()
    fresh = Batch(solver, [(before, scenes.cube_scene(N, 51)[1])])  # the solver goes on
    fresh.step(1)
    assert fresh.error_flags() == 0
    fresh.close()
    solver.close()

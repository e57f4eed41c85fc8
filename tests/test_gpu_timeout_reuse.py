"""A sort whose look-back wait gives up leaves entries of its outputs unwritten.  What lies
there is a key and an index of the batch all the same, whatever the solver's pool handed out:
the failed call stays within its arrays, and the next upload or frame on the same batch gives
the bits of a fresh one."""
import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu

FIELDS = ("id", "type", "mass", "position", "velocity", "colour")


@pytest.fixture()
def fault():
    lib = capi.load()

    def set_to(on):
        # tile 0 never publishes; the next tile gives up after a few thousand polls
        capi.check(lib.fgb_test_lookback_fault(0 if on else 0xFFFFFFFF, 4096 if on else 0))

    yield set_to
    set_to(False)


def _scene(n, seed):
    parts, cfg = scenes.cube_scene(n, seed)
    cfg.surface = 1
    return parts, cfg


def _used_pool(solver, made):
    """The solver's pool holds blocks of a batch of the same sizes, full of its state."""
    b = Batch(solver, [(scenes.copy_particles(p), c) for p, c in made])
    b.step(3)
    b.surface(0)
    b.close()


def _valid(batch, made):
    keys, order = batch.probe(capi.PROBE_KEYS, np.uint32), batch.probe(capi.PROBE_ORDER, np.uint32)
    info = [batch.grid_info(k) for k in range(len(made))]
    scene, code = keys >> info[0].morton_bits, keys & ((1 << info[0].morton_bits) - 1)
    assert scene.max() < len(made)
    assert (code < np.array([i.table_size for i in info])[scene]).all()
    assert order.max() < max(len(p["mass"]) for p, _ in made)


@pytest.mark.parametrize("n", [13824, 40000])  # sorts of short and of long tiles
@pytest.mark.parametrize("count", [1, 3])
def test_a_batch_steps_on_after_a_sort_that_gave_up(fault, n, count):
    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    made = [_scene(n, 7 + k) for k in range(count)]
    _used_pool(solver, made)
    fault(True)
    batch = Batch(solver, [(scenes.copy_particles(p), c) for p, c in made])
    batch.step(1)
    assert batch.error_flags() & 1
    _valid(batch, made)
    fault(False)
    capi.check(batch.lib.fgb_batch_set_timing(batch.handle, 1))  # graphs without the fault
    for k, (p, _) in enumerate(made):
        batch.upload(k, scenes.copy_particles(p))
    batch.step(2)
    fresh = Batch(solver, [(scenes.copy_particles(p), c) for p, c in made])
    fresh.step(2)
    for k in range(count):
        got, want = batch.download(k), fresh.download(k)
        for f in FIELDS:
            assert got[f].tobytes() == want[f].tobytes(), f
    assert batch.error_flags() == 0
    # a surface that gives up, and the next one
    fault(True)
    with pytest.raises(capi.FluidError) as e:
        batch.surface(0)
    assert e.value.code == capi.FGB_ERR_TIMEOUT
    fault(False)
    batch.error_flags()
    assert batch.surface(0).tobytes() == fresh.surface(0).tobytes()
    batch.close()
    fresh.close()
    solver.close()


def test_a_frame_after_one_that_gave_up_is_a_fresh_solvers(fault):
    params = capi.params(capi.PROFILE_BASELINE, 0.1)
    parts, cfg = _scene(13824, 5)
    cfg.surface = 0
    solver, plain = SphSolver(params=params), SphSolver(params=params)
    _used_pool(solver, [(parts, cfg)])
    fault(True)
    with pytest.raises(capi.FluidError) as e:
        solver.advance(cfg, scenes.copy_particles(parts))
    assert e.value.code == capi.FGB_ERR_TIMEOUT
    fault(False)
    # colliders far above the fluid: more of them than before, so the graphs are recorded anew
    far = np.array([[90 + k, 90, 90, 91 + k, 90, 90, 90 + k, 91, 90] for k in range(3)], np.float32)
    got, want = scenes.copy_particles(parts), scenes.copy_particles(parts)
    for _ in range(2):
        solver.advance(cfg, got, far)
        plain.advance(cfg, want, far)
    for f in FIELDS:
        assert got[f].tobytes() == want[f].tobytes(), f
    solver.close()
    plain.close()

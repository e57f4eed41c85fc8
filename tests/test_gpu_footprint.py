"""The footprint of a scene (admission against a budget) counts the rows of neighbours that its
batch has: as long as they are at first, and as long as they have grown."""
import ctypes

import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu


def _footprint(solver, cfg, n):
    out = ctypes.c_uint64()
    capi.check(solver.lib.fgb_scene_footprint(solver.handle, ctypes.byref(cfg), n, 0, ctypes.byref(out)))
    return out.value


def _per_particle(solver, cfg, n):
    """Of scenes of n to n + 1000 particles, which share a size class."""
    return (_footprint(solver, cfg, n + 1000) - _footprint(solver, cfg, n)) / 1000


# words of a row at first, and bytes of a particle's other arrays: two states of 44, keys and
# indices 20, sort 8, positions 64, lambda and density 8, id 8, row count and groups 15, and
# by profile colour sums 20, or vorticity terms and records 80
@pytest.mark.parametrize("profile,words,rest", [(capi.PROFILE_REF, 256, 231), (capi.PROFILE_BASELINE, 96, 291)])
def test_footprints_count_the_rows_at_hand(profile, words, rest):
    solver = SphSolver(params=capi.params(profile, 0.1))
    n = 3000
    rng = np.random.default_rng(3)
    parts = scenes.block((n, 1, 1), (0.0, 0.0, 0.0), 3)
    parts["position"] = (rng.random(3 * n) * 0.2).astype(np.float32)
    cfg = scenes.config((0.0, 0.0, 0.0), (0.3, 0.2, 0.2))
    held = 4 * words + rest
    before = _per_particle(solver, cfg, 2100)
    # at least what it holds; at most that and a quarter, or the 160 words of the list kernels
    assert held <= before <= max(1.1 * held, 4 * 160 + 64 + 178 + 1)
    batch = Batch(solver, [(parts, cfg)])
    for _ in range(5):  # hundreds of neighbours: rows grow by half, once or more
        batch.step(1)
        batch.sync()
    after = _per_particle(solver, cfg, 2100)
    lengths = [words]
    while lengths[-1] < 3000:
        lengths.append((lengths[-1] * 3 // 2 + 3) & ~3)
    assert any(4 * g + rest <= after <= 1.1 * (4 * g + rest) for g in lengths[1:])
    assert _per_particle(solver, cfg, 200000) == before  # another size class
    batch.close()
    solver.close()


def test_a_clump_does_not_set_the_rows_of_a_large_scene():
    """Four clumps of 6000 obstacles among 262 k particles: far fewer than one in a hundred have
    more than 1024 neighbours, and those walk their cells."""
    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    rng = np.random.default_rng(5)
    side, clumps, each = 64, 4, 6000
    calm = scenes.block((side, side, side), (0.0, 0.0, 0.0), 5)
    n = side ** 3 + clumps * each
    parts = scenes.block((n, 1, 1), (0.0, 0.0, 0.0), 5)
    pos = parts["position"].reshape(-1, 3)
    pos[: side ** 3] = calm["position"].reshape(-1, 3)
    for k in range(clumps):
        at = slice(side ** 3 + k * each, side ** 3 + (k + 1) * each)
        pos[at] = 1.0 + 0.3 * k + 0.12 * (rng.random((each, 3)).astype(np.float32) - np.float32(0.5))
        parts["type"][at] = capi.TYPE_OBSTACLE
    e = side * scenes.SPACING
    cfg = scenes.config((0.0, 0.0, 0.0), (e, e, e))
    batch = Batch(solver, [(parts, cfg)])
    for _ in range(14):
        batch.step(1)
        batch.sync()
    words = (_per_particle(solver, cfg, n - 2000) - 242) / 4 - 16
    assert words == 1024
    batch.close()
    solver.close()

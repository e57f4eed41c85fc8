"""The kernels on hit rows from one warp per cell (the default) give the bits of the list
kernels (FGB_VERLET=0), which walk the 27 cells: at the edges of their groups, segments and
rows, with equal and different masses, obstacles, crowded cells, several scenes, a solver
length at which the shared root does not apply, and rows that grow."""
import os

import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu

FIELDS = ("id", "type", "mass", "position", "velocity", "colour")


def _cloud(n, side, seed, h=0.1, masses=False, obstacles=0, speed=1.0):
    """n particles uniform in a cube of `side` cells."""
    rng = np.random.default_rng(seed)
    parts = scenes.block((n, 1, 1), (0.0, 0.0, 0.0), seed)
    parts["position"] = (rng.random(3 * n) * side * h).astype(np.float32)
    parts["velocity"] = ((rng.random(3 * n) - 0.5) * speed * h * 10).astype(np.float32)
    parts["mass"] = (parts["mass"] * (h / 0.1) ** 3).astype(np.float32)
    if masses:
        parts["mass"] = (parts["mass"] * (0.5 + rng.random(n))).astype(np.float32)
    if obstacles:
        parts["type"][::obstacles] = capi.TYPE_OBSTACLE
    e = float(side) * h
    return parts, scenes.config((0.0, 0.0, 0.0), (1.5 * e, e, e))


def _run(profile, made, steps, h=0.1, lists=False):
    env = {"FGB_VERLET": "0"} if lists else {}
    os.environ.update(env)
    try:
        solver = SphSolver(h=h, profile=profile)
        b = Batch(solver, [(scenes.copy_particles(p), c) for p, c in made])
    finally:
        for k in env:
            del os.environ[k]
    for _ in range(steps):  # one call each: rows grow between calls
        b.step(1)
    got = [b.download(k) for k in range(len(made))]
    assert b.error_flags() == 0
    b.close()
    solver.close()
    return got


def _same(profile, made, steps, h=0.1):
    for a, b in zip(_run(profile, made, steps, h), _run(profile, made, steps, h, lists=True)):
        for f in FIELDS:
            assert a[f].tobytes() == b[f].tobytes(), f


PROFILES = [capi.PROFILE_BASELINE, capi.PROFILE_REF]


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("n,side", [
    (1, 2), (2, 1), (31, 1), (33, 1), (300, 1),   # one cell: a lone particle, groups and segments overrun
    (3000, 2),                                      # 375 in a cell: 3000 candidates, rows that overflow and grow
    (6000, 9), (23999, 14), (24001, 14),            # ordinary density around the group sizes' line
])
def test_clouds(profile, n, side):
    _same(profile, [_cloud(n, side, n)], 4)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("masses,obstacles", [(True, 0), (False, 5), (True, 7)])
def test_masses_and_obstacles(profile, masses, obstacles):
    _same(profile, [_cloud(9000, 10, 3, masses=masses, obstacles=obstacles)], 5)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("h", [1.0, 0.005, 0.37])  # the IEEE root at the first two
def test_lengths(profile, h):
    _same(profile, [_cloud(5000, 8, 4, h=h)], 4, h)


@pytest.mark.parametrize("profile", PROFILES)
def test_scenes_of_several_sizes_and_a_violent_one(profile):
    # the last one's particles move far within a step: its rows do not last
    made = [_cloud(700, 4, 5), scenes.cube_scene(13824, 6), _cloud(64, 6, 7, obstacles=3), _cloud(8000, 10, 8, speed=40.0)]
    _same(profile, made, 12)


def test_calm_scene_over_many_steps():
    _same(capi.PROFILE_BASELINE, [scenes.cube_scene(8192, 9)], 40)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8, 9, 255, 256, 257, 259])
def test_row_ends(profile, n):
    # all of one cell: rows of n entries end at every place of a quad, and in a second segment
    _same(profile, [_cloud(n, 1, n, masses=True)], 3)


@pytest.mark.parametrize("n", [399999, 400001])
def test_rows_asked_for_ahead(n):
    # at either side of the size from which the passes prefetch their rows
    _same(capi.PROFILE_BASELINE, [_cloud(n, 36, n, obstacles=11)], 3)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("n", [7999, 8001, 65535, 65537])
def test_group_sizes(profile, n):
    _same(profile, [_cloud(n, 10 if n < 10000 else 20, n)], 3)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("first", [False, True])
def test_particles_far_from_their_cell(profile, first):
    # outside the grid, where the edge cells hold them at any distance; beyond 16 bits; not a
    # number; and (crowded) pushed across several cells by the first correction
    made, crowd = _cloud(6000, 8, 11), _cloud(2000, 2, 12, speed=300.0)
    p = made[0]["position"].reshape(-1, 3)
    at = slice(0, 40) if first else slice(5000, 5040)
    p[at] = np.linspace(-3.0, 4.0, 120, dtype=np.float32).reshape(40, 3)
    p[at.start + 40] = (1e30, 0.1, 0.1)
    p[at.start + 41] = (np.nan, 0.2, 0.2)
    _same(profile, [made, crowd], 3)


@pytest.mark.parametrize("n", [99999, 100001])
def test_stale_groups_listed_first(n):
    # at either side of the size from which a later search lists its groups first, calm and not
    _same(capi.PROFILE_BASELINE, [_cloud(n, 24, n, obstacles=13, speed=0.2)], 6)
    _same(capi.PROFILE_BASELINE, [_cloud(n - 700, 24, n), _cloud(700, 5, n, speed=30.0)], 4)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("n", [23997, 24003, 44998, 45001])
@pytest.mark.parametrize("h,masses,obstacles", [(0.1, False, 0), (0.1, True, 9), (1.0, True, 9)])
def test_four_lanes_or_one(profile, n, h, masses, obstacles):
    # at either side of the sizes below which a particle has four lanes, in both forms of the root
    _same(profile, [_cloud(n - 500, 15, n, h, masses, obstacles), _cloud(500, 1, 1, h, masses)], 3, h)


@pytest.mark.parametrize("n,side", [(1, 2), (31, 1), (65, 3), (4097, 7)])
@pytest.mark.parametrize("obstacles", [0, 3])
def test_colours_diffuse_as_the_oracle_has_them(n, side, obstacles):
    from oracle import oracle
    oracle.build()
    params = capi.params(capi.PROFILE_REF, 0.1)
    parts, cfg = _cloud(n, side, n, obstacles=obstacles)
    parts["colour"][:] = np.random.default_rng(n).integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    want = scenes.copy_particles(parts)
    solver = SphSolver(params=params)
    b = Batch(solver, [(parts, cfg)])
    for _ in range(3):
        b.step(1)
        oracle.step(params, cfg, want)
        assert (b.download(0)["colour"] == want["colour"]).all()
    b.close()
    solver.close()

"""Scenes with hardly more than a particle a cell, whose searches go by particles, give the bits
of the list kernels: at either side of the sizes and densities of the rule, with obstacles,
particles far outside and not numbers, rows that end anywhere in a quad or overflow, several
scenes at once, and scenes that change sides as they gather."""
import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu

PROFILES = [capi.PROFILE_BASELINE, capi.PROFILE_REF]
FIELDS = ("id", "type", "mass", "position", "velocity", "colour")


def _cloud(n, per_cell, seed, obstacles=0, clump=0, masses=False):
    side = max(1, round((n / per_cell) ** (1 / 3)))
    rng = np.random.default_rng(seed)
    parts = scenes.block((n, 1, 1), (0.0, 0.0, 0.0), seed)
    parts["position"] = (rng.random(3 * n) * side * 0.1).astype(np.float32)
    parts["velocity"] = (4 * (rng.random(3 * n) - 0.5)).astype(np.float32)
    if masses:
        parts["mass"] = (parts["mass"] * (0.5 + rng.random(n))).astype(np.float32)
    if clump:
        parts["position"].reshape(-1, 3)[:clump] = 0.1 * side / 2 + 0.12 * rng.random((clump, 3)).astype(np.float32)
    if obstacles:
        parts["type"][::obstacles] = capi.TYPE_OBSTACLE
    e = side * 0.1
    return parts, scenes.config((0.0, 0.0, 0.0), (e, e, e))


def _same(profile, made, monkeypatch, steps=4):
    got = []
    for lists in (False, True):
        if lists:
            monkeypatch.setenv("FGB_VERLET", "0")
        solver = SphSolver(params=capi.params(profile, 0.1))
        batch = Batch(solver, [(scenes.copy_particles(p), c) for p, c in made])
        for _ in range(steps):
            batch.step(1)
            batch.sync()
        got.append([batch.download(k) for k in range(len(made))])
        assert batch.error_flags() == 0
        batch.close()
        solver.close()
    monkeypatch.delenv("FGB_VERLET")
    for a, b in zip(*got):
        for f in FIELDS:
            assert a[f].tobytes() == b[f].tobytes(), f


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("n", [29999, 30001, 99999, 100001])
@pytest.mark.parametrize("per_cell", [0.1, 0.5, 1.5])
def test_sizes_and_densities(profile, n, per_cell, monkeypatch):
    _same(profile, [_cloud(n, per_cell, n)], monkeypatch)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("n", [399999, 400001])
def test_large_ones(profile, n, monkeypatch):
    _same(profile, [_cloud(n, 1.8, n, obstacles=9)], monkeypatch, 2)


@pytest.mark.parametrize("profile", PROFILES)
@pytest.mark.parametrize("obstacles,clump,masses", [(3, 0, True), (0, 200, False), (5, 1500, True)])
def test_obstacles_masses_and_clumps_among_them(profile, obstacles, clump, masses, monkeypatch):
    # clumps: rows of any length, and rows that overflow and grow
    _same(profile, [_cloud(40000, 0.2, 7, obstacles, clump, masses)], monkeypatch, 6)


@pytest.mark.parametrize("profile", PROFILES)
def test_far_particles_and_several_scenes(profile, monkeypatch):
    made = [_cloud(35000, 0.3, 1), _cloud(64, 2, 2), _cloud(20000, 0.5, 3, obstacles=4)]
    p = made[0][0]["position"].reshape(-1, 3)
    p[:40] = np.linspace(-9.0, 40.0, 120, dtype=np.float32).reshape(40, 3)
    p[50] = (1e30, 0.1, 0.1)
    p[51] = (np.nan, 0.2, 0.2)
    _same(profile, made, monkeypatch)


def test_a_scene_that_gathers(monkeypatch):
    # thrown at a wall: sparse at first, then several particles a cell
    parts, cfg = _cloud(60000, 0.9, 5)
    parts["velocity"].reshape(-1, 3)[:, 1] -= 60.0
    _same(capi.PROFILE_BASELINE, [(parts, cfg)], monkeypatch, 10)

"""The cell table is emptied only where the last grid, a step's or a surface's, had cells, and
the digit counts of a sort come from the kernel that makes the keys.  The oracle's cells of
each step, and the meshes and states of a fresh batch, hold after every order of steps,
surfaces, uploads, copies and edits."""
import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu

H = 0.1


def _scene(profile, n, seed):
    parts, cfg = scenes.cube_scene(n, seed)
    cfg.surface = 1
    if profile == capi.PROFILE_REF:
        cfg.isolevel = 100.0
    return parts, cfg


def _check(solver, batch, k, cfg):
    """The batch's cells are those of its keys; its scene k gives what a fresh batch gives."""
    keys = batch.probe(capi.PROBE_KEYS, np.uint32)
    cells = batch.probe(capi.PROBE_CELLS, np.uint32).reshape(-1, 2)
    assert (cells[:, 1] - cells[:, 0]).sum() == len(keys)
    assert np.count_nonzero(cells.any(1)) == len(np.unique(keys))
    fresh = Batch(solver, [(batch.download(k), cfg)])
    mesh, want = batch.surface(k), fresh.surface(0)
    assert mesh.tobytes() == want.tobytes()
    batch.step(1)
    fresh.step(1)
    got, ref = batch.download(k), fresh.download(0)
    for f in ("type", "mass", "position", "velocity", "colour"):
        assert got[f].tobytes() == ref[f].tobytes(), f
    assert batch.error_flags() == 0
    fresh.close()


@pytest.mark.parametrize("profile", [capi.PROFILE_BASELINE, capi.PROFILE_REF])
@pytest.mark.parametrize("n", [27, 4095, 4097, 13824])
def test_steps_surfaces_and_uploads_in_any_order(profile, n):
    solver = SphSolver(params=capi.params(profile, H))
    parts, cfg = _scene(profile, n, 5)
    other, _ = _scene(profile, n, 6)
    batch = Batch(solver, [(scenes.copy_particles(parts), cfg), (scenes.copy_particles(other), cfg)])
    for move in ("s", "ss", "msm", "mms", "us", "mus", "sus", "ssmmuss"):
        for m in move:
            if m == "s":
                batch.step(1)
            elif m == "m":
                batch.surface(0)
                batch.surface(1)
            else:
                batch.upload(0, scenes.copy_particles(other))
        if move[-1] == "s":
            _check(solver, batch, 0, cfg)
    batch.close()
    solver.close()

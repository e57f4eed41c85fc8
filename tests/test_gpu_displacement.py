"""The displacement probe gives how far a step's corrections moved each particle from its grid
position, on the row kernels as on the list kernels."""
import numpy as np
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", [capi.PROFILE_BASELINE, capi.PROFILE_REF])
@pytest.mark.parametrize("iterations", [1, 4, 5])
def test_displacements_are_those_of_the_list_kernels(profile, iterations, monkeypatch):
    parts, cfg = scenes.cube_scene(4096, 3, iterations)
    parts["type"][::9] = capi.TYPE_OBSTACLE
    solver = SphSolver(params=capi.params(profile, 0.1))
    got = []
    for lists in (False, True):
        if lists:
            monkeypatch.setenv("FGB_LIST_CAP", "96")
        batch = Batch(solver, [(scenes.copy_particles(parts), cfg)])
        assert batch.row_kernels() != lists
        batch.step(1)
        got.append(batch.probe(capi.PROBE_DISPLACEMENT, np.float32))
        batch.close()
    assert (got[0] > 0).sum() > 3000 and (got[0] == 0).sum() >= 4096 // 9
    assert got[0].tobytes() == got[1].tobytes()
    solver.close()

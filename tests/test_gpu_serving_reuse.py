"""A server whose clients fetch their results before the next request arrives: each request runs
on its own particles, whatever became of the memory of the one before."""
import pytest

from libfluid_gb300 import capi, scenes
from libfluid_gb300.serve import Server
from libfluid_gb300.solver import Batch, SphSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(4096, 4096), (4096, 13824, 8000), (13824, 4096, 13824)])
@pytest.mark.parametrize("together", [1, 2])
def test_requests_after_fetched_ones_run_on_their_own_particles(sizes, together):
    solver, plain = (SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1)) for _ in range(2))
    sv = Server(solver)
    for turn in range(6):
        made = [scenes.cube_scene(sizes[(turn + k) % len(sizes)], 100 + 10 * turn + k) for k in range(together)]
        tickets = [sv.submit(cfg, parts, 2 + turn % 3 + k) for k, (parts, cfg) in enumerate(made)]
        sv.drain(60)
        for k, (ticket, (parts, cfg)) in enumerate(zip(tickets, made)):
            got, _ = sv.fetch(ticket)
            alone = Batch(plain, [(scenes.copy_particles(parts), cfg)])
            alone.step(2 + turn % 3 + k)
            want = alone.download(0)
            for f in ("id", "position", "velocity", "colour"):
                assert got[f].tobytes() == want[f].tobytes(), (turn, k, f)
            alone.close()
    sv.close()
    solver.close()
    plain.close()

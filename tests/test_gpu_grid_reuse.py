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


def test_mesh_arrays_outlive_their_solver_and_welds_share_their_pool():
    import gc
    import threading

    from libfluid_gb300.weld import weld

    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, H))
    parts, cfg = _scene(capi.PROFILE_BASELINE, 4096, 3)
    batch = Batch(solver, [(parts, cfg)])
    batch.step(2)
    mesh = batch.surface(0)
    want = mesh.copy()
    view = mesh[5:, :18]
    again = batch.surface(0)  # another buffer: the first array is not written again
    again[:] = 0
    assert mesh.tobytes() == want.tobytes()
    index, vertices = weld(mesh)
    seen = []

    def work():
        for _ in range(5):
            i, v = weld(want)
            seen.append(i.tobytes() == index.tobytes() and v.tobytes() == vertices.tobytes())

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == [True] * 20
    batch.close()
    solver.close()
    del mesh, again
    gc.collect()
    assert view.tobytes() == want[5:, :18].tobytes()
    i, v = weld(want)  # after the pool was trimmed
    assert i.tobytes() == index.tobytes() and v.tobytes() == vertices.tobytes()


@pytest.mark.parametrize("n", [4095, 4097, 32 * 4096, 33 * 4096, 33 * 4096 + 1, 66 * 4096 + 7, 1200007])
def test_scans_that_look_back_a_warp_at_a_time(n):
    # around one tile and 32 of them, the most that a warp sees at once
    import ctypes

    torch = pytest.importorskip("torch")
    lib = capi.load()
    x = torch.from_numpy(np.random.default_rng(n).integers(0, 9, n, dtype=np.int32)).cuda()
    out, total = torch.empty_like(x), torch.zeros(1, dtype=torch.int32, device="cuda")
    size = lib.fgb_scan_scratch_bytes(n)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    capi.check(lib.fgb_exclusive_scan_u32(x.data_ptr(), out.data_ptr(), total.data_ptr(), n, scratch.data_ptr(),
                                          size, stream))
    want = np.cumsum(x.cpu().numpy())
    assert (out.cpu().numpy()[1:] == want[:-1]).all() and int(out[0]) == 0 and int(total[0]) == want[-1]


@pytest.mark.parametrize("n", [1023, 1025, 5000, 32767, 32768])
def test_steps_on_short_sorts_order_as_the_oracle(n):
    # around a short sort's tile, and the size from which tiles are longer
    from oracle import oracle
    oracle.build()
    params = capi.params(capi.PROFILE_BASELINE, H)
    parts, cfg = scenes.cube_scene(32768, 7)
    keep = np.sort(np.random.default_rng(n).permutation(32768)[:n])
    parts = {f: (v.reshape(32768, -1)[keep].ravel() if len(v) != n else v).copy() for f, v in parts.items()}
    solver = SphSolver(params=params)
    b = Batch(solver, [(scenes.copy_particles(parts), cfg)])
    for _ in range(3):
        b.step(1)
        pr = oracle.step(params, cfg, parts, probe=True)
        assert (b.probe(capi.PROBE_KEYS, np.uint32) == np.sort(b.probe(capi.PROBE_KEYS, np.uint32))).all()
        assert (b.download(0)["id"] == parts["id"]).all()
    b.close()
    solver.close()

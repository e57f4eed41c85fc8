"""The groups of a cell's particles (fgb_device.cuh: group_begins, group_end): those that begin where the grid
is built are, end by end, all particles once, each group of one cell, and small in a crowd.  On
the GPU crowded scenes give the bits of the list kernels."""
import os
import subprocess

import numpy as np
import pytest

from libfluid_gb300 import build, capi, scenes
from libfluid_gb300.solver import Batch, SphSolver

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "fgb_device.cuh"
// cells of the sizes read from the input: prints how many groups, or what is wrong with them
int main(int, char **v) {
    const uint32_t mask = (uint32_t)atoi(v[1]);
    std::vector<uint32_t> keys, to;
    uint32_t size;
    for (uint32_t cell = 0; scanf("%u", &size) == 1; ++cell) {
        const uint32_t at = (uint32_t)keys.size();
        for (uint32_t k = 0; k < size; ++k) keys.push_back(cell), to.push_back(at + size);
    }
    const uint32_t n = (uint32_t)keys.size();
    uint32_t groups = 0, next = 0;
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t warp = i & ~31u;
        const bool crowd = warp + 31 < n && keys[warp] == keys[warp + 31];
        if (!(i == 0 || keys[i - 1] != keys[i] || fgb::group_begins(i, mask, crowd))) continue;
        if (i != next) return printf("a group begins at %u, the last one ended at %u\n", i, next), 1;
        next = fgb::group_end(i, to[i], mask);
        if (next > to[i] || next > n) return printf("the group of %u ends outside its cell, at %u\n", i, next), 1;
        if (next - i > mask + 1 || next - i > 63) return printf("the group of %u has %u particles\n", i, next - i), 1;
        ++groups;
    }
    if (next != n) return printf("the last group ends at %u of %u\n", next, n), 1;
    printf("%u\n", groups);
}
"""


@pytest.fixture(scope="module")
def groups(tmp_path_factory):
    d = tmp_path_factory.mktemp("groups")
    src, exe = d / "g.cu", d / "g"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I" + os.path.join(ROOT, "libfluid_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)

    def run(mask, sizes):
        r = subprocess.run([str(exe), str(mask)], input=" ".join(map(str, sizes)), capture_output=True, text=True)
        assert r.returncode == 0, (mask, sizes, r.stdout)
        return int(r.stdout)

    return run


@pytest.mark.parametrize("mask", [3, 7, 15, 255])
def test_groups_cover_every_particle_once(groups, mask):
    for first in (0, 1, 7, 8, 31, 32, 37):
        for size in (1, 8, 31, 32, 33, 62, 63, 64, 65, 95, 96, 127, 128, 255, 256, 257, 287, 288, 700):
            groups(mask, ([first] if first else []) + [size])
            groups(mask, ([first] if first else []) + [size, 1, size, 64, 3])
    rng = np.random.default_rng(1)
    for _ in range(60):
        groups(mask, np.maximum(1, (2.0 ** rng.uniform(0, 9.5, 40)).astype(int)).tolist())


def test_a_crowd_has_small_groups_and_other_cells_one(groups):
    assert groups(255, [8000]) == 250
    assert groups(255, [20] * 12) == 12  # within the first 256 particles


@pytest.mark.gpu
@pytest.mark.parametrize("profile", [capi.PROFILE_BASELINE, capi.PROFILE_REF])
@pytest.mark.parametrize("n,side,obstacles", [(8064, 1, 0), (8101, 2, 3), (9000, 3, 0), (16000, 4, 7)])
def test_crowds_have_the_bits_of_the_list_kernels(profile, n, side, obstacles, monkeypatch):
    rng = np.random.default_rng(n)
    parts = scenes.block((n, 1, 1), (0.0, 0.0, 0.0), n)
    parts["position"] = (rng.random(3 * n) * side * 0.1).astype(np.float32)
    parts["velocity"] = (rng.random(3 * n) - 0.5).astype(np.float32)
    parts["mass"] = (parts["mass"] * (0.5 + rng.random(n))).astype(np.float32)
    if obstacles:
        parts["type"][::obstacles] = capi.TYPE_OBSTACLE
    e = 0.1 * side
    cfg = scenes.config((0.0, 0.0, 0.0), (1.5 * e, e, e))
    got = []
    for lists in (False, True):
        if lists:
            monkeypatch.setenv("FGB_VERLET", "0")
        solver = SphSolver(params=capi.params(profile, 0.1))
        batch = Batch(solver, [(scenes.copy_particles(parts), cfg)])
        for _ in range(4):
            batch.step(1)
            batch.sync()
        got.append(batch.download(0))
        assert batch.error_flags() == 0
        batch.close()
        solver.close()
    for f in ("id", "position", "velocity", "colour"):
        assert got[0][f].tobytes() == got[1][f].tobytes(), f

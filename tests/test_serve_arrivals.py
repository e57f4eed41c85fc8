"""When a lone request waits for its successor (serve_arrivals.h): in a stream that the client
does not wait for, never for a client that takes its requests one after the other."""
import os
import subprocess
import time

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "serve_arrivals.h"
// each argument triple: time in ms, in turn (0/1), waited in vain (0/1); prints how long each waits, in ms
int main() {
    fgb::Arrivals a;
    double t;
    int in_turn, vain;
    while (scanf("%lf %d %d", &t, &in_turn, &vain) == 3) {
        a.arrived(t * 1e-3, in_turn);
        printf("%.3f ", (a.wait_until() - t * 1e-3) * 1e3);
        if (vain) a.in_vain();
    }
}
"""


@pytest.fixture(scope="module")
def waits(tmp_path_factory):
    d = tmp_path_factory.mktemp("arrivals")
    src, exe = d / "a.cpp", d / "a"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "libfluid_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)

    def run(arrivals):
        text = "".join("%g %d %d\n" % a for a in arrivals)
        out = subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True).stdout
        return [float(x) for x in out.split()]

    return run


def test_a_sequential_client_never_waits(waits):
    assert waits([(k * 1.0, 1, 0) for k in range(6)]) == [0] * 6


def test_a_stream_waits_from_its_third_request(waits):
    assert waits([(k * 2.0, 0, 0) for k in range(5)]) == [0, 0, 2.5, 2.5, 2.5]


def test_requests_far_apart_never_wait(waits):
    assert waits([(k * 4.0, 0, 0) for k in range(5)]) == [0] * 5
    assert waits([(0, 0, 0), (2, 0, 0), (50, 0, 0), (52, 0, 0)]) == [0] * 4


def test_a_wait_in_vain_is_not_repeated_at_once(waits):
    assert waits([(0, 0, 0), (2, 0, 0), (4, 0, 1), (7, 0, 0), (9, 0, 0), (11, 0, 0)]) == [0, 0, 2.5, 0, 2.5, 2.5]


@pytest.mark.gpu
@pytest.mark.parametrize("ask", ["poll", "drain", "stats"])
def test_a_sequential_client_is_admitted_at_once(ask):
    from libfluid_gb300 import capi, scenes
    from libfluid_gb300.serve import Server
    from libfluid_gb300.solver import SphSolver

    solver = SphSolver(params=capi.params(capi.PROFILE_BASELINE, 0.1))
    parts, cfg = scenes.cube_scene(4096, 3)
    sv = Server(solver)
    tickets = []
    for k in range(24):
        tickets.append(sv.submit(cfg, parts, 2))
        if ask == "drain":
            sv.drain(60)
            continue
        end = time.time() + 60
        while time.time() < end:
            if ask == "poll" and sv.poll(tickets[-1]).status == capi.SERVE_DONE:
                break
            if ask == "stats" and sv.stats().completed > k:
                break
    seen = [sv.poll(t) for t in tickets]
    assert all(r.status == capi.SERVE_DONE for r in seen)
    sv.close()
    solver.close()
    # a wait for a successor would be 1.25 times the gap between two requests, milliseconds
    assert np.median([r.t_admit - r.t_submit for r in seen[4:]]) < 0.001

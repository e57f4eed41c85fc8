"""The pair sums' shared root and quotient (pbf_sums.cuh: root_and_spiky) give the bits of
the IEEE square root and division.

On the CPU: the mantissas whose reciprocals lie near the midpoint of two floats, which the
host checks one by one for the solver's h, are all of them.  On the GPU: every float of the
range is put through the device function wherever the host lets a solver take it."""
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "libfluid_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "fast_root.h"
#include "pbf_sums.cuh"
using namespace fgb;
__global__ void check(Phys ph, uint32_t lo, uint32_t hi, unsigned long long *bad) {
    unsigned long long wrong = 0;
    for (uint64_t i = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= hi; i += (uint64_t)gridDim.x * blockDim.x) {
        const float q = __uint_as_float((uint32_t)i);
        Two r, s, r0, s0;
        root_and_spiky<true>(ph, Two(q, q), r, s);
        root_and_spiky<false>(ph, Two(q, q), r0, s0);
        wrong += r.lo() != r0.lo() || r.hi() != r0.hi() || s.lo() != s0.lo() || s.hi() != s0.hi();
    }
    if (wrong) atomicAdd(bad, wrong);
}
int main(int, char **v) {
    Phys ph{};
    ph.h = (float)atof(v[1]);
    ph.corr_n = 4.f;
    ph.rho0 = 1000.f;
    ph.corr_ref = 3.f;
    ph.profile = kRef;
    const float first = 1e-16f, last = ph.h * ph.h;
    uint32_t lo, hi;
    memcpy(&lo, &first, 4);
    memcpy(&hi, &last, 4);
    unsigned long long *d, bad = 1;
    cudaMalloc(&d, 8);
    cudaMemset(d, 0, 8);
    check<<<152 * 8, 256>>>(ph, lo, hi, d);
    cudaMemcpy(&bad, d, 8, cudaMemcpyDeviceToHost);
    printf("%d %u %llu\n", fast_root_exact(ph) ? 1 : 0, hi - lo, cudaGetLastError() == cudaSuccess ? bad : ~0ull);
}
"""


def _listed():
    src = open(os.path.join(CSRC, "fast_root.h")).read()
    body = src[src.index("kNearTieReciprocals[] = {"):]
    return [int(x, 16) for x in re.findall(r"0x[0-9a-f]{6}", body[:body.index("};")])]


def test_near_tie_reciprocals_are_complete():
    # r = m / 2^23, m in [2^23, 2^24): 1 / r in units of half an ulp is 2^48 / m, and a
    # midpoint an odd integer
    m = np.arange(1 << 23, 1 << 24, dtype=np.uint64)
    whole, rest = np.divmod(np.uint64(1 << 48), m)
    near = np.where(whole & np.uint64(1), rest, m - rest).astype(np.float64) / m
    rel = near / ((1 << 48) / m.astype(np.float64))
    want = np.nonzero(rel < 2.0 ** -43)[0]
    assert sorted(_listed()) == want.tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("h", ["0.1", "0.0078125001", "0.37", "7.7"])
def test_every_root_and_quotient_has_the_ieee_bits(h, tmp_path):
    from libfluid_gb300 import build
    src, exe = tmp_path / "root.cu", tmp_path / "root"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-I" + CSRC, str(src), "-o", str(exe)],
                   check=True)
    taken, count, bad = (int(x) for x in subprocess.run([str(exe), h], check=True, capture_output=True, text=True).stdout.split())
    assert count > 1 << 26
    # the shortest h is a power of two (as a float), where some quotients do not come out:
    # the host leaves such a solver to the IEEE functions
    assert taken == (np.log2(np.float32(h)) % 1 != 0)
    assert bad == 0 or not taken

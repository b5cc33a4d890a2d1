"""The status that a record of a cell gives a pass (ahead_status), against the
pass itself: the neighbours clipped one by one under its caps.  The records'
function is compiled for the host."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
VERTEX, PLANE, RADIUS, SUCCESS, TRIANGLES = 0, 1, 3, 4, 8
LEVELS, NONE = 6, 255

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
using std::max;
using std::min;
#include "cell.cuh"
int main() {
  rpd::AheadRecord r{};
  int need, ntri, K, T, lP, lV, p;
  while (std::scanf("%d %d %d %d %d %d", &need, &ntri, &K, &T, &lP, &lV) == 6) {
    r.need = (unsigned short)need;
    r.ntri = (unsigned short)ntri;
    for (unsigned char *a : {r.jP, r.jV})
      for (int k = 0; k < rpd::kAheadLevels; ++k) {
        if (std::scanf("%d", &p) != 1) return 1;
        a[k] = (unsigned char)p;
      }
    std::printf("%d\n", rpd::ahead_status(r, K, T, lP, lV));
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def status(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("ahead")
    src, exe = d / "ahead.cpp", d / "ahead"
    src.write_text(PROGRAM)
    inc = os.path.join(ROOT, "gpu-restricted-power-diagrams_b200", "csrc")
    subprocess.run([cxx, "-std=c++17", "-I", inc, "-I", os.path.join(CUDA, "include"), str(src), "-o", str(exe)], check=True)

    def run(rows):
        text = "\n".join(" ".join(map(str, r)) for r in rows) + "\n"
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
        return [int(x) for x in out.split()]

    return run


def one_pass(cuts, need, ntri, K, P, V, T):
    """cuts: neighbour -> vertices after its cut; the cell is finished by
    neighbour need - 1."""
    planes = 6
    for i in range(K):
        if planes >= P:
            return PLANE
        if i in cuts:
            if cuts[i] > V:
                return VERTEX
            planes += 1
        if i == need - 1:
            return TRIANGLES if ntri > T else SUCCESS
    return RADIUS


def ladder(P, V):
    out = []
    for _ in range(LEVELS):
        out.append((P, V))
        P, V = int(P * 1.5), min(int(V * 1.5), 256)
    return out


def test_first_pass_records(status):
    """Records as a first pass that clips past its caps writes them."""
    rng = random.Random(1)
    rows, want = [], []
    for _ in range(4000):
        need = rng.randint(1, 200)
        cuts, v = {}, 8
        for i in range(need):
            if rng.random() < 0.25:
                v = max(4, v + rng.randint(-4, 4))
                cuts[i] = v
        lad = ladder(rng.randint(7, 30), rng.randint(8, 32))
        jP, jV, planes = [NONE] * LEVELS, [NONE] * LEVELS, 6
        for i in sorted(cuts):
            planes += 1
            for k, (P, V) in enumerate(lad):
                if jP[k] == NONE and planes >= P:
                    jP[k] = i + 1
                if jV[k] == NONE and cuts[i] > V:
                    jV[k] = i
        K, lP, lV = rng.randint(1, 200), rng.randrange(LEVELS), rng.randrange(LEVELS)
        rows.append([need, 0, K, 100, lP, lV] + jP + jV)
        want.append(one_pass(cuts, need, 0, K, lad[lP][0], lad[lV][1], 100))
    assert status(rows) == want


@pytest.mark.parametrize("need", [1, 171, 172, 254, 255, 256])
def test_retry_records(status, need):
    """Records of a retry pass, whose caps stop the cell nowhere, up to the
    longest neighbour list."""
    rows, want = [], []
    for K in (34, 76, 114, 171, 254, 255, 256):
        for ntri in (0, 101):
            for T in (100, 150):
                rows.append([need, ntri, K, T, 3, 7] + [NONE] * (2 * LEVELS))
                want.append(one_pass({}, need, ntri, K, 255, 256, T))
    assert status(rows) == want

"""Freed device blocks kept for reuse.  Beside a server's memory budget: when a
request is admitted, those that do not fit beside it are given back.  A
solver of a smaller size takes the blocks that a larger one left.  In a
process of its own, whose device memory is what it allocated."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MB = 1 << 20

HEAD = """
import numpy as np, rpd, sys
from cuda.bindings import runtime as rt
from rpd import synth

def pool_used():  # bytes that allocations hold of the device's memory pool, the kept blocks among them
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    err, used = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    return int(used)

ctx = rpd.Context(0)
"""

BUDGET = HEAD + """
s = rpd.Solver(ctx).set_points(synth.uniform(2_000_000, seed=1))
s.launch(K=70, P=30, V=40)
s.close()
print(pool_used())  # kept: the context is alive
x = synth.uniform(20_000, seed=2)
with rpd.Server(slots=2, mem_budget=int(sys.argv[1])) as sv:
    for _ in range(3):
        t, session = sv.solve(x, K=50, P=30, V=40)
        assert np.isfinite(sv.wait(t)[0]).all()
        print(pool_used())
    print(sv.bytes_in_use())
"""

SMALLER = HEAD + """
grid = rpd.Grid.cube(40)
def solve(n):
    s = rpd.Solver(ctx).set_points(synth.uniform(n, seed=n)).set_grid(grid)
    s.launch(K=50, P=30, V=40)
    return s
solve(300_000).close()
print(pool_used())
for n in (290_000, 250_000, 200_000):
    s = solve(n)
    print(pool_used())
    s.close()
"""


def run(program, *args):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "gpu-restricted-power-diagrams_b200"))
    out = subprocess.run([sys.executable, "-c", program, *map(str, args)], env=env, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr
    return [int(v) for v in out.stdout.split()]


@pytest.mark.parametrize("budget", [128 * MB, 512 * MB])
def test_kept_blocks_within_the_budget(budget):
    kept, *held = run(BUDGET, budget)
    assert kept > 700 * MB
    assert max(held) <= budget


def test_smaller_solvers_take_kept_blocks():
    first, *then = run(SMALLER)
    assert first > 200 * MB
    assert max(then) <= first + first // 50

"""Freed device blocks handed out again by size class: solvers of many sizes
made and dropped by several threads, each with its own context, give the bits
that a solver gives alone, also after the last context is gone and a new one
is made."""
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rpd():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import rpd as m

    return m


SIZES = [1, 33, 700, 4095, 4096, 9000, 30000]


def solve(rpd, ctx, n):
    from rpd import synth

    s = rpd.Solver(ctx).set_points(synth.uniform(n, seed=n))
    s.set_grid_blob(36, 5, 2)
    s.launch(K=30, P=30, V=40, T=40)
    return s.status(), s.moments()


@pytest.mark.parametrize("threads", [1, 4])
def test_blocks_reused_across_solvers(rpd, threads):
    ctx = rpd.Context(0)
    want = {n: solve(rpd, ctx, n) for n in SIZES}
    del ctx
    gc.collect()
    bad = []

    def work(k):
        try:
            c = rpd.Context(0)
            order = np.random.default_rng(k).permutation(SIZES * 3)
            for n in order:
                st, m = solve(rpd, c, int(n))
                if not (np.array_equal(st, want[n][0]) and np.array_equal(m, want[n][1])):
                    bad.append((k, int(n)))
        except Exception as e:  # shown by the assertion below
            bad.append((k, repr(e)))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad

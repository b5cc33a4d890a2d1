"""Batched solves of tiny diagrams, whose cells' neighbour lists end before
their security radius, against single solves: status, moments and pass
schedule.  A larger diagram beside them makes the batch one that records
cells."""
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


def result(s):
    """Status, moments and pass schedule; the solver is closed."""
    out = s.status(), s.moments(), [(p["cells"], p["K"], p["P"], p["V"], p["T"]) for p in s.stats()["passes"]]
    s.close()
    return out


def equal(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2]


@pytest.mark.parametrize("extra", [1, 5])
@pytest.mark.parametrize("n", [8, 12, 16, 21, 27, 33, 47])
def test_batch_of_tiny_diagrams(rpd, n, extra):
    from rpd import synth

    ctx = rpd.Context(0)
    caps = [(K, P) for K in range(5, 25, 2) for P in (9, 11, 13, 14, 16, 18, 20, 24, 32)]
    xs = [synth.uniform(n, seed=100 * n + i) for i in range(len(caps))] + [synth.uniform(5000, seed=1)]
    par = [rpd.Params.default(K=K, P=P, V=64, T=100, max_extra_passes=extra) for K, P in caps + [(20, 25)]]
    solvers = [rpd.Solver(ctx).set_points(x) for x in xs]
    batch = rpd.Batch(solvers, par, ctx)
    batch.launch()
    batch.close()
    got = [result(s) for s in solvers]
    want = []
    for x, p in zip(xs, par):
        s = rpd.Solver(ctx).set_points(x)
        s.launch(p)
        want.append(result(s))
    bad = [c for c, a, b in zip(caps, got, want) if not equal(a, b)]
    assert not bad

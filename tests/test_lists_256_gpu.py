"""Neighbour lists of up to 256, settled from records of the pass before,
against launches that collect counters (which clip every pass again)."""
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


@pytest.mark.parametrize("n,K", [(256, 34), (256, 51), (256, 76), (256, 114), (257, 76), (255, 114), (3000, 76),
                                 (3000, 114)])
@pytest.mark.parametrize("domain", ["box", "cube"])
def test_lists_of_256(rpd, n, K, domain):
    """Schedules of 171 and 256 neighbours; the hull cells of one cluster
    reach across the box and need nearly all of the seeds."""
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = 500 + np.random.default_rng(n).normal(0, 30, (n, 3))
    ctx = rpd.Context(0)
    out = []
    for flags in (0, rpd.FLAG_COUNTERS):
        s = rpd.Solver(ctx).set_points(x)
        if domain == "cube":
            s.set_grid(rpd.Grid.cube(20))
        s.launch(K=K, P=60, V=100, T=3000, flags=flags | rpd.FLAG_NO_T_AHEAD)
        out.append(result(s))
    assert equal(*out)

"""Clipping with eight lanes per cell against the warp-per-cell kernel
(launches with work counters use the latter): the same statuses, pass
schedule and moments bit for bit, at the edges of the octets' caps (32 and 48
planes, 32 and 64 vertices), of the rows that fill a block, and with walls,
ties and domains."""
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


def seeds(n, kind, seed=3):
    from rpd import synth

    if kind == "lattice":  # exact ties between neighbours
        m = int(round(n ** (1 / 3)))
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
        x = np.zeros((m**3, 4), np.float32)
        x[:, :3] = (g + 0.5) * (1000.0 / m)
        return x
    x = synth.uniform(n, seed=seed)
    h2 = n ** (-2 / 3) * 1e6
    x[:, 3] = np.random.default_rng(seed).uniform(0, 0.1 * h2, n)
    if kind == "walls":
        x[::7, 3] = -200000.0
    return x


def solve(rpd, x, domain, flags=0, **kw):
    s = rpd.Solver().set_points(x)
    if domain == "cube":
        s.set_grid(rpd.Grid.cube(30))
    elif domain == "blob":
        s.set_grid_blob(40, 5, 2)
    s.launch(flags=flags, **kw)
    st = s.stats()
    return s.status(), s.moments(), [(p["cells"], p["K"], p["P"], p["V"], p["T"]) for p in st["passes"]]


CASES = [
    (4096, "uniform", "box", 50, 30, 40), (4097, "uniform", "cube", 50, 32, 32), (5003, "uniform", "blob", 50, 33, 33),
    (6001, "uniform", "blob", 9, 9, 12), (6001, "uniform", "cube", 90, 47, 64), (6001, "uniform", "box", 90, 48, 65),
    (6001, "uniform", "cube", 90, 49, 100), (4913, "lattice", "box", 50, 40, 60), (4913, "lattice", "cube", 33, 25, 30),
    (8009, "walls", "blob", 50, 30, 40), (20011, "uniform", "blob", 20, 16, 24),
]


@pytest.mark.parametrize("n,kind,domain,K,P,V", CASES)
def test_octet_equals_warp(rpd, n, kind, domain, K, P, V):
    x = seeds(n, kind)
    a = solve(rpd, x, domain, rpd.FLAG_NO_T_AHEAD, K=K, P=P, V=V)
    b = solve(rpd, x, domain, rpd.FLAG_NO_T_AHEAD | rpd.FLAG_COUNTERS, K=K, P=P, V=V)
    assert np.array_equal(a[0], b[0]) and a[2] == b[2]
    assert np.array_equal(a[1], b[1])

"""The neighbour search's selection from the 5x5x5 bins and its hand-over to
the shell scan, against the oracle's exact lists: K at the edges of the sorted
slots, grids of few bins, bins past the candidate registers, and exact ties
across the threshold."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rpd():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import rpd as m

    return m


def seeds(kind, n):
    rng = np.random.default_rng(n)
    x = np.zeros((n, 4), np.float32)
    if kind == "ties":
        m = int(round(n ** (1 / 3)))
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
        x = np.zeros((m**3, 4), np.float32)
        x[:, :3] = (g + 0.5) * (1000.0 / m)
    elif kind == "clusters":
        c = rng.random((8, 3)) * 1000
        x[:, :3] = np.clip(c[rng.integers(8, size=n)] + rng.normal(0, 30, (n, 3)), 0, 999.9)
    else:
        x[:, :3] = rng.random((n, 3)) * 1000
    return x


@pytest.mark.parametrize("kind,n", [("uniform", 60), ("uniform", 200), ("uniform", 3000), ("uniform", 20000),
                                    ("clusters", 4000), ("ties", 8000)])
@pytest.mark.parametrize("K", [1, 13, 31, 32, 33, 63, 64, 65, 95, 96, 97])
def test_select_bitexact(rpd, kind, n, K):
    x = seeds(kind, n)
    got = rpd.Solver(rpd.Context(0)).set_points(x).knn(K)
    assert np.array_equal(got, oracle.knn(x.astype(np.float64), K, knn_mode=1))

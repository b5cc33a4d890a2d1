"""The neighbour search's selection from the 5x5x5 bins where its bounds are
close: seeds exactly on the faces of bins (exact ties, and distances that
round to the bound), near and past the box's faces, and grids of so few bins
that the block has none beyond; against the oracle's exact lists."""
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
    if kind == "faces":  # 10 bins of 100 for 3,100 seeds
        x[:, :3] = rng.integers(0, 31, (n, 3)) * np.float32(100 / 3)
        x = np.unique(x, axis=0)
    elif kind == "outside":
        x[:, :3] = rng.uniform(-20, 1020, (n, 3))
    else:
        x[:, :3] = rng.random((n, 3)) * 1000
    return x


@pytest.mark.parametrize("kind,n", [("faces", 3100), ("faces", 900), ("outside", 3000), ("uniform", 150), ("uniform", 420),
                                    ("uniform", 1200)])
@pytest.mark.parametrize("K", [5, 6, 7, 8, 12, 20, 33, 50, 80, 95, 96])
def test_bounds_bitexact(rpd, kind, n, K):
    x = seeds(kind, n)
    got = rpd.Solver(rpd.Context(0)).set_points(x).knn(K)
    assert np.array_equal(got, oracle.knn(x.astype(np.float64), K, knn_mode=1))

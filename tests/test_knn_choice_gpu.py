"""The neighbour-search variant chosen for a search depends on its own rows,
not on the size that a context searched first: K and sizes where a warp or a
thread per seed is faster by far."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WARP, THREAD = 0, 1


@pytest.fixture(scope="module")
def rpd():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import rpd as m

    return m


# uniform seeds, warp / thread: K 8, 0.08 / 0.13 ms for 32K seeds and 2.3 / 0.7
# for 1M; K 12, 0.08 / 0.14 and 2.1 / 0.9
@pytest.mark.parametrize("K", [8, 12])
@pytest.mark.parametrize("sizes", [[(32_000, WARP), (1_000_000, THREAD)], [(1_000_000, THREAD), (32_000, WARP)],
                                   [(32_000, WARP), (40_000, WARP)]])
def test_choice_by_rows(rpd, K, sizes):
    from rpd import synth

    ctx = rpd.Context(0)
    for n, want in sizes:
        x = synth.uniform(n, seed=n)
        s = rpd.Solver(ctx).set_points(x)
        first, again = s.knn(K), s.knn(K)
        s.close()
        assert np.array_equal(first, again)  # the trial's own lists, then the choice's
        assert ctx.knn_variant(K) == want

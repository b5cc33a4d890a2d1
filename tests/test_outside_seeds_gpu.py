"""Seeds outside the box of the domain: the statuses and moments of launches
that clip with a warp per cell (with work counters), where the cells may end
empty but are proven outside the domain before."""
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


@pytest.mark.parametrize("n,size,K,P,V", [(4200, 21, 200, 60, 120), (6000, 37, 50, 60, 120), (9000, 30, 20, 60, 120),
                                          (8600, 8, 171, 120, 8)])
@pytest.mark.parametrize("how", ["launch", "batch"])
def test_seeds_outside_the_box(rpd, n, size, K, P, V, how):
    ctx = rpd.Context(0)
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = np.random.default_rng(n).uniform(-40, 1040, (n, 3))
    kw = dict(K=K, P=P, V=V, T=60)
    out = []
    for flags in (rpd.FLAG_NO_T_AHEAD, rpd.FLAG_NO_T_AHEAD | rpd.FLAG_COUNTERS):
        s = rpd.Solver(ctx).set_points(x).set_grid_blob(size, 5, 2)
        if how == "batch" and not flags & rpd.FLAG_COUNTERS:
            b = rpd.Batch([s], rpd.Params.default(flags=flags, **kw), ctx)
            b.launch()
            b.close()
        else:
            s.launch(flags=flags, **kw)
        out.append((s.status(), s.moments()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])

"""Triangle overflows settled ahead in the retry passes too: statuses and
moments of RPD_FLAG_NO_T_AHEAD launches bit for bit, single and batched, with
domains whose cells hold many times T triangles."""
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


@pytest.mark.parametrize("n,K,P,V,T,size", [(3000, 20, 16, 24, 20, 40), (3000, 50, 30, 40, 60, 64),
                                            (9000, 33, 20, 28, 16, 60), (700, 90, 60, 80, 100, 50)])
def test_settled_ahead_in_every_pass(rpd, n, K, P, V, T, size):
    from rpd import synth

    x = synth.uniform(n, seed=8)
    ctx = rpd.Context(0)
    out, cells = [], []
    for flags in (0, rpd.FLAG_NO_T_AHEAD):
        s = rpd.Solver(ctx).set_points(x).set_grid_blob(size, 5, 2)
        s.launch(K=K, P=P, V=V, T=T, flags=flags)
        out.append((s.status(), s.moments()))
        cells.append(sum(p["cells"] for p in s.stats()["passes"]))
    b = rpd.Solver(ctx).set_points(x).set_grid_blob(size, 5, 2)
    rpd.Batch([b], rpd.Params.default(K=K, P=P, V=V, T=T), ctx).launch()
    out.append((b.status(), b.moments()))
    assert cells[0] < cells[1]
    for st, m in out[1:]:
        assert np.array_equal(st, out[0][0])
        assert np.array_equal(m, out[0][1])

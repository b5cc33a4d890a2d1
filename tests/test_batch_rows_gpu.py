"""Batched launches of few rows clip with a warp per cell, of more with eight
lanes: batches whose rows in all lie on either side of the line, and whose
retry passes do, against single solves."""
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


# rows of the batch, and first-pass caps: K 12 leaves most cells to the second
# pass (more and fewer than 4,096 rows), K 60 few
@pytest.mark.parametrize("sizes", [(700, 300), (2000, 2095), (2000, 2096), (2000, 2097), (9000, 400), (6000, 6000)])
@pytest.mark.parametrize("domains", ["box", "blob", "both"])
@pytest.mark.parametrize("K,P,V,rows", [(12, 30, 40, 0), (60, 30, 40, 0), (60, 20, 28, 0), (33, 30, 40, 30)])
def test_batch_equals_single(rpd, sizes, domains, K, P, V, rows):
    from rpd import synth

    ctx = rpd.Context(0)
    kw = dict(K=K, P=P, V=V, T=40)
    if rows:
        kw.update(hessian_h=rows, hessian_hc=1)

    def solver(i, n):
        x = synth.uniform(n, seed=n + i)
        x[:, 3] = np.random.default_rng(i).uniform(0, 0.1 * n ** (-2 / 3) * 1e6, n)
        s = rpd.Solver(ctx).set_points(x)
        if domains == "blob" or (domains == "both" and i == 0):
            s.set_grid_blob(30, 5, 2)
        return s

    def result(s):
        out = [s.status(), s.moments()]
        if rows:
            out += list(s.hessian(rows, 1))
        sched = [(p["cells"], p["K"], p["P"], p["V"], p["T"]) for p in s.stats()["passes"]]
        s.close()
        return out, sched

    batch = [solver(i, n) for i, n in enumerate(sizes)]
    b = rpd.Batch(batch, rpd.Params.default(**kw), ctx)
    b.launch()
    b.close()
    for i, s in enumerate(batch):
        got, sched = result(s)
        alone = solver(i, sizes[i])
        alone.launch(rpd.Params.default(**kw))
        want, sched1 = result(alone)
        assert sched == sched1
        for u, v in zip(got, want):
            assert np.array_equal(u, v)

"""Retry passes of few cells clip with the next pass's K and restrict up to
the last pass's T; the passes after them settle the cells from records.
Against launches that collect counters (every pass clips again): the same
statuses and moments bit for bit, and without triangle overflows settled
ahead the same pass schedule; where the schedule ends before a cell's need,
for lists at and above one block's size, and mixed precision."""
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


@pytest.mark.parametrize("n", [1, 40, 1500, 4096, 4097, 9000])
@pytest.mark.parametrize("domain", ["box", "cube", "blob"])
@pytest.mark.parametrize("K,P,V,T,extra", [(30, 30, 40, 20, 5), (8, 30, 40, 8, 5), (12, 14, 20, 8, 3), (40, 30, 40, 30, 2),
                                           (8, 20, 30, 20, 1), (180, 30, 40, 40, 5)])
def test_retry_records_equal_passes(rpd, n, domain, K, P, V, T, extra):
    from rpd import synth

    x = synth.uniform(n, seed=n)
    x[:, 3] = np.random.default_rng(n).uniform(0, 0.2 * n ** (-2 / 3) * 1e6, n)
    ctx = rpd.Context(0)
    for flags in (0, rpd.FLAG_NO_T_AHEAD):
        out = []
        for more in (0, rpd.FLAG_COUNTERS):
            s = rpd.Solver(ctx).set_points(x)
            if domain == "cube":
                s.set_grid(rpd.Grid.cube(12))
            elif domain == "blob":
                s.set_grid_blob(36, 5, 2)
            s.launch(K=K, P=P, V=V, T=T, max_extra_passes=extra, flags=flags | more)
            out.append((s.status(), s.moments(), [[p[k] for k in "KPVT"] + [p["cells"]] for p in s.stats()["passes"]]))
        (s0, m0, p0), (s1, m1, p1) = out
        assert np.array_equal(s0, s1) and np.array_equal(m0, m1)
        if flags:
            assert p0 == p1


def test_retry_records_mixed_precision(rpd):
    from rpd import synth

    x = synth.uniform(6000, seed=3)
    ctx = rpd.Context(0)
    out = []
    for more in (0, rpd.FLAG_COUNTERS):
        s = rpd.Solver(ctx).set_points(x)
        s.set_grid_blob(36, 5, 2)
        s.launch(K=24, P=30, V=40, T=20, precision=rpd.PRECISION_MIXED, flags=rpd.FLAG_NO_T_AHEAD | more)
        out.append((s.status(), s.moments()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])

"""Cells clipped past the first pass's caps and settled from their records,
against launches that collect counters (which clip every pass again): the
same statuses, pass schedule and moments bit for bit, where K, P and V each
stop the cells first, where the schedule ends before a cell's need, and for
batches."""
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


def seeds(kind, n):
    from rpd import synth

    if kind == "lattice":
        return synth.jittered_lattice(int(round(n ** (1 / 3))), seed=5)
    x = synth.uniform(n, seed=6)
    x[:, 3] = np.random.default_rng(1).uniform(0, 0.1 * n ** (-2 / 3) * 1e6, n)
    return x


@pytest.mark.parametrize("kind", ["uniform", "lattice"])
@pytest.mark.parametrize("domain", ["box", "cube", "blob"])
@pytest.mark.parametrize("K,P,V,extra", [(20, 25, 30, 5), (8, 30, 40, 5), (24, 9, 64, 5), (50, 40, 12, 5),
                                         (20, 12, 14, 1), (14, 48, 32, 2), (70, 10, 9, 5)])
def test_clip_ahead_equals_passes(rpd, kind, domain, K, P, V, extra):
    x = seeds(kind, 6000)
    ctx = rpd.Context(0)

    def solver():
        s = rpd.Solver(ctx).set_points(x)
        if domain == "cube":
            s.set_grid(rpd.Grid.cube(30))
        elif domain == "blob":
            s.set_grid_blob(36, 5, 2)
        return s

    kw = dict(K=K, P=P, V=V, T=60, max_extra_passes=extra)
    out = []
    for flags in (0, rpd.FLAG_COUNTERS):
        s = solver()
        s.launch(flags=flags | rpd.FLAG_NO_T_AHEAD, **kw)
        out.append((s.status(), s.moments(), [(p["cells"], p["K"], p["P"], p["V"], p["T"]) for p in s.stats()["passes"]]))
    (s0, m0, p0), (s1, m1, p1) = out
    assert p0 == p1 and np.array_equal(s0, s1) and np.array_equal(m0, m1)
    b = solver()
    rpd.Batch([b], rpd.Params.default(flags=rpd.FLAG_NO_T_AHEAD, **kw), ctx).launch()
    assert np.array_equal(b.status(), s0) and np.array_equal(b.moments(), m0)

"""A kept neighbour table whose rows are longer than a launch needs serves it
too: launches with and without Hessian rows by turns at a small K, whose first
passes hold 20 and 48 neighbours per row, search once; the results are those
of launches that search afresh."""
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


@pytest.mark.parametrize("domain", ["box", "cube"])
def test_rows_by_turns_search_once(rpd, domain):
    from rpd import synth

    s = rpd.Solver(rpd.Context(0)).set_points(synth.uniform(8000, seed=3))
    if domain == "cube":
        s.set_grid(rpd.Grid.cube(24))
    plain, rows = dict(K=20, P=25, V=30), dict(K=20, P=25, V=30, hessian_h=20, hessian_hc=1)

    def launch(kw, flags=0):
        s.launch(flags=flags, **kw)
        out = [s.status(), s.moments()]
        if "hessian_h" in kw:
            out += list(s.hessian(20, 1))
        return s.stats()["kernel_launches"], out

    launch(plain)
    for kw in (rows, plain, rows):
        kept, got = launch(kw)
        fresh, want = launch(kw, rpd.FLAG_FRESH_NEIGHBOURS)
        launch(plain)  # the table that the turns leave
        assert kept == fresh - 1
        for u, v in zip(got, want):
            assert np.array_equal(u, v)

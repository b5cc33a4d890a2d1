"""Launches whose every cell goes on in a warp after the clipping (Hessian
rows, used cells) have a record for each: none is clipped a second time, which
would take one launch more."""
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


OPTIONS = [("box", dict(hessian_h=30, hessian_hc=1)), ("cube", dict(hessian_h=30, hessian_hc=4)),
           ("cube", dict(keep_distance=0, keep_volume=1.0))]


@pytest.mark.parametrize("domain,options", OPTIONS)
def test_no_cell_is_clipped_twice(rpd, domain, options):
    from rpd import synth

    ctx = rpd.Context(0)
    launches, out = [], []
    # 130K cells are more than the records of a launch with boundary cells only
    for m, flags in ((40, 0), (51, 0), (51, rpd.FLAG_SAFE_RADIUS)):
        s = rpd.Solver(ctx).set_points(synth.jittered_lattice(m, seed=5, weights=False))
        if domain == "cube":
            s.set_grid(rpd.Grid.cube(m))
        s.launch(K=50, P=30, V=40, T=100, flags=rpd.FLAG_FIRST_PASS_ONLY | flags, **options)
        launches.append(s.stats()["kernel_launches"])
        out.append((s.status(), s.moments()))
        s.close()
    assert launches[0] == launches[1]
    # equal weights: the weighted security radius is the reference's, and its
    # launches clip with a warp per cell
    assert np.array_equal(out[1][0], out[2][0]) and np.array_equal(out[1][1], out[2][1])


def test_batch_with_rows(rpd):
    from rpd import synth

    ctx = rpd.Context(0)
    xs = [synth.jittered_lattice(m, seed=m, weights=False) for m in (44, 40, 12)]
    par = [rpd.Params.default(K=50, P=30, V=40, hessian_h=h, hessian_hc=1) for h in (30, 0, 30)]
    solvers = [rpd.Solver(ctx).set_points(x).set_grid(rpd.Grid.cube(24)) for x in xs]
    b = rpd.Batch(solvers, par, ctx)
    b.launch()
    b.close()
    for x, p, got in zip(xs, par, solvers):
        s = rpd.Solver(ctx).set_points(x).set_grid(rpd.Grid.cube(24))
        s.launch(p)
        assert np.array_equal(got.status(), s.status()) and np.array_equal(got.moments(), s.moments())
        if p.hessian_h:
            for u, v in zip(got.hessian(30, 1), s.hessian(30, 1)):
                assert np.array_equal(u, v)
        s.close()
        got.close()

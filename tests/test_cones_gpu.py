"""Facet pieces of the inner apex, eight lanes per triangle, against the
reference's cone clipping from its start corner: at layouts where the cone
work space changes size (planes 28, 56 and 57, 128 and more), with work items
of one to many triangles, parked and in the cell's own warp, and the facet
areas of the Hessian rows against the moments (the areas' divergence)."""
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


@pytest.mark.parametrize("P,V", [(25, 30), (28, 32), (32, 32), (56, 32), (57, 32), (76, 40), (128, 64), (200, 200)])
@pytest.mark.parametrize("size,domain", [(12, "blob"), (60, "blob"), (24, "cube")])
def test_inner_apex_equals_start_corner(rpd, P, V, size, domain):
    from rpd import synth

    x = synth.jittered_lattice(12, seed=4)
    out = []
    for flags in (0, rpd.FLAG_NO_DEFER, rpd.FLAG_REFERENCE_APEX):
        s = rpd.Solver().set_points(x)
        if domain == "cube":
            s.set_grid(rpd.Grid.cube(size))
        else:
            s.set_grid_blob(size, 5, 2)
        s.launch(K=60, P=P, V=V, T=700, flags=flags)
        out.append((s.status(), s.moments()))
    (s0, m0), (s1, m1), (s2, m2) = out
    # a cone of the start corner may overflow caps that the facet pieces do
    # not use; where every form succeeds the moments agree
    ok = (s0 == 4) & (s1 == 4) & (s2 == 4)
    assert ok.sum() > 0.9 * len(x) and np.array_equal(s0, s1)
    # a typical cell's mass is h^3 = 5.8e5; FP64 sums of up to ~700 pieces
    assert np.abs(m0[ok, 3] - m1[ok, 3]).max() <= 1e-12 * 5.8e5 * 700
    assert np.abs(m0[ok, 3] - m2[ok, 3]).max() <= 1e-12 * 5.8e5 * 700
    # moments: mass times the frame
    assert np.abs(m0[ok, :3] - m2[ok, :3]).max() <= 1e-12 * 5.8e8 * 700

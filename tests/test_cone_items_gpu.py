"""Parked cells that find no work items left run again with their cones in
their own warp: the bits of launches without parking.  Seeds on a diagonal,
whose cells' voxel ranges each hold most of the surface, with the cones of
the start corner, which take every triangle of the range."""
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


def diagonal(n):
    x = np.zeros((n, 4), np.float32)
    t = 200 + 600 * (np.arange(n) + 0.5) / n
    x[:, :3] = t[:, None] + np.random.default_rng(n).uniform(-0.2, 0.2, (n, 3)) * 600 / n
    return x


def field(S):
    """A rippled ball that holds the seeds."""
    g = np.linspace(0.0, 1.0, S + 1) - 0.5
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    return (np.sqrt(x * x + y * y + z * z) - 0.42 + 0.01 * np.sin(30 * x)).astype(np.float32)


@pytest.mark.parametrize("n,S,items", [(4, 12, "enough"), (60, 12, "too few"), (200, 12, "too few")])
@pytest.mark.parametrize("how", ["launch", "batch"])
def test_items_run_out(rpd, n, S, items, how):
    x = diagonal(n)
    ctx = rpd.Context(0)
    kw = dict(K=min(n + 10, 250), P=40, V=60, T=4096, max_extra_passes=0)
    out = []
    for flags in (rpd.FLAG_REFERENCE_APEX, rpd.FLAG_REFERENCE_APEX | rpd.FLAG_NO_DEFER):
        s = rpd.Solver(ctx).set_points(x)
        s.set_grid_field(field(S))
        if how == "batch":
            b = rpd.Batch([s], rpd.Params.default(flags=flags, **kw), ctx)
            b.launch()
            b.close()
        else:
            s.launch(flags=flags, **kw)
        out.append((s.status(), s.moments()))
        triangles = s.export_grid().info()[2]
        s.close()
    (s0, m0), (s1, m1) = out
    # a slab's voxel range holds at least half of the surface: the items of 8
    # triangles that the cells ask for, against the arrays' bound (T / 32 a cell)
    asked = (s0 == 4).sum() * (triangles // 2) // 8
    held = max(4096 // 32 * n, n + triangles)
    assert (asked > held) == (items == "too few"), (asked, held, triangles)
    assert (s0 == 4).sum() > 0 and np.array_equal(s0, s1) and np.array_equal(m0, m1)


def pool_used():
    from cuda.bindings import runtime as rt

    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    err, used = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    return int(used)


def test_items_take_less_than_their_cells(rpd):
    """A launch with room for 4,096 triangles a cell: the work items (40 bytes
    for 32 triangles, 5.1 KB a cell) beside the parked cells (20 KB) and the
    seeds' own arrays (under 0.6 KB).  Items for every triangle of every cell
    would take as much as the cells."""
    import gc

    from rpd import synth

    gc.collect()
    n = 400_000
    ctx = rpd.Context(0)
    before = pool_used()
    s = rpd.Solver(ctx).set_points(synth.uniform(n, seed=1)).set_grid(rpd.Grid.cube(32))
    s.launch(K=20, P=25, V=30, T=4096, max_extra_passes=0)
    used = pool_used() - before
    s.close()
    cells = n // 8 * (144 + 32 * 28 + 44 * 64 + 4 * 4096)
    assert used < 1.125 * (1.25 * cells + 600 * n)

"""Freed device blocks kept for reuse, beside a server's memory budget: when a
request is admitted, those that do not fit beside it are given back."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(scope="module")
def rpd():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import rpd as m

    return m


def pool_used():
    """Bytes that allocations hold of the device's memory pool, the kept
    blocks among them."""
    from cuda.bindings import runtime as rt

    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    err, used = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    return int(used)


@pytest.mark.parametrize("budget", [128, 512])
def test_kept_blocks_within_the_budget(rpd, budget):
    from rpd import synth

    gc.collect()
    ctx = rpd.Context(0)
    before = pool_used()
    s = rpd.Solver(ctx).set_points(synth.uniform(2_000_000, seed=1))
    s.launch(K=70, P=30, V=40)
    s.close()
    assert pool_used() - before > 700 * MB  # kept: the context is alive
    x = synth.uniform(20_000, seed=2)
    with rpd.Server(slots=2, mem_budget=budget * MB) as sv:
        for _ in range(3):
            t, session = sv.solve(x, K=50, P=30, V=40)
            assert np.isfinite(sv.wait(t)[0]).all()
            assert pool_used() - before <= budget * MB
        assert sv.bytes_in_use() <= budget * MB
    ctx.close()

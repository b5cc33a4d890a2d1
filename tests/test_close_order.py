"""Solvers and batches are destroyed before their context and once, also where
the garbage collector closes the context first (a reference cycle that holds
them all).  The library is a fake that records its calls; no GPU."""
import gc

import pytest

import rpd


class FakeLib:
    def __init__(self):
        self.calls, self.next = [], 1

    def __getattr__(self, name):
        def call(*args):
            if name.endswith("_create"):
                self.next += 1
                return self.next
            if name.endswith("_destroy"):
                self.calls.append((name, args[0]))
            return 0

        return call


@pytest.mark.parametrize("how", ["cycle", "context first", "solver first"])
def test_destroyed_in_order(monkeypatch, how):
    fake = FakeLib()
    monkeypatch.setattr(rpd, "lib", lambda: fake)
    ctx = rpd.Context(0)
    solvers = [rpd.Solver(ctx), rpd.Solver(ctx)]
    batch = rpd.Batch(solvers, rpd.Params(), ctx)
    want = {("rpd_context_destroy", ctx.h), ("rpd_batch_destroy", batch.h)} | {("rpd_solver_destroy", s.h) for s in solvers}
    if how == "context first":
        ctx.close()
    elif how == "solver first":
        solvers[0].close()
    node = [ctx, solvers, batch]
    node.append(node)
    del ctx, solvers, batch, node
    gc.collect()
    assert len(fake.calls) == len(want) and set(fake.calls) == want
    assert fake.calls[-1][0] == "rpd_context_destroy"

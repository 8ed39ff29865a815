"""Plan executions recorded into a caller's CUDA graph: the field's pair
records are never left to the graph, and executions of one plan that overlap on
several streams keep their own work units."""

from __future__ import annotations

import ctypes

import pytest

import giaoint_gb300 as gi
from giaoint_gb300 import _native as nat
from giaoint_gb300.plan import EriPlan

from helpers import molecule

pytestmark = pytest.mark.gpu


@pytest.fixture
def setup():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = nat.Context(0)

    def use(stream):
        nat.check(nat.lib().gx_context_set_stream(
            ctx.handle, ctypes.c_void_p(stream.cuda_stream) if stream is not None else None))

    yield torch, ctx, use
    torch.cuda.synchronize()
    use(None)


def _values(torch, ctx, basis, field, precision="fp64", quartets=None):
    plan = EriPlan(basis, quartets, context=ctx)
    out = torch.empty(plan.total, dtype=torch.complex128, device="cuda:0")
    plan.execute(out, field, precision=precision)
    plan.synchronize()
    return out


def test_new_field_under_capture_is_refused(setup):
    torch, ctx, use = setup
    _, basis = molecule(seed=7, natoms=2)
    first, second = gi.MagneticField((0.05, -0.1, 0.12)), gi.MagneticField((-0.15, 0.02, 0.08))
    plan = EriPlan(basis, context=ctx)
    out = torch.empty(plan.total, dtype=torch.complex128, device="cuda:0")
    plan.execute(out, first)
    plan.synchronize()
    ref = out.clone()
    stream = torch.cuda.Stream()
    use(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        with pytest.raises(RuntimeError, match="captured"):
            plan.execute(out, second)
        plan.execute(out, first)
    # what was refused left no trace: the second field is evaluated, not taken as evaluated
    plan.execute(out, second)
    plan.synchronize()
    other = nat.Context(0)
    fresh = gi.Basis(basis.shells)
    assert torch.equal(out, _values(torch, other, fresh, second))
    # and a replay evaluates the first field again once its records are back
    plan.execute(out, first)
    plan.synchronize()
    out.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)

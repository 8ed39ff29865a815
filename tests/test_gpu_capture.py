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


def test_replay_beside_eager_executions_of_the_same_plan(setup):
    """A captured execution has work units of its own: its replays on one stream and eager executions with
    another cutoff (other units) on a second one give what each gives alone."""
    torch, ctx, use = setup
    _, basis = molecule(seed=7, natoms=3)
    field = gi.MagneticField((0.05, -0.1, 0.12))
    plan = EriPlan(basis, context=ctx)
    outs = [torch.empty(plan.total, dtype=torch.complex128, device="cuda:0") for _ in range(2)]
    refs = []
    for out, precision in zip(outs, ("fp64", "mixed")):
        plan.execute(out, field, precision=precision)
        plan.synchronize()
        refs.append(out.clone())
    streams = [torch.cuda.Stream() for _ in range(2)]
    use(streams[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        plan.execute(outs[0], field, precision="fp64")
    use(streams[1])
    for _ in range(10):
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            graph.replay()
        plan.execute(outs[1], field, precision="mixed")
        torch.cuda.synchronize()
        for out, ref in zip(outs, refs):
            assert torch.equal(out, ref)


def test_one_plan_and_two_fields_on_alternating_streams(setup):
    """Executions on alternating streams without a wait between them, with the field (and so the pair records that
    all of them read) changing every second time."""
    torch, ctx, use = setup
    _, basis = molecule(seed=11, natoms=3)
    fields = [gi.MagneticField((0.05, -0.1, 0.12)), gi.MagneticField((-0.15, 0.02, 0.08))]
    plan = EriPlan(basis, context=ctx)
    refs = [_values(torch, ctx, basis, f) for f in fields]
    outs = [torch.zeros(plan.total, dtype=torch.complex128, device="cuda:0") for _ in range(8)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        use(streams[i % 2])
        plan.execute(out, fields[(i // 2) % 2])
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        assert torch.equal(out, refs[(i // 2) % 2]), i


def test_plans_on_two_streams_do_not_wait_for_each_other(setup):
    """A plan's execution finishes while another plan's is still queued behind a long kernel of its own stream.
    (One class, so that the launches are on that stream alone; streams can share a hardware queue: one of several
    suffices.)"""
    torch, ctx, use = setup
    _, basis = molecule(seed=7, natoms=2)
    field = gi.MagneticField((0.05, -0.1, 0.12))
    plans = [EriPlan(basis, [(0, 0, 0, 0)], context=ctx) for _ in range(2)]
    outs = [torch.empty(p.total, dtype=torch.complex128, device="cuda:0") for p in plans]
    streams = [torch.cuda.Stream() for _ in range(5)]
    overlapped = False
    for other in streams[1:]:
        for plan, out, stream in zip(plans, outs, (streams[0], other)):
            use(stream)
            plan.execute(out, field)
            plan.synchronize()
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(400_000_000)
        use(streams[0])
        plans[0].execute(outs[0], field)
        queued = torch.cuda.Event()
        queued.record(streams[0])
        use(other)
        plans[1].execute(outs[1], field)
        other.synchronize()
        overlapped = overlapped or not queued.query()
        torch.cuda.synchronize()
    assert overlapped
    assert torch.equal(outs[0], outs[1])

"""The launch count of a plan is the number of kernels that an execution enqueues, in every precision, before and
after tuning, and what a replayed graph holds."""

from __future__ import annotations

import ctypes

import pytest

import giaoint_gb300 as gi
from giaoint_gb300 import _native as nat
from giaoint_gb300 import synthetic as syn
from giaoint_gb300.plan import EriPlan

pytestmark = pytest.mark.gpu


def _kernels_captured(torch, ctx, run):
    """Kernel nodes of what `run` enqueues on a stream that is being captured."""
    cuda = ctypes.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    nat.check(nat.lib().gx_context_set_stream(ctx.handle, ctypes.c_void_p(stream.cuda_stream)))
    handle = ctypes.c_void_p(stream.cuda_stream)
    graph, count = ctypes.c_void_p(), ctypes.c_size_t()
    assert cuda.cuStreamBeginCapture_v2(handle, 1) == 0  # thread local
    try:
        run()
    finally:
        assert cuda.cuStreamEndCapture(handle, ctypes.byref(graph)) == 0
    assert cuda.cuGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cuda.cuGraphGetNodes(graph, nodes, ctypes.byref(count)) == 0
    kernels = 0
    for node in nodes:
        kind = ctypes.c_int()
        assert cuda.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kernels += kind.value == 0
    assert cuda.cuGraphDestroy(graph) == 0
    nat.check(nat.lib().gx_context_set_stream(ctx.handle, None))
    return kernels


@pytest.mark.parametrize("recipe", [((0, 2), (1, 1)), syn.MOLECULE_RECIPE, ((0, 1), (2, 1), (3, 1))])
@pytest.mark.parametrize("B", [(0.0, 0.0, 0.0), (0.05, -0.1, 0.12)])
def test_launches_are_the_kernels_enqueued(recipe, B):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = nat.Context(0)
    basis = gi.Basis([gi.Shell.from_record(r) for r in syn.random_molecule(3, natoms=3, box=5.0, recipe=recipe)])
    field = gi.MagneticField(B)
    plan = EriPlan(basis, context=ctx)
    before = plan.launches
    out = torch.empty(plan.total, dtype=torch.complex128, device="cuda:0")
    for i, precision in enumerate(("fp64", "mixed", "fp64_exact")):
        plan.execute(out, field, precision=precision)  # (buffers and pair records exist from here on)
        plan.synchronize()
        eager = plan.launches
        if i == 0 and any(B):
            assert before == eager
        assert _kernels_captured(torch, ctx, lambda: plan.execute(out, field, precision=precision)) == eager
        for _ in range(3):
            plan.execute(out, field, precision=precision)
        plan.synchronize()
        assert plan.launches == eager  # replayed
    plan.autotune(out, field, precision="mixed", repeats=1)
    plan.execute(out, field, precision="mixed")
    plan.synchronize()
    tuned = plan.launches
    assert _kernels_captured(torch, ctx, lambda: plan.execute(out, field, precision="mixed")) == tuned
    profile = plan.profile(out, field, precision="mixed")
    assert all(p["groups"] > 0 for p in profile)

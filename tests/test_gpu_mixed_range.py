"""Mixed precision: primitive quartets whose Hermite seeds leave the FP32 range are evaluated in FP64, whatever
their size (classes of total order 5 and up)."""

from __future__ import annotations

import math

import numpy as np
import pytest

import giaoint_gb300 as gi
from giaoint_gb300.plan import EriPlan

pytestmark = pytest.mark.gpu

# every entry is in the FP32 range of the screening
ALL_FP32 = 1.0e30


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _run(basis, field, precision, quartets=None, **kw):
    torch = _torch()
    plan = EriPlan(basis, quartets)
    out = torch.empty(plan.total, dtype=torch.complex128, device="cuda:0")
    plan.execute(out, field, precision=precision, **kw)
    plan.synchronize()
    return out.cpu().numpy(), plan.counts(), plan


@pytest.mark.parametrize("ls", [(2, 1, 1, 1), (2, 1, 2, 1), (2, 2, 2, 1), (2, 2, 2, 2), (2, 2, 3, 2), (2, 2, 3, 3)])
@pytest.mark.parametrize("apart", [0.0, 1.0e-3])
def test_one_tight_quartet(ls, apart):
    """One primitive quartet of exponent 1e5 a shell: its top seed is far above 1e25, so mixed precision gives the
    FP64 value (FP64 rounding of some hundred terms of the block's size)."""
    centers = [(0.1, -0.2, 0.3), (0.1, -0.2, 0.3 + apart)] * 2
    basis = gi.Basis([gi.Shell(c, l, [1.0e5], [1.0]) for c, l in zip(centers, ls)])
    field = gi.MagneticField((0.1, 0.05, -0.2)) if apart else None
    exact, _, _ = _run(basis, field, "fp64_exact", [(0, 1, 2, 3)])
    mixed, counts, _ = _run(basis, field, "mixed", [(0, 1, 2, 3)], mixed_cutoff=ALL_FP32)
    assert np.abs(mixed - exact).max() <= 1e-12 * np.abs(exact).max()
    assert (counts["fp64_quartets"], counts["fp32_quartets"]) == (1, 0)


def test_many_quartets_in_and_out_of_the_range():
    """A class with unit arrays (more than 512 shell quartets), uncontracted d shells from diffuse to tight on two
    near centres: every quartet whose top seed C (2 rho)^8 / 17 is above 1e25 comes out in FP64, others stay FP32."""
    exponents = [0.8, 8.0, 80.0, 3.0e3, 1.0e4, 3.0e4, 1.0e5, 3.0e5]
    centers = [(0.0, 0.0, 0.0) if i % 2 else (2.0e-4, 0.0, 1.0e-4) for i in range(len(exponents))]
    basis = gi.Basis([gi.Shell(c, 2, [e], [1.0]) for c, e in zip(centers, exponents)])
    field = gi.MagneticField((0.1, 0.05, -0.2))
    exact, _, plan = _run(basis, field, "fp64_exact")
    mixed, counts, _ = _run(basis, field, "mixed", mixed_cutoff=ALL_FP32)
    assert len(plan.quartets) > 512
    assert counts["fp64_quartets"] + counts["fp32_quartets"] == len(plan.quartets)
    assert counts["fp64_quartets"] > 0 and counts["fp32_quartets"] > 0

    def norm(a):  # radial part of the primitive normalisation, l = 2
        return (2.0 * a / math.pi) ** 0.75 * 4.0 * a

    out_of_range = 0
    for i, (a, b, c, d) in enumerate(plan.quartets):
        ea, eb, ec, ed = (exponents[k] for k in (a, b, c, d))
        p, q = ea + eb, ec + ed
        rho = p * q / (p + q)
        if rho * 5.0e-8 > 0.1:  # (then F_8 is no longer 1/17)
            continue
        pre = 2.0 * math.pi**2.5 / (p * q * math.sqrt(p + q)) * math.prod(norm(e) for e in (ea, eb, ec, ed))
        top = 0.5 * pre * (2.0 * rho) ** 8 / 17.0  # (0.5: the overlap factors of near centres, below this exponent)
        lo, hi = plan.offsets[i], plan.offsets[i + 1]
        error = np.abs(mixed[lo:hi] - exact[lo:hi]).max() / np.abs(exact[lo:hi]).max()
        if top >= 1.0e25:
            out_of_range += 1
            assert error <= 1e-12, (i, a, b, c, d, error)
        else:
            assert error <= 1e-3, (i, a, b, c, d, error)
    assert out_of_range > 50

"""Streamed Cholesky around the length (65,536 ordered pairs) up to which the
residual comes to the host with every reduction, and beyond it.  Every element
of the residual is bounded by its diagonal (Cauchy-Schwarz), so the factors
reproduce the integrals within the threshold, plus 1e-10 for rounding."""

from __future__ import annotations

import numpy as np
import pytest

import giaoint_gb300 as gi
from giaoint_gb300 import synthetic as syn
from giaoint_gb300.eri import _eri_batch

pytestmark = pytest.mark.gpu

THRESHOLD = 1e-3


@pytest.mark.parametrize("counts,functions", [((23, 12, 12, 8, 3), 256), ((20, 14, 12, 8, 3), 259)])
def test_factors_reproduce_integrals(counts, functions):
    basis = gi.Basis([gi.Shell.from_record(r) for r in syn.atom_even_tempered(counts, [0.05] * 5, ratio=1.7)])
    n = basis.ao_count
    assert n == functions
    chol = gi.cholesky_eri(basis, field=gi.MagneticField((0.0, 0.0, 0.1)), threshold=THRESHOLD)
    assert chol.max_residual_diagonal <= THRESHOLD
    first = np.concatenate([[0], np.cumsum([s.ao_count for s in basis.shells])])
    rng = np.random.default_rng(functions)
    q = rng.integers(0, len(basis.shells), (60, 4)).astype(np.uint32)
    q[:20, 2:] = q[:20, 1::-1]  # diagonal blocks among them
    _, shapes, offsets, values, _, _ = _eri_batch(basis, q)  # (one centre: the field's phases cancel)
    L = np.asarray(chol.vectors)
    for i, (a, b, c, d) in enumerate(q.astype(int)):
        left = L[:, first[a]:first[a + 1], first[b]:first[b + 1]]
        right = L[:, first[d]:first[d + 1], first[c]:first[c + 1]]
        got = np.einsum("pij,plk->ijkl", left, right.conj())
        want = values[offsets[i]:offsets[i + 1]].reshape(shapes[i])
        assert np.abs(got - want).max() <= THRESHOLD + 1e-10

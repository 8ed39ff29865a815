"""Default quartet list of the batch generators: the canonical quartets in the
reference's order, cut into runs of at most target_bytes (a larger block makes a
run of its own), against the plain enumeration."""

from __future__ import annotations

import sys
from itertools import product
from math import prod
from types import SimpleNamespace

import numpy as np
import pytest

import giaoint_gb300  # noqa: F401

eri = sys.modules["giaoint_gb300.eri"]


def _plain(sizes, element_bytes, target_bytes):
    runs, packed, held = [], [], 0
    for q in product(range(len(sizes)), repeat=4):
        a, b, c, d = q
        if min(q, (c, d, a, b), (b, a, d, c), (d, c, b, a)) != q:
            continue
        block = element_bytes * prod(sizes[i] for i in q)
        if packed and held + block > target_bytes:
            runs.append(packed)
            packed, held = [], 0
        packed.append(list(q))
        held += block
    return runs + [packed] if packed else runs


@pytest.mark.parametrize("target", [1, 16, 100, 5000, 77777, 10**6, 10**30])
@pytest.mark.parametrize("shells", [1, 2, 5, 9])
@pytest.mark.parametrize("element_bytes", [16, 192])
def test_runs(shells, target, element_bytes):
    sizes = [int(x) for x in np.random.default_rng(shells).choice([1, 3, 6, 10], shells)]
    basis = SimpleNamespace(shells=[SimpleNamespace(ao_count=n) for n in sizes])
    want = _plain(sizes, element_bytes, target)
    got = [np.asarray(r).tolist() for r in eri._packed_quartets(basis, None, element_bytes, target)]
    assert got == want
    listed = [q for r in want for q in r]
    assert [np.asarray(r).tolist() for r in eri._packed_quartets(basis, listed, element_bytes, target)] == want


def test_runs_over_several_enumerations():
    basis = SimpleNamespace(shells=[SimpleNamespace(ao_count=1)] * 40)
    runs = list(eri._packed_quartets(basis, None, 16, 100_000))
    assert all(len(r) == 6250 for r in runs[:-1])
    assert np.array_equal(np.concatenate(runs), eri.canonical_quartets(40))

"""Lane-per-quartet kernels (L <= 2 and lane-dense classes, and the real
arithmetic of q = 0 pairs in all of them) at the places where their unit cutting
and batching can go wrong: classes of one task, of 31 to 33 and of more than 512
tasks, contracted tasks that span batches, units without a survivor, general
contractions (strided blocks), and batches of every kind of pair.  FP64 within
1e-12 of the oracle (the bar of the FP64 path) and the same bits however the
quartet list is cut; mixed precision within 1e-10."""

from __future__ import annotations

import numpy as np
import pytest

import giaoint_gb300 as gi
from giaoint_gb300 import synthetic as syn
from giaoint_gb300.eri import _eri_batch

from helpers import basis_from_records

pytestmark = pytest.mark.gpu


def _records(seed, ls, nprims, centers, contractions=1, far=0.0):
    """One shell per (l, primitive count, centre index)."""
    rng = np.random.default_rng(seed)
    sites = rng.uniform(0.0, 2.5, (max(centers) + 1, 3))
    sites[-1] += far
    out = []
    for l, k, c in zip(ls, nprims, centers):
        e = np.exp(rng.uniform(np.log(0.2), np.log(20.0), k))
        co = rng.uniform(0.1, 1.0, (contractions, k))
        out.append(syn.ShellRecord(tuple(map(float, sites[c])), l, tuple(map(float, e)),
                                   tuple(tuple(map(float, r)) for r in co)))
    return out


CASES = {
    # every template pair and its mirror, L up to 8 and beyond (class-generic), mixed sites
    "shells_spdf": (dict(ls=(0, 1, 2, 3, 1), nprims=(3, 2, 1, 1, 1), centers=(0, 0, 1, 1, 2)), (0.1, -0.07, 0.12), 160),
    # one centre in a field: every pair real although B != 0
    "one_site": (dict(ls=(0, 1, 2, 3), nprims=(4, 2, 2, 1), centers=(0, 0, 0, 0)), (0.2, 0.1, -0.3), 120),
    # zero field, several sites: every pair real
    "zero_field": (dict(ls=(0, 1, 2, 3, 2), nprims=(5, 3, 1, 1, 2), centers=(0, 1, 2, 2, 1)), (0.0, 0.0, 0.0), 120),
    # general contractions: blocks written with strides
    "contractions": (dict(ls=(0, 1, 2), nprims=(4, 3, 2), centers=(0, 1, 0), contractions=2), (0.05, 0.1, 0.0), 60),
    # deep contractions: one task fills many batches
    "deep": (dict(ls=(0, 0, 1), nprims=(9, 7, 6), centers=(0, 1, 1)), (-0.1, 0.02, 0.3), 81),
    # order above the Schwarz factors' limit, beyond a warp's lanes of component pairs
    "high_l": (dict(ls=(5, 4, 0), nprims=(1, 2, 2), centers=(0, 1, 1)), (0.1, 0.2, -0.1), 12),
    # a distant site: tasks and whole units without a surviving primitive quartet
    "distant": (dict(ls=(0, 1, 2, 0, 1), nprims=(3, 2, 1, 3, 1), centers=(0, 0, 0, 1, 1), far=60.0), (0.01, 0.02, 0.0),
                200),
}


@pytest.mark.parametrize("name", CASES)
def test_blocks_against_oracle(name, oracle):
    spec, B, count = CASES[name]
    recs = _records(11, **spec)
    basis = basis_from_records(recs)
    ns = len(recs)
    q = np.array([(a, b, c, d) for a in range(ns) for b in range(ns) for c in range(ns) for d in range(ns)], np.uint32)
    rng = np.random.default_rng(5)
    q = q[np.sort(rng.choice(len(q), min(count, len(q)), replace=False))]
    field = gi.MagneticField(B)
    _, _, offsets, values, _, _ = _eri_batch(basis, q, field=field)
    ref, roff = oracle.eri_batch(recs, q, B, None, 8)
    np.testing.assert_array_equal(offsets, roff)
    assert np.abs(values - ref).max() <= 1e-12
    _, _, _, exact, _, _ = _eri_batch(basis, q, field=field, precision="fp64_exact")
    assert np.abs(exact - ref).max() <= 1e-12
    _, _, _, mixed, _, _ = _eri_batch(basis, q, field=field, precision="mixed")
    assert np.abs(mixed - ref).max() <= 1e-10
    # the bits of a quartet do not depend on what it is evaluated with
    lmax = np.array([r.angular_momentum for r in recs])[q.astype(int)].sum(1)
    for part in (slice(0, 1), slice(3, 36), slice(1, None, 2)):
        _, _, off2, val2, _, _ = _eri_batch(basis, q[part], field=field)
        for i, k in enumerate(np.arange(len(q))[part]):
            if lmax[k] <= 8:  # (beyond, the class-generic kernel splits by class size)
                assert np.array_equal(val2[off2[i]:off2[i + 1]], values[offsets[k]:offsets[k + 1]])


@pytest.mark.parametrize("tasks", [1, 31, 32, 33, 511, 512, 513, 1500])
@pytest.mark.parametrize("key", [(0, 1, 0, 0), (1, 1, 0, 2), (2, 1, 2, 2)])
def test_class_sizes(key, tasks, oracle):
    """Classes around a batch and around the size from which the units are cut
    by kernels of their own; the tasks repeat over few shells."""
    rng = np.random.default_rng(tasks)
    recs = _records(3, ls=key * 2, nprims=(2, 1, 1, 2, 1, 2, 3, 1), centers=(0, 1, 2, 0, 1, 1, 0, 2))
    basis = basis_from_records(recs)
    slots = [[i for i in (k, 4 + k)] for k in range(4)]
    q = np.array([[rng.choice(s) for s in slots] for _ in range(tasks)], dtype=np.uint32)
    B = (0.12, -0.2, 0.07)
    _, _, offsets, values, _, _ = _eri_batch(basis, q, field=gi.MagneticField(B))
    uniq, inv = np.unique(q, axis=0, return_inverse=True)
    ref, roff = oracle.eri_batch(recs, uniq.astype(np.uint32), B, None, 8)
    size = int(offsets[1])
    want = ref.reshape(-1, size)[inv.reshape(-1)]
    assert np.abs(values.reshape(-1, size) - want).max() <= 1e-12


def test_equal_schwarz_factors(oracle):
    """Shells with repeated primitives: the order of equal factors is that of
    the records, and 24 primitives fill several rounds of the ranking."""
    e = tuple([0.8] * 12 + [1.7] * 12)
    c = ((0.1,) * 24,)
    recs = [syn.ShellRecord((0.0, 0.0, 0.1 * k), l, e, c) for k, l in enumerate((0, 1))]
    basis = basis_from_records(recs)
    q = np.array([(0, 1, 0, 1), (1, 1, 0, 0)], np.uint32)
    B = (0.3, -0.1, 0.2)
    _, _, _, values, _, _ = _eri_batch(basis, q, field=gi.MagneticField(B))
    # (the oracle adds the 331,776 terms one by one and is itself 1.6e-12 off
    # the sum: it gets the same shells with the repeated primitives merged)
    merged = [syn.ShellRecord(r.center, r.angular_momentum, (0.8, 1.7), ((1.2, 1.2),)) for r in recs]
    ref, _ = oracle.eri_batch(merged, q, B, None, 8)
    assert np.abs(values - ref).max() <= 1e-12


@pytest.mark.parametrize("nuclei", [1, 31, 33, 70])
@pytest.mark.parametrize("B", [(0.0, 0.0, 0.0), (0.1, -0.2, 0.15)])
def test_nuclear_batches(nuclei, B, oracle):
    """Nuclear attraction with lanes that hold (primitive pair, nucleus): fewer
    nuclei than lanes, more, and shells on both sides of the table limit
    (la + lb <= 8).  Tolerance: that of the reference comparison."""
    recs = _records(17, ls=(0, 1, 2, 3, 5, 4), nprims=(5, 3, 2, 1, 1, 1), centers=(0, 0, 1, 2, 1, 2))
    basis = basis_from_records(recs)
    rng = np.random.default_rng(nuclei)
    nucs = [(float(rng.integers(1, 9)), tuple(map(float, rng.uniform(-2.0, 4.0, 3)))) for _ in range(nuclei)]
    got = gi.nuclear_attraction(basis, [gi.Nucleus(z, c) for z, c in nucs], field=gi.MagneticField(B))
    ref = oracle.nuclear(recs, nucs, B, None)
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-12 * np.abs(ref).max())


@pytest.mark.parametrize("key", [(2, 1, 3, 3), (3, 0, 3, 3), (2, 2, 2, 3), (3, 3, 1, 3), (3, 3, 2, 2), (3, 2, 3, 2)])
@pytest.mark.parametrize("tasks", [1, 40, 600])
def test_real_orders_9_and_10(key, tasks, oracle):
    """Classes that the lane-dense kernel takes at zero field alone, their
    mirrors and one without a template pair, with units cut by the blocks and by
    kernels of their own; then the same plan in a field (class-generic kernel)
    and at zero field again.  Tolerances: the bars of the two precision modes."""
    rng = np.random.default_rng(tasks + sum(key))
    recs = _records(23, ls=key * 2, nprims=(2, 1, 1, 2, 1, 1, 2, 1), centers=(0, 1, 1, 2, 2, 1, 0, 2))
    basis = basis_from_records(recs)
    q = np.array([[rng.choice([k, 4 + k]) for k in range(4)] for _ in range(tasks)], dtype=np.uint32)
    uniq, inv = np.unique(q, axis=0, return_inverse=True)
    bits = {}
    for turn, B in enumerate([(0.0, 0.0, 0.0), (0.12, -0.2, 0.07), (0.0, 0.0, 0.0)]):
        ref, _ = oracle.eri_batch(recs, uniq.astype(np.uint32), B, None, 8)
        for precision, bar in (("fp64", 1e-12), ("mixed", 1e-10)):
            _, _, offsets, values, _, _ = _eri_batch(basis, q, field=gi.MagneticField(B), precision=precision)
            want = ref.reshape(len(uniq), -1)[inv.reshape(-1)].reshape(-1)
            assert np.abs(values - want).max() <= bar * max(1.0, np.abs(ref).max())
            if turn == 0:
                bits[precision] = values.copy()
            elif turn == 2:
                assert np.array_equal(values, bits[precision])


def test_cost_of_an_entry_does_not_grow_with_the_contraction():
    """One (ss|ss) of 20 primitives a shell against one of 14: 4.2 times the entries.  (Sought from the task's first
    bra pair for every batch, they took 6.6 times as long.)"""
    import time

    field = gi.MagneticField((0.1, 0.05, 0.0))
    seconds = []
    for nprim in (14, 20):
        rng = np.random.default_rng(1)
        shells = [gi.Shell((0.3 * i, 0.0, 0.1 * i), 0, np.exp(rng.uniform(-2.0, 8.0, nprim)),
                           rng.uniform(0.1, 1.0, nprim)) for i in range(2)]
        best = np.inf
        for _ in range(5):
            start = time.perf_counter()
            gi.eri_shell(shells[0], shells[1], shells[0], shells[1], field=field)
            best = min(best, time.perf_counter() - start)
        seconds.append(best)
    assert seconds[1] <= 5.2 * seconds[0], seconds


def test_pair_records_of_deep_contractions_stay_cheap():
    """Ordering the primitive pairs of two s shells of 128 primitives (16,384 pairs each way): 10 to 20 ms, 0.6 s when
    every shell pair had a warp and FP64 comparisons."""
    import time

    rng = np.random.default_rng(2)
    shells = [gi.Shell((0.3 * i, 0.0, 0.0), 0, np.exp(rng.uniform(-2.0, 6.0, 128)), rng.uniform(0.1, 1.0, 128))
              for i in range(2)]
    best = np.inf
    for k in range(3):  # (a new basis and field every time)
        start = time.perf_counter()
        gi.nuclear_attraction(gi.Basis(shells), [gi.Nucleus(1.0, (0.0, 0.0, 0.5))],
                              field=gi.MagneticField((0.1, 0.01 * k, 0.0)))
        best = min(best, time.perf_counter() - start)
    assert best <= 0.2, best


def test_mixed_precision_of_very_deep_contractions():
    """An (ss|ss) of 66,049 bra pairs whose FP32 entries wait in a queue: every entry keeps its own pair (a sum of
    FP32 values, all entries in the FP32 range: 66,049 roundings of 6e-8 of at most the largest entry, and the FP32
    recurrence of a few more)."""
    from giaoint_gb300.plan import EriPlan

    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4)
    deep = [gi.Shell((0.1 * k, 0.0, 0.0), 0, np.exp(rng.uniform(-1.0, 6.0, 257)), rng.uniform(0.1, 1.0, 257))
            for k in range(2)]
    basis = gi.Basis(deep + [gi.Shell((0.0, 0.2, 0.0), 0, [0.7], [1.0]), gi.Shell((0.0, 0.0, 0.3), 0, [1.1], [1.0])])
    plan = EriPlan(basis, [(0, 1, 2, 3), (2, 3, 1, 0)])
    out = torch.empty(plan.total, dtype=torch.complex128, device="cuda:0")
    field = gi.MagneticField((0.1, -0.1, 0.05))
    plan.execute(out, field, precision="fp64_exact")
    plan.synchronize()
    exact = out.cpu().numpy()
    plan.execute(out, field, precision="mixed", mixed_cutoff=1.0e30)
    plan.synchronize()
    assert plan.counts()["fp32_quartets"] > 2 * 65536
    assert np.abs(out.cpu().numpy() - exact).max() <= 1e-6 * np.abs(exact).max()

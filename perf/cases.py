"""The electron-repulsion workloads whose speed is watched, through the public entry points.

``listed()`` names the cases, ``prepare(case, seed)`` makes what a program has in hand before the call (a basis, a
field, a plan with its output buffer), ``run(state)`` is one pass, ``work(case)`` the bytes and operations that a
pass cannot do without and ``exact(case, seed)`` the same results from a separate 64-bit evaluation: complex
McMurchie-Davidson integrals written with torch only (Hermite coefficients about the complex Gaussian centre, Boys
function by Gauss-Legendre quadrature).
"""

from __future__ import annotations

import math

import numpy as np
import torch

import giaoint_gb300 as gi
from giaoint_gb300 import synthetic as syn
from giaoint_gb300.boys import boys_many
from giaoint_gb300.plan import EriPlan

# (angular momentum, primitive count) of each atom's shells: the package's own s/p/d recipe, the same with an f
# shell, and a small s/p one
RECIPES = {
    "sp": ((0, 3), (0, 1), (1, 2)),
    "spd": syn.MOLECULE_RECIPE,
    "spdf": ((0, 6), (0, 1), (1, 3), (1, 1), (2, 1), (3, 1)),
}
# shells per angular momentum of the uncontracted even-tempered atoms
ATOMS = {"19ao": "4,3,1", "40ao": "6,4,2,1"}


def listed():
    return [
        # one contracted shell quartet on four centres: the smallest call, where launches and allocations count
        {"name": "shell_quartet", "kind": "shell", "ls": "1,1,2,1", "nprim": "3,1,1,3"},
        # the complex Boys function of many arguments, host array in and out (tables, checks of other codes)
        {"name": "boys_values", "kind": "boys", "count": 50000, "order": 8},
        # the whole tensor of a 19-function atom in a field (SCF on small systems)
        {"name": "full_tensor_atom", "kind": "full", "counts": ATOMS["19ao"], "field": True},
        # the default call of the package, eri(basis): every block of a molecule without a field, on the host
        {"name": "blocks_molecule", "kind": "blocks", "atoms": 4, "recipe": "spd", "field": False},
        # the 12-atom molecule in a field, all canonical quartets into device memory, in FP64 ...
        {"name": "plan_fp64_12", "kind": "plan", "atoms": 12, "recipe": "spd", "field": True, "precision": "fp64"},
        # ... and in mixed precision: the benchmark's step
        {"name": "plan_mixed_12", "kind": "plan", "atoms": 12, "recipe": "spd", "field": True, "precision": "mixed"},
        # a molecule with f shells without a field (the usual quantum-chemistry call)
        {"name": "plan_fp64_zero_f", "kind": "plan", "atoms": 5, "recipe": "spdf", "field": False,
         "precision": "fp64"},
        # a sweep over magnetic fields: the pair records change with every field
        {"name": "field_sweep", "kind": "sweep", "atoms": 5, "recipe": "spd", "fields": 4, "precision": "mixed"},
        # pivoted Cholesky factors of an atom (real) and of a molecule in a field (complex)
        {"name": "cholesky_atom", "kind": "cholesky", "counts": ATOMS["40ao"], "atoms": 0, "recipe": "",
         "field": False},
        {"name": "cholesky_molecule", "kind": "cholesky", "counts": "", "atoms": 2, "recipe": "spd", "field": True},
        # nuclear gradient: centre derivatives contracted with a density
        {"name": "gradient_molecule", "kind": "gradient", "atoms": 3, "recipe": "spd", "field": True},
        # the nuclear-attraction matrix of the 12-atom molecule in a field
        {"name": "nuclear_12", "kind": "nuclear", "atoms": 12, "recipe": "spd", "field": True},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("shell", "boys", "full", "blocks", "plan", "plan", "plan", "sweep", "cholesky", "gradient",
                       "nuclear"))
    field = rng.random() < 0.6
    if kind == "shell":
        ls = [rng.randint(0, 3) for _ in range(4)]
        return {"kind": kind, "ls": ",".join(map(str, ls)),
                "nprim": ",".join(str(rng.randint(1, 6 if l == 0 else 3)) for l in ls)}
    if kind == "boys":
        return {"kind": kind, "count": log_int(1, 200000), "order": rng.randint(0, 16)}
    if kind == "full":
        return {"kind": kind, "counts": "%d,%d,%d" % (rng.randint(1, 5), rng.randint(1, 3), rng.randint(0, 1)),
                "field": field}
    spread = round(rng.uniform(0.8, 1.3), 3)
    if kind == "blocks":
        return {"kind": kind, "atoms": rng.randint(1, 4), "recipe": rng.choice(("sp", "spd")), "field": field,
                "spread": spread}
    if kind == "plan":
        recipe = rng.choice(("sp", "spd", "spd", "spdf"))
        atoms = rng.randint(1, 5 if recipe == "spdf" else 11)
        return {"kind": kind, "atoms": atoms, "recipe": recipe, "field": field, "spread": spread,
                "precision": rng.choice(("fp64", "mixed") if atoms > 7 or recipe == "spdf" else
                                        ("fp64", "fp64", "mixed", "mixed", "fp64_exact"))}
    if kind == "sweep":
        return {"kind": kind, "atoms": rng.randint(1, 5), "recipe": rng.choice(("sp", "spd")),
                "fields": rng.randint(2, 5), "precision": rng.choice(("fp64", "mixed")), "spread": spread}
    if kind == "cholesky":
        if rng.random() < 0.5:
            return {"kind": kind, "counts": "%d,%d,%d,%d" % (rng.randint(2, 6), rng.randint(1, 4), rng.randint(1, 2),
                                                            rng.randint(0, 1)),
                    "atoms": 0, "recipe": "", "field": False, "ratio": round(2.5 * spread, 3)}
        return {"kind": kind, "counts": "", "atoms": rng.randint(1, 2), "recipe": rng.choice(("sp", "spd")),
                "field": field, "spread": spread}
    if kind == "gradient":
        return {"kind": kind, "atoms": rng.randint(1, 3), "recipe": rng.choice(("sp", "spd")), "field": field,
                "spread": spread}
    return {"kind": kind, "atoms": rng.randint(1, 12), "recipe": rng.choice(("sp", "spd", "spdf")), "field": field,
            "spread": spread}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _records(case, seed):
    """Shell records of the case; the molecule's density is that of 12 atoms in a cube of side 10 (times ``spread``)."""
    if case["kind"] == "shell":
        rng = np.random.default_rng(seed)
        return [syn.ShellRecord(tuple(map(float, rng.uniform(0.0, 3.0, 3))), int(l),
                                tuple(map(float, np.exp(rng.uniform(math.log(0.1), math.log(50.0), int(k))))),
                                (tuple(map(float, rng.uniform(0.1, 1.0, int(k)))),))
                for l, k in zip(case["ls"].split(","), case["nprim"].split(","))]
    if case.get("counts"):
        counts = [int(c) for c in case["counts"].split(",")]
        first = np.random.default_rng(seed).uniform(0.15, 0.3, len(counts))
        return syn.atom_even_tempered(counts, [float(f) for f in first], ratio=case.get("ratio", 2.5))
    box = 10.0 * case.get("spread", 1.0) * (case["atoms"] / 12.0) ** (1.0 / 3.0)
    return syn.random_molecule(seed, natoms=case["atoms"], box=max(box, 4.0), recipe=RECIPES[case["recipe"]])


def _field(case, seed, k=0):
    if not case.get("field", True):
        return None
    return syn.random_field(seed + 1000 * k, bmax=0.2)


def _boys_arguments(case, seed):
    """Arguments as primitive quartets give them: rho X'.X', mostly moderate, some far out, small imaginary part."""
    rng = np.random.default_rng(seed)
    x = np.where(rng.random(case["count"]) < 0.8, rng.uniform(0.0, 60.0, case["count"]),
                 np.exp(rng.uniform(math.log(1e-4), math.log(155.0), case["count"])))
    y = 0.4 * np.minimum(x + 0.5, 8.0) * rng.uniform(-1.0, 1.0, case["count"])
    return x + 1j * y


def _nuclei(case, seed):
    rng = np.random.default_rng(seed + 17)
    centers = sorted({r.center for r in _records(case, seed)})
    return [(float(rng.integers(1, 10)), c) for c in centers]


def _density(n, seed):
    rng = np.random.default_rng(seed + 29)
    m = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return (m + m.conj().T) / (2.0 * n)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "boys":
        return {"kind": kind, "z": _boys_arguments(case, seed), "order": case["order"]}
    records = _records(case, seed)
    shells = [gi.Shell.from_record(r) for r in records]
    state = {"kind": kind}
    b = _field(case, seed)
    state["field"] = None if b is None else gi.MagneticField(b)
    if kind == "shell":
        return dict(state, shells=shells)
    basis = gi.Basis(shells)
    state["basis"] = basis
    if kind in ("plan", "sweep"):
        plan = EriPlan(basis)
        count = case["fields"] if kind == "sweep" else 1
        state.update(plan=plan, precision=case["precision"],
                     fields=[gi.MagneticField(_field(case, seed, k)) for k in range(count)] if kind == "sweep"
                     else [state["field"]],
                     out=[torch.empty(plan.total, dtype=torch.complex128, device="cuda") for _ in range(count)])
    elif kind == "gradient":
        atoms = {c: i for i, c in enumerate(sorted({r.center for r in records}))}
        state.update(atoms=[atoms[r.center] for r in records], natom=len(atoms), density=_density(basis.ao_count, seed))
    elif kind == "nuclear":
        state["nuclei"] = [gi.Nucleus(z, c) for z, c in _nuclei(case, seed)]
    return state


def run(state):
    kind = state["kind"]
    if kind == "shell":
        return gi.eri_shell(*state["shells"], field=state["field"])
    if kind == "boys":
        return boys_many(state["z"], state["order"])[0]
    if kind == "full":
        n = state["basis"].ao_count
        return gi.eri(state["basis"], field=state["field"], storage="full", max_bytes=16 * n**4)
    if kind == "blocks":
        return [batch.values for batch in gi.eri(state["basis"], field=state["field"])]
    if kind in ("plan", "sweep"):
        for field, out in zip(state["fields"], state["out"]):
            state["plan"].execute(out, field, precision=state["precision"])
        return state["out"]
    if kind == "cholesky":
        # the factors' row order rests on ties between equal diagonal elements, so what they stand for is returned:
        # (mu nu|lam sig) = sum_P L[P,mu,nu] conj(L[P,sig,lam])
        chol = gi.cholesky_eri(state["basis"], field=state["field"], threshold=1e-10)
        r, n, _ = chol.vectors.shape
        v = torch.as_tensor(chol.vectors if state["field"] is not None else np.ascontiguousarray(chol.vectors.real),
                            device="cuda").reshape(r, n * n)
        return (v.T @ v.conj()).reshape(n, n, n, n).permute(0, 1, 3, 2)
    if kind == "gradient":
        pair = [(state["density"], state["density"])]
        return gi.eri_derivative_contraction(state["basis"], state["atoms"], state["natom"], field=state["field"],
                                             coulomb_pairs=pair, exchange_pairs=pair)
    return gi.nuclear_attraction(state["basis"], state["nuclei"], field=state["field"])


# ---------------------------------------------------------------------------
# work of a pass
# ---------------------------------------------------------------------------


def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _components(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _nherm(L):
    return (L + 1) * (L + 2) * (L + 3) // 6


def _box(la, lb):
    """Hermite terms of all component pairs of (la, lb)."""
    return sum((a[0] + b[0] + 1) * (a[1] + b[1] + 1) * (a[2] + b[2] + 1)
               for a in _components(la) for b in _components(lb))


def _quartet_flops(la, lb, lc, ld, real):
    """One primitive quartet: Boys values, Hermite table, ket and bra transform (multiply-adds count two)."""
    L = la + lb + lc + ld
    table = 2 * sum(_nherm(k) for k in range(1, L + 1))
    ket = 2 * _nherm(la + lb) * _box(lc, ld)
    bra = 2 * _ncart(lc) * _ncart(ld) * _box(la, lb)
    return (1 if real else 4) * (table + ket + bra) + 60 + 20 * L


def work(case):
    kind = case["kind"]
    if kind == "boys":
        n = case["count"]
        return {"bytes": 16.0 * n * (case["order"] + 2), "flops": n * (80.0 + 12.0 * case["order"])}
    shells = [(r.angular_momentum, len(r.exponents)) for r in _records(case, 1)]
    real = not case.get("field", True)
    nao = sum(_ncart(l) for l, _ in shells)
    by_l = {l: sum(1 for x, _ in shells if x == l) for l, _ in shells}
    if kind == "shell":
        ls = [l for l, _ in shells]
        prims = math.prod(k for _, k in shells)
        return {"bytes": 16.0 * math.prod(_ncart(l) for l in ls), "flops": prims * _quartet_flops(*ls, real)}
    if kind == "nuclear":
        flops = sum(ka * kb * case["atoms"] * (2 * _box(la, lb) + 60 + 20 * (la + lb)) * (1 if real else 4) / 2
                    for la, ka in shells for lb, kb in shells)
        return {"bytes": 16.0 * nao**2, "flops": flops}
    # at least one primitive quartet of every canonical shell quartet (orbits of at most four)
    flops = sum(by_l[a] * by_l[b] * by_l[c] * by_l[d] / 4.0 * _quartet_flops(a, b, c, d, real)
                for a in by_l for b in by_l for c in by_l for d in by_l)
    if kind == "cholesky":
        rank = 0.25 * nao**2  # about, at this threshold
        flops = rank**2 * nao**2 * (1 if real else 4)
        return {"bytes": 16.0 * nao**4 + (8.0 if real else 16.0) * rank * nao**2, "flops": flops}
    if kind == "gradient":
        return {"bytes": 32.0 * nao**2, "flops": 12 * flops}
    if kind == "full":
        return {"bytes": 16.0 * nao**4, "flops": flops}
    count = case["fields"] if kind == "sweep" else 1
    return {"bytes": 4.0 * nao**4 * count, "flops": flops * count}


# ---------------------------------------------------------------------------
# the same results in 64 bits, with torch alone
# ---------------------------------------------------------------------------

_GL = np.polynomial.legendre.leggauss(96)
_LIMIT = 2.5e6  # primitive quartets (weighted) beyond which the separate evaluation takes too long


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _boys(z, order):
    """F_0 .. F_order of complex z (Re z > -20): quadrature below Re z = 45, erf asymptotics above."""
    t = torch.as_tensor(0.5 * (_GL[0] + 1.0), device=z.device)
    w = torch.as_tensor(0.5 * _GL[1], device=z.device)
    out = torch.empty(order + 1, z.numel(), dtype=torch.complex128, device=z.device)
    far = z.real >= 45.0
    if bool(far.any()):
        zf = z[far]
        f = 0.5 * torch.sqrt(math.pi / zf)
        e = torch.exp(-zf)
        for n in range(order + 1):
            out[n, far] = f
            f = ((2 * n + 1) * f - e) / (2.0 * zf)
    near = torch.nonzero(~far).reshape(-1)
    for part in near.split(100000):
        e = torch.exp(-z[part][:, None] * (t * t)[None, :])
        for n in range(order + 1):
            out[n, part] = (e * (w * t ** (2 * n))[None, :]).sum(1)
    return out


def _hermite_indices(L):
    return [(k, l, s - k - l) for s in range(L + 1) for k in range(s, -1, -1) for l in range(s - k, -1, -1)]


def _hermite_table(L, x, seeds):
    """R_{tuv}, t + u + v <= L, of the complex separation x[3] from seeds[n] = C (-2 rho)^n F_n: [N, count]."""
    level = {(0, 0, 0): seeds[L]}
    for n in range(L - 1, -1, -1):
        new = {(0, 0, 0): seeds[n]}
        for k in _hermite_indices(L - n)[1:]:
            axis = 0 if k[0] else 1 if k[1] else 2
            low = tuple(v - (i == axis) for i, v in enumerate(k))
            value = x[axis] * level[low]
            if low[axis]:
                value = value + low[axis] * level[tuple(v - (i == axis) for i, v in enumerate(low))]
            new[k] = value
        level = new
    return torch.stack([level[k] for k in _hermite_indices(L)], 1)


def _odd_factorial(n):
    return math.prod(range(2 * n - 1, 0, -2)) if n > 0 else 1


def _primitive_norm(a, comp):
    return ((2.0 * a / math.pi) ** 0.75 * (4.0 * a) ** (0.5 * sum(comp))
            / math.sqrt(math.prod(_odd_factorial(c) for c in comp)))


def _normalised(record):
    """Contraction coefficients with unit self-overlap of the (l, 0, 0) component."""
    l, e = record.angular_momentum, np.asarray(record.exponents)
    c = np.asarray(record.raw_coefficients[0], dtype=float)
    p = e[:, None] + e[None, :]
    n = _primitive_norm(e, (l, 0, 0))
    overlap = (c * n)[:, None] * (c * n)[None, :] * _odd_factorial(l) / (2.0 * p) ** l * (math.pi / p) ** 1.5
    return c / math.sqrt(overlap.sum())


class _Pairs:
    """Primitive pairs of every ordered shell pair, by pair class: exponent sum p, complex centre P', prefactor K,
    Hermite coefficients E[pair, component pair, Hermite index]."""

    def __init__(self, records, field):
        dev = _device()
        B = np.zeros(3) if field is None else np.asarray(field)
        coefs = [_normalised(r) for r in records]
        rows, self.where = {}, {}
        for a, ra in enumerate(records):
            for b, rb in enumerate(records):
                key = (ra.angular_momentum, rb.angular_momentum)
                group = rows.setdefault(key, [])
                self.where[a, b] = (len(group), len(ra.exponents) * len(rb.exponents))
                for i, ea in enumerate(ra.exponents):
                    for j, eb in enumerate(rb.exponents):
                        group.append((ea, eb, coefs[a][i] * coefs[b][j], *ra.center, *rb.center))
        self.of = {}
        for (la, lb), group in rows.items():
            g = torch.as_tensor(np.asarray(group), device=dev)
            ea, eb, cc, A, C = g[:, 0], g[:, 1], g[:, 2], g[:, 3:6], g[:, 6:9]
            p = ea + eb
            P = (ea[:, None] * A + eb[:, None] * C) / p[:, None]
            half = 0.5 * torch.as_tensor(B, device=dev).expand_as(A)
            q = torch.linalg.cross(half, C) - torch.linalg.cross(half, A)
            K = (cc * torch.exp(-ea * eb / p * ((A - C) ** 2).sum(1) - (q * q).sum(1) / (4.0 * p))
                 * torch.exp(-1j * (q * P).sum(1)))
            Pc = P - 0.5j * q / p[:, None]
            axis = [self._axis(la, lb, Pc[:, x] - A[:, x], Pc[:, x] - C[:, x], 0.5 / p) for x in range(3)]
            index = {h: i for i, h in enumerate(_hermite_indices(la + lb))}
            E = torch.zeros(len(group), _ncart(la) * _ncart(lb), len(index), dtype=torch.complex128, device=dev)
            for ab, (ca, cb) in enumerate((x, y) for x in _components(la) for y in _components(lb)):
                norm = _primitive_norm(ea, ca) * _primitive_norm(eb, cb)
                ex, ey, ez = (axis[x][ca[x], cb[x]] for x in range(3))
                for k, vx in enumerate(ex):
                    for l, vy in enumerate(ey):
                        for m, vz in enumerate(ez):
                            E[:, ab, index[k, l, m]] = norm * vx * vy * vz
            self.of[la, lb] = (p, Pc, K, E)

    @staticmethod
    def _axis(la, lb, PA, PB, half):
        """{(i, j): [E_0 .. E_{i+j}]} along one axis."""
        def raised(e, d):
            old = e + [torch.zeros_like(d)] * 2
            return [(half * old[t - 1] if t else 0.0) + d * old[t] + (t + 1) * old[t + 1] for t in range(len(e) + 1)]

        out = {(0, 0): [torch.ones_like(PA)]}
        for i in range(la + 1):
            if i:
                out[i, 0] = raised(out[i - 1, 0], PA)
            for j in range(1, lb + 1):
                out[i, j] = raised(out[i, j - 1], PB)
        return out


def _eri(records, field, quartets):
    """Packed blocks of the quartets in C order, complex128."""
    pairs = _Pairs(records, field)
    dev = _device()
    ls = np.array([r.angular_momentum for r in records])
    nc = (ls + 1) * (ls + 2) // 2
    quartets = np.asarray(quartets, dtype=np.int64)
    sizes = np.prod(nc[quartets], axis=1)
    starts = np.concatenate([[0], np.cumsum(sizes)])
    out = torch.zeros(int(starts[-1]), dtype=torch.complex128, device=dev)
    keys = ls[quartets]
    for key in np.unique(keys, axis=0):
        la, lb, lc, ld = (int(x) for x in key)
        members = np.nonzero((keys == key).all(1))[0]
        bra = np.array([pairs.where[a, b] for a, b in quartets[members][:, :2]])
        ket = np.array([pairs.where[c, d] for c, d in quartets[members][:, 2:]])
        count = bra[:, 1] * ket[:, 1]
        task = np.repeat(np.arange(len(members)), count)
        r = np.arange(len(task)) - np.repeat(np.cumsum(count) - count, count)
        ip = torch.as_tensor(bra[task, 0] + r // ket[task, 1], device=dev)
        iq = torch.as_tensor(ket[task, 0] + r % ket[task, 1], device=dev)
        task = torch.as_tensor(task, device=dev)
        L, hab, hcd = la + lb + lc + ld, _hermite_indices(la + lb), _hermite_indices(lc + ld)
        index = {h: i for i, h in enumerate(_hermite_indices(L))}
        gather = torch.as_tensor([[index[tuple(x + y for x, y in zip(h, g))] for g in hcd] for h in hab], device=dev)
        sign = torch.as_tensor([(-1.0) ** sum(g) for g in hcd], device=dev, dtype=torch.complex128)
        p1, P1, K1, E1 = pairs.of[la, lb]
        p2, P2, K2, E2 = pairs.of[lc, ld]
        block = torch.zeros(len(members), _ncart(la) * _ncart(lb), _ncart(lc) * _ncart(ld), dtype=torch.complex128,
                            device=dev)
        step = max(256, int(3e7 / (len(hab) * len(hcd) + block.shape[1] * block.shape[2])))
        for lo in range(0, len(task), step):
            i, j = ip[lo:lo + step], iq[lo:lo + step]
            p, q = p1[i], p2[j]
            rho = p * q / (p + q)
            X = P1[i] - P2[j]
            F = _boys(rho * (X * X).sum(1), L)
            C = 2.0 * math.pi**2.5 / (p * q * torch.sqrt(p + q)) * K1[i] * K2[j]
            R = _hermite_table(L, X.T, [C * (-2.0 * rho) ** n * F[n] for n in range(L + 1)])
            W = torch.bmm(R[:, gather] * sign, E2[j].transpose(1, 2))
            block.index_add_(0, task[lo:lo + step], torch.bmm(E1[i], W))
        where = torch.as_tensor(starts[members], device=dev)[:, None] + torch.arange(int(sizes[members[0]]), device=dev)
        out[where.reshape(-1)] = block.reshape(-1)
    return out


def _full(records, field):
    n = len(records)
    quartets = [(a, b, c, d) for a in range(n) for b in range(n) for c in range(n) for d in range(n)]
    nc = [_ncart(r.angular_momentum) for r in records]
    off = np.concatenate([[0], np.cumsum(nc)])
    values = _eri(records, field, quartets).cpu().numpy()
    full = np.empty((off[-1],) * 4, dtype=np.complex128)
    at = 0
    for q in quartets:
        shape = tuple(nc[s] for s in q)
        size = math.prod(shape)
        full[tuple(slice(off[s], off[s + 1]) for s in q)] = values[at:at + size].reshape(shape)
        at += size
    return full


def _nuclear(records, field, nuclei):
    pairs = _Pairs(records, field)
    nc = [_ncart(r.angular_momentum) for r in records]
    off = np.concatenate([[0], np.cumsum(nc)])
    out = np.zeros((off[-1],) * 2, dtype=np.complex128)
    sums = {}
    for (la, lb), (p, P, K, E) in pairs.of.items():
        total = torch.zeros(E.shape[:2], dtype=torch.complex128, device=p.device)
        for charge, center in nuclei:
            X = P - torch.as_tensor(center, dtype=torch.float64, device=p.device)
            F = _boys(p * (X * X).sum(1), la + lb)
            R = _hermite_table(la + lb, X.T, [-charge * 2.0 * math.pi / p * K * (-2.0 * p) ** n * F[n]
                                              for n in range(la + lb + 1)])
            total += torch.bmm(E, R[:, :, None])[:, :, 0]
        sums[la, lb] = total.cpu().numpy()
    for (a, b), (first, count) in pairs.where.items():
        block = sums[records[a].angular_momentum, records[b].angular_momentum][first:first + count].sum(0)
        out[off[a]:off[a + 1], off[b]:off[b + 1]] = block.reshape(nc[a], nc[b])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        return None
    if kind == "boys":
        z = torch.as_tensor(_boys_arguments(case, seed), device=_device())
        return _boys(z, case["order"]).T.cpu().numpy()
    records = _records(case, seed)
    field = _field(case, seed)
    weight = sum(len(r.exponents) * (1 + r.angular_momentum) for r in records) ** 4 / 16.0
    if kind == "nuclear":
        return _nuclear(records, field, _nuclei(case, seed))
    if kind == "shell":
        return _eri(records, field, [(0, 1, 2, 3)]).reshape([_ncart(r.angular_momentum) for r in records])
    if weight > _LIMIT:
        return None
    if kind in ("full", "cholesky"):
        return _full(records, field)
    n = len(records)
    every = [(a, b, c, d) for a in range(n) for b in range(n) for c in range(n) for d in range(n)
             if (a, b, c, d) == min((a, b, c, d), (c, d, a, b), (b, a, d, c), (d, c, b, a))]
    if kind == "sweep":
        return [_eri(records, _field(case, seed, k), every) for k in range(case["fields"])]
    return [_eri(records, field, every)]

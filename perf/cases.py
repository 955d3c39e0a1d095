"""Workloads of the DF engine, as a user's program runs them through the public entry points.

Each case is a dict of plain values; ``kind`` names the call:

* ``step``      one geometry step: DF two-electron energy, J, K and dE/dR
                (``grad.df_energy`` + ``torch.autograd.grad``), the inner call of an SCF-converged
                optimisation or dynamics step, in FP64 or in the mixed mode;
* ``build``     the whitened DF tensor from packed bases (``df.build_df_B_from_cueri_packed_bases``),
                once at the start of every SCF run with stored factors;
* ``jk``        one SCF cycle's J and K from stored factors (``jk.DFJKWorkspace.jk_from_bq_cw``);
* ``context``   a correlated method's gradient: dE/dB in packed-Qp layout contracted through a
                ``DFGradContractionContext`` kept for the geometry;
* ``batch``     the J/K builds of several molecules replayed as one CUDA graph
                (``batch.BatchedDFJK``);
* ``streamed``  energy and gradient of a cluster too large to store its 3c tensor in earnest
                (``grad.df_energy_grad_streamed``).

Geometries are the seeded generators of ``asuka_b200.geometry`` (N2, n-decane, water clusters);
the occupied orbitals are random orthonormal columns scaled by sqrt(2).

``exact`` restates the integrals by the McMurchie-Davidson scheme in plain torch FP64 (Hermite
expansion, Boys functions by their series) and differentiates them with autograd.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from asuka_b200 import basis as bm
from asuka_b200 import geometry as geo

F64 = torch.float64
EXACT_MAX_NAO = 130  # largest molecule whose integrals ``exact`` evaluates


# ---------------------------------------------------------------- cases

def listed():
    return [
        # a diatomic in the smallest basis: the smallest call there is, bound by launches and latency
        {"name": "step n2 svp", "kind": "step", "mol": "n2", "n": 1, "basis": "ma-svp", "precision": "fp64"},
        # one small molecule, f shells (aux up to l = 6): a geometry optimisation of a fragment
        {"name": "step water tzvp", "kind": "step", "mol": "water", "n": 1, "basis": "ma-tzvp", "precision": "fp64"},
        # a chain in a small basis, mixed mode: the early steps of an ordinary organic molecule
        {"name": "step decane svp mixed", "kind": "step", "mol": "decane", "n": 10, "basis": "ma-svp",
         "precision": "mixed"},
        # the benchmark cluster of bench.py in FP64 and in the mixed mode
        {"name": "step water8 tzvp", "kind": "step", "mol": "water", "n": 8, "basis": "ma-tzvp", "precision": "fp64"},
        {"name": "step water8 tzvp mixed", "kind": "step", "mol": "water", "n": 8, "basis": "ma-tzvp",
         "precision": "mixed"},
        # g shells and aux shells up to l = 8: high angular momentum, a benchmark-quality basis
        {"name": "step water3 qzvp", "kind": "step", "mol": "water", "n": 3, "basis": "ma-qzvp", "precision": "fp64"},
        # set-up of an SCF run with stored factors in the reference's layout
        {"name": "build water4 tzvp", "kind": "build", "mol": "water", "n": 4, "basis": "ma-tzvp", "layout": "mnQ"},
        # one SCF cycle with stored factors, in FP64 and in the mixed mode of the early cycles
        {"name": "jk water8 tzvp", "kind": "jk", "mol": "water", "n": 8, "basis": "ma-tzvp", "precision": "fp64"},
        {"name": "jk decane svp mixed", "kind": "jk", "mol": "decane", "n": 10, "basis": "ma-svp",
         "precision": "mixed"},
        # the gradient of a correlated method (dE/dB in packed form) at an odd cluster size
        {"name": "context water5 tzvp", "kind": "context", "mol": "water", "n": 5, "basis": "ma-tzvp"},
        # several small molecules per call, as in a data-set run
        {"name": "batch 6 tzvp", "kind": "batch", "mol": "water", "n": 4, "count": 6, "basis": "ma-tzvp",
         "precision": "fp64"},
        # the largest: recomputed integrals, nothing of size naux nao^2 stored
        {"name": "streamed water12 tzvp", "kind": "streamed", "mol": "water", "n": 12, "basis": "ma-tzvp",
         "precision": "fp64"},
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "build", "jk", "context", "batch", "streamed"])
    basis = rng.choice(["ma-svp", "ma-tzvp", "ma-tzvp", "ma-qzvp"])
    top = {"ma-svp": 14, "ma-tzvp": 10, "ma-qzvp": 3}[basis]
    if kind in ("context", "build", "batch"):
        top = max(2, top // 2)
    n = int(round(math.exp(rng.uniform(0.0, math.log(top)))))
    case = {"kind": kind, "mol": "water", "n": n, "basis": basis}
    if kind in ("step", "jk", "batch", "streamed"):
        case["precision"] = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "build":
        case["layout"] = rng.choice(["mnQ", "Qmn"])
    if kind == "batch":
        case["count"] = rng.randint(2, 6)
    case["shift"] = rng.randint(1, 1 << 20)  # another family of geometries
    return case


# ---------------------------------------------------------------- inputs

def _molecule(case, seed):
    s = (int(seed) * 7919 + int(case.get("shift", 0))) % (1 << 31)
    if case["mol"] == "n2":
        return geo.n2(case["basis"], r_angstrom=1.0977 + 0.05 * float(np.random.default_rng(s).uniform(-1, 1)))
    if case["mol"] == "decane":
        return geo.decane(s, case["basis"])
    return geo.water_cluster(case["n"], s, case["basis"])


def _molecules(case, seed):
    """Members of a batch: n, n-1, ... monomers, each from a seed of its own."""
    return [_molecule(dict(case, n=max(1, case["n"] - i)), int(seed) * 101 + i) for i in range(case["count"])]


def _bases(mol):
    atoms = list(mol.atoms_bohr)
    return bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux")


def _randn(shape, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn(shape, generator=g, dtype=F64, device="cuda")


def _orbitals(nao, nocc, seed):
    return (torch.linalg.qr(_randn((nao, nocc), seed))[0] * math.sqrt(2.0)).contiguous()


def _factors(naux, nao, seed):
    """Symmetric DF-like factors B_Q whose size falls with Q, as whitened factors do."""
    B = _randn((naux, nao, nao), seed)
    B = B + B.transpose(1, 2)
    return B * torch.exp(-4.0 * torch.arange(naux, dtype=F64, device="cuda") / naux).view(-1, 1, 1)


def _packed(T):
    """(q, nao, nao) symmetric -> (q, ntri) lower triangle, p = m (m + 1) / 2 + n."""
    i, j = torch.tril_indices(T.shape[1], T.shape[1], device=T.device)
    return T[:, i, j].contiguous()


def _sizes(case):
    mol = _molecule(case, 0)
    ao, aux = _bases(mol)
    return ao.nao, aux.nao, mol.nelectron // 2


def prepare(case, seed):
    from asuka_b200.batch import BatchedDFJK
    from asuka_b200.df import DFEngine
    from asuka_b200.grad_context import DFGradContractionContext
    from asuka_b200.jk import DFJKWorkspace

    kind = case["kind"]
    if kind == "batch":
        mols = _molecules(case, seed)
        b = BatchedDFJK(mols, precision=case["precision"])
        Cws = [_orbitals(nao, nocc, seed * 31 + i) for i, (nao, _naux, nocc, _s) in enumerate(b.sizes)]
        b.set_orbitals(Cws)
        b.capture()
        return {"case": case, "batch": b, "Cws": Cws}
    mol = _molecule(case, seed)
    ao, aux = _bases(mol)
    nao, naux, nocc = ao.nao, aux.nao, mol.nelectron // 2
    if kind == "build":
        return {"case": case, "ao": ao, "aux": aux}
    if kind == "jk":
        Cw = _orbitals(nao, nocc, seed)
        return {"case": case, "ws": DFJKWorkspace(precision=case["precision"]), "B": _factors(naux, nao, seed + 1),
                "Cw": Cw, "D": Cw @ Cw.T, "J": torch.empty((nao, nao), dtype=F64, device="cuda"),
                "K": torch.empty((nao, nao), dtype=F64, device="cuda")}
    if kind == "context":
        ctx = DFGradContractionContext.build(ao, aux, atom_coords_bohr=mol.coords_bohr)
        return {"case": case, "ctx": ctx, "B": _packed(_factors(naux, nao, seed + 1)),
                "bar": _packed(_factors(naux, nao, seed + 2))}
    return {"case": case, "eng": DFEngine(ao, aux), "Cw": _orbitals(nao, nocc, seed),
            "R": torch.as_tensor(mol.coords_bohr, dtype=F64, device="cuda")}


def run(state):
    from asuka_b200.df import build_df_B_from_cueri_packed_bases
    from asuka_b200.grad import df_energy, df_energy_grad_streamed

    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        R = state["R"].detach().requires_grad_(True)
        E, J, K = df_energy(R, state["Cw"], state["eng"], case["precision"])
        (g,) = torch.autograd.grad(E, R)
        return {"E": E.detach(), "J": J, "K": K, "g": g}
    if kind == "build":
        return {"B": build_df_B_from_cueri_packed_bases(state["ao"], state["aux"], layout=case["layout"])}
    if kind == "jk":
        state["ws"].jk_from_bq_cw(state["B"], state["Cw"], state["D"], state["J"], state["K"],
                                  stream=torch.cuda.current_stream().cuda_stream)
        return {"J": state["J"], "K": state["K"]}
    if kind == "context":
        return {"g": state["ctx"].contract_device(B_ao=state["B"], bar_L_ao=state["bar"])}
    if kind == "batch":
        return [{"J": J, "K": K} for J, K in state["batch"].run(state["Cws"])]
    E, g, K = df_energy_grad_streamed(state["eng"], state["Cw"], precision=case["precision"])
    return {"E": E, "g": g, "K": K}


# ---------------------------------------------------------------- work and tolerance

def _distinct_prims(aux):
    """Per l: the number of distinct (centre, exponent) pairs, the fewest primitive aux functions
    from which every contracted aux shell follows by a linear combination."""
    out = {}
    seen = set()
    for s in range(aux.nshell):
        l = int(aux.shell_l[s])
        a, n = int(aux.shell_prim_start[s]), int(aux.shell_nprim[s])
        for e in aux.prim_exp[a:a + n]:
            key = (l, int(aux.shell_atom[s]), float(e))
            if key not in seen:
                seen.add(key)
                out[l] = out.get(l, 0) + 1
    return out


def _integral_flops(ao, aux, deriv):
    """Rys model: every primitive triplet takes n_r roots, each the 2D recurrence tables and three
    multiply-adds per Cartesian element (the six centre derivatives of a contracted element: ten)."""
    sp = bm.build_shell_pairs_l_order(ao)
    la, lb = ao.shell_l[sp.sp_A], ao.shell_l[sp.sp_B]
    d = 1 if deriv else 0
    tot = 0.0
    for lp, kp in _distinct_prims(aux).items():
        for a in np.unique(la):
            for b in np.unique(lb):
                kab = float(sp.sp_npair[(la == a) & (lb == b)].sum())
                nr = (int(a) + int(b) + lp + d) // 2 + 1
                n3 = bm.ncart(int(a)) * bm.ncart(int(b)) * bm.ncart(lp)
                tot += kab * kp * nr * ((10 if deriv else 3) * n3 + 9 * (int(a) + int(b) + d + 1) * (lp + 1))
    return tot


def _jk_flops(nao, naux, nocc):
    return 4.0 * naux * nao * nao + 2.0 * naux * nao * nao * nocc + 1.0 * naux * nao * nao * nocc


def work(case):
    kind = case["kind"]
    if kind == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for mol in _molecules(case, 0):
            ao, aux = _bases(mol)
            nao, naux, nocc = ao.nao, aux.nao, mol.nelectron // 2
            tot["flops"] += (_integral_flops(ao, aux, False) + _jk_flops(nao, naux, nocc)
                             + 1.0 * naux * naux * nao * nocc)
            tot["bytes"] += 8.0 * (naux * naux / 2 + nao * nocc + 2 * nao * nao)
        return tot
    mol = _molecule(case, 0)
    ao, aux = _bases(mol)
    nao, naux, nocc = ao.nao, aux.nao, mol.nelectron // 2
    if kind == "jk":
        return {"bytes": 8.0 * (naux * nao * nao + nao * nocc + 3 * nao * nao), "flops": _jk_flops(nao, naux, nocc)}
    if kind == "build":
        return {"bytes": 8.0 * naux * nao * nao,
                "flops": _integral_flops(ao, aux, False) + naux ** 3 / 3 + 0.5 * naux * naux * nao * nao}
    if kind == "context":
        ntri = nao * (nao + 1) / 2
        return {"bytes": 8.0 * (2 * naux * ntri + naux * naux / 2),
                "flops": _integral_flops(ao, aux, True) + 3.0 * naux * naux * ntri + 2.0 * naux ** 3}
    adj = (2.0 * naux * nao * nocc * nocc + 2.0 * naux * naux * nocc * nocc + 2.0 * naux * nocc * nocc * nao
           + 1.0 * naux * nao * nao * nocc)
    return {"bytes": 8.0 * (nao * nocc + 2 * nao * nao),
            "flops": (_integral_flops(ao, aux, False) + _integral_flops(ao, aux, True) + naux ** 3 / 3
                      + _jk_flops(nao, naux, nocc) + 1.0 * naux * naux * nao * nocc + adj)}


def tolerance(case):
    if case.get("precision") == "mixed":
        # the exchange matrix is a three-term BF16 tensor-core sum with FP32 accumulation: 1.4e-6 to
        # 5e-6 against FP64
        return {"rel": 2e-5, "max": 2e-3}
    if case["kind"] == "jk":
        return {"rel": 1e-13, "max": 1e-11}
    # FP64 sums, whose rounding the solves with the metric amplify by its condition number: 1e-14 to
    # 1e-11 against the restatement below on small molecules, larger for the larger metrics it leaves out
    return {"rel": 1e-9, "max": 1e-6}


# ---------------------------------------------------------------- 64-bit restatement

class _Boys(torch.autograd.Function):
    """F_0 .. F_M at T (stacked in front), by the ascending series of F_M and downward recursion,
    or the asymptotic form where exp(-T) is negligible; dF_m/dT = -F_{m+1}."""

    @staticmethod
    def forward(ctx, T, M):
        F = torch.empty((M + 2,) + tuple(T.shape), dtype=F64, device=T.device)
        big = T > 150.0
        Ts = torch.where(big, torch.ones_like(T), T)
        e = torch.exp(-Ts)
        term = torch.full_like(Ts, 1.0 / (M + 1.5))
        acc = term.clone()
        for i in range(1, 420):
            term = term * Ts / (M + 1.5 + i)
            acc += term
            if i % 32 == 0 and float((term / acc).max()) < 1e-17:
                break
        F[M + 1] = 0.5 * e * acc
        for m in range(M, -1, -1):
            F[m] = (2.0 * Ts * F[m + 1] + e) / (2 * m + 1)
        Tb = torch.where(big, T, torch.full_like(T, 200.0))
        f = 0.5 * torch.sqrt(math.pi / Tb)
        for m in range(M + 2):
            F[m] = torch.where(big, f, F[m])
            f = f * (2 * m + 1) / (2.0 * Tb)
        ctx.save_for_backward(F)
        return F[: M + 1].clone()

    @staticmethod
    def backward(ctx, g):
        (F,) = ctx.saved_tensors
        return -(g * F[1: g.shape[0] + 1]).sum(0), None


def _comps(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _herm(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _E1d(la, lb, PA, PB, hp):
    """Hermite expansion coefficients E[a][b][t] of one direction (tensors over primitive pairs)."""
    E = {(0, 0, 0): torch.ones_like(PA)}

    def get(a, b, t):
        return E.get((a, b, t))

    def step(a, b, a0, b0, X):
        for t in range(a + b + 1):
            v = None
            for c, w in ((get(a0, b0, t - 1), hp), (get(a0, b0, t), X), (get(a0, b0, t + 1), float(t + 1))):
                if c is not None:
                    v = c * w if v is None else v + c * w
            E[(a, b, t)] = v

    for a in range(1, la + 1):
        step(a, 0, a - 1, 0, PA)
    for b in range(1, lb + 1):
        for a in range(la + 1):
            step(a, b, a, b - 1, PB)
    return E


def _E3d(la, lb, PA, PB, hp):
    """(npair, components of a x b, Hermite functions up to la + lb)."""
    Ed = [_E1d(la, lb, PA[:, d], PB[:, d], hp) for d in range(3)]
    z = torch.zeros_like(hp)
    rows = []
    for ca in _comps(la):
        for cb in _comps(lb):
            row = []
            for h in _herm(la + lb):
                f = [Ed[d].get((ca[d], cb[d], h[d])) for d in range(3)]
                row.append(z if any(x is None for x in f) else f[0] * f[1] * f[2])
            rows.append(torch.stack(row, 1))
    return torch.stack(rows, 1)


def _R_table(PQ, alpha, L):
    """Hermite Coulomb integrals R_tuv, t+u+v <= L, over the leading shape of alpha."""
    F = _Boys.apply(alpha * (PQ * PQ).sum(-1), L)
    cur = {n: {(0, 0, 0): F[n] * (-2.0 * alpha) ** n} for n in range(L + 1)}
    for k in range(1, L + 1):
        for n in range(L - k + 1):
            for t in range(k + 1):
                for u in range(k + 1 - t):
                    h = (t, u, k - t - u)
                    d = 0 if h[0] else (1 if h[1] else 2)
                    lo = tuple(x - (i == d) for i, x in enumerate(h))
                    v = PQ[..., d] * cur[n + 1][lo]
                    if lo[d] > 0:
                        lo2 = tuple(x - (i == d) for i, x in enumerate(lo))
                        v = v + lo[d] * cur[n + 1][lo2]
                    cur[n][h] = v
    return cur[0]


def _prims(b, l):
    """(shell, exponent, coefficient) of every primitive of the shells with angular momentum l."""
    sh = np.nonzero(b.shell_l == l)[0]
    idx = np.concatenate([np.arange(b.shell_prim_start[s], b.shell_prim_start[s] + b.shell_nprim[s]) for s in sh])
    own = np.repeat(np.arange(sh.size), b.shell_nprim[sh])
    t = lambda a, dt=F64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")  # noqa: E731
    return sh, t(own, torch.long), t(b.prim_exp[idx]), t(b.prim_coef[idx])


def _rows(b, sh, l):
    """AO indices (len(sh), ncart(l)) of the listed shells."""
    return torch.as_tensor(b.shell_ao_start[sh][:, None] + np.arange(bm.ncart(l))[None, :], dtype=torch.long,
                           device="cuda")


def _tile(A, B, C, ea, eb, ca, cb, eq, cq, la, lb, lc, with_b):
    """Primitive Coulomb integrals (npair, nab, nprim_c, nc) for centres A, B (pairs) and C (aux)."""
    p = ea + eb if with_b else ea
    P = (ea[:, None] * A + eb[:, None] * B) / p[:, None] if with_b else A
    K = ca * cb * torch.exp(-ea * eb / p * ((A - B) ** 2).sum(1)) if with_b else ca
    Eab = _E3d(la, lb, P - A, (P - B) if with_b else (P - A), 0.5 / p) * K[:, None, None]
    zero = torch.zeros((eq.shape[0], 3), dtype=F64, device="cuda")
    Ec = _E3d(lc, 0, zero, zero, 0.5 / eq) * cq[:, None, None]
    alpha = p[:, None] * eq[None, :] / (p[:, None] + eq[None, :])
    R = _R_table(P[:, None, :] - C[None, :, :], alpha, la + lb + lc)
    pre = 2.0 * math.pi ** 2.5 / (p[:, None] * eq[None, :] * torch.sqrt(p[:, None] + eq[None, :]))
    hab, hc = _herm(la + lb), _herm(lc)
    out = 0.0
    for k, s in enumerate(hc):
        sign = -1.0 if sum(s) % 2 else 1.0
        M = torch.stack([R[tuple(x + y for x, y in zip(h, s))] for h in hab], -1)  # (npair, nq, nh)
        t = torch.einsum("pah,pqh->paq", Eab, M) * (sign * pre)[:, None, :]
        out = out + t[..., None] * Ec[:, :, k][None, None, :, :]
    return out


def _integrals(ao, aux, R, sink3, sink2):
    """Hand every contracted block of (mu nu|P) and (P|Q) to the sinks, at atom positions R."""
    Rao, Rax = R[torch.as_tensor(ao.shell_atom, dtype=torch.long)], R[torch.as_tensor(aux.shell_atom, dtype=torch.long)]
    for lc in range(aux.lmax + 1):
        if not (aux.shell_l == lc).any():
            continue
        shc, oc, eq, cq = _prims(aux, lc)
        Cs = Rax[torch.as_tensor(shc, dtype=torch.long)]
        for la in range(ao.lmax + 1):
            for lb in range(la + 1):
                if not ((ao.shell_l == la).any() and (ao.shell_l == lb).any()):
                    continue
                sha, oa, ea, ca = _prims(ao, la)
                shb, ob, eb, cb = _prims(ao, lb)
                ia, ib = torch.meshgrid(torch.arange(len(ea), device="cuda"), torch.arange(len(eb), device="cuda"),
                                        indexing="ij")
                ia, ib = ia.reshape(-1), ib.reshape(-1)
                A, B = Rao[torch.as_tensor(sha)][oa][ia], Rao[torch.as_tensor(shb)][ob][ib]
                per = len(eq) * len(_herm(la + lb + lc)) * 12
                n = max(1, int(2e8) // per)
                for q0 in range(0, len(ia), n):
                    s = slice(q0, q0 + n)
                    T = _tile(A[s], B[s], Cs[oc], ea[ia[s]], eb[ib[s]], ca[ia[s]], cb[ib[s]], eq, cq, la, lb, lc, True)
                    na, nb, nc = bm.ncart(la), bm.ncart(lb), bm.ncart(lc)
                    T = T.reshape(T.shape[0], na, nb, len(eq), nc)
                    T = torch.zeros(T.shape[:3] + (len(shc), nc), dtype=F64, device="cuda").index_add(3, oc, T)
                    sink3(T, _rows(ao, sha, la)[oa[ia[s]]], _rows(ao, shb, lb)[ob[ib[s]]], _rows(aux, shc, lc), la != lb)
        for ld in range(lc + 1):
            if not (aux.shell_l == ld).any():
                continue
            shd, od, ed, cd = _prims(aux, ld)
            T = _tile(Cs[oc], None, Rax[torch.as_tensor(shd, dtype=torch.long)][od], eq, None, cq, None, ed, cd, lc, 0,
                      ld, False)
            T = torch.zeros((len(shc),) + tuple(T.shape[1:]), dtype=F64, device="cuda").index_add(0, oc, T)
            T = torch.zeros(T.shape[:2] + (len(shd), T.shape[3]), dtype=F64, device="cuda").index_add(2, od, T)
            sink2(T, _rows(aux, shc, lc), _rows(aux, shd, ld), lc != ld)


def _build_XV(ao, aux, R):
    X = torch.zeros((aux.nao, ao.nao, ao.nao), dtype=F64, device="cuda")
    V = torch.zeros((aux.nao, aux.nao), dtype=F64, device="cuda")

    def sink3(T, ra, rb, rc, both):
        v = T.permute(0, 3, 4, 1, 2)  # (pair, c, nc, na, nb)
        i = rc[None, :, :, None, None].expand(v.shape)
        a = ra[:, None, None, :, None].expand(v.shape)
        b = rb[:, None, None, None, :].expand(v.shape)
        X.index_put_((i, a, b), v, accumulate=True)
        if both:
            X.index_put_((i, b, a), v, accumulate=True)

    def sink2(T, rc, rd, both):
        i = rc[:, :, None, None].expand(T.shape)
        j = rd[None, None, :, :].expand(T.shape)
        V.index_put_((i, j), T, accumulate=True)
        if both:
            V.index_put_((j, i), T, accumulate=True)

    with torch.no_grad():
        _integrals(ao, aux, R, sink3, sink2)
    return X, V


def _gradient(ao, aux, R, G3, G2):
    """d/dR of sum G3 . X(R) + sum G2 . V(R) for symmetric adjoints."""
    R = R.clone().requires_grad_(True)
    total = torch.zeros_like(R)

    def add(s):
        nonlocal total
        (g,) = torch.autograd.grad(s, R, retain_graph=True, allow_unused=True)
        total = total + g

    def sink3(T, ra, rb, rc, both):
        g = G3[rc[None, None, None], ra[:, :, None, None, None], rb[:, None, :, None, None]]
        add((T * g).sum() * (2.0 if both else 1.0))

    def sink2(T, rc, rd, both):
        add((T * G2[rc[:, :, None, None], rd[None, None, :, :]]).sum() * (2.0 if both else 1.0))

    _integrals(ao, aux, R, sink3, sink2)
    return total


def _sym(A):
    return 0.5 * (A + A.transpose(-1, -2))


def _exact_energy(ao, aux, R, Cw):
    X, V = _build_XV(ao, aux, R)
    X.requires_grad_(True)
    V.requires_grad_(True)
    D = Cw @ Cw.T
    Li = torch.linalg.inv(torch.linalg.cholesky(_sym(V)))
    rho = torch.einsum("pmn,mn->p", X, D)
    d = Li.T @ (Li @ rho)
    J = torch.einsum("p,pmn->mn", d, X)
    W = torch.einsum("qp,pmi->qmi", Li, X @ Cw)
    K = torch.einsum("qmi,qni->mn", W, W)
    E = 0.5 * rho @ d - 0.25 * (D * K).sum()
    G3, G2 = torch.autograd.grad(E, (X, V))
    return E.detach(), J.detach(), K.detach(), _gradient(ao, aux, R, _sym(G3), _sym(G2))


def exact(case, seed):
    kind = case["kind"]
    if kind == "jk":
        s = prepare(case, seed)
        B, Cw, D = s["B"], s["Cw"], s["D"]
        J = torch.einsum("q,qmn->mn", torch.einsum("qmn,mn->q", B, D), B)
        K = torch.zeros_like(D)
        for q in range(0, B.shape[0], 256):
            U = B[q:q + 256] @ Cw
            K += torch.einsum("qmi,qni->mn", U, U)
        return {"J": J, "K": K}
    if kind == "batch":
        mols = _molecules(case, seed)
        if any(_bases(m)[0].nao > EXACT_MAX_NAO for m in mols):
            return None
        out = []
        for i, m in enumerate(mols):
            ao, aux = _bases(m)
            X, V = _build_XV(ao, aux, torch.as_tensor(m.coords_bohr, dtype=F64, device="cuda"))
            Cw = _orbitals(ao.nao, m.nelectron // 2, seed * 31 + i)
            Li = torch.linalg.inv(torch.linalg.cholesky(_sym(V)))
            d = Li.T @ (Li @ torch.einsum("pmn,mn->p", X, Cw @ Cw.T))
            W = torch.einsum("qp,pmi->qmi", Li, X @ Cw)
            out.append({"J": torch.einsum("p,pmn->mn", d, X), "K": torch.einsum("qmi,qni->mn", W, W)})
        return out
    mol = _molecule(case, seed)
    ao, aux = _bases(mol)
    if ao.nao > EXACT_MAX_NAO:
        return None
    R = torch.as_tensor(mol.coords_bohr, dtype=F64, device="cuda")
    if kind == "build":
        X, V = _build_XV(ao, aux, R)
        B = torch.linalg.solve_triangular(torch.linalg.cholesky(_sym(V)), X.reshape(aux.nao, -1), upper=False)
        B = B.reshape(X.shape)
        return {"B": B.permute(1, 2, 0).contiguous() if case["layout"] == "mnQ" else B}
    if kind == "context":
        # dE/dB is given on the whitened factors B = L^-1 X, but E depends on X and V through B only:
        # B here is the caller's tensor, so the chain is written out with B as a constant
        B = _factors(aux.nao, ao.nao, seed + 1)
        bar = _factors(aux.nao, ao.nao, seed + 2)
        _X, V = _build_XV(ao, aux, R)
        L = torch.linalg.cholesky(_sym(V))
        Li = torch.linalg.inv(L)
        G3 = torch.einsum("qp,qmn->pmn", Li, bar)
        gL = -torch.tril(torch.einsum("pmn,qmn->pq", G3, B))  # dE/dL
        Phi = torch.tril(L.T @ gL)
        Phi.diagonal().mul_(0.5)
        return {"g": _gradient(ao, aux, R, G3, _sym(Li.T @ Phi @ Li))}
    Cw = _orbitals(ao.nao, mol.nelectron // 2, seed)
    E, J, K, g = _exact_energy(ao, aux, R, Cw)
    if kind == "streamed":
        return {"E": E, "g": g, "K": K}
    return {"E": E, "J": J, "K": K, "g": g}

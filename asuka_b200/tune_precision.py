"""Per-class precision autotuner for the mixed mode.

The FP32-component integral kernels (``dfb_prim_integrals`` with f32 set) add about 1e-7 relative error
per integral; summed over a whole molecule that error reaches the 1e-6 Eh accuracy contract of the mixed
step if every class runs in FP32.  This tool measures, on the GPU and on the kernels that the mixed mode
runs, every angular class's contribution separately: one J/K + gradient step with only that class's 3c
integrals in FP32, against the all-FP64 step at the same density -- the first-order energy and gradient
change the class causes -- and the class's integrals in FP64 and in FP32, timed in turn.  It then admits
the classes that FP32 makes faster by more than the runs differ, greedily by time saved per unit of error,
until the summed absolute energy change or any summed absolute gradient component reaches its budget
(a fortieth of the contract by default), and writes them to ``asuka_b200/data/class_precision.json``
(read by ``asuka_b200.df.mixed_class_table``).  The derivative contractions of the mixed mode run in FP64.

    python -m asuka_b200.tune_precision [--workload w8] [--e-budget 2.5e-8] [--g-budget 2.5e-8]

The reference has no counterpart: its mixed mode is all-or-nothing per kernel family
(``asuka/integrals/cueri_df.py:61-65``).
"""

from __future__ import annotations

import argparse
import json
import os
import time
from contextlib import contextmanager

import numpy as np
import torch

from . import df as dfmod
from .grad import df_backward, df_forward
from .profile_step import WORKLOADS

OUT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "data", "class_precision.json")


def _density(mol, eng):
    """Converged FP64 RHF occupied block Cw of the workload (stored-B SCF)."""
    from .df import cholesky_metric, whiten_3c2e
    from .int1e import build_int1e
    from .scf import rhf_df

    int1e = build_int1e(eng.ao, mol.coords_bohr, mol.charges)
    L = cholesky_metric(eng.metric())
    B = whiten_3c2e(eng.int3c("Qmn"), L, layout="Qmn")
    res = rhf_df(int1e.S, int1e.hcore, B, nelec=mol.nelectron, enuc=mol.energy_nuc())
    del B
    torch.cuda.empty_cache()
    nocc = mol.nelectron // 2
    return (res.mo_coeff[:, :nocc] * 2.0**0.5).contiguous(), res.e_tot


def _step(eng, Cw, R, X, precision):
    eng.set_coords(R)
    E, _J, _K, saved = df_forward(eng, Cw, precision, X=X, with_adjoints=True)
    g = df_backward(eng, Cw, saved, precision=precision)
    return float(E), g.cpu().numpy()


@contextmanager
def _table(*classes):
    """The engine's mixed mode with these classes only in FP32."""
    orig = dfmod.mixed_class_table
    dfmod.mixed_class_table = lambda _t={"int3c": set(classes)}: _t  # type: ignore[assignment]
    try:
        yield
    finally:
        dfmod.mixed_class_table = orig  # type: ignore[assignment]


def _class_times(eng, entry, X, reps=15):
    """Milliseconds of one class's integrals, (FP64 runs, FP32 runs), timed in turn."""
    cls = tuple(entry[:3])
    every = eng.classes3c
    eng.classes3c = [entry]
    s = (eng.nao * eng.nao, eng.nao, 1)
    times: tuple = ([], [])
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    try:
        for i in range(reps + 2):
            for f32, ts in enumerate(times):
                with _table(*([cls] if f32 else [])):
                    work = eng._int3c_work(X, s, "mixed")
                    torch.cuda._sleep(2000000)  # the launches queue up behind it
                    e0.record()
                    eng._run_int([work])
                    e1.record()
                torch.cuda.synchronize()
                if i >= 2:
                    ts.append(e0.elapsed_time(e1))
    finally:
        eng.classes3c = every
    return times


def measure(workload: str = "w8") -> dict:
    mol = WORKLOADS[workload]()
    from . import basis as bm

    atoms = list(mol.atoms_bohr)
    ao = bm.pack_basis(atoms, mol.basis, "ao")
    aux = bm.pack_basis(atoms, mol.basis, "aux")
    eng = dfmod.DFEngine(ao, aux)
    Cw, e_scf = _density(mol, eng)
    R = torch.as_tensor(mol.coords_bohr, dtype=torch.float64, device=eng.device)
    X = torch.empty((eng.naux, eng.nao, eng.nao), dtype=torch.float64, device=eng.device)
    E64, g64 = _step(eng, Cw, R, X, "fp64")
    Eall, gall = _step(eng, Cw, R, X, "mixed_all")
    rows = []
    t0 = time.time()
    for entry in list(eng.classes3c):
        cls = tuple(entry[:3])
        with _table(cls):
            Ec, gc = _step(eng, Cw, R, X, "mixed")
        ms64, ms32 = _class_times(eng, entry, X)
        dg = gc - g64
        m64, m32 = float(np.median(ms64)), float(np.median(ms32))
        spread = float(np.percentile(ms64, 75) - np.percentile(ms64, 25))
        rows.append({"kind": "int3c", "cls": list(cls), "dE": Ec - E64, "dg": dg.tolist(),
                     "dg_max": float(np.abs(dg).max()), "ms_fp64": m64, "ms_fp32": m32, "spread": spread})
    return {"workload": workload, "nao": eng.nao, "naux": eng.naux, "natm": eng.natm, "e_scf": e_scf, "E64": E64,
            "dE_all_mixed": Eall - E64, "dg_all_mixed": float(np.abs(gall - g64).max()), "rows": rows,
            "seconds": time.time() - t0}


def select(data: dict, e_budget: float, g_budget: float) -> dict:
    """Greedy admission by time saved per unit of (budget-normalised) error."""
    natm = data["natm"]
    cand = []
    for r in data["rows"]:
        gain = r["ms_fp64"] - r["ms_fp32"]
        if gain <= r["spread"] or r["dE"] == 0.0:  # no clear gain, or a class without an FP32 kernel
            continue
        cost = max(abs(r["dE"]) / e_budget, r["dg_max"] / g_budget, 1e-12)
        cand.append((gain / cost, r))
    cand.sort(key=lambda t: -t[0])
    e_sum = 0.0
    g_sum = np.zeros((natm, 3))
    chosen = {"int3c": []}
    saved = 0.0
    for _score, r in cand:
        e_new = e_sum + abs(r["dE"])
        g_new = g_sum + np.abs(np.asarray(r["dg"]))
        if e_new <= e_budget and float(g_new.max()) <= g_budget:
            e_sum, g_sum = e_new, g_new
            chosen[r["kind"]].append(r["cls"])
            saved += r["ms_fp64"] - r["ms_fp32"]
    return {"int3c": sorted(chosen["int3c"]), "bound_abs_dE": e_sum, "bound_max_abs_dg": float(g_sum.max()),
            "class_ms_saved": saved, "e_budget": e_budget, "g_budget": g_budget}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--workload", default="w8", choices=sorted(WORKLOADS))
    ap.add_argument("--e-budget", type=float, default=2.5e-8)
    ap.add_argument("--g-budget", type=float, default=2.5e-8)
    ap.add_argument("--raw", default=None, help="also write the per-class measurements here (JSON)")
    ap.add_argument("--out", default=OUT)
    args = ap.parse_args()
    data = measure(args.workload)
    if args.raw:
        with open(args.raw, "w") as f:
            json.dump(data, f)
    sel = select(data, args.e_budget, args.g_budget)
    sel.update(workload=args.workload, device=torch.cuda.get_device_name(),
               dE_all_mixed=data["dE_all_mixed"], dg_all_mixed=data["dg_all_mixed"])
    with open(args.out, "w") as f:
        json.dump(sel, f, indent=1)
    print(json.dumps({k: v for k, v in sel.items() if k != "int3c"}))
    print(json.dumps({"int3c": len(sel["int3c"])}))


if __name__ == "__main__":
    main()

"""Primitive-group integral and derivative kernels (``dfb_prim_integrals``, ``dfb_grad_contract``)
against the generic shell-by-shell kernels, over the forms their route accepts.

Both sides evaluate the same FP64 recurrences and differ in the order of sums (the group kernels
contract the auxiliary primitives last, the adjoint first): 2000 ulp (4e-13) of the largest element for integrals, and for the metric
and the derivatives, where the largest primitive terms exceed the contracted result by up to 1e4,
1e-11 as in the oracle tests of the shell-by-shell kernels.
"""

import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _bases(case):
    from asuka_b200 import basis as bm
    from asuka_b200 import geometry as geo

    mol = {"n2": lambda: geo.n2(), "svp": lambda: geo.water_cluster(2, 3, "ma-svp"),
           "tzvp": lambda: geo.water("ma-tzvp"), "qzvp": lambda: geo.water("ma-qzvp"),
           "unshared": lambda: geo.water("ma-svp"), "many": lambda: geo.water("ma-svp"),
           "far": lambda: geo.water_cluster(2, 3, "ma-svp")}[case]()
    atoms = [(el, np.array(x) + (case == "far") * 40.0 * (i >= 3)) for i, (el, x) in enumerate(mol.atoms_bohr)]
    ao, aux = bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux")
    if case == "unshared":  # every shell gets an exponent list of its own: groups of one shell
        e = aux.prim_exp.copy()
        for s in range(aux.nshell):
            a = aux.shell_prim_start[s]
            e[a:a + aux.shell_nprim[s]] *= 1.0 + 1e-3 * s
        aux = dataclasses.replace(aux, prim_exp=e)
    if case == "many":  # groups of 9 to 27 shells: more than one register batch of the contractions
        rep = 9
        idx = np.tile(np.arange(aux.nshell), rep)
        scale = np.repeat(1.0 + 0.1 * np.arange(rep), aux.prim_exp.size)
        l = aux.shell_l[idx]
        nc = (l + 1) * (l + 2) // 2
        start = aux.shell_prim_start[idx] + np.repeat(np.arange(rep) * aux.prim_exp.size, aux.nshell)
        aux = dataclasses.replace(aux, shell_cxyz=aux.shell_cxyz[idx], shell_prim_start=start.astype(np.int32),
                                  shell_nprim=aux.shell_nprim[idx], shell_l=l,
                                  shell_ao_start=(np.cumsum(nc) - nc).astype(np.int32),
                                  prim_exp=np.tile(aux.prim_exp, rep), prim_coef=np.tile(aux.prim_coef, rep) * scale,
                                  shell_atom=aux.shell_atom[idx])
    return ao, aux


def _rel(a, b):
    return float((a - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("wave", [1 << 23, 1], ids=["one-wave", "many-waves"])
@pytest.mark.parametrize("case", ["n2", "svp", "tzvp", "qzvp", "unshared", "many", "far"])
def test_group_kernels_match_shell_kernels(monkeypatch, case, wave):
    """AO l <= 4, aux l <= 8; one and several primitives per chunk (the small-task rule is switched off
    with the small wave); wave 1: one group (or one chunk) per wave."""
    from asuka_b200 import df

    monkeypatch.setattr(df, "PRIM_WAVE", wave)
    if wave == 1:
        monkeypatch.setattr(df, "GRAD_THREADS", 1)
    eng = df.DFEngine(*_bases(case))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)
    bar = torch.randn((eng.naux, eng.nao, eng.nao), generator=gen, dtype=torch.float64, device="cuda")
    bar = bar + bar.transpose(1, 2)
    barm = bar.permute(1, 2, 0).contiguous()
    b2 = torch.randn((eng.naux, eng.naux), generator=gen, dtype=torch.float64, device="cuda")
    b2 = b2 + b2.T

    def run():
        g = [torch.zeros((eng.natm, 3), dtype=torch.float64, device="cuda") for _ in range(4)]
        out = [eng.int3c("Qmn"), eng.int3c("mnQ").permute(2, 0, 1).contiguous(), eng.metric()]
        eng.deriv3c(bar, g[0])
        eng.deriv3c(barm, g[1], layout="mnQ")
        eng.deriv2c(b2, g[2])
        X = torch.empty_like(out[0])
        for p0, p1, blk in eng.aux_blocks(40):  # blocks cut through groups
            X[p0:p1] = eng.int3c_block(blk, p0, p1)
            eng.deriv3c_block(blk, bar[p0:p1], g[3])
        torch.cuda.synchronize()
        return out + [X], g

    new, gnew = run()
    monkeypatch.setenv("DFB_DISABLE_TMPL", "1")
    old, gold = run()
    for i, (a, b) in enumerate(zip(new, old)):
        assert _rel(a, b) < (1e-11 if i == 2 else 4e-13), (i, _rel(a, b))
    assert torch.equal(new[0], new[0].transpose(1, 2)) or _rel(new[0], new[0].transpose(1, 2).contiguous()) < 4e-13
    for i, (a, b) in enumerate(zip(gnew, gold)):
        assert _rel(a, b) < 1e-11, (i, _rel(a, b))
    # one fan-out for both contractions, and the energy step's overlapped integrals
    monkeypatch.delenv("DFB_DISABLE_TMPL")
    g = torch.zeros_like(gold[0])
    eng.deriv3c_2c(bar, b2, g)
    assert _rel(g, gold[0] + gold[2]) < 1e-11
    if case == "many":  # proportional shells: the metric is singular
        return
    V, _L, X = eng.metric_cholesky_int3c()
    assert _rel(V, old[2]) < 1e-11 and _rel(X, old[0]) < 4e-13


def test_ao_shells_above_g_keep_the_shell_kernels():
    """An h shell on the AO side: its classes run shell by shell beside the group classes."""
    from asuka_b200 import basis as bm
    from asuka_b200 import df, geometry as geo

    mol = geo.n2()
    atoms = list(mol.atoms_bohr)
    ao, aux = bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux")
    nsh, npr = ao.nshell, ao.prim_exp.size
    big = dataclasses.replace(
        ao, shell_cxyz=np.vstack([ao.shell_cxyz, ao.shell_cxyz[:1]]),
        shell_prim_start=np.append(ao.shell_prim_start, npr).astype(np.int32),
        shell_nprim=np.append(ao.shell_nprim, 1).astype(np.int32), shell_l=np.append(ao.shell_l, 5).astype(np.int32),
        shell_ao_start=np.append(ao.shell_ao_start, ao.nao).astype(np.int32), prim_exp=np.append(ao.prim_exp, 0.9),
        prim_coef=np.append(ao.prim_coef, 0.3), shell_atom=np.append(ao.shell_atom, 0).astype(np.int32))
    assert big.nshell == nsh + 1
    e0, e1 = df.DFEngine(ao, aux), df.DFEngine(big, aux)
    X0, X1 = e0.int3c("Qmn"), e1.int3c("Qmn")
    n = ao.nao
    assert _rel(X1[:, :n, :n], X0) < 1e-14
    bar = torch.zeros_like(X1)
    bar[:, :n, :n] = X0
    g0 = torch.zeros((e0.natm, 3), dtype=torch.float64, device="cuda")
    g1 = torch.zeros_like(g0)
    e0.deriv3c(X0, g0)
    e1.deriv3c(bar, g1)
    assert _rel(g1, g0) < 1e-12

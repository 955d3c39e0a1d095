"""Host lists of an engine against their definition, on CPU tensors (the kernels are not called)."""

import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _bases(mol):
    from asuka_b200 import basis as bm

    atoms = list(mol.atoms_bohr)
    return bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux")


@pytest.mark.parametrize("screen", [1e-20, 1e-4, 0.0])
@pytest.mark.parametrize("stretch", [1.0, 4.0, 1e3])
def test_pair_lists_of_a_geometry(screen, stretch):
    """Kept primitive pairs, the pairs of a class by (-count, A, B) and the derivative segments by (-length, A, B,
    position), pair by pair; the static part is shared by all geometries."""
    from asuka_b200 import df
    from asuka_b200 import geometry as geo
    from asuka_b200.basis import build_shell_pairs_l_order

    ao, aux = _bases(geo.water_cluster(2, 3, "ma-svp"))
    eng = df.DFEngine.__new__(df.DFEngine)
    eng.ao, eng.aux, eng.device, eng.prim_screen = ao, aux, torch.device("cpu"), screen
    eng.sp = sp = build_shell_pairs_l_order(ao)
    t = torch.zeros(1)
    eng.sp_A = eng.sp_B = eng.ao_cxyz = eng.ao_aostart = eng.ao_atom = t
    eng.aux_by_l = {0: t}
    eng._pair_static = df._PairStatic(ao, sp)
    eng._build_ao_pairs(ao.shell_cxyz)  # another geometry first
    c = ao.shell_cxyz * stretch
    eng._build_ao_pairs(c)

    pairs, segs, dropped = {}, {}, []
    owner, local, start = [], [], []
    for i in range(sp.nsp):
        A, B = int(sp.sp_A[i]), int(sp.sp_B[i])
        R2 = float(((c[A] - c[B]) ** 2).sum())
        kept = []
        for j in range(int(ao.shell_nprim[A]) * int(ao.shell_nprim[B])):
            pa = ao.shell_prim_start[A] + j // ao.shell_nprim[B]
            pb = ao.shell_prim_start[B] + j % ao.shell_nprim[B]
            a, b = ao.prim_exp[pa], ao.prim_exp[pb]
            w = abs(ao.prim_coef[pa] * ao.prim_coef[pb]) * math.exp(-a * b / (a + b) * R2) * (math.pi / (a + b)) ** 1.5
            if w >= screen:
                kept.append(j)
        start.append(len(owner))
        owner += [i] * len(kept)
        local += kept
        key = (int(ao.shell_l[A]), int(ao.shell_l[B]))
        if not kept:
            dropped.append(i)
            continue
        pairs.setdefault(key, []).append((-len(kept), A, B, i))
        for k in range(0, len(kept), df.SEG_PRIMS):
            n = min(df.SEG_PRIMS, len(kept) - k)
            segs.setdefault(key, []).append((-n, A, B, start[-1] + k))
    assert eng.pp_sp.tolist() == owner and eng.pp_local.tolist() == local
    assert eng.sp_pstart.tolist() == start and eng.n_prim_pairs == len(owner)
    assert eng._dropped[0].tolist() == dropped and eng.n_dropped_pairs == len(dropped)
    assert {k: v.tolist() for k, v in eng._pairs3c.items()} == {k: [x[3] for x in sorted(v)] for k, v in pairs.items()}
    assert list(eng._pairs3c) == sorted(pairs)
    A, B, s0, n = (x.tolist() for x in eng._segs)
    assert {k: [(-n[e], A[e], B[e], s0[e]) for e in v.tolist()] for k, v in eng._seg_lists.items()} == \
        {k: sorted(v) for k, v in segs.items()}


@pytest.mark.parametrize("hi", [3, 300, 40000, 1 << 40])
def test_stable_order(hi):
    from asuka_b200.df import _stable_order

    key = np.random.default_rng(hi).integers(-hi, hi, 5000)
    assert np.array_equal(_stable_order(key), np.lexsort((np.arange(5000), key)))
    assert _stable_order(key[:0]).size == 0

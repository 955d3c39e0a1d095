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


def _ints(address, n):
    import ctypes

    return np.array((ctypes.c_int * n).from_address(address)) if n else np.zeros(0, int)


def _doubles(address, n):
    import ctypes

    return np.array((ctypes.c_double * n).from_address(address))


def _longs(address, n):
    import ctypes

    return np.array((ctypes.c_long * n).from_address(address))


@pytest.mark.parametrize("mol", ["n2", "tzvp", "qzvp", "unshared"])
@pytest.mark.parametrize("max_naux", [10 ** 6, 60, 1])
def test_aux_groups_and_their_blocks(mol, max_naux):
    """What the kernels read, from the addresses they get: every shell of a block in one group with its own
    coefficients, rows numbered per l, chunk lists that cover each primitive once, and the first bra entries of the
    metric's lists."""
    import dataclasses

    from asuka_b200 import auxgroups, geometry as geo
    from asuka_b200.auxgroups import NQ, PLO, AuxGroups

    _ao, aux = _bases({"n2": geo.n2("ma-svp"), "tzvp": geo.water("ma-tzvp"), "qzvp": geo.water("ma-qzvp"),
                       "unshared": geo.water("ma-svp")}[mol])
    if mol == "unshared":
        aux = dataclasses.replace(aux, prim_exp=aux.prim_exp * (1.0 + 1e-3 * np.arange(aux.prim_exp.size)))
    dev, t = torch.device("cpu"), torch.zeros(1)
    nc = (aux.shell_l + 1) * (aux.shell_l + 2) // 2
    cuts, s0 = [], 0
    while s0 < aux.nshell:
        s1 = s0 + 1
        while s1 < aux.nshell and nc[s0:s1 + 1].sum() <= max_naux:
            s1 += 1
        cuts.append(np.arange(s0, s1))
        s0 = s1
    shifted = [torch.as_tensor((aux.shell_ao_start - aux.shell_ao_start[c[0]]).astype(np.int32)) for c in cuts]
    whole = AuxGroups(aux, np.arange(aux.nshell), dev, t, t, t)
    sets = AuxGroups.blocks(aux, whole.shell_ids, cuts, dev, t, shifted, t) if max_naux < 10 ** 6 else [whole]
    assert len(sets) == len(cuts)
    for gr, shells, sh in zip(sets, cuts, shifted):
        if gr is not whole:
            assert gr.c.aostart == sh.data_ptr()
        assert sorted(gr.fam) == sorted({int(v) for v in aux.shell_l[shells]})
        seen = []
        for l in gr.fam:
            glist, rows, _first, ng = gr.group_rows(l, 1)
            gl = _ints(glist, 2 * ng).reshape(ng, 2)
            rows = _longs(rows, ng + 1)
            assert np.array_equal(gl[:, 1], rows[:-1])
            ids = _ints(*gr.group_ids(l))
            assert np.array_equal(ids, gl[:, 0])
            lo, hi = gr.prims[l]
            assert np.array_equal(_ints(*gr.prim_ids(l)), np.arange(lo, hi)) and rows[-1] == hi - lo
            most = 0
            info = {}
            for g, row in gl.tolist():
                rep, p0, n, ns, c0, m0 = _ints(gr.c.info + 24 * g, 6).tolist()
                assert (p0 - lo, n) == (row, rows[list(ids).index(g) + 1] - row)
                members = _ints(gr.c.shells + 4 * m0, ns).tolist()
                seen += members
                assert rep == members[0]
                most = max(most, ns)
                info[g] = (p0, n)
                e = aux.prim_exp[aux.shell_prim_start[rep]:][:n]
                assert np.array_equal(_doubles(gr.c.pexp + 8 * p0, n), e)
                assert np.array_equal(_doubles(gr.c.rexp + 8 * p0, n), 1.0 / e)
                for i, s in enumerate(members):
                    a = int(aux.shell_prim_start[s])
                    assert (aux.shell_l[s], aux.shell_atom[s], aux.shell_nprim[s]) == (l, aux.shell_atom[rep], n)
                    assert np.array_equal(aux.prim_exp[a:a + n], e)
                    assert np.array_equal(_doubles(gr.c.coef + 8 * (c0 + i * n), n), aux.prim_coef[a:a + n])
                for k in range(p0, p0 + n):  # the primitives as bra entries
                    assert _ints(gr.bra.shA + 4 * k, 1)[0] == rep and _ints(gr.bra.shB + 4 * k, 1)[0] == g
                    assert _ints(gr.bra.pstart + 4 * k, 1)[0] == k and _ints(gr.bra.npair + 4 * k, 1)[0] == 1
                    assert _doubles(gr.bra.rec + 64 * k, 1)[0] == aux.prim_exp[aux.shell_prim_start[rep] + k - p0]
            assert gr.max_shells[l] == most
            for nq in NQ:
                first = _longs(gr.group_rows(l, nq)[2], ng + 1)
                for plo in PLO[nq]:
                    at, n = gr.chunk_range(l, nq, plo)
                    ch = _ints(at, 5 * n).reshape(n, 5)
                    assert first[-1] == n
                    got = []
                    for i, (g, p, cnt, row, pl) in enumerate(ch.tolist()):
                        j = list(ids).index(g)
                        assert first[j] <= i < first[j + 1] and 1 <= cnt <= nq and row == p - lo
                        assert pl == {"all": 0, "own": info[g][0] - lo, "after": sum(info[g]) - lo}[plo]
                        got += range(p, p + cnt)
                    assert got == list(range(lo, hi))
        assert sorted(seen) == list(shells)
        if mol == "unshared":
            assert set(gr.max_shells.values()) == {1}
    assert len(np.unique(auxgroups.shell_group_ids(aux))) == sum(g1 - g0 for _f, g0, g1 in whole.fam.values())


def test_plan_records_match_the_c_structs():
    import ctypes

    from asuka_b200 import _lib, df

    for dt, cls in ((df._GRAD_CLASS, _lib.GradClass), (df._PRIM_CLASS, _lib.PrimClass)):
        assert dt.itemsize == ctypes.sizeof(cls)
        for name, _t in cls._fields_:
            assert dt.fields[name][1] == getattr(cls, name).offset
            assert dt.fields[name][0].itemsize == getattr(cls, name).size

"""Class lists that a program assigns or edits (``DFEngine.classes3c``): every entry is evaluated with its own
pairs and aux shells, by the integrals and by the derivatives alike."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _bases():
    from asuka_b200 import basis as bm
    from asuka_b200 import geometry as geo

    mol = geo.water_cluster(2, 3, "ma-svp")
    atoms = list(mol.atoms_bohr)
    return bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux")


def _edits(classes):
    """Name -> edited list: a shorter pair list, a class split in two, a shorter aux list, entries left out."""
    i = next(k for k, c in enumerate(classes) if c[3].numel() > 2 and c[4].numel() > 1)
    la, lb, lc, pairs, auxs = classes[i]
    n = pairs.numel() // 2
    parts = [(la, lb, lc, pairs[:n].clone(), auxs), (la, lb, lc, pairs[n:].clone(), auxs)]
    return {"pairs": classes[:i] + parts[:1] + classes[i + 1:], "split": classes[:i] + parts + classes[i + 1:],
            "aux": classes[:i] + [(la, lb, lc, pairs, auxs[:1].clone())] + classes[i + 1:],
            "fewer": classes[:i] + classes[i + 1:], "twice": classes + classes[i:i + 1]}


def test_plans_follow_the_list():
    """Host side on CPU tensors: whole classes go to the group kernels, others keep their lists for the shell
    kernels, and assigned and edited lists both take effect at the next call."""
    import os

    from asuka_b200 import _lib, df
    from asuka_b200.auxgroups import AuxGroups

    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("library not built")
    _ao, aux = _bases()
    dev = torch.device("cpu")
    eng = df.DFEngine.__new__(df.DFEngine)
    t = torch.zeros(1)
    eng.groups = AuxGroups(aux, np.arange(aux.nshell), dev, t, t, t)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    eng._pairs3c = {(0, 0): i32(0, 1, 2, 3), (1, 0): i32(4, 5, 6)}
    eng._seg_lists = {k: v.clone() for k, v in eng._pairs3c.items()}
    eng.aux_by_l = {int(l): i32(*np.nonzero(aux.shell_l == l)[0]) for l in np.unique(aux.shell_l)}
    built = [(a, b, c, p, x) for (a, b), p in eng._pairs3c.items() for c, x in eng.aux_by_l.items()]
    eng.classes3c = list(built)
    for kind in ("int", "der"):
        arr, n, old, _per = eng._plan(kind, eng.groups, "fp64")
        assert n == len(built) and not old
        assert eng._plan(kind, eng.groups, "fp64")[0] is arr  # kept
    n_new = {"pairs": -1, "split": -1, "aux": -1, "fewer": -1, "twice": 1}
    n_old = {"pairs": 1, "split": 2, "aux": 1, "fewer": 0, "twice": 0}
    for name, edited in _edits(built).items():
        for in_place in (False, True):
            if in_place:
                eng.classes3c = list(built)
                eng._plan("int", eng.groups, "fp64")
                eng.classes3c[:] = edited
            else:
                eng.classes3c = edited
            for kind in ("int", "der"):
                _arr, n, old, _per = eng._plan(kind, eng.groups, "fp64")
                assert (n, len(old)) == (len(built) + n_new[name], n_old[name]), (name, kind)
                for c in old:
                    assert any(c[3] is e[3] and c[4] is e[4] for e in edited)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["pairs", "split", "aux", "fewer", "twice"])
def test_edited_lists_match_the_shell_kernels(monkeypatch, name):
    """Integrals (over a zero-filled tensor) and derivatives of an edited list against the shell kernels with the
    same list; blocks of aux shells too."""
    from asuka_b200 import df

    eng = df.DFEngine(*_bases(), prim_screen=0.0)
    eng.classes3c = _edits(eng.classes3c)[name]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    bar = torch.randn((eng.naux, eng.nao, eng.nao), generator=gen, dtype=torch.float64, device="cuda")
    bar = bar + bar.transpose(1, 2)

    def run():
        X = eng.int3c("Qmn", out=torch.zeros_like(bar))
        Xb = torch.zeros_like(bar)
        g, gb = (torch.zeros((eng.natm, 3), dtype=torch.float64, device="cuda") for _ in range(2))
        eng.deriv3c(bar, g)
        for p0, p1, blk in eng.aux_blocks(50):
            eng.int3c_block(blk, p0, p1, out=Xb[p0:p1])
            eng.deriv3c_block(blk, bar[p0:p1], gb)
        return X, Xb, g, gb

    new = run()
    monkeypatch.setenv("DFB_DISABLE_TMPL", "1")
    old = run()
    for i, (a, b) in enumerate(zip(new, old)):
        assert float((a - b).abs().max()) <= (4e-13 if i < 2 else 1e-11) * float(b.abs().max()), i


@pytest.mark.gpu
def test_one_block_takes_the_engines_lists():
    """A block that holds the whole aux basis shares the engine's groups (nothing is built for it twice), and is
    bit for bit the whole tensor; smaller blocks have groups of their own."""
    from asuka_b200 import df

    eng = df.DFEngine(*_bases())
    ((p0, p1, blk),) = eng.aux_blocks(10 ** 6)
    assert (p0, p1) == (0, eng.naux) and blk[3] is eng.groups
    assert torch.equal(eng.int3c_block(blk, p0, p1), eng.int3c("Qmn"))
    assert all(b[2][3] is not eng.groups for b in eng.aux_blocks(50))

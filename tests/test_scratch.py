"""Scratch of the integral calls: rows of primitive integrals belong to one call."""

import ctypes

import pytest

torch = pytest.importorskip("torch")


class _FakeLib:
    """Records the scratch range of every integral call."""

    def __init__(self):
        self.ranges = []

    def dfb_prim_integrals(self, _bra, _groups, _arr, _ncls, _out, _sp, _sm, _sn, ptr, doubles, _streams, _n):
        self.ranges.append((ptr, ptr + 8 * doubles))
        return 0


def _overlap(a, b):
    return a[0] < b[1] and b[0] < a[1]


def test_calls_in_flight_have_their_own_rows(monkeypatch):
    """Two calls of one engine before the first has ended (its fork is open), larger and smaller needs first."""
    from types import SimpleNamespace as NS

    from asuka_b200 import _lib, df

    fake = _FakeLib()
    monkeypatch.setattr(_lib, "lib", lambda: fake)
    eng = df.DFEngine.__new__(df.DFEngine)
    eng.device = torch.device("cpu")
    eng._scratch = df.ScratchHolder()
    monkeypatch.setattr(df.DFEngine, "_fork", lambda self: (0, 8, (ctypes.c_void_p * 8)()))
    monkeypatch.setattr(df.DFEngine, "_join", lambda self, fork: None)
    out = torch.zeros(1)
    groups = NS(c=_lib.Groups())
    for first, second in ((1000, 40), (40, 1000), (64, 64)):
        fake.ranges.clear()
        held = [eng._run_int([(_lib.Bra(), groups, None, 1, need, out, (0, 0, 0), [])]) for need in (first, second)]
        a, b = fake.ranges
        assert a[1] - a[0] >= 64 * first and b[1] - b[0] >= 64 * second  # eight slices of 8-byte doubles
        assert not _overlap(a, b)
        assert len(held) == 2


def _engine(n=2):
    from asuka_b200 import basis as bm
    from asuka_b200 import geometry as geo
    from asuka_b200.df import DFEngine

    mol = geo.water_cluster(n, 3, "ma-svp")
    atoms = list(mol.atoms_bohr)
    return DFEngine(bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux"))


@pytest.mark.gpu
def test_calls_from_two_streams():
    """Metric and 3c integrals of one engine issued from two streams, whose kernels run beside each other."""
    eng = _engine()
    V0, X0 = eng.metric(), eng.int3c("Qmn")
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(5):
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            torch.cuda._sleep(200000)
            V = eng.metric()
        with torch.cuda.stream(b):
            X = eng.int3c("Qmn")
        with torch.cuda.stream(a):
            V2 = eng.metric()
        torch.cuda.synchronize()
        assert torch.equal(V, V0) and torch.equal(V2, V0) and torch.equal(X, X0)


@pytest.mark.gpu
def test_captured_call_outlives_larger_ones():
    """A captured metric replayed after a call with a larger need, with the freed memory written over."""
    eng = _engine()
    V0 = eng.metric()
    eng2 = _engine()
    eng2.metric()
    torch.cuda.synchronize()
    V = torch.empty_like(V0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        eng2.metric(out=V)
    eng2.int3c("Qmn")
    junk = [torch.full((1 << 20,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(8)]
    for _ in range(2):
        V.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(V, V0)
    assert all(bool(torch.isnan(t).all()) for t in junk)  # the replay wrote to none of it


@pytest.mark.parametrize("l", [(0, 0, 0), (1, 1, 2), (2, 1, 4), (4, 4, 6)])
@pytest.mark.parametrize("npair", [1, 32, 33, 5000])
def test_rows_stay_within_the_target(l, npair):
    """Scratch of one class on the host: the target, or one group over all pairs up to four times as much, or one
    group over one tile of 32 pairs, unless all rows take less; the pair count does not enter otherwise."""
    import numpy as np

    from asuka_b200 import _lib

    if not __import__("os").path.exists(_lib.LIB_PATH):
        pytest.skip("library not built")
    L = _lib.lib()
    rows = np.array([0, 5, 27, 30], dtype=np.int64)  # groups of 5, 22 and 3 primitives
    nc = [(k + 1) * (k + 2) // 2 for k in range(10)]
    la, lb, lc = l
    tile = 32 * nc[lc] * sum(nc[la:la + lb + 1])
    c = _lib.PrimClass(la, lb, lc, npair, 0, 0, 0, rows.ctypes.data, rows.ctypes.data, 3, 2, 0, 0, 0, 0)
    for target in (1, 1 << 16, 1 << 20, 1 << 30):
        need = L.dfb_prim_scratch(ctypes.byref(c), 1, target)
        tiles = -(-npair // 32)
        assert need <= max(4 * target, 22 * tile)
        group = 22 * tile * tiles if 22 * tile * tiles <= 4 * target else max(4 * target, 22 * tile)
        assert need == min(max(target, group), 30 * tile * tiles)
    c.bra_groups = 1  # metric: all pairs
    need = L.dfb_prim_scratch(ctypes.byref(c), 1, 1)
    assert need == 22 * tile * -(-npair // 32)


@pytest.mark.gpu
@pytest.mark.parametrize("share", [0.0, 1.0], ids=["memset", "blocks"])
def test_zeros_of_dropped_pairs(monkeypatch, share):
    """Both ways of clearing the dropped pairs leave the same integrals in both layouts, over a NaN-filled tensor
    for the blocks of which there are some and none."""
    import numpy as np

    from asuka_b200 import basis as bm
    from asuka_b200 import df, geometry as geo

    monkeypatch.setattr(df, "ZERO_SHARE", (share, share))
    mol = geo.water_cluster(2, 3, "ma-svp")
    atoms = [(el, np.array(x) + 40.0 * (i >= 3)) for i, (el, x) in enumerate(mol.atoms_bohr)]  # far apart
    eng = df.DFEngine(bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux"))
    assert eng.n_dropped_pairs
    full = df.DFEngine(eng.ao, eng.aux, prim_screen=0.0)
    assert not full.n_dropped_pairs
    ref = full.int3c("Qmn")
    for layout, back in (("Qmn", (0, 1, 2)), ("mnQ", (2, 0, 1))):
        shape = (eng.naux, eng.nao, eng.nao) if layout == "Qmn" else (eng.nao, eng.nao, eng.naux)
        X = torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")
        X = eng.int3c(layout, out=X).permute(back)
        assert float((X - ref).abs().max()) <= 1e-13 * float(ref.abs().max())
        assert float((X == 0).double().mean()) > 0.3


@pytest.mark.parametrize("layout,share,blocks", [("Qmn", 0.05, True), ("Qmn", 0.1, False), ("Qmn", 0.2, False),
                                                 ("mnQ", 0.1, True), ("mnQ", 0.2, True), ("mnQ", 0.3, False)])
def test_rule_of_the_zeros(monkeypatch, layout, share, blocks):
    """The measured crossing, about 0.07 of a 'Qmn' tensor and 0.3 of a large 'mnQ' one."""
    from asuka_b200 import _lib, df

    calls = []
    fake = type("L", (), {"dfb_zero_pairs": lambda self, *a: calls.append(a) or 0})()
    monkeypatch.setattr(_lib, "lib", lambda: fake)
    monkeypatch.setattr(df, "_stream", lambda: 0)
    eng = df.DFEngine.__new__(df.DFEngine)
    eng.n_dropped_pairs, eng.bra_ao = 3, _lib.Bra()
    lst = torch.zeros(3, dtype=torch.int32)
    eng._dropped = (lst, lst, share)
    X = torch.ones(8)
    eng._clear_dropped(X, (16, 4, 1) if layout == "Qmn" else (1, 32, 8), 8)
    assert bool(calls) == blocks and bool((X == 0).all()) != blocks


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["whole", "edited", "h shell", "generic"])
def test_first_call_under_capture(monkeypatch, form):
    """The first integral, metric and derivative calls of an engine, recorded into a graph, for the classes of the
    group kernels and for those that stay on the shell kernels: nothing is uploaded by a call."""
    import dataclasses

    import numpy as np

    from asuka_b200 import basis as bm
    from asuka_b200 import df, geometry as geo

    if form == "generic":
        monkeypatch.setenv("DFB_DISABLE_TMPL", "1")
    mol = geo.n2()
    atoms = list(mol.atoms_bohr)
    ao, aux = bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux")
    if form == "h shell":
        ao = dataclasses.replace(
            ao, shell_cxyz=np.vstack([ao.shell_cxyz, ao.shell_cxyz[:1]]),
            shell_prim_start=np.append(ao.shell_prim_start, ao.prim_exp.size).astype(np.int32),
            shell_nprim=np.append(ao.shell_nprim, 1).astype(np.int32), shell_l=np.append(ao.shell_l, 5).astype(np.int32),
            shell_ao_start=np.append(ao.shell_ao_start, ao.nao).astype(np.int32), prim_exp=np.append(ao.prim_exp, 0.9),
            prim_coef=np.append(ao.prim_coef, 0.3), shell_atom=np.append(ao.shell_atom, 0).astype(np.int32))

    def engine():
        eng = df.DFEngine(ao, aux)
        if form == "edited":
            eng.classes3c = [(a, b, c, p.clone(), x) for a, b, c, p, x in eng.classes3c]
        return eng

    ref = engine()
    bar = torch.ones((ref.naux, ref.nao, ref.nao), dtype=torch.float64, device="cuda")
    bar2 = torch.ones((ref.naux, ref.naux), dtype=torch.float64, device="cuda")

    def calls(eng, X, V, g):
        eng.int3c("Qmn", out=X)
        eng.metric(out=V)
        eng.deriv3c(bar, g)
        eng.deriv2c(bar2, g)

    def outputs(eng):
        return (torch.zeros_like(bar), torch.zeros_like(bar2), torch.zeros((eng.natm, 3), dtype=torch.float64, device="cuda"))

    want = outputs(ref)
    calls(ref, *want)
    eng = engine()
    got = outputs(eng)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls(eng, *got)
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())

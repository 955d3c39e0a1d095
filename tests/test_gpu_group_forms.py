"""Group kernels in the forms that the small molecules of the other tests do not reach by themselves: tasks of
sixteen primitives, FP32 classes and the gradient of many atoms."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _engine(n=2, basis="ma-svp"):
    from asuka_b200 import basis as bm
    from asuka_b200 import geometry as geo
    from asuka_b200.df import DFEngine

    mol = geo.water_cluster(n, 3, basis)
    atoms = list(mol.atoms_bohr)
    return DFEngine(bm.pack_basis(atoms, mol.basis, "ao"), bm.pack_basis(atoms, mol.basis, "aux"))


def _bars(eng):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    b3 = torch.randn((eng.naux, eng.nao, eng.nao), generator=gen, dtype=torch.float64, device="cuda")
    b2 = torch.randn((eng.naux, eng.naux), generator=gen, dtype=torch.float64, device="cuda")
    return b3 + b3.transpose(1, 2), b2 + b2.T


def _grads(eng, bars, natm):
    out = [torch.zeros((natm, 3), dtype=torch.float64, device="cuda") for _ in range(2)]
    eng.deriv3c(bars[0], out[0])
    eng.deriv2c(bars[1], out[1])
    return out


@pytest.mark.parametrize("n,basis", [(2, "ma-svp"), (1, "ma-tzvp"), (1, "ma-qzvp")])
def test_tasks_of_sixteen_primitives(monkeypatch, n, basis):
    """All derivative classes with the largest task size (groups hold 1 to 22 primitives, so the last chunk of a
    group is shorter), against the shell kernels and the size that the rule gives."""
    from asuka_b200 import df

    eng = _engine(n, basis)
    bars = _bars(eng)
    rule = _grads(eng, bars, eng.natm)
    monkeypatch.setattr(df, "GRAD_THREADS", 1)
    monkeypatch.setattr(df, "GRAD_BIG", 1)
    eng.groups.plans.clear()
    arr, ncls, old, _per = eng._plan("der", eng.groups, "fp64")
    assert ncls and not old and {arr[i].nq for i in range(ncls)} == {16}
    big = _grads(eng, bars, eng.natm)
    monkeypatch.setenv("DFB_DISABLE_TMPL", "1")
    ref = _grads(eng, bars, eng.natm)
    for a, b, c in zip(big, rule, ref):
        scale = float(c.abs().max())
        assert float((a - c).abs().max()) <= 1e-11 * scale and float((b - c).abs().max()) <= 1e-11 * scale


@pytest.mark.parametrize("natm", [682, 683, 2000])
def test_gradient_of_many_atoms(natm):
    """Up to 682 atoms the gradient is summed in shared memory, beyond in global memory."""
    eng = _engine()
    bars = _bars(eng)
    ref = _grads(eng, bars, eng.natm)
    n = eng.natm
    eng.natm = natm
    for a, b in zip(_grads(eng, bars, natm), ref):
        assert float((a[:n] - b).abs().max()) <= 1e-12 * float(b.abs().max())
        assert float(a[n:].abs().max()) == 0.0


@pytest.mark.parametrize("basis", ["ma-svp", "ma-tzvp"])
@pytest.mark.parametrize("layout", ["Qmn", "mnQ"])
def test_fp32_classes(monkeypatch, basis, layout):
    """Every class in FP32: about twelve recurrence steps of 2^-24 on primitive terms up to ten times the result,
    1e-5 of the largest element; and really another arithmetic than FP64."""
    from asuka_b200 import df

    eng = _engine(1, basis)
    ref = eng.int3c(layout)
    monkeypatch.setattr(df, "mixed_class_table", lambda: {"int3c": {tuple(c[:3]) for c in eng.classes3c}})
    X = eng.int3c(layout, precision="mixed")
    err = float((X - ref).abs().max() / ref.abs().max())
    assert 1e-12 < err < 1e-5

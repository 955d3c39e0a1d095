"""The precision table of the mixed mode: admitted by measurements of the kernels that the mode runs."""

import json
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def test_table_names_integral_classes_within_the_budget():
    from asuka_b200 import df, tune_precision

    with open(tune_precision.OUT) as f:
        t = json.load(f)
    assert set(df.mixed_class_table()) == {"int3c"} and "deriv3c" not in t and "deriv2c" not in t
    assert t["int3c"] and t["bound_abs_dE"] <= t["e_budget"] <= 2.5e-8 and t["bound_max_abs_dg"] <= t["g_budget"]
    assert os.path.getsize(tune_precision.OUT) < 4096


def test_selection_takes_clear_gains_only():
    """Classes whose FP32 runs are slower, equal within the spread of the FP64 runs or without an FP32 kernel
    (no change of the energy at all) stay in FP64, and the sums stay within the budgets."""
    from asuka_b200.tune_precision import select

    def row(cls, dE, gain, spread=0.01):
        return {"kind": "int3c", "cls": cls, "dE": dE, "dg": np.full((2, 3), dE).tolist(), "dg_max": abs(dE),
                "ms_fp64": 1.0, "ms_fp32": 1.0 - gain, "spread": spread}

    rows = [row([0, 0, 0], 1e-9, -0.1), row([0, 0, 1], 1e-9, 0.005), row([0, 0, 2], 0.0, 0.2), row([0, 0, 3], -1e-9, 0.1),
            row([0, 0, 4], 1.5e-8, 0.1), row([0, 0, 5], 1.5e-8, 0.1)]
    sel = select({"natm": 2, "rows": rows}, 2e-8, 2e-8)
    assert sel["int3c"] == [[0, 0, 3], [0, 0, 4]]
    assert sel["bound_abs_dE"] == pytest.approx(1.6e-8)


@pytest.mark.gpu
@pytest.mark.parametrize("name,g_tol", [("w8_matzvp", 2e-8), ("decane_masvp", 2e-8), ("h2o_maqzvp", 1.7e-7)])
def test_mixed_energy_and_gradient_stay_close(name, g_tol):
    """The FP32 classes move the energy and the gradient at the converged density by less than 4e-8 Eh and
    2e-8 Eh/bohr (the table's budget is 2.5e-8 on (H2O)8; the shell kernels' table moved (H2O)8 by 3.9e-8).  In a
    basis that the table was not measured on: FP32 rounding, 2^-24, of gradient elements up to 2.8 Eh/bohr."""
    from _util import bases_of, golden

    from asuka_b200.df import DFEngine
    from asuka_b200.grad import df_energy

    g = golden(name)
    ao, aux, _sp = bases_of(g)
    eng = DFEngine(ao, aux)
    Cw = torch.as_tensor(g["Cw"], device="cuda").contiguous()
    out = []
    for precision in ("fp64", "mixed"):
        R = torch.as_tensor(g["coords_bohr"], device="cuda").requires_grad_(True)
        E, _J, _K = df_energy(R, Cw, eng, precision)
        (gR,) = torch.autograd.grad(E, R)
        out.append((float(E.detach()), gR.cpu().numpy()))
    (E0, g0), (E1, g1) = out
    assert abs(E1 - E0) <= 4e-8, E1 - E0
    assert np.abs(g1 - g0).max() <= g_tol, np.abs(g1 - g0).max()

"""Non-affine hexahedra beyond test_gpu_general.py: set-up, and the column form's sizes.

Creation of a mixed-precision case: the residual of the
uniform state, which every later residual subtracts, is formed from a state
that has arrived on the device.  A previous case leaves its freed memory
behind, so a kernel that runs ahead of the upload reads something else; the
sizes are those at which it did (states of 1.1 to 1.6 MB).

Bar: creation and arithmetic are deterministic, so every case gives the bits of
the first one."""
import numpy as np
import pytest

import dg_b200
from test_gpu_general import bent_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [15, 16, 17])
def test_mixed_case_on_reused_memory(n):
    mesh = bent_box((n, n, n))
    first = None
    for _ in range(3):
        other = dg_b200.Case(mesh, 1, gas_constant=1.0)
        U = other.project_ic("IsentropicVortexXY", [1.0, 1.0, 1.0, 1.0, 2.0, 5.0, 5.0, 10.0, 10.0])
        other.close()
        case = dg_b200.Case(mesh, 1, gas_constant=1.0, precision="mixed_fp32")
        case.set_state(U)
        R = case.residual()
        case.close()
        assert np.isfinite(R).all()
        first = R if first is None else first
        assert np.array_equal(R, first)


@pytest.mark.parametrize("flux", ["LaxFriedrichs", "HLLC"])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_general_column_form_over_many_batches(p, flux):
    """FP64 column form on bent, turned elements, more of them than CTAs (13 x 13 x
    11) and fewer: residual, one mass-inverse update and RK4 steps against the
    one-launch kernel.  Sums differ in order only: 1e-12 of the largest entry, as
    between the kernels' forms elsewhere (1e-10 for the update, which cancels)."""
    for n in ((13, 13, 11), (2, 3, 1)):
        case = dg_b200.Case(bent_box(n, rotate_seed=3, amplitude=0.05), p, flux=flux, gas_constant=1.0)
        vs = [(i, v[4].split("+")) for i, v in enumerate(case.stage_variants()) if v[3] == "fp64"]
        plain = next(i for i, o in vs if "ge" in o and "fx" not in o)
        column = next(i for i, o in vs if "ge" in o and "cf" in o)
        U = case.project_ic("IsentropicVortexXY", [1.0, 1.0, 1.0, 1.0, 2.0, 5.0, 5.0, 10.0, 10.0])
        dt = case.cfl_time_step(U, 0.05)
        out = {}
        for i in (plain, column):
            case.stage_variant = i
            case.set_state(U)
            R, K = case.residual(), case.mass_inverse_residual(dt)
            case.rk4(dt, 2)
            out[i] = R, K, case.get_state()
        for a, b, bar in zip(out[plain], out[column], (1e-12, 1e-10, 1e-12)):
            assert np.abs(a - b).max() <= bar * np.abs(a).max()
        case.close()

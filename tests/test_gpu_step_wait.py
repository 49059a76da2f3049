"""The waits between blocks of the one-launch RK4 steps, made to run out: a step with an
arrival withheld ends with DG_ERR_TIMEOUT after its short limit, the state stays, and the
context's counters start again -- the next steps give the bits of a context that never
gave up."""
import time

import numpy as np
import pytest

import dg_b200

pytestmark = pytest.mark.gpu

XY = [1.0, 0.4, -0.3, 1.0, 2.0, 5.0, 4.5, 10.0, 9.0]
LIMIT = 2_000_000  # SM cycles, about 1 ms


def gives_up_and_goes_on(make):
    case, other = make(), make()
    U = case.project_ic("IsentropicVortexXY", XY)
    other.set_state(U)
    case.rk4(1e-4, 3)
    other.rk4(1e-4, 3)
    U = case.get_state()
    for limit in (0, LIMIT):
        t = time.perf_counter()
        with pytest.raises(dg_b200.DGError, match="TIMEOUT"):
            case.probe_step_wait(limit)
        assert time.perf_counter() - t < 0.5
        assert np.array_equal(case.get_state(), U)
        case.rk4(1e-4, 2)
        other.rk4(1e-4, 2)
        U = case.get_state()
        assert np.array_equal(U, other.get_state())
    case.status()  # (reports the timeouts)
    case.fe(1e-4, 3)
    other.fe(1e-4, 3)
    assert np.array_equal(case.get_state(), other.get_state())
    assert case.status() == 0


@pytest.mark.parametrize("precision", ["fp64", "mixed_fp32"])
@pytest.mark.parametrize("n,p", [((1, 1, 1), 3), ((8, 7, 6), 1), ((6, 6, 6), 5)])
def test_small_mesh_steps(n, p, precision):
    gives_up_and_goes_on(lambda: dg_b200.Case(dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (10.0, 9.0, 10.0), rotate_seed=2), p,
                                              gas_constant=1.0, precision=precision))


@pytest.mark.parametrize("n,p", [((1, 1), 2), ((20, 19), 0), ((40, 41), 3)])
def test_small_mesh_steps_2d(n, p):
    gives_up_and_goes_on(lambda: dg_b200.Case2D(dg_b200.periodic_box_2d(n, (0.0, 0.0), (10.0, 9.0)), p, gas_constant=1.0))


def test_probe_refuses_meshes_that_do_not_wait():
    case = dg_b200.Case(dg_b200.periodic_box((16, 16, 16)), 3)
    case2 = dg_b200.Case2D(dg_b200.periodic_box_2d((120, 120)), 3)
    for c in (case, case2):
        with pytest.raises(dg_b200.DGError, match="UNSUPPORTED"):
            c.probe_step_wait(LIMIT)
        with pytest.raises(dg_b200.DGError, match="ARG"):
            c.probe_step_wait(-1)

"""The column form on meshes of more elements than its CTAs take at once."""
import numpy as np
import pytest

import dg_b200

pytestmark = pytest.mark.gpu

XY = [1.0, 1.0, 1.0, 1.0, 2.0, 5.0, 5.0, 10.0, 10.0]


@pytest.mark.parametrize("precision", ["fp64", "mixed_fp32"])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5])
def test_forward_euler_steps_of_a_call_follow_one_another(p, precision):
    """The face kernel of a step may start before the step ahead has ended: the
    steps of one call give the bits of as many calls, on a mesh that fits at once and
    on one that does not."""
    for n in ((3, 4, 3), (13, 12, 14)):
        mesh = dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (10.0, 10.0, 10.0), rotate_seed=5)
        case = dg_b200.Case(mesh, p, gas_constant=1.0, precision=precision)
        case.stage_variant = next(i for i, v in enumerate(case.stage_variants())
                                  if v[3] == precision and {"cf", "sm"} & set(v[4].split("+")) == {"cf"} and "ge" not in v[4])
        U = case.project_ic("IsentropicVortexXY", XY)
        dt = case.cfl_time_step(U, 0.1)
        for _ in range(6):
            case.fe(dt, 1)
        one_by_one = case.get_state()
        case.set_state(U)
        case.fe(dt, 6)
        assert np.array_equal(case.get_state(), one_by_one)
        assert case.status() == 0
        case.close()


def more_than_resident(per_batch):
    """A mesh of more batches than the 32 one-warp CTAs to an SM, which is the most one
    holds, the last batch partly filled."""
    import torch

    n = int(np.ceil((32 * torch.cuda.get_device_properties(0).multi_processor_count * per_batch) ** (1.0 / 3.0)))
    while per_batch > 1 and n % per_batch == 0:
        n += 1
    return n, n, n  # (per_batch is 1 or a prime)


def outputs(case, v, U, dt):
    case.stage_variant = v
    case.set_state(U)
    out = [case.residual(), case.mass_inverse_residual(dt)]
    case.rk4(dt, 2)
    out.append(case.get_state())
    case.set_state(U)
    case.fe(dt, 2)
    return out + [case.get_state()]


@pytest.mark.parametrize("flux", ["LaxFriedrichs", "HLLC"])
@pytest.mark.parametrize("precision", ["fp64", "mixed_fp32"])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5])
def test_column_form_over_many_batches(p, precision, flux):
    """Against the stage kernel: FP64 to rounding (sums in another order: 1e-12 of the
    largest entry, 1e-10 for the update, which cancels), mixed precision bit for
    bit on an unturned mesh and to the mixed bar of 1e-6 on a turned one."""
    for turned in (0, 9):
        if precision == "fp64" and not turned:
            continue
        case = dg_b200.Case(dg_b200.periodic_box((2, 2, 2)), p, precision=precision)
        vs = [(i, v[0], v[4].split("+")) for i, v in enumerate(case.stage_variants()) if v[3] == precision and "ge" not in v[4]]
        column, batch = next((i, e) for i, e, o in vs if "cf" in o and "sm" not in o)
        stage = next(i for i, _, o in vs if "cf" not in o and "fx" in o or "cf" not in o and p == 1)
        n = more_than_resident(batch)
        mesh = dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (10.0, 10.0, 10.0), rotate_seed=turned)
        case = dg_b200.Case(mesh, p, flux=flux, gas_constant=1.0, precision=precision)
        U = case.project_ic("IsentropicVortexXY", XY)
        dt = case.cfl_time_step(U, 0.1)
        want, got = outputs(case, stage, U, dt), outputs(case, column, U, dt)
        for a, b, bar in zip(want, got, (1e-12, 1e-10, 1e-12, 1e-12)):
            if precision == "fp64":
                assert np.abs(a - b).max() <= bar * np.abs(a).max()
            elif not turned:
                assert np.array_equal(a, b)
        if precision != "fp64" and turned:
            for a, b in zip(want[2:], got[2:]):
                assert np.linalg.norm(a - b) < 1e-6 * np.linalg.norm(a)
        assert case.status() == 0
        case.close()


@pytest.mark.parametrize("flux", ["LaxFriedrichs", "HLLC"])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_general_column_form_beyond_what_is_resident(p, flux):
    """FP64 column form on bent, turned elements against the one-launch kernel, bars as above."""
    from test_gpu_general import bent_box

    case = dg_b200.Case(bent_box(more_than_resident(1), rotate_seed=3, amplitude=0.05), p, flux=flux, gas_constant=1.0)
    vs = [(i, v[4].split("+")) for i, v in enumerate(case.stage_variants()) if v[3] == "fp64"]
    plain = next(i for i, o in vs if "ge" in o and "fx" not in o)
    column = next(i for i, o in vs if "ge" in o and "cf" in o)
    U = case.project_ic("IsentropicVortexXY", XY)
    dt = case.cfl_time_step(U, 0.05)
    for a, b, bar in zip(outputs(case, plain, U, dt), outputs(case, column, U, dt), (1e-12, 1e-10, 1e-12, 1e-12)):
        assert np.abs(a - b).max() <= bar * np.abs(a).max()
    case.close()

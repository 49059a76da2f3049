"""The tuner's choice on meshes whose RK4 steps may run in one launch (option
"sm"): the variant it returns is the one it timed as the fastest, a batch, which
launches stages by themselves, never gets the one-launch form, and forward Euler
runs the fastest stage that is launched by itself.  That choice is read off the
bits of an update (the kernels' sums differ in order), at p = 5, where the
fastest is ahead by a third."""
import numpy as np
import pytest

import dg_b200

pytestmark = pytest.mark.gpu

XY = [1.0, 1.0, 1.0, 1.0, 2.0, 5.0, 5.0, 10.0, 10.0]


def options(case):
    return [v[4].split("+") for v in case.stage_variants()]


@pytest.mark.parametrize("precision", ["fp64", "mixed_fp32"])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5])
def test_tuner_returns_what_it_measured(p, precision):
    mesh = dg_b200.periodic_box((3, 3, 2), (0.0, 0.0, 0.0), (10.0, 10.0, 10.0))
    case = dg_b200.Case(mesh, p, gas_constant=1.0, precision=precision)
    U = case.project_ic("IsentropicVortexXY", XY)
    U[:, :, 3] = -0.0  # a state is put back to the bit
    case.set_state(U)
    best, ms = case.tune_stage(reps=20)
    assert np.array_equal(case.get_state().view(np.int64), U.view(np.int64)) and case.status() == 0
    assert best == case.stage_variant and ms[best] == min(t for t in ms if t > 0)
    if p != 5:
        return
    one_launch = [i for i, o in enumerate(options(case)) if "sm" in o]
    alone = min((t, i) for i, t in enumerate(ms) if t > 0 and i not in one_launch)[1]
    dt = case.cfl_time_step(U, 0.1)
    case.fe(dt, 2)
    other = dg_b200.Case(mesh, p, gas_constant=1.0, precision=precision)
    other.stage_variant = alone
    other.set_state(U)
    other.fe(dt, 2)
    assert np.array_equal(case.get_state(), other.get_state())


def test_tuned_batch_launches_stages():
    mesh = dg_b200.periodic_box((3, 2, 2), (0.0, 0.0, 0.0), (10.0, 10.0, 10.0))
    batch = dg_b200.Batch([(mesh, p) for p in (1, 2, 3, 4, 5)], gas_constant=1.0)
    for i in range(5):
        batch.project_ic(i, "IsentropicVortexXY", XY)
        batch.set_time_step(i, 1e-3)
    batch.tune(reps=5)
    batch.single_launch = False  # each group its own variant
    for order, _, _, variant in batch.groups():
        case = dg_b200.Case(mesh, order)
        assert "sm" not in options(case)[variant], order
        case.close()
    batch.rk4(1)
    assert batch.status() == 0

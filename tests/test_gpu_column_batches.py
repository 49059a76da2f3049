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

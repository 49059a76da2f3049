"""The 2D steps on both sides of the size up to which they run in one launch
(every stage warp one batch of 32 / (p+2) elements, four to an SM), on counts
that leave the last batch and the last edge batch partly filled, against the
oracle (1e-12 after time steps, the bar of test_gpu_2d.py)."""
import numpy as np
import pytest

import dg_b200
import pyoracle
from test_gpu_2d import rel_l2

pytestmark = pytest.mark.gpu

XY = [1.0, 0.4, -0.3, 1.0, 3.0, 5.0, 4.5, 10.0, 9.0]


@pytest.mark.parametrize("flux", ["LaxFriedrichs", "HLLC"])
@pytest.mark.parametrize("side", ["one launch", "two launches"])
@pytest.mark.parametrize("p", [0, 1, 2, 3, 4, 5])
def test_steps_on_both_sides_of_the_one_launch_size(p, side, flux):
    import torch

    most = 32 // (p + 2) * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    n = int(np.sqrt(most)) - (1 if side == "one launch" else -2)
    mesh = dg_b200.periodic_box_2d((n, n - 1 if side == "one launch" else n + 1), (0.0, 0.0), (10.0, 9.0), rotate_seed=3)
    assert (mesh.nelem <= most) == (side == "one launch")
    gpu = dg_b200.Case2D(mesh, p, flux=flux, gas_constant=1.0)
    orc = pyoracle.OracleCase2D.from_mesh(mesh, p, flux=flux, gas_constant=1.0)
    U = orc.project_ic("IsentropicVortexXY", XY)
    gpu.set_state(U)
    gpu.rk4(1e-3, 2)
    assert rel_l2(gpu.get_state(), orc.rk4(U, 1e-3, 2)).max() < 1e-12
    assert gpu.status() == 0

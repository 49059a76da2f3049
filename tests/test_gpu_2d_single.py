"""2D forward Euler and residuals on both sides of the size up to which they run in
one launch, on counts that leave batches partly filled and blocks with one to four
batches, on meshes whose unlisted edges keep a zero lift, and on one element whose
edges are its own neighbours'; against the oracle (residual 1e-11, time steps 1e-12, the bars
of test_gpu_2d.py).  Steps of one call, in one or several launches, give the bits of
as many calls."""
import numpy as np
import pytest

import dg_b200
import pyoracle
from test_gpu_2d import rel_l2

pytestmark = pytest.mark.gpu

XY = [1.0, 0.4, -0.3, 1.0, 2.0, 5.0, 4.5, 10.0, 9.0]


def sizes(p):
    """(nx, ny): one element, few, about one, two and three batches to a block, four, and more than one launch takes."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = 32 // (p + 2) * sms
    return [(1, 1), (3, 2)] + [(n, n - 1) for n in (int(np.sqrt(per * k)) for k in (0.9, 1.7, 2.6, 4.0))] + [(int(np.sqrt(4 * per)) + 2,) * 2]


@pytest.mark.parametrize("flux", ["LaxFriedrichs", "HLLC"])
@pytest.mark.parametrize("p", [0, 1, 2, 3, 4, 5])
def test_single_stages_match_oracle_2d(p, flux):
    for i, n in enumerate(sizes(p)):
        mesh = dg_b200.periodic_box_2d(n, (0.0, 0.0), (10.0, 9.0), rotate_seed=i)
        if i % 2:  # some edges not listed
            mesh = dg_b200.Mesh(mesh.node_coords, mesh.elem_to_node_ids, np.ascontiguousarray(mesh.interior_faces[::2 + i]))
        gpu = dg_b200.Case2D(mesh, p, flux=flux, gas_constant=1.0)
        orc = pyoracle.OracleCase2D.from_mesh(mesh, p, flux=flux, gas_constant=1.0)
        U = orc.project_ic("IsentropicVortexXY", XY)
        gpu.set_state(U)
        R = orc.residual(U)
        assert np.abs(gpu.residual() - R).max() <= 1e-11 * max(np.abs(R).max(), 1e-3)
        assert np.array_equal(gpu.get_state(), U)
        gpu.fe(1e-4, 3)
        want = orc.fe(U, 1e-4, 3)
        assert rel_l2(gpu.get_state(), want).max() < 1e-12
        gpu.rk4(1e-4, 2)  # (after an odd number of steps)
        assert rel_l2(gpu.get_state(), orc.rk4(want, 1e-4, 2)).max() < 1e-12
        assert gpu.status() == 0


@pytest.mark.parametrize("p", [0, 3, 5])
def test_steps_of_a_call_are_single_calls_2d(p):
    mesh = dg_b200.periodic_box_2d((23, 21), (0.0, 0.0), (10.0, 9.0), rotate_seed=2)
    gpu = dg_b200.Case2D(mesh, p, gas_constant=1.0)
    U = gpu.project_ic("IsentropicVortexXY", XY)
    for step, nsteps in ((gpu.fe, 259), (gpu.rk4, 258)):  # more than one launch takes, odd and even
        gpu.set_state(U)
        for _ in range(nsteps):
            step(1e-4, 1)
        one_by_one = gpu.get_state()
        gpu.set_state(U)
        step(1e-4, nsteps)
        assert np.array_equal(gpu.get_state(), one_by_one)
        assert gpu.status() == 0


@pytest.mark.parametrize("p", [0, 1, 3, 5])
def test_states_return_whatever_their_size_2d(p):
    """Set and get return every bit at the sizes around the 16384 values up to which
    the host transposes a state; a non-physical residual leaves an error, not values."""
    per = 4 * (p + 1) ** 2
    rng = np.random.default_rng(p)
    for ne in (1, 16384 // per, 16384 // per + 1):
        mesh = dg_b200.periodic_box_2d((ne, 1), (0.0, 0.0), (10.0, 9.0))
        gpu = dg_b200.Case2D(mesh, p, gas_constant=1.0)
        U = rng.standard_normal((ne, (p + 1) ** 2, 4))
        gpu.set_state(U)
        assert np.array_equal(gpu.get_state(), U)
        U[:, :, 0] = -1.0
        gpu.set_state(U)
        with pytest.raises(dg_b200.DGError, match="NONPHYSICAL"):
            gpu.residual()

"""The device reductions (L2 error, kinetic energy) at element counts around
the elements per CTA of every order: the error against the oracle (1e-10
relative, the bar of test_gpu_parity.py), the kinetic energy against the
allocation-free kernel's dense sums (1e-12, two orders of summation)."""
import numpy as np
import pytest

import dg_b200
import pyoracle

pytestmark = pytest.mark.gpu

VORTEX_XY = [1.0, 1.0, 1.0, 1.0, 2.0, 5.0, 5.0, 10.0, 10.0]


@pytest.mark.parametrize("n,turned", [((1, 1, 1), 0), ((3, 3, 1), 0), ((4, 3, 5), 6)])
@pytest.mark.parametrize("p", [0, 1, 2, 3, 4, 5])
def test_reductions_match_oracle_and_dense_sums(p, n, turned):
    import torch

    mesh = dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (10.0, 10.0, 10.0), rotate_seed=turned)
    case = dg_b200.Case(mesh, p, gas_constant=1.0)
    orc = pyoracle.OracleCase.from_mesh(mesh, p, gas_constant=1.0)
    U = case.project_ic("IsentropicVortexXY", VORTEX_XY)
    for name, data in (("IsentropicVortexXY", VORTEX_XY), ("TaylorGreen", [0.1])):
        np.testing.assert_allclose(case.l2_error(name, data, 0.4), orc.l2_error(U, name, data, 0.4), rtol=1e-10, atol=1e-13)
    djac = torch.full((case.ne,), case.total_volume() / case.ne / 8.0, dtype=torch.float64, device="cuda")
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    dg_b200.kinetic_energy_noalloc(p, case.ne, case.device_state_ptr(), djac.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    assert abs(case.kinetic_energy() / float(out.item()) - 1.0) < 1e-12

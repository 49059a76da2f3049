"""Creation of a mixed-precision case on non-affine hexahedra: the residual of the
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

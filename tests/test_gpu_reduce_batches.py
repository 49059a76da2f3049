"""The device reductions at the sizes their launch depends on: up to one element per SM,
where the error spreads an element's points over more threads, one more, and more
batches than CTAs, with a last batch that is partly filled.  Bars of test_gpu_reduce.py:
the error against the oracle 1e-10, the kinetic energy against dense sums 1e-12."""
import numpy as np
import pytest

import dg_b200
import pyoracle

pytestmark = pytest.mark.gpu

VORTEX_XY = [1.0, 1.0, 1.0, 1.0, 2.0, 5.0, 5.0, 10.0, 10.0]


def elements(p, where, sms):
    """The element count: exactly, or at least that many and no multiple of a batch."""
    if where == "one per SM":
        return sms
    if where == "one per SM and one more":
        return sms + 1
    per_cta = [max(1, 128 // m ** 2) for m in (2 * max(p, 1) + 2, p + 2)]  # error, kinetic energy
    n = 8 * sms * max(per_cta) + 1
    while any(e > 1 and n % e == 0 for e in per_cta):
        n += 1
    return n


@pytest.mark.parametrize("where", ["one per SM", "one per SM and one more", "more batches than CTAs"])
@pytest.mark.parametrize("p", [0, 1, 2, 3, 4, 5])
def test_reductions_at_their_launch_limits(p, where):
    import torch

    ne = elements(p, where, torch.cuda.get_device_properties(0).multi_processor_count)
    a = next(k for k in (4, 3, 2, 1) if ne % k == 0)
    # (turned numberings: columns of points along every axis)
    mesh = dg_b200.periodic_box((a, 1, ne // a), (0.0, 0.0, 0.0), (10.0, 10.0, 10.0), rotate_seed=6)
    case = dg_b200.Case(mesh, p, gas_constant=1.0)
    orc = pyoracle.OracleCase.from_mesh(mesh, p, gas_constant=1.0)
    assert case.ne == ne
    U = case.project_ic("IsentropicVortexXY", VORTEX_XY)
    for name, data in (("IsentropicVortexXY", VORTEX_XY), ("TaylorGreen", [0.1])):
        np.testing.assert_allclose(case.l2_error(name, data, 0.4), orc.l2_error(U, name, data, 0.4), rtol=1e-10, atol=1e-13)
    djac = torch.full((ne,), case.total_volume() / ne / 8.0, dtype=torch.float64, device="cuda")
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    dg_b200.kinetic_energy_noalloc(p, ne, case.device_state_ptr(), djac.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    assert abs(case.kinetic_energy() / float(out.item()) - 1.0) < 1e-12
    case.close()

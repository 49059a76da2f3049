"""Lax-Friedrichs, FP64: a state at rest whose pressure is positive at every volume point
and negative in a face's trace.  On the left side of a face it has no wave speed (the
square root of a negative number): the flux is NaN, so that the next state is and a step
does not go on from it, on small and larger meshes and in 2D."""
import numpy as np
import pytest

import dg_b200

pytestmark = pytest.mark.gpu


def at_rest(ne, nb, nv, p, end):
    """rho = 1, no momentum; pressure along x from 2 to -0.05 (linear, 0.18 at the outer
    volume point of p = 1), the negative end at x = +1 (end 1) or -1 (end 0)."""
    U = np.zeros((ne, nb, nv))
    U[:, :, 0] = 1.0
    x = np.linspace(0.0, 1.0, p + 1)[np.arange(nb) % (p + 1)]
    U[:, :, nv - 1] = (2.0 - 2.05 * (x if end else 1.0 - x)) / 0.4
    return U


def noticed(case, U):
    case.set_state(U)
    return not np.isfinite(case.residual()).all()


@pytest.mark.parametrize("n", [(2, 2, 2), (12, 12, 12)])
def test_negative_trace_pressure(n):
    case = dg_b200.Case(dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)), 1, gas_constant=1.0)
    assert any(noticed(case, at_rest(case.ne, 8, 5, 1, end)) for end in (0, 1))


@pytest.mark.parametrize("n", [(3, 3), (90, 90)])
def test_negative_trace_pressure_2d(n):
    mesh = dg_b200.periodic_box_2d(n, (0.0, 0.0), (1.0, 1.0))
    case = dg_b200.Case2D(mesh, 1, gas_constant=1.0)
    assert any(noticed(case, at_rest(mesh.nelem, 4, 4, 1, end)) for end in (0, 1))

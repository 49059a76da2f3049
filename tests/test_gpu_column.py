"""The column form of the RK stage (launch option "cf": face_lift_kernel and
column_kernel) where it can go wrong: one element, element counts that do not
fill the last batch, turned and sheared elements, both fluxes and precisions,
every output mode.

Bars: FP64 against the oracle as in test_gpu_parity.py (1e-11 for a residual,
1e-12 after time steps).  Mixed precision performs the stage kernel's FP32
operations in their order, so on meshes whose face orders agree (unturned
boxes) it gives the same bits as the stage kernel; on turned elements, where a
lift is summed in the neighbour's order, it stays within the mixed bar of 1e-6.
"""
import numpy as np
import pytest

import dg_b200
import pyoracle
from test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu

# strength 2: the projected state of the coarse sheared meshes stays physical
VORTEX_XY = [1.0, 1.0, 1.0, 1.0, 2.0, 5.0, 5.0, 10.0, 10.0]


def column_variants(case, precision):
    """(column variants, the first stage-kernel variant) of an affine case."""
    vs = [(i, v[4].split("+")) for i, v in enumerate(case.stage_variants()) if v[3] == precision]
    cf = [i for i, o in vs if "cf" in o and "ge" not in o]
    assert cf, "every order from 1 on compiles a column variant"
    return cf, [i for i, o in vs if "cf" not in o and "ge" not in o][0]


def box(n, turned=0, shear=False):
    mesh = dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (10.0, 10.0, 10.0), rotate_seed=turned)
    if shear:  # parallelepipeds: every entry of the metric terms is used
        x = mesh.node_coords
        y = x @ np.array([[1.0, 0.05, 0.1], [0.2, 1.0, 0.15], [0.1, 0.25, 1.0]])
        mesh = dg_b200.Mesh(np.ascontiguousarray(y), mesh.elem_to_node_ids, mesh.interior_faces)
    return mesh


@pytest.mark.parametrize("flux", ["LaxFriedrichs", "HLLC"])
@pytest.mark.parametrize("n,turned,shear", [((1, 1, 1), 0, False), ((3, 2, 3), 7, False), ((5, 3, 3), 4, True)])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5])
def test_column_fp64_matches_oracle(p, n, turned, shear, flux):
    mesh = box(n, turned, shear)
    orc = pyoracle.OracleCase.from_mesh(mesh, p, flux=flux, gas_constant=1.0)
    case = dg_b200.Case(mesh, p, flux=flux, gas_constant=1.0)
    U = orc.project_ic("IsentropicVortexXY", VORTEX_XY)
    dt = case.cfl_time_step(U, 0.1)
    R, S, F = orc.residual(U), orc.rk4(U, dt, 3), orc.fe(U, dt, 2)
    for v in column_variants(case, "fp64")[0]:
        case.stage_variant = v
        case.set_state(U)
        assert rel_l2(case.residual(), R).max() < 1e-11
        # dt M^-1 R is the forward-Euler increment, a difference that cancels U
        assert rel_l2(case.mass_inverse_residual(dt), orc.fe(U, dt, 1) - U).max() < 1e-10
        case.rk4(dt, 3)
        assert rel_l2(case.get_state(), S).max() < 1e-12
        case.set_state(U)
        case.fe(dt, 2)
        assert rel_l2(case.get_state(), F).max() < 1e-12
        assert case.status() == 0


@pytest.mark.parametrize("flux", ["LaxFriedrichs", "HLLC"])
@pytest.mark.parametrize("n,turned,shear", [((1, 1, 1), 0, False), ((5, 3, 4), 0, False), ((4, 3, 3), 0, True), ((3, 2, 3), 7, False)])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5])
def test_column_mixed_is_the_stage_kernels(p, n, turned, shear, flux):
    mesh = box(n, turned, shear)
    case = dg_b200.Case(mesh, p, flux=flux, gas_constant=1.0, precision="mixed_fp32")
    U = case.project_ic("IsentropicVortexXY", VORTEX_XY)
    dt = case.cfl_time_step(U, 0.1)
    cf, stage = column_variants(case, "mixed_fp32")

    def outputs(v):
        case.stage_variant = v
        case.set_state(U)
        out = [case.residual(), case.mass_inverse_residual(dt)]
        case.rk4(dt, 3)
        out.append(case.get_state())
        case.set_state(U)
        case.fe(dt, 2)
        return out + [case.get_state()]

    want = outputs(stage)
    for v in cf:
        got = outputs(v)
        if turned:
            assert rel_l2(got[2], want[2]).max() < 1e-6 and rel_l2(got[3], want[3]).max() < 1e-6
        else:
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert case.status() == 0


@pytest.mark.parametrize("precision", ["fp64", "mixed_fp32"])
def test_column_batch_is_a_contexts(precision):
    """Cases of a batch (several geometry classes and time steps in one launch)
    give the bits of single contexts that run the same column variant."""
    meshes = [box((12, 11, 10)), box((9, 12, 13), turned=5)]
    batch = dg_b200.Batch([(m, 2) for m in meshes], gas_constant=1.0, precision=precision)
    v = batch.groups()[0][3]
    dts = [2e-3, 3e-3]
    for i, dt in enumerate(dts):
        batch.project_ic(i, "IsentropicVortexXY", VORTEX_XY)
        batch.set_time_step(i, dt)
    batch.rk4(2)
    for i, (m, dt) in enumerate(zip(meshes, dts)):
        case = dg_b200.Case(m, 2, gas_constant=1.0, precision=precision)
        case.stage_variant = v
        assert "cf" in case.stage_variants()[v][4].split("+")
        case.project_ic("IsentropicVortexXY", VORTEX_XY)
        case.rk4(dt, 2)
        assert np.array_equal(batch.get_state(i), case.get_state())


def test_default_form_follows_the_mesh_size():
    """The column form is the default of affine meshes: its one-launch steps while
    every element can have its own threads, its stage launches above; bent meshes
    run general geometry's kernel."""
    def options(mesh, p=3):
        c = dg_b200.Case(mesh, p)
        return c.stage_variants()[c.stage_variant][4].split("+")

    assert {"cf", "sm"} <= set(options(box((3, 3, 3))))
    assert "cf" in options(box((16, 16, 16))) and "sm" not in options(box((16, 16, 16)))
    bent = box((4, 4, 4))
    bent.node_coords[:, 0] += 0.1 * np.sin(2 * np.pi * bent.node_coords[:, 1] / 10.0) * np.sin(2 * np.pi * bent.node_coords[:, 2] / 10.0)
    assert "ge" in options(bent)

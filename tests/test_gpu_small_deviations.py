"""Deviations from the reference level far below the FP32 spacing of the level itself: the
mixed step reads zeta - zeta_reference with FP32 precision, whatever its size.  From rest the
discharge after a step is -g h grad(zeta) dt to first order, so it shows the deviations that
the kernel read."""
import numpy as np
import pytest

from oceano_gb300 import uniform_mesh
from oceano_gb300.icbc import nodal_points

pytestmark = pytest.mark.gpu

# FP32 arithmetic on deviations that round once (6e-8) and their differences over a cell
TOL = 1e-5


@pytest.mark.parametrize("level", [1.0, 10.0, 2.0, 1.0 / 3.0])
@pytest.mark.parametrize("units", [1, 40, 3000, 1 << 20, 1 << 28])
@pytest.mark.parametrize("degree", [1, 4])
def test_from_rest(gpu_lib, degree, units, level):
    from oceano_gb300.operator import OceanoOperator
    mesh = uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, degree)
    x = nodal_points(mesh)
    unit = np.spacing(level)  # FP64 spacing of zeta
    k = np.rint(units * (2 + np.sin(np.pi * x[:, 0]) * np.cos(np.pi * x[:, 1])) * 4)
    z = level + k * unit
    assert np.array_equal((z - level) / unit, np.rint((z - level) / unit))
    dt, out = 1e-4, []
    # the same deviations, exact in FP32, about a reference level of 0 (the FP64 form)
    for precision, zeta in (("mixed", z), ("fp64", z - level)):
        op = OceanoOperator(mesh, precision=precision,
                            zeta_reference=level if precision == "mixed" else 0.0)
        for b in (0, 1, 2):
            op.set_wall_boundary(b)
        if precision == "fp64":  # the depth of the level as bathymetry
            op.initialize_data_at_quadrature(
                lambda px, py: np.stack([np.full_like(px, level)] + [0 * px] * 4))
        else:
            op.set_reference_state(level, (0.0, 0.0))
        zeta, q = zeta.copy(), np.zeros(2 * op.n_dofs)
        op.perform_time_step("forward_euler", 0.0, dt, zeta, q)
        out.append(q)
        op.close()
    assert np.linalg.norm(out[0] - out[1]) < TOL * np.linalg.norm(out[1])

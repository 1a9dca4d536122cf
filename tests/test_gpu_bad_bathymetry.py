"""A bathymetry value that is not finite at a Gauss-Lobatto point is reported by the FP64
stage and time step, as the literal zeta iteration reports it."""
import numpy as np
import pytest

from cases import bump_problem_data
from oceano_gb300 import uniform_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("degree", [1, 2, 3, 4])
def test_reported(gpu_lib, degree, bad):
    from oceano_gb300._lib import OceanoError
    from oceano_gb300.operator import OceanoOperator
    op = OceanoOperator(uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), False, degree))
    for b in (0, 1, 2):
        op.set_wall_boundary(b)
    arrays = op.initialize_data_at_quadrature(bump_problem_data)
    n = (degree + 2) ** 2
    for point in (0, n // 2, 5 * n - 1):  # first, inner and last point of a cell
        broken = [a.copy() for a in arrays]
        broken[1][point] = bad
        op.set_static_data(*broken)
        with pytest.raises(OceanoError):
            op.perform_time_step("ssp33", 0.0, 1e-4, np.full(op.n_dofs, 0.01),
                                 np.zeros(2 * op.n_dofs))
    op.set_static_data(*arrays)
    z = np.full(op.n_dofs, 0.01)
    op.perform_time_step("ssp33", 0.0, 1e-4, z, np.zeros(2 * op.n_dofs))
    assert np.isfinite(z).all()
    op.close()

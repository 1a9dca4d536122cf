"""compute_cell_transport_speed is the largest of cell_transport_speed, bit for bit: a point's
speed does not depend on which cells are evaluated beside it.  Smooth states whose speed is
largest inside a cell."""
import numpy as np
import pytest

from cases import bump_problem_data, hanging_mesh, mixed_degree
from oceano_gb300 import uniform_mesh
from oceano_gb300.icbc import nodal_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bathymetry", [False, True])
@pytest.mark.parametrize("mesh", ["1", "2", "3", "4", "hp"])
def test_largest_of_the_cells(gpu_lib, mesh, bathymetry):
    import torch
    from oceano_gb300.operator import OceanoOperator
    m = (mixed_degree(hanging_mesh(2, seed=11)) if mesh == "hp" else
         uniform_mesh(23, 11, (0.0, 2.0, 0.0, 1.0), True, int(mesh)))
    op = OceanoOperator(m)
    if bathymetry:
        op.initialize_data_at_quadrature(bump_problem_data)
    x = nodal_points(m)
    rng = np.random.default_rng(4)
    for _ in range(40):
        cx, cy, w, amp = rng.uniform((0.2, 0.2, 0.05, 0.05), (1.8, 0.8, 0.3, 0.4))
        bump = amp * np.exp(-((x[:, 0] - cx) ** 2 + (x[:, 1] - cy) ** 2) / w ** 2)
        z = (0.0 if bathymetry else 1.0) + bump
        q = np.zeros(2 * op.n_dofs)
        off, nd = m.offsets(), np.diff(m.offsets())
        c = np.repeat(np.arange(m.n_cells), nd)
        q[off[c] + np.arange(len(c))] = 0.3 + bump
        q[off[c] + np.arange(len(c)) + nd[c]] = 0.5 * bump
        zt, qt = torch.from_numpy(z).cuda(), torch.from_numpy(q).cuda()
        torch.cuda.synchronize()
        speed = op.compute_cell_transport_speed(zt, qt)
        assert speed == op.cell_transport_speed(zt, qt).max().item()
    op.close()

"""Batches of 9 and 10 cells of the zeta stop rule (degree 1): the lean mixed step runs the
two-lanes form of cell_kernel, as smaller batches run the four-lanes form.  Against the
oracle, and in time against the general kernel.  (Below the depth of the literal iteration
test_gpu_cell_stage.py compares the two kernels; there the mixed form keeps hu = q over a
flat bottom, where the oracle's desingularised velocity does not.)"""
import numpy as np
import pytest

from oceano_gb300 import uniform_mesh
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-6  # the bar of the mixed form


def state(mesh, depth):
    rng = np.random.default_rng(2)
    n = mesh.n_dofs()
    z = depth * (1 + 0.1 * rng.standard_normal(n).clip(-2, 2))
    return z, 0.1 * depth * rng.standard_normal(2 * n)


@pytest.mark.parametrize("batch", [9, 10])
@pytest.mark.parametrize("cells", [(9, 7), (10, 8)])
def test_against_oracle(gpu_lib, cells, batch):
    from oceano_gb300.operator import OceanoOperator
    mesh, depth = uniform_mesh(*cells, (0.0, 2.0, 0.0, 1.0), True, 1), 1.0
    orc = O.Oracle(mesh, bcs={b: ("wall",) for b in (0, 1, 2)}, batch=batch)
    op = OceanoOperator(mesh, precision="mixed", zeta_reference=depth, batch_width=batch)
    for b in (0, 1, 2):
        op.set_wall_boundary(b)
    op.set_reference_state(depth, (0.0, 0.0))
    z, q = state(mesh, depth)
    zo, qo = z.copy(), q.copy()
    tb = O.TABLEAUX["ssp33"]
    for k in range(2):
        O.erk_step(orc, tb["a"], tb["b"], tb["c"], 0.0, 1e-4, zo, qo)
        op.perform_time_step("ssp33", 0.0, 1e-4, z, q)
    op.close()
    for a, b in ((z, zo), (q, qo)):
        assert np.linalg.norm(a - b) < TOL * np.linalg.norm(b)


def test_not_the_general_kernel(gpu_lib):
    import torch
    from oceano_gb300.operator import OceanoOperator
    mesh, best = uniform_mesh(320, 160, (0.0, 2.0, 0.0, 1.0), True, 1), []
    for friction in ("none", "linear"):
        op = OceanoOperator(mesh, precision="mixed", zeta_reference=1.0, batch_width=10,
                            friction=friction)
        for b in (0, 1, 2):
            op.set_wall_boundary(b)
        z = torch.ones(op.n_dofs, dtype=torch.float64, device="cuda")
        q = torch.zeros(2 * op.n_dofs, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        stream, ms = torch.cuda.ExternalStream(op.stream), []
        for k in range(23):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record(stream)
            op.perform_time_step("ssp33", 0.0, 1e-5, z, q)
            b.record(stream)
            op.synchronize()
            ms.append(a.elapsed_time(b))
        best.append(min(ms[3:]))
        op.close()
    assert best[0] < 0.75 * best[1]  # (the general kernel takes more than twice as long)

"""The zeta inverse of fully wet cells in closed form against the oracle's literal
sweeps: every degree, sweep limits at which the closed sums are empty or short, and
updates small enough to meet the stop rule (1e-12 in the l1 norm of a cell batch)
at the first sweep, in between and never."""
import numpy as np
import pytest

from cases import hanging_mesh, mixed_degree, perturbed_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# one sweep more or less where a norm meets 1e-12 within rounding moves zeta (about 1)
# by less than 1e-12 in each cell; the other differences are FP64 rounding
TOL = 1e-12


@pytest.mark.parametrize("scale", [1e-3, 1e-8, 3e-10, 1e-13])
@pytest.mark.parametrize("max_iter", [0, 1, 2, 3, 15])
@pytest.mark.parametrize("batch", [1, 3])
def test_closed_sweeps(gpu_lib, scale, max_iter, batch):
    from oceano_gb300.operator import OceanoOperator
    mesh = mixed_degree(hanging_mesh(2, seed=11))
    if batch > 1:  # batches hold cells of one degree
        mesh = mesh.with_degree(np.full(mesh.n_cells, 3, np.int32))
    bcs = {0: ("wall",)}
    orc = O.Oracle(mesh, bcs=bcs, batch=batch, max_iter=max_iter, vortex=[1, 1, .2, .1, .5, .5, 0, 0])
    op = OceanoOperator(mesh, batch_width=batch, max_iteration_height=max_iter)
    op.set_wall_boundary(0)
    z, q = perturbed_state(orc, 3)
    rng = np.random.default_rng(8)
    kz0 = [np.zeros(orc.n)] + [1e-2 * rng.standard_normal(orc.n) for _ in range(3)]
    kq0 = [np.zeros(2 * orc.n) for _ in range(4)]
    f, out = np.array([scale, 0.5 * scale]), []
    for who in (orc, op):
        kz, kq = [k.copy() for k in kz0], [k.copy() for k in kq0]
        sz, sq, nz, nq = z.copy(), q.copy(), np.zeros(orc.n), np.zeros(2 * orc.n)
        if who is orc:
            orc.stage_erk(1, 3, 0.0, f, z, q, kz, kq, sz, sq, nz, nq)
        else:
            op.perform_stage_hydro(1, 3, 0.0, f, [z, q], kz, kq, sz, sq, nz, nq)
        out.append(nz)
    op.close()
    assert np.linalg.norm(out[1] - out[0]) < TOL * np.linalg.norm(out[0])
    # the update itself, down to the stop rule and the rounding of zeta
    assert np.abs(out[1] - out[0]).max() < 3e-12

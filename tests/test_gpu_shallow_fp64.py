"""FP64 stages where the depth lies on both sides of Threshold_for_wetdry: the velocity as
q / h above it, the desingularised form below, reconstructed depths that fall below it over
a bathymetry step, against the oracle."""
import numpy as np
import pytest

from cases import hanging_mesh, static_arrays
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-12  # the bar of the FP64 form


def step_data(x, y):
    """A bathymetry that jumps by 0.06 at x = 1 (depths of 0.07 and 0.13 around the threshold 0.1)."""
    zb = np.where(x < 1.0, 0.13, 0.07)
    return np.stack([zb, 0.02 + 0 * x, 0 * x, 0 * x, 0 * x])


@pytest.mark.parametrize("bottom", ["flat", "step"])
@pytest.mark.parametrize("degree", [1, 2, 3, 4])
@pytest.mark.parametrize("stage", [0, 2])
def test_stage(gpu_lib, degree, bottom, stage):
    from oceano_gb300.operator import OceanoOperator
    mesh = hanging_mesh(degree, seed=4, periodic=False)
    bcs = {b: ("wall",) for b in (0, 1, 2)}
    friction = 2 if bottom == "step" else 0
    orc = O.Oracle(mesh, bcs=bcs, friction=friction)
    op = OceanoOperator(mesh, friction="manning" if friction else "none")
    for b in bcs:
        op.set_wall_boundary(b)
    if bottom == "step":
        arrs = static_arrays(orc, step_data)
        orc.set_static(*arrs)
        op.set_static_data(*arrs)
    n = orc.n
    rng = np.random.default_rng(degree)
    z = (0.0 if bottom == "step" else 0.1) + 0.02 * rng.standard_normal(n).clip(-2, 2)
    q = 0.05 * rng.standard_normal(2 * n)
    kz0 = [np.zeros(n)] + [1e-4 * rng.standard_normal(n) for _ in range(3)]
    kq0 = [np.zeros(2 * n)] + [1e-4 * rng.standard_normal(2 * n) for _ in range(3)]
    f = np.array([[1e-4], [], [1e-4 / 6, 1e-4 / 6, 2e-4 / 3]][stage])
    out = []
    for who in (orc, op):
        kz, kq = [k.copy() for k in kz0], [k.copy() for k in kq0]
        sz, sq, nz, nq = z.copy(), q.copy(), np.zeros(n), np.zeros(2 * n)
        if who is orc:
            orc.stage_erk(stage, 3, 0.0, f, z, q, kz, kq, sz, sq, nz, nq)
        else:
            op.perform_stage_hydro(stage, 3, 0.0, f, [z, q], kz, kq, sz, sq, nz, nq)
        out.append((kz[stage + 1], kq[stage + 1], sz if stage == 2 else nz, sq if stage == 2 else nq))
    op.close()
    for a, b in zip(out[1], out[0]):
        assert np.linalg.norm(a - b) < TOL * np.linalg.norm(b)

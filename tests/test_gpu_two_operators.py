"""Operators with different sweep limits in one process: what an operator computes does not
depend on the operators made after it (every form that applies the zeta sweeps in closed
form, one degree and several)."""
import numpy as np
import pytest

from cases import hanging_mesh, mixed_degree, perturbed_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def make(mesh, form, max_iter):
    from oceano_gb300.operator import OceanoOperator
    mixed = form != "fp64"
    op = OceanoOperator(mesh, max_iteration_height=max_iter,
                        precision="mixed" if mixed else "fp64",
                        zeta_reference=1.0 if mixed else 0.0,
                        friction="linear" if form == "mixed general" else "none")
    op.set_wall_boundary(0)
    if form == "mixed one launch":
        op.set_launch_mode("one")
    return op


def run(op, form, z, q):
    z, q, n = z.copy(), q.copy(), len(z)
    if form != "mixed stage":
        op.perform_time_step("ssp33", 0.0, 1e-3, z, q)
        return z, q
    kz, kq = [np.zeros(n) for _ in range(4)], [np.zeros(2 * n) for _ in range(4)]
    nz, nq = np.zeros(n), np.zeros(2 * n)
    op.perform_stage_hydro(0, 3, 0.0, np.array([1e-3]), [z, q], kz, kq, z, q, nz, nq)
    return nz, nq


FORMS = ["fp64", "mixed", "mixed general", "mixed stage"]


@pytest.mark.parametrize("form,degrees", [(f, d) for f in FORMS for d in ("3", "1-4")] +
                         [("mixed one launch", "1-4")])
def test_sweep_limits_stay_apart(gpu_lib, form, degrees):
    mesh = hanging_mesh(3, seed=11)
    if degrees == "1-4":
        mesh = mixed_degree(mesh)
    orc = O.Oracle(mesh, bcs={0: ("wall",)}, vortex=[1, 1, .2, .1, .5, .5, 0, 0])
    z, q = perturbed_state(orc, 3)
    first = make(mesh, form, 15)
    alone = run(first, form, z, q)
    second = make(mesh, form, 2)
    other = run(second, form, z, q)
    again = run(first, form, z, q)
    for a, b, c in zip(alone[:1], again, other):
        assert np.linalg.norm(c - a) > 1e-9 * np.linalg.norm(a)  # the limit matters here
    for a, b in zip(alone, again):
        assert np.array_equal(a, b)
    first.close()
    second.close()

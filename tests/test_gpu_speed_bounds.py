"""Transport speed with FP32 bounds in front of the FP64 evaluation: the maximum and every
cell's own maximum against FP64, on states where many points tie (uniform flow), where
one stands out, near the wet/dry threshold, over bathymetry and with a large offset."""
import numpy as np
import pytest

from cases import bump_problem_data, hanging_mesh, mixed_degree, static_arrays
from oceano_gb300 import uniform_mesh
from oceano_gb300.basis import lagrange_matrix, lobatto
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-12  # FP64 against FP64


def cell_speeds(mesh, z, q, g=9.81, cu=0.1, zb=None):
    """Per-cell maxima in NumPy (rectangular cells)."""
    off, out = mesh.offsets(), np.zeros(mesh.n_cells)
    for c in range(mesh.n_cells):
        p = int(mesh.degree[c])
        n, B = (p + 1) ** 2, lagrange_matrix(lobatto(p + 1)[0], lobatto(p + 2)[0])
        ev = lambda v: (B @ v.reshape(p + 1, p + 1) @ B.T).ravel()  # noqa: E731
        h, a, b = (ev(v) for v in (z[off[c]:off[c] + n], q[2 * off[c]:2 * off[c] + n],
                                   q[2 * off[c] + n:2 * off[c] + 2 * n]))
        h = np.maximum(h + (0 if zb is None else zb[c]), 1e-12)
        f = np.sqrt(2.) * h / np.sqrt(h ** 4 + np.maximum(h ** 4, cu ** 4))
        v = mesh.vertices[c]
        J = np.array([1 / (v[2] - v[0]), 1 / (v[5] - v[1])])
        e = np.ones(2)
        for _ in range(5):
            e = J * J * e
            e /= np.abs(e).max()
        s = np.linalg.norm(J * e) / np.linalg.norm(e)
        out[c] = (s * np.sqrt(g * h) + np.maximum(abs(J[0] * a * f), abs(J[1] * b * f))).max()
    return out


def states(kind, n, rng):
    z, q = np.ones(n), np.zeros(2 * n)
    if kind == "uniform":
        q[:] = 0.3
    elif kind == "noise":
        z += 1e-3 * rng.standard_normal(n)
        q += 1e-1 * rng.standard_normal(2 * n)
    elif kind == "peak":
        z += 1e-9 * rng.standard_normal(n)
        z[n // 2] += 1e-7
    elif kind == "shallow":
        z = 0.1 + 0.05 * rng.standard_normal(n)  # across the threshold, some points dry
        q += 0.05 * rng.standard_normal(2 * n)
    return z, q


@pytest.mark.parametrize("kind", ["uniform", "rest", "noise", "peak", "shallow"])
@pytest.mark.parametrize("mesh", ["1", "2", "3", "4", "hp"])
def test_speed(gpu_lib, mesh, kind):
    import torch
    from oceano_gb300.operator import OceanoOperator
    m = (mixed_degree(hanging_mesh(2, seed=11)) if mesh == "hp" else
         uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, int(mesh)))
    op = OceanoOperator(m)
    z, q = states(kind, op.n_dofs, np.random.default_rng(5))
    ref = cell_speeds(m, z, q)
    zt, qt = torch.from_numpy(z).cuda(), torch.from_numpy(q).cuda()
    torch.cuda.synchronize()
    assert abs(op.compute_cell_transport_speed(zt, qt) - ref.max()) <= TOL * ref.max()
    got = op.cell_transport_speed(zt, qt).cpu().numpy()
    assert np.abs(got - ref).max() <= TOL * ref.max()
    op.close()


@pytest.mark.parametrize("offset", [0.0, 1e4])
def test_speed_over_bathymetry(gpu_lib, offset):
    """zb and zeta with a common offset that cancels in the depth."""
    from oceano_gb300.operator import OceanoOperator
    m = uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), False, 3)
    orc = O.Oracle(m, bcs={0: ("wall",)})

    def data(x, y):
        d = bump_problem_data(x, y)
        d[0] -= offset
        return d
    arrs = static_arrays(orc, data)
    orc.set_static(*arrs)
    op = OceanoOperator(m)
    op.set_static_data(*arrs)
    rng = np.random.default_rng(6)
    z = offset + 1e-3 * rng.standard_normal(op.n_dofs)
    q = 0.1 * rng.standard_normal(2 * op.n_dofs)
    ref = orc.transport_speed(z, q)
    # the depth carries the rounding of zeta and zb, 1e-16 of the offset
    assert abs(op.compute_cell_transport_speed(z, q) - ref) <= max(TOL, 1e-15 * offset * 10) * ref
    op.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["zeta", "q"])
def test_non_finite(gpu_lib, bad, where):
    """Reported where a point's speed is not finite (the running maximum of |J^-1 u| drops a
    NaN discharge, as std::max does)."""
    if where == "q" and np.isnan(bad):
        pytest.skip("dropped by the maximum")
    from oceano_gb300._lib import OceanoError
    from oceano_gb300.operator import OceanoOperator
    op = OceanoOperator(uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, 3))
    z, q = states("noise", op.n_dofs, np.random.default_rng(5))
    v = z if where == "zeta" else q
    v[7] = bad
    with pytest.raises(OceanoError):
        op.compute_cell_transport_speed(z, q)
    v[7] = 1.0
    assert np.isfinite(op.compute_cell_transport_speed(z, q))  # the flag was cleared
    op.close()

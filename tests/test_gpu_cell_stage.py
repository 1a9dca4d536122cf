"""The four-lanes-per-cell stage of the mixed time step (operators without static data)
against the team kernel, which the same operator runs with a friction model whose
coefficient is zero (none given): cell counts that do not fill a warp, every degree, zeta stop batches, depths above the
wet/dry threshold, across it, and below the depth where the literal zeta iteration takes
over; schemes of one to four stages."""
import numpy as np
import pytest

from cases import hanging_mesh, mixed_degree
from oceano_gb300 import uniform_mesh

pytestmark = pytest.mark.gpu

# two FP32 evaluations of one scheme: the bar of the mixed form
TOL = 1e-6


def meshes(name):
    if name == "hp":
        return mixed_degree(hanging_mesh(2, seed=11))
    if name.startswith("hanging"):
        return hanging_mesh(int(name[-1]), seed=4, periodic=False)
    p, nx, ny = (int(v) for v in name.split("_"))
    return uniform_mesh(nx, ny, (0.0, 2.0, 0.0, 1.0), True, p)


def state(mesh, depth, seed=2):
    """Depth varying by 20% over the domain, 1e-3 of noise; the discharge of 0.5 m/s."""
    rng = np.random.default_rng(seed)
    off = mesh.offsets()
    nd = np.diff(off)
    c = np.repeat(np.arange(mesh.n_cells), nd)
    x = mesh.vertices[c, 0]
    h = depth * (1 + 0.2 * np.sin(np.pi * x) + 1e-3 * rng.standard_normal(len(c)))
    q = np.zeros(2 * len(c))
    for e, u in ((0, 0.5), (1, 0.1)):
        q[off[c] + np.arange(len(c)) + e * nd[c]] = u * h
    return h, q


def run(mesh, general, z, q, scheme, dt, steps=2, **kw):
    import torch
    from oceano_gb300.operator import OceanoOperator
    h = float(z.mean())
    op = OceanoOperator(mesh, precision="mixed", zeta_reference=h,
                        friction="linear" if general else "none", **kw)
    op.set_reference_state(h, (0.5 * h, 0.1 * h))
    for b in (0, 1, 2):
        op.set_wall_boundary(b)
    zt, qt = torch.from_numpy(z).cuda(), torch.from_numpy(q).cuda()
    for k in range(steps):
        op.perform_time_step(scheme, k * dt, dt, zt, qt)
    op.synchronize()
    op.close()
    return zt.cpu().numpy(), qt.cpu().numpy()


def compare(mesh, depth, scheme="ssp33", **kw):
    z, q = state(mesh, depth)
    dt = 2e-4
    a, b = (run(mesh, g, z, q, scheme, dt, **kw) for g in (False, True))
    for x, y in zip(a, b):
        assert np.isfinite(x).all()
        assert np.linalg.norm(x - y) < TOL * np.linalg.norm(y)
    assert np.linalg.norm(a[0] - z) > 10 * TOL * np.linalg.norm(z)  # the step moved the state


@pytest.mark.parametrize("depth", [1.0, 0.1, 8e-4])
@pytest.mark.parametrize("mesh", ["1_5_3", "2_3_3", "3_9_7", "4_5_5", "3_4_2", "hp", "hanging1",
                                  "hanging4"])
def test_against_team_kernel(gpu_lib, mesh, depth):
    compare(meshes(mesh), depth)


@pytest.mark.parametrize("scheme", ["forward_euler", "ssp22", "rk4", "stage3_order2"])
@pytest.mark.parametrize("mesh", ["3_9_7", "hp"])
def test_schemes(gpu_lib, mesh, scheme):
    compare(meshes(mesh), 1.0, scheme)


@pytest.mark.parametrize("batch,mesh", [(2, "2_9_7"), (3, "3_9_7"), (8, "1_9_7"), (10, "1_9_7")])
@pytest.mark.parametrize("depth", [1.0, 8e-4])
def test_batches(gpu_lib, mesh, batch, depth):
    compare(meshes(mesh), depth, batch_width=batch)


@pytest.mark.parametrize("rule", ["default", "p+1"])
def test_cell_rules(gpu_lib, rule):
    compare(meshes("4_5_3"), 1.0, cell_quadrature=rule)


@pytest.mark.parametrize("depth", [1.0, 0.1, 8e-4])
@pytest.mark.parametrize("batch", [1, 3])
def test_large_degree_1(gpu_lib, depth, batch):
    """Above 16,384 cells of degree 1: two lanes per cell."""
    compare(meshes("1_167_101"), depth, batch_width=batch)


@pytest.mark.parametrize("depth", [1.0, 0.1, 8e-4])
@pytest.mark.parametrize("mesh,batch,rule", [("4_9_7", 4, "default"), ("4_9_7", 5, "p+1"),
                                             ("4_101_97", 1, "default")])
def test_lanes_of_degree_4(gpu_lib, depth, mesh, batch, rule):
    """Eight lanes per cell, or four where a batch does not fit and above 9,728 cells."""
    compare(meshes(mesh), depth, batch_width=batch, cell_quadrature=rule)

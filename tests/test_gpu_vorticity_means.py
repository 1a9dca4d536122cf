"""Vorticity and means of the indicator features straight from the state, and the
sum-factorised velocity field, on rectangular and sheared cells of every degree, several
members in a warp, with and without bathymetry, against the oracle's separate passes."""
import numpy as np
import pytest

from cases import bump_problem_data, hanging_mesh, mixed_degree, perturbed_state, static_arrays
from oceano_gb300.indicator import cell_info
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shear", [0.0, 0.3])
@pytest.mark.parametrize("degree", ["1", "2", "3", "4", "hp"])
@pytest.mark.parametrize("bottom", [False, True])
def test_features(gpu_lib, degree, shear, bottom):
    import torch
    from oceano_gb300.indicator import features
    from oceano_gb300.operator import OceanoOperator
    mesh = hanging_mesh(2, seed=11)
    mesh = mixed_degree(mesh) if degree == "hp" else mesh.with_degree(
        np.full(mesh.n_cells, int(degree), np.int32))
    mesh.vertices[:, 0::2] += shear * mesh.vertices[:, 1::2]
    bcs = {0: ("wall",)}
    orc = O.Oracle(mesh, bcs=bcs, vortex=[1, 1, .2, .1, .5, .5, 0, 0])
    op = OceanoOperator(mesh)
    if bottom:
        arrs = static_arrays(orc, bump_problem_data)
        orc.set_static(*arrs)
        op.set_static_data(*arrs)
    z, q = perturbed_state(orc, 1)
    u = orc.velocity_field(z, q)
    w = orc.vorticity(u, int(mesh.degree.max()))
    zt, qt = torch.from_numpy(z).cuda(), torch.from_numpy(q).cuda()
    ut = torch.empty_like(qt)
    member = np.arange(mesh.n_cells, dtype=np.int32) % 5
    info = torch.from_numpy(cell_info(mesh, member)).cuda()
    torch.cuda.synchronize()
    op.evaluate_velocity_field(zt, qt, ut)
    assert np.linalg.norm(ut.cpu().numpy() - u) < 1e-12 * np.linalg.norm(u)  # FP64
    feat, _, vort = features(op, zt, qt, info, 5, want_vorticity=True)
    top = np.array([w[member == k].max() for k in range(5)])
    # FP64 values rounded to FP32 (2^-24 each) and divided by another one
    assert np.abs(vort.cpu().numpy() - w / top[member]).max() < 4e-7
    feat, off = feat.cpu().numpy(), mesh.offsets()
    for c in range(mesh.n_cells):
        p = int(mesh.degree[c])
        n = (p + 1) ** 2
        wts = np.kron(mass_row(p), mass_row(p))
        mean = [wts @ v for v in (z[off[c]:off[c] + n], q[2 * off[c]:2 * off[c] + n],
                                  q[2 * off[c] + n:2 * off[c] + 2 * n])]
        assert np.abs(feat[c, :3] - mean).max() < 1e-6 * max(1.0, np.abs(mean).max())
    op.close()


def mass_row(p):
    """Integrals of the basis on [0, 1]: the Gauss-Lobatto weights."""
    from oceano_gb300.basis import lobatto
    return lobatto(p + 1)[1]

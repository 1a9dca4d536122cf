"""The time step on page-locked host vectors runs stage 0 by chunks of cells as the state
arrives; the batches of the zeta stop rule are those of the device step, bit for bit.  A
shallow state (literal iteration everywhere) with updates on both sides of the stop rule, and
cell counts whose thirds are no multiples of the batch."""
import numpy as np
import pytest

from oceano_gb300 import uniform_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("batch", [1, 3, 4])
def test_host_equals_device(gpu_lib, batch, general):
    import torch
    from oceano_gb300.operator import OceanoOperator
    degree, depth, dt = 2, 8e-4, 1e-5
    mesh = uniform_mesh(241, 163, (0.0, 2.0, 0.0, 1.0), True, degree)
    assert 24 * mesh.n_dofs() >= 8 << 20 and mesh.n_cells // 3 % 3  # chunked; see setup_chunks
    rng = np.random.default_rng(5)
    nn = (degree + 1) ** 2
    scale = 10.0 ** rng.uniform(-12, -5, mesh.n_cells).repeat(nn)
    z = depth + scale * rng.standard_normal(mesh.n_dofs())
    q = 1e-3 * scale.repeat(2) * rng.standard_normal(2 * mesh.n_dofs())
    out = []
    for host in (False, True):
        op = OceanoOperator(mesh, precision="mixed", zeta_reference=depth, batch_width=batch,
                            friction="linear" if general else "none")
        for b in (0, 1, 2):
            op.set_wall_boundary(b)
        op.set_reference_state(depth, (0.0, 0.0))
        zt, qt = torch.from_numpy(z.copy()), torch.from_numpy(q.copy())
        if host:
            zt, qt = zt.pin_memory(), qt.pin_memory()
        else:
            zt, qt = zt.cuda(), qt.cuda()
            torch.cuda.synchronize()
        for _ in range(3):  # (the first step tunes, without chunks)
            op.perform_time_step("ssp33", 0.0, dt, *((zt.numpy(), qt.numpy()) if host else (zt, qt)))
        op.synchronize()
        out.append((zt.cpu().numpy().copy(), qt.cpu().numpy().copy()))
        op.close()
    assert not np.array_equal(out[0][0], z)
    for a, b in zip(*out):
        assert np.isfinite(a).all()
        assert np.array_equal(a, b)

"""Launch configurations belong to the kernel they were timed with: the lean mixed step
reports its own block size, an operator that goes over to the general kernel (static data, the
additive scheme) and back tunes each kernel once, and the states are those of operators that
ran one kernel only."""
import numpy as np
import pytest

from cases import hanging_mesh, mixed_degree
from oceano_gb300 import uniform_mesh

pytestmark = pytest.mark.gpu


def make(mesh):
    from oceano_gb300.operator import OceanoOperator
    op = OceanoOperator(mesh, precision="mixed", zeta_reference=1.0)
    for b in (0, 1, 2):
        op.set_wall_boundary(b)
    op.set_reference_state(1.0, (0.0, 0.0))
    return op


def state(op):
    rng = np.random.default_rng(1)
    n = op.n_dofs
    return 1.0 + 1e-2 * rng.standard_normal(n), 1e-2 * rng.standard_normal(2 * n)


def flat(px, py):
    return np.stack([np.zeros_like(px)] * 5)


@pytest.mark.parametrize("memory", ["host", "pinned"])
@pytest.mark.parametrize("mesh", ["uniform", "large", "hp"])
def test_kernels_in_turn(gpu_lib, mesh, memory):
    import torch
    m = {"uniform": lambda: uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, 2),
         "large": lambda: uniform_mesh(241, 163, (0.0, 2.0, 0.0, 1.0), True, 2),  # in chunks
         "hp": lambda: mixed_degree(hanging_mesh(2, seed=11))}[mesh]()
    both, lean, general = make(m), make(m), make(m)
    general.initialize_data_at_quadrature(flat)
    assert not both.launch_config["tuned"]

    def step(op, scheme, z, q):
        if memory == "pinned":
            zt, qt = torch.from_numpy(z).pin_memory(), torch.from_numpy(q).pin_memory()
            op.perform_time_step(scheme, 0.0, 1e-4, zt.numpy(), qt.numpy())
            z[:], q[:] = zt.numpy(), qt.numpy()
        else:
            op.perform_time_step(scheme, 0.0, 1e-4, z, q)

    z0, q0 = state(both)
    for k in range(2):
        for other, static, scheme in ((lean, False, "ssp33"), (general, True, "ssp33"),
                                      (general, True, "ark_stage3_order2"),
                                      (lean, False, "ssp33")):
            if static:
                both.initialize_data_at_quadrature(flat)
            else:
                both.set_static_data()
            a, b = (z0.copy(), q0.copy()), (z0.copy(), q0.copy())
            step(both, scheme, *a)
            step(other, scheme, *b)
            cfg = both.launch_config
            assert cfg["tuned"]
            if not static:
                assert set(cfg["group_warps"].values()) == {2} and cfg["one_launch_warps"] == 2
            for x, y in zip(a, b):
                assert np.isfinite(x).all() and np.array_equal(x, y)
    for op in (both, lean, general):
        op.close()

"""The forms of cell_kernel with two, four and eight lanes per cell where they differ most:
two lanes above 128 cells per SM (conforming and not), eight lanes at inflow, outflow and
absorbing boundaries, per-cell time scales with each, and cells whose reference frame is
turned by half a turn (faces met in the opposite direction), the latter also in the other
kernels.  Against the team kernel (a friction model without coefficients), the oracle, or the
same mesh unturned."""
import numpy as np
import pytest

from cases import CASES, VORTEX, hanging_mesh, mixed_degree
from oceano_gb300 import QuadForest, uniform_mesh
from oceano_gb300.mesh import Mesh
from oceano_gb300.workloads import apply_bcs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-6  # two FP32 evaluations: the bar of the mixed form
WALLS = {b: ("wall",) for b in (0, 1, 2)}


def state(mesh, seed=2):
    rng = np.random.default_rng(seed)
    off = mesh.offsets()
    nd = np.diff(off)
    c = np.repeat(np.arange(mesh.n_cells), nd)
    h = 1 + 0.2 * np.sin(np.pi * mesh.vertices[c, 0]) + 1e-3 * rng.standard_normal(len(c))
    q = np.zeros(2 * len(c))
    for e, u in ((0, 0.5), (1, 0.1)):
        q[off[c] + np.arange(len(c)) + e * nd[c]] = u * h
    return h, q


def run(mesh, z, q, general=False, precision="mixed", scale=None, bcs=WALLS, steps=2, dt=1e-4,
        mode=None):
    from oceano_gb300.operator import OceanoOperator
    mixed = precision == "mixed"
    op = OceanoOperator(mesh, precision=precision, zeta_reference=1.0 if mixed else 0.0,
                        friction="linear" if general else "none")
    if mixed:
        op.set_reference_state(1.0, (0.5, 0.1))
    apply_bcs(op, bcs)
    op.set_vortex(*VORTEX)
    if scale is not None:
        op.set_cell_time_scale(scale)
    if mode:
        op.set_launch_mode(mode)
    z, q = z.copy(), q.copy()
    for k in range(steps):
        op.perform_time_step("ssp33", k * dt, dt, z, q)
    op.close()
    return z, q


def close(a, b, tol=TOL):
    for x, y in zip(a, b):
        assert np.isfinite(x).all()
        assert np.linalg.norm(x - y) < tol * np.linalg.norm(y)


def refined(nx, ny, degree):
    """Conforming but for one refined corner of the coarse grid."""
    f = QuadForest(nx, ny, (0.0, 2.0, 0.0, 1.0), periodic_x=True)
    for leaf in sorted(f.leaves):
        if leaf[1] < 7 and leaf[2] < 9:
            f.refine(leaf)
    f.balance()
    return f.build(degree)


@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("mesh", ["1 conforming", "1 hanging", "4 conforming", "4 hanging", "hp"])
def test_against_team_kernel(gpu_lib, mesh, scaled):
    m = {"1 conforming": lambda: uniform_mesh(197, 103, (0.0, 2.0, 0.0, 1.0), True, 1),
         "1 hanging": lambda: refined(197, 103, 1),
         "4 conforming": lambda: uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, 4),
         "4 hanging": lambda: hanging_mesh(4, seed=4, periodic=False),
         "hp": lambda: mixed_degree(hanging_mesh(2, seed=11))}[mesh]()
    scale = np.random.default_rng(3).uniform(0.2, 1.0, m.n_cells) if scaled else None
    z, q = state(m)
    a, b = (run(m, z, q, general=g, scale=scale) for g in (False, True))
    close(a, b)
    assert np.linalg.norm(a[0] - z) > 10 * TOL * np.linalg.norm(z)


@pytest.mark.parametrize("case", ["open_bcs_p2", "absorbing_p3"])
@pytest.mark.parametrize("degree", [1, 2, 3, 4])
def test_open_boundaries(gpu_lib, case, degree):
    mf, bcs, _, _ = CASES[case]
    m = mf().with_degree(degree)
    orc = O.Oracle(m, bcs=bcs, vortex=VORTEX + [0, 0])
    z, q = orc.project_vortex(0.0)
    zo, qo = z.copy(), q.copy()
    tb = O.TABLEAUX["ssp33"]
    for k in range(2):
        O.erk_step(orc, tb["a"], tb["b"], tb["c"], k * 1e-4, 1e-4, zo, qo)
    close(run(m, z, q, bcs=bcs), (zo, qo))


def turned(mesh, seed=6):
    """The mesh with the frames of half of the cells turned by half a turn, and the DoF order
    of zeta that goes with it."""
    rng = np.random.default_rng(seed)
    t = rng.random(mesh.n_cells) < 0.5
    v = mesh.vertices.reshape(-1, 4, 2).copy()
    v[t] = v[t][:, ::-1]
    ni = mesh.n_inner
    fm, fp, sub = mesh.face_m.copy(), mesh.face_p.copy(), mesh.subface.copy()
    tm, tp = t[mesh.cell_m], t[mesh.cell_p]
    fm[tm] ^= 1
    fp[tp] ^= 1
    flip = tp & (sub >= 0)
    sub[flip] = 1 - sub[flip]  # the half of the plus cell's face, in its frame
    orient = (tm[:ni] ^ tp).astype(mesh.orient.dtype)
    order = np.arange(mesh.n_dofs())
    off = mesh.offsets()
    for c in np.nonzero(t)[0]:
        order[off[c]:off[c + 1]] = order[off[c]:off[c + 1]][::-1]
    return Mesh(mesh.degree, v.reshape(-1, 8), mesh.cell_m, mesh.cell_p, fm, fp, sub, orient,
                mesh.bid, mesh.level, mesh.domain), order


@pytest.mark.parametrize("form", ["fp64", "fp64 one launch", "lean", "lean one launch", "general"])
@pytest.mark.parametrize("mesh", ["1 large", "2", "3", "4", "4 hanging", "hp"])
def test_turned_cells(gpu_lib, mesh, form):
    m = {"1 large": lambda: uniform_mesh(197, 103, (0.0, 2.0, 0.0, 1.0), True, 1),
         "2": lambda: uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, 2),
         "3": lambda: uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, 3),
         "4": lambda: uniform_mesh(9, 7, (0.0, 2.0, 0.0, 1.0), True, 4),
         "4 hanging": lambda: hanging_mesh(4, seed=4, periodic=False),
         "hp": lambda: mixed_degree(hanging_mesh(2, seed=11))}[mesh]()
    t, order = turned(m)
    off, nd = m.offsets(), np.diff(m.offsets())
    c = np.repeat(np.arange(m.n_cells), nd)
    qo = np.zeros(2 * m.n_dofs(), np.int64)  # the same order for both components
    for e in (0, 1):
        qo[off[c] + np.arange(len(c)) + e * nd[c]] = off[c] + order + e * nd[c]
    z, q = state(m)
    kw = dict(precision="fp64" if form.startswith("fp64") else "mixed", general=form == "general",
              mode="one" if form.endswith("one launch") else None)
    a, b = run(m, z, q, **kw), run(t, z[order], q[qo], **kw)
    # FP64: rounding of the same sums in another order
    close((b[0], b[1]), (a[0][order], a[1][qo]), 1e-12 if kw["precision"] == "fp64" else TOL)

"""The launch forms of the multilevel V-cycle's level kernels.

A level runs in one of several forms by its size: one node per thread with
one, two or four planes per thread (the coefficients of the first two loaded
ahead of the wait on small grids), or one column per thread on wide levels;
level 1's pre-smoothing runs in the fine pass's blocks or as a kernel.  Each
form is held to a NumPy FP64 restatement of M^-1 r = T^-1 r + Z_1 V_1(Z_1^T r)
built on the device's own coarse stencils (which other tests pin to the
Galerkin products), so that boards too wide for an assembled operator can be
checked.  The boards of test_level_forms reach their forms by size; a test
switch has every level of the boards of test_wide_forms run in its wide form,
so that each plane count's kernel is reached by a board of modest size.
Tolerance: 1e-4 of the result's norm, what the assembled restatement
is held to.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OMEGA = 2.0 / 3.0


def _board(ns, slabs, rows, cols, fixed):
    rng = np.random.default_rng(slabs * rows + cols)
    k = np.full((slabs, rows, cols), 0.3)
    for z in range(0, slabs, 3):
        k[z][rng.random((rows, cols)) < 0.7] = 385.0
    mesh = ns.LayeredThermalMesh(
        slab_thickness_m=tuple(35e-6 if z % 3 == 0 else 0.3e-3 for z in range(slabs)), pitch_x_m=0.25e-3,
        pitch_y_m=0.25e-3, conductivity_w_per_m_k=k)
    kwargs = {}
    if fixed:
        mask = np.zeros(mesh.node_shape, dtype=bool)
        mask[:, :, :9] = True  # two whole level-1 columns, and a ninth that splits an aggregate
        kwargs = dict(fixed_temperature_mask=mask, fixed_temperature_k=298.15)
    return ns.ThermalConductionProblem(mesh, convection=(ns.ConvectionBoundary("top", 10.0, 298.15),), **kwargs)


def _zline(d, e, f):
    """Tridiagonal solves along axis 0 (diagonal d, coupling e[z] between z and z + 1)."""

    planes = d.shape[0]
    p, g = [d[0]], [f[0]]
    for z in range(1, planes):
        l = e[z - 1] / p[-1]
        p.append(d[z] - l * e[z - 1])
        g.append(f[z] - l * g[-1])
    w = [g[-1] / p[-1]]
    for z in range(planes - 2, -1, -1):
        w.append(g[z] / p[z] - e[z] / p[z] * w[-1])
    return np.stack(w[::-1])


def _shift(n, d):
    """Slices (i, i + d) of an axis of n nodes."""

    return slice(max(0, -d), n - max(0, d)), slice(max(0, d), n - max(0, -d))


def _stencil(st, x):
    y = st[0] * x
    for k in range(1, 14):
        o = 13 + k
        pairs = [_shift(n, d) for n, d in zip(x.shape, (o // 9 - 1, (o // 3) % 3 - 1, o % 3 - 1))]
        i, j = tuple(p[0] for p in pairs), tuple(p[1] for p in pairs)
        y[i] += st[k][i] * x[j]
        y[j] += st[k][i] * x[i]
    return y


def _restrict(v, b):
    planes, rows, cols = v.shape
    padded = np.zeros((planes, -(-rows // b) * b, -(-cols // b) * b))
    padded[:, :rows, :cols] = v
    return padded.reshape(planes, padded.shape[1] // b, b, padded.shape[2] // b, b).sum(axis=(2, 4))


def _prolong(c, b, shape):
    return np.repeat(np.repeat(c, b, axis=1), b, axis=2)[:, : shape[1], : shape[2]]


def _vcycle(levels, inverse, grids, r, l=0):
    if l + 1 == len(grids):
        return (inverse @ r.reshape(-1)).reshape(r.shape)
    st = levels[l]
    live = ~((st[0] == 1.0) & (np.abs(st[1:]).sum(axis=0) == 0.0) & (r == 0.0))
    smooth = lambda f: OMEGA * _zline(st[0], st[9], f)
    b = -(-grids[l][1] // grids[l + 1][1])
    x = smooth(r)
    c = _vcycle(levels, inverse, grids, _restrict(np.where(live, r - _stencil(st, x), 0.0), b), l + 1)
    x = x + np.where(live, _prolong(c, b, x.shape), 0.0)
    return x + smooth(r - _stencil(st, x))


@pytest.mark.parametrize(
    "slabs, rows, cols, fixed",
    [
        (1, 1449, 1447, False),  # 363 x 362 columns on level 1: every step in its wide form
        (2, 820, 813, False),    # 206 x 204: wide pre-smoothing and up, node-per-thread down
        (9, 643, 655, False),    # 161 x 164, ten planes: pre-smoothing as a kernel, two planes per thread
        (8, 37, 130, True),      # nine planes: one plane per thread, loads ahead of the wait, empty aggregates
        (12, 130, 71, True),     # thirteen planes in two rounds of seven groups
        (19, 66, 90, False),     # twenty planes: more than two per thread
        (32, 41, 50, True),      # thirty-three planes, the most the preconditioner takes
    ],
)
def test_level_forms(ns_local, slabs, rows, cols, fixed):
    _check(ns_local, slabs, rows, cols, fixed)


# Level 1 is more than 200 columns long, so that the aggregates below it are 2 x 2
# (the wide forms are built for those) but for the last board's 4 x 4.
@pytest.mark.parametrize(
    "slabs, rows, cols, fixed",
    [
        (8, 811, 21, False),    # nine planes, the most of the nine-plane kernels
        (9, 23, 817, True),     # ten: the next kernels up
        (16, 811, 30, True),    # seventeen: the most of the seventeen-plane pre-smoothing
        (17, 26, 809, False),   # eighteen: the most of the eighteen-plane kernels
        (18, 812, 17, True),    # nineteen
        (32, 811, 22, False),   # thirty-three
        (19, 66, 90, True),     # 4 x 4 aggregates: only the pre-smoothing is wide
    ],
)
def test_wide_forms(ns_local, slabs, rows, cols, fixed):
    _check(ns_local, slabs, rows, cols, fixed, wide=True)


def _check(ns, slabs, rows, cols, fixed, wide=False):
    problem = _board(ns, slabs, rows, cols, fixed)
    op = ns.MatrixFreeThermalOperator(problem, preconditioner="multilevel")
    try:
        system = op.device_system
        if wide:
            system.set_test("wide_columns", 0)
        grids = system.multilevel_grids()
        levels = [system.multilevel_stencil(l + 1).astype(np.float64) for l in range(len(grids) - 1)]
        inverse = system.coarse()[1]
        shape = problem.mesh.node_shape
        free = op.free_nodes
        d = op.diagonal_high().reshape(shape)
        ax, ay, az = problem.mesh.element_coefficients()
        element = ax / 18.0 + ay / 18.0 - az / 9.0
        e = np.zeros((slabs,) + shape[1:])
        for dy in (0, 1):
            for dx in (0, 1):
                e[:, dy : dy + rows, dx : dx + cols] += element
        e *= free[:-1] & free[1:]
        r = np.random.default_rng(1).standard_normal(shape)
        expected = _zline(d, e, r)
        coarse = _vcycle(levels, inverse, grids, _restrict(np.where(free, r, 0.0), 4))
        expected += np.where(free, _prolong(coarse, 4, shape), 0.0)
        got = system.precondition_f32(r).reshape(shape)
    finally:
        op.close()
    assert np.linalg.norm(got - expected) <= 1e-4 * np.linalg.norm(expected)

"""The cooperative PCG kernel of small boards against the graph-captured kernels.

A launch plan set by the caller selects the graph-captured kernels, so each
solve runs both ways: the same stopping rules on the same FP32 recurrences,
rounded differently.  Tolerances: two converged refinements (FP64 residual
1e-10) agree like any two of them, 1e-7 of the peak rise; the residual one
inner solve can attain in FP32 is within a factor of two.  Iteration counts are
not compared: an inner residual that lingers above its tolerance crosses it
hundreds of iterations apart in two roundings (the graph-captured plans among
themselves: 4,220 and 4,637 on one of these boards).
"""

from __future__ import annotations

import numpy as np
import pytest

from pcb_analysis_b200 import workloads
from pcb_analysis_b200.mpir import MPIRConfig

pytestmark = pytest.mark.gpu

CONFIG = MPIRConfig(inner_relative_tolerance=1e-3, max_outer_iterations=40, max_inner_iterations=100000)


def _board(ns, slabs, rows, cols, fixed, void):
    rng = np.random.default_rng(rows + 7 * cols + slabs)
    k = np.full((slabs, rows, cols), 0.3)
    for z in range(0, slabs, 3):
        k[z] = np.where(rng.random((rows, cols)) < 0.6, 385.0, 0.3)
    kwargs = {}
    if void:
        active = np.ones((slabs, rows, cols), dtype=bool)
        active[:, rows // 2 :, cols // 2 :] = False
        kwargs["active"] = active
    mesh = ns.LayeredThermalMesh(
        slab_thickness_m=tuple(35e-6 if z % 3 == 0 else 0.3e-3 for z in range(slabs)),
        pitch_x_m=np.linspace(0.2e-3, 0.3e-3, cols), pitch_y_m=0.25e-3, conductivity_w_per_m_k=k,
        through_plane_conductivity_w_per_m_k=0.5 * k, **kwargs)
    problem = {}
    if fixed:
        mask = np.zeros(mesh.node_shape, dtype=bool)
        mask[0, :, 0] = True
        problem = dict(fixed_temperature_mask=mask, fixed_temperature_k=310.0)
    return ns.ThermalConductionProblem(
        mesh, convection=(ns.ConvectionBoundary("top", 12.0, 298.15),),
        heat_sources=(ns.HeatSource(((slabs, rows // 3, cols // 3),), 0.2),), **problem)


def _both(ns, problem, preconditioner, config):
    out = []
    for graph in (False, True):
        op = ns.MatrixFreeThermalOperator(problem, preconditioner=preconditioner)
        try:
            if graph:
                op.device_system.apply_plan = op.device_system.apply_plan
            rhs = op.build_rhs(op.default_reference_temperature())
            launches = op.device_system.launch_count()
            out.append(op.device_system.solve_mpir(rhs, config) | {"rhs": rhs})
            out[-1]["launches"] = op.device_system.launch_count() - launches
        finally:
            op.close()
    return out


@pytest.mark.parametrize("preconditioner", ["jacobi", "two-level"])
@pytest.mark.parametrize(
    "slabs, rows, cols, fixed, void",
    [
        (1, 1, 1, False, False),      # one element: one block
        (2, 9, 130, True, False),     # rows longer than a block's nodes
        (5, 37, 44, False, True),     # void elements: rows without an unknown
        (8, 100, 101, True, False),   # one node per thread
        (8, 128, 128, False, False),  # two nodes per thread
        (12, 118, 127, True, True),   # near the largest board the kernel takes
    ],
)
def test_small_boards_solve_alike(ns_local, preconditioner, slabs, rows, cols, fixed, void):
    one, graph = _both(ns_local, _board(ns_local, slabs, rows, cols, fixed, void), preconditioner, CONFIG)
    assert one["converged"] and graph["converged"]
    assert one["launches"] < graph["launches"]
    peak = np.max(np.abs(graph["solution"]))
    assert np.max(np.abs(one["solution"] - graph["solution"])) <= 1e-7 * peak


@pytest.mark.parametrize("preconditioner", ["jacobi", "two-level"])
@pytest.mark.parametrize("slabs, rows, cols, fixed, void", [(2, 9, 130, True, False), (5, 37, 44, False, True),
                                                            (8, 128, 128, False, False)])
def test_attainable_residual(ns_local, preconditioner, slabs, rows, cols, fixed, void):
    """One inner solve run far past FP32: what its correction leaves in FP64."""

    config = MPIRConfig(inner_relative_tolerance=1e-9, max_outer_iterations=2, max_inner_iterations=4000)
    one, graph = _both(ns_local, _board(ns_local, slabs, rows, cols, fixed, void), preconditioner, config)
    assert one["history"][1][1] <= 2.0 * graph["history"][1][1]


@pytest.mark.parametrize("preconditioner", ["jacobi", "two-level"])
@pytest.mark.parametrize("limit", [1, 7, 540])
def test_iteration_limit(ns_local, preconditioner, limit):
    """Stops at the limit with the last step still owed, and across launches
    (540 iterations are more than one launch runs; the inner tolerance is out
    of FP32's reach)."""

    config = MPIRConfig(inner_relative_tolerance=1e-30, max_outer_iterations=1, max_inner_iterations=limit)
    one, graph = _both(ns_local, _board(ns_local, 6, 60, 70, True, False), preconditioner, config)
    assert [h[2] for h in one["history"]] == [h[2] for h in graph["history"]] == [limit]
    assert one["low_operator_applications"] == graph["low_operator_applications"]
    if limit < 540:  # before the two roundings of the recurrence drift apart
        peak = np.max(np.abs(graph["solution"]))
        assert np.max(np.abs(one["solution"] - graph["solution"])) <= 1e-4 * peak


def test_same_bits_every_time(ns_local):
    problem = workloads.board_c1(3, None, 70, 61)
    op = ns_local.MatrixFreeThermalOperator(problem, preconditioner="two-level")
    try:
        rhs = op.build_rhs(op.default_reference_temperature())
        first, second = (op.device_system.solve_mpir(rhs, CONFIG) for _ in range(2))
    finally:
        op.close()
    np.testing.assert_array_equal(first["solution"], second["solution"])
    assert first["history"] == second["history"]


def test_a_wait_that_runs_out_is_reported(ns_local):
    op = ns_local.MatrixFreeThermalOperator(workloads.board_c1(0, None, 40, 48), preconditioner="two-level")
    try:
        system = op.device_system
        rhs = op.build_rhs(op.default_reference_temperature())
        before = system.solve_mpir(rhs, CONFIG)
        system.set_stage_test(64)  # block 0 posts nothing
        with pytest.raises(TimeoutError):
            system.solve_mpir(rhs, CONFIG)
        system.set_stage_test(0)
        after = system.solve_mpir(rhs, CONFIG)
    finally:
        op.close()
    np.testing.assert_array_equal(before["solution"], after["solution"])


@pytest.mark.parametrize(
    "preconditioner, words",
    [("jacobi", 1), ("jacobi", 2), ("jacobi", 16), ("two-level", 1), ("two-level", 2), ("two-level", 4),
     ("two-level", 8), ("two-level", 16), ("two-level", 0)],
)
@pytest.mark.parametrize("block, slice_", [(0, 0), (7, 0), (119, 1)])
def test_every_wait_that_runs_out_is_reported(ns_local, preconditioner, words, block, slice_):
    """One block keeps back one kind of word: direction, p.q, patch sums, coarse
    solution or r.z (0: all of them).  With launches of one iteration the last
    block's coarse solution is missed by blocks that nobody waits for any more."""

    op = ns_local.MatrixFreeThermalOperator(workloads.board_c1(0, None, 40, 48), preconditioner=preconditioner)
    try:
        system = op.device_system
        rhs = op.build_rhs(op.default_reference_temperature())
        before = system.solve_mpir(rhs, CONFIG)
        system.set_test("pcg_mute", words)
        system.set_test("pcg_mute_block", block)
        system.set_test("pcg_slice", slice_)
        system.set_stage_test(64)
        with pytest.raises(TimeoutError, match="PCG kernel"):
            system.solve_mpir(rhs, CONFIG)
        system.set_stage_test(0)
        after = system.solve_mpir(rhs, CONFIG)
    finally:
        op.close()
    np.testing.assert_array_equal(before["solution"], after["solution"])


@pytest.mark.parametrize("preconditioner", ["jacobi", "two-level"])
@pytest.mark.parametrize("refused", [1, 2])
def test_a_refused_kernel_leaves_the_solve_to_the_graph_kernels(ns_local, preconditioner, refused):
    """Its buffers (1) or its cooperative launch (2) are refused by the runtime."""

    problem = workloads.board_c1(0, None, 40, 48)
    out = []
    for graph in (False, True):
        op = ns_local.MatrixFreeThermalOperator(problem, preconditioner=preconditioner)
        try:
            system = op.device_system
            rhs = op.build_rhs(op.default_reference_temperature())
            if graph:
                system.apply_plan = system.apply_plan
            else:
                system.set_test("pcg_refuse", refused)
            out.append(system.solve_mpir(rhs, CONFIG))
            if not graph:  # allowed again: the kernel is taken up again
                system.set_test("pcg_refuse", 0)
                launches = system.launch_count()
                again = system.solve_mpir(rhs, CONFIG)
                assert again["converged"]
                assert system.launch_count() - launches < 1000
        finally:
            op.close()
    assert out[0]["converged"]
    np.testing.assert_array_equal(out[0]["solution"], out[1]["solution"])
    assert out[0]["history"] == out[1]["history"]


@pytest.mark.parametrize("cols, taken", [(4799, True), (4803, False), (7000, False)])
def test_boards_with_long_rows_stay_on_the_graph_kernels(ns_local, cols, taken):
    config = MPIRConfig(inner_relative_tolerance=1e-30, max_outer_iterations=1, max_inner_iterations=30)
    one, graph = _both(ns_local, _board(ns_local, 2, 1, cols, False, False), "jacobi", config)
    assert (one["launches"] < graph["launches"]) == taken
    if not taken:
        np.testing.assert_array_equal(one["solution"], graph["solution"])


def _rows(mesh):
    """The operator's rows in FP64: couplings [27, nodes] in the order (dz, dy, dx)
    ascending, the centre left out."""

    a = np.zeros((27,) + mesh.node_shape)
    parts = [c.reshape(mesh.conductivity_w_per_m_k.shape) for c in mesh.element_coefficients()]
    slabs, rows, cols = parts[0].shape
    ends = [(o, b) for o in np.ndindex(2, 2, 2) for b in np.ndindex(2, 2, 2) if b != (0, 0, 0)]
    for corner, other in ends:
        m = [1.0 / 6.0 if t else 2.0 / 6.0 for t in other]
        s = [-1.0 if t else 1.0 for t in other]
        k = parts[0] * (m[0] * m[1] * s[2]) + parts[1] * (m[0] * s[1] * m[2]) + parts[2] * (s[0] * m[1] * m[2])
        step = [(1 - 2 * c) * t for c, t in zip(corner, other)]
        o = (step[0] + 1) * 9 + (step[1] + 1) * 3 + step[2] + 1
        a[o][corner[0] : corner[0] + slabs, corner[1] : corner[1] + rows, corner[2] : corner[2] + cols] += k
    return a


@pytest.mark.parametrize(
    "slabs, rows, cols, fixed, void",
    [(8, 37, 44, True, True), (16, 30, 41, False, False), (16, 80, 100, True, False), (3, 210, 19, False, True)],
)
@pytest.mark.parametrize("smooth", [False, True])
def test_two_iterations_match_fp64(ns_local, slabs, rows, cols, fixed, void, smooth):
    """Two inner iterations against the same in FP64, node by node.

    The second direction holds the first action of the kernel's own operator at
    every node, so a wrong coefficient shows where it stands.  Bound: the
    magnitudes that a node's value is made of (the action's taken on differences,
    as the kernel does) times 32 units of FP32 rounding: some 24 roundings of half
    a unit each along the way, and as much again for the scalars."""

    problem = _board(ns_local, slabs, rows, cols, fixed, void)
    op = ns_local.MatrixFreeThermalOperator(problem, preconditioner="jacobi")
    config = MPIRConfig(inner_relative_tolerance=1e-30, max_outer_iterations=1, max_inner_iterations=2)
    try:
        shape = problem.mesh.node_shape
        free = op.free_nodes.reshape(-1)
        d = op.diagonal_high().reshape(-1)
        rng = np.random.default_rng(slabs + rows)
        v = rng.standard_normal(shape)
        if smooth:  # nearly constant through the stack
            v = v[:1] + 1e-3 * v
        r0 = d * v.reshape(-1) * free
        got = op.device_system.solve_mpir(r0, config)["solution"]
        action = op.apply_high
        p0 = r0 / d
        q0 = action(p0)
        rz0 = r0 @ p0
        a0 = rz0 / (p0 @ q0)
        r1 = r0 - a0 * q0
        z1 = r1 / d
        b0 = (r1 @ z1) / rz0
        p1 = z1 + b0 * p0
        a1 = (r1 @ z1) / (p1 @ action(p1))
    finally:
        op.close()
    expected = a0 * p0 + a1 * p1
    rows27 = _rows(problem.mesh)
    u = np.pad((p0 * free).reshape(shape), 1)
    centre = p0.reshape(shape)
    size = np.zeros(shape)
    view = lambda dz, dy, dx: u[1 + dz : u.shape[0] - 1 + dz, 1 + dy : u.shape[1] - 1 + dy, 1 + dx : u.shape[2] - 1 + dx]
    total = np.zeros(shape)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            k = (dy + 1) * 3 + dx + 1
            low, mid, high = rows27[k], rows27[9 + k], rows27[18 + k]
            side = view(0, dy, dx)
            size += np.abs(low * (view(-1, dy, dx) - side)) + np.abs(high * (view(1, dy, dx) - side))
            size += np.abs((low + mid + high) * (side - centre))
            total += low + mid + high
    robin = np.maximum(d.reshape(shape) + total, 0.0)  # the diagonal less the element part: R
    size += robin * np.abs(centre)
    size = size.reshape(-1)
    bound = np.abs(a0 * p0) + np.abs(a1) * ((np.abs(r0) + np.abs(a0) * size) / d + np.abs(b0 * p0))
    eps = np.finfo(np.float32).eps
    assert np.all(np.abs(got - expected)[free] <= 32 * eps * bound[free])
    assert np.linalg.norm((got - expected)[free]) <= 8 * eps * np.linalg.norm(bound[free])


def test_small_solves_leave_a_batch_engine_its_share(ns_local):
    """A thread of small solves beside a batch: both get on, with the same bits as
    alone.  The batch took six times as long with launches that did not wait for
    the engine's; the bound is three."""

    import threading
    import time

    from pcb_analysis_b200 import serve
    from pcb_analysis_b200._native import BatchEngine

    requests = [serve.board_request(workloads.board_random(i, side=(150 + 5 * i, 150 + 5 * i), slabs=(8, 8)))
                for i in range(6)]
    op = ns_local.MatrixFreeThermalOperator(workloads.board_c1(0, None, 96, 80), preconditioner="two-level")
    try:
        with BatchEngine(capacity=6, max_slabs=8, tile_rows=16, preconditioner="two-level") as engine:
            def batch():
                start = time.perf_counter()
                results = serve.solve_batch(requests, CONFIG, engine=engine)
                return time.perf_counter() - start, results

            rhs = op.build_rhs(op.default_reference_temperature())
            alone = op.device_system.solve_mpir(rhs, CONFIG)
            batch()
            seconds, expected = batch()
            beside, stop = [], threading.Event()

            def small():
                while not stop.is_set():
                    beside.append(op.device_system.solve_mpir(rhs, CONFIG))

            thread = threading.Thread(target=small)
            thread.start()
            try:
                shared_seconds, shared = batch()
            finally:
                stop.set()
                thread.join()
    finally:
        op.close()
    assert beside
    for result in beside:
        np.testing.assert_array_equal(result["solution"], alone["solution"])
    for got, want in zip(shared, expected):
        np.testing.assert_array_equal(got.solution, want.solution)
    assert shared_seconds <= 3.0 * seconds

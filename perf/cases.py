"""The work a user of this framework has it do, as measurable cases.

Three ways in, as programs use them:

* ``call``: the whole public call from host arrays (``solve_thermal_conduction``,
  ``solve_thermal_transient``, ``solve_pcb_dc``) -- prepare, solve, post-process;
* ``resident``: an operator kept in HBM by a program that solves one board
  again and again (parameter sweeps, coupled loops, a service), the right-hand
  side and the iterate being device tensors;
* ``batch``: boards handed to a running ``BatchEngine``;

and the two operator actions by themselves (``action``), for programs that run
their own iteration around the operator.

Boards come from the package's seeded workload generators: the stack-ups c1
(8 slabs), c2 (12 slabs), c3 (16 slabs, a fixed edge strip), and the mixed
boards of the batch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import pcb_analysis_b200.electrical as electrical
import pcb_analysis_b200.thermal as thermal
from pcb_analysis_b200 import serve, workloads
from pcb_analysis_b200._native import BatchEngine
from pcb_analysis_b200.mpir import MPIRConfig

DEVICE = "cuda:0"
SLABS = {"c1": 8, "c2": 12, "c3": 16}
# The refinement settings of the repository's own benchmark: FP32 PCG to 1e-4
# inside, the FP64 residual to 1e-10.
TIGHT = MPIRConfig(inner_relative_tolerance=1e-4, max_outer_iterations=40, max_inner_iterations=400000)


def listed():
    return [
        # One small module through the public call with its defaults (two-level,
        # the facade's own limits): an interactive what-if.
        dict(name="call_small_default", kind="call", rules="c1", rows=128, cols=128, preconditioner="two-level",
             settings="default"),
        # The same call on an ordinary board of ragged size, multilevel.
        dict(name="call_ragged_multilevel", kind="call", rules="c2", rows=311, cols=257, preconditioner="multilevel",
             settings="tight"),
        # Smallest resident solve: latency and launches count.
        dict(name="resident_tiny_multilevel", kind="resident", rules="c1", rows=71, cols=93,
             preconditioner="multilevel"),
        # The plain Jacobi PCG that the method is named after, on a small board.
        dict(name="resident_small_jacobi", kind="resident", rules="c1", rows=96, cols=80, preconditioner="jacobi"),
        # An ordinary board, swept: the reference's default preconditioner ...
        dict(name="resident_board_two_level", kind="resident", rules="c2", rows=512, cols=512,
             preconditioner="two-level"),
        # ... and the one for larger boards.
        dict(name="resident_board_multilevel", kind="resident", rules="c2", rows=512, cols=512,
             preconditioner="multilevel"),
        # The largest single board.
        dict(name="resident_large_multilevel", kind="resident", rules="c3", rows=2048, cols=2048,
             preconditioner="multilevel"),
        # A short backward-Euler march of a board warming up.
        dict(name="transient_march", kind="transient", rules="c1", rows=150, cols=122, preconditioner="two-level",
             steps=5),
        # Uneven boards through the batch engine.
        dict(name="batch_mixed", kind="batch", count=10, low=72, high=288, preconditioner="two-level"),
        # The electrical package's DC solve of a four-layer power net.
        dict(name="call_dc_net", kind="dc", rows=384, cols=512, vias=600, preconditioner="two-level"),
        # One FP32 action of the operator on an ordinary board, one FP64 action on a ragged one.
        dict(name="action_low", kind="action", rules="c2", rows=512, cols=512, precision="low"),
        dict(name="action_high", kind="action", rules="c2", rows=333, cols=701, precision="high"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["call", "resident", "resident", "resident", "transient", "batch", "dc", "action", "action"])
    if kind == "call":
        two = rng.random() < 0.5
        return dict(kind=kind, rules=rng.choice(["c1", "c2"]), rows=_log_int(rng, 64, 160 if two else 512),
                    cols=_log_int(rng, 64, 160 if two else 512), preconditioner="two-level" if two else "multilevel",
                    settings="tight")
    if kind == "resident":
        preconditioner = rng.choice(["multilevel", "multilevel", "two-level", "jacobi"])
        top = {"multilevel": 1024, "two-level": 480, "jacobi": 112}[preconditioner]
        rules = rng.choice(["c1", "c2", "c3"])
        return dict(kind=kind, rules=rules, rows=_log_int(rng, 64, top), cols=_log_int(rng, 64, top),
                    preconditioner=preconditioner)
    if kind == "transient":
        return dict(kind=kind, rules=rng.choice(["c1", "c2"]), rows=_log_int(rng, 64, 160),
                    cols=_log_int(rng, 64, 160), preconditioner=rng.choice(["two-level", "multilevel"]),
                    steps=rng.randint(2, 5))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 10), low=64, high=_log_int(rng, 96, 288),
                    preconditioner="two-level")
    if kind == "dc":
        return dict(kind=kind, rows=_log_int(rng, 128, 512), cols=_log_int(rng, 128, 512), vias=_log_int(rng, 100, 800),
                    preconditioner="two-level")
    return dict(kind=kind, rules=rng.choice(["c1", "c2", "c3"]), rows=_log_int(rng, 64, 1024),
                cols=_log_int(rng, 64, 1024), precision=rng.choice(["low", "high"]))


# ------------------------------------------------------------------ building
def _board(case, seed):
    build = {"c1": workloads.board_c1, "c2": workloads.board_c2, "c3": workloads.board_c3}[case["rules"]]
    return build(seed, None, case["rows"], case["cols"])


def _heat_capacity(problem):
    """The board with volumetric heat capacities (copper 3.45, FR-4 1.9 MJ/m3K)."""

    mesh = problem.mesh
    k = np.asarray(mesh.conductivity_w_per_m_k)
    capacity = np.where(k > 100.0, 3.45e6, 1.9e6)
    mesh = thermal.LayeredThermalMesh(
        slab_thickness_m=mesh.slab_thickness_m, pitch_x_m=mesh.pitch_x_m, pitch_y_m=mesh.pitch_y_m,
        conductivity_w_per_m_k=k, volumetric_heat_capacity_j_per_m3_k=capacity)
    return thermal.ThermalConductionProblem(mesh, convection=problem.convection, heat_sources=problem.heat_sources)


def _schedule(case):
    return thermal.TimeSchedule.geometric(0.5, 0.5 * (1.5 ** case["steps"] - 1.0) / 0.5, growth=1.5)


def _batch_problems(case, seed):
    """Boards by the batch rules; every board's size is fixed by the case, its copper by the seed."""

    out = []
    for i in range(case["count"]):
        t = i / max(1, case["count"] - 1)
        side = int(round(case["low"] * (case["high"] / case["low"]) ** t))
        slabs = 4 + (5 * i) % 9
        out.append(workloads.board_random(seed * 1000 + i, side=(side, side), slabs=(slabs, slabs)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "call":
        return dict(case=case, problem=_board(case, seed), config=None if case["settings"] == "default" else TIGHT)
    if kind == "transient":
        return dict(case=case, problem=_heat_capacity(_board(case, seed)), schedule=_schedule(case))
    if kind == "dc":
        return dict(case=case, problem=workloads.dc_power_net(seed, None, case["rows"], case["cols"], case["vias"]),
                    config=MPIRConfig(relative_tolerance=1e-12, inner_relative_tolerance=1e-4,
                                      max_outer_iterations=40, max_inner_iterations=100000))
    if kind == "batch":
        requests = [serve.board_request(p) for p in _batch_problems(case, seed)]
        engine = BatchEngine(capacity=case["count"], max_slabs=12, preconditioner=case["preconditioner"])
        return dict(case=case, requests=requests, engine=engine)
    if kind == "action":
        operator = thermal.MatrixFreeThermalOperator(_board(case, seed), preconditioner="jacobi")
        generator = torch.Generator(device=DEVICE).manual_seed(seed)
        dtype = torch.float32 if case["precision"] == "low" else torch.float64
        x = torch.randn(operator.size, generator=generator, device=DEVICE, dtype=dtype)
        return dict(case=case, operator=operator, x=x, y=torch.empty_like(x))
    operator = thermal.MatrixFreeThermalOperator(_board(case, seed), preconditioner=case["preconditioner"])
    reference = operator.default_reference_temperature()
    rhs = torch.empty(operator.size, device=DEVICE, dtype=torch.float64)
    operator.device_system.build_rhs_device(reference, rhs)
    return dict(case=case, operator=operator, reference=reference, rhs=rhs)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        s = thermal.solve_thermal_conduction(state["problem"], config=state["config"],
                                             preconditioner=case["preconditioner"])
        return dict(temperature_k=s.temperature_k, heat_flux=s.heat_flux_w_per_m2, convective_w=s.convective_heat_w)
    if kind == "transient":
        s = thermal.solve_thermal_transient(state["problem"], state["schedule"], preconditioner=case["preconditioner"],
                                            config=TIGHT)
        return dict(temperature_k=s.temperature_k, stored_w=s.final.stored_heat_w)
    if kind == "dc":
        s = electrical.solve_pcb_dc(state["problem"], config=state["config"], preconditioner=case["preconditioner"])
        return dict(potential_v=np.nan_to_num(s.potential_v), current_density=s.current_density_a_per_m2,
                    via_current_a=s.via_current_a, loss_w=s.joule_loss_w)
    if kind == "batch":
        results = serve.solve_batch(state["requests"], TIGHT, engine=state["engine"])
        return [q.tag + r.solution for q, r in zip(state["requests"], results)]
    if kind == "action":
        system = state["operator"].device_system
        if case["precision"] == "low":
            system.apply_f32_device(state["x"], state["y"])
        else:
            system.apply_f64_device(state["x"], state["y"])
        return state["y"]
    rise = torch.zeros_like(state["rhs"])
    state["operator"].device_system.solve_mpir_device(state["rhs"], rise, TIGHT)
    return rise + state["reference"]


def work(case):
    """Each input read once and each output written once; for a solve one FP64
    residual's arithmetic per digit that it gains over the start."""

    kind = case["kind"]
    per_element = 110.0  # forward and inverse Haar transforms, seven scalings, of one element
    if kind == "dc":
        elements, nodes = 4 * case["rows"] * case["cols"], 4 * (case["rows"] + 1) * (case["cols"] + 1)
        return dict(bytes=9.0 * elements + 8.0 * nodes + 16.0 * elements, flops=10 * 40.0 * elements)
    if kind == "batch":
        elements = nodes = 0
        for i in range(case["count"]):
            side = int(round(case["low"] * (case["high"] / case["low"]) ** (i / max(1, case["count"] - 1))))
            slabs = 4 + (5 * i) % 9
            elements += slabs * side * side
            nodes += (slabs + 1) * (side + 1) ** 2
        return dict(bytes=16.0 * elements + 25.0 * nodes, flops=10 * per_element * elements)
    slabs = SLABS[case["rules"]]
    elements = slabs * case["rows"] * case["cols"]
    nodes = (slabs + 1) * (case["rows"] + 1) * (case["cols"] + 1)
    if kind == "action":
        word = 4 if case["precision"] == "low" else 8
        return dict(bytes=word * (2.0 * elements + 2.0 * nodes), flops=per_element * elements)
    if kind == "resident":
        return dict(bytes=16.0 * elements + 16.0 * nodes, flops=10 * per_element * elements)
    if kind == "transient":
        return dict(bytes=24.0 * elements + 8.0 * nodes * (case["steps"] + 1),
                    flops=10 * per_element * elements * case["steps"])
    return dict(bytes=40.0 * elements + 8.0 * nodes, flops=10 * per_element * elements)


# ------------------------------------------------- the same in plain torch FP64
_S = np.array([[1.0, -1.0], [-1.0, 1.0]])
_M = np.array([[2.0, 1.0], [1.0, 2.0]]) / 6.0
EXACT_NODES = 260_000  # a plain Jacobi PCG of more nodes takes too long


def _unit(z, y, x):
    return torch.tensor(np.kron(np.kron(z, y), x), device=DEVICE)


class _Hex:
    """K u of the trilinear hexahedra, from the conductivities and the grid."""

    def __init__(self, mesh):
        f64 = dict(device=DEVICE, dtype=torch.float64)
        k = torch.tensor(np.asarray(mesh.conductivity_w_per_m_k), **f64)
        kz = torch.tensor(np.asarray(mesh.through_plane_conductivity_w_per_m_k), **f64)
        hz = torch.tensor(np.asarray(mesh.slab_thickness_m), **f64)[:, None, None]
        hy = torch.tensor(np.asarray(mesh.pitch_y_m), **f64)[None, :, None]
        hx = torch.tensor(np.asarray(mesh.pitch_x_m), **f64)[None, None, :]
        self.k, self.kz, self.h = k, kz, (hz, hy, hx)
        self.a = [(k * hy * hz / hx).reshape(-1), (k * hx * hz / hy).reshape(-1), (kz * hx * hy / hz).reshape(-1)]
        self.u = [_unit(_M, _M, _S), _unit(_M, _S, _M), _unit(_S, _M, _M)]
        self.shape = k.shape
        s, r, c = k.shape
        self.nodes = (s + 1, r + 1, c + 1)

    def _views(self, grid):
        s, r, c = self.shape
        return [grid[i >> 2 : (i >> 2) + s, (i >> 1) % 2 : (i >> 1) % 2 + r, i % 2 : i % 2 + c] for i in range(8)]

    def __call__(self, v):
        e = torch.stack(self._views(v.reshape(self.nodes))).reshape(8, -1)
        f = sum(a * (u @ e) for a, u in zip(self.a, self.u))
        out = torch.zeros(self.nodes, device=DEVICE, dtype=torch.float64)
        for view, part in zip(self._views(out), f.reshape((8,) + tuple(self.shape))):
            view += part
        return out.reshape(-1)

    def diagonal(self):
        f = sum(a * u[0, 0] for a, u in zip(self.a, self.u)).reshape(self.shape)
        out = torch.zeros(self.nodes, device=DEVICE, dtype=torch.float64)
        for view in self._views(out):
            view += f
        return out.reshape(-1)

    def flux(self, t):
        v = self._views(t.reshape(self.nodes))
        parts = []
        for bit, h, k in ((1, self.h[2], self.k), (2, self.h[1], self.k), (4, self.h[0], self.kz)):
            up = sum(v[i] for i in range(8) if i & bit)
            down = sum(v[i] for i in range(8) if not i & bit)
            parts.append(-k * (up - down) / (4.0 * h))
        return torch.stack(parts, dim=-1)


def _pcg(apply, diagonal, b, tolerance=1e-13, limit=60000):
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diagonal
    p = z.clone()
    rz = r @ z
    target = float(b @ b) * tolerance**2
    for i in range(limit):
        q = apply(p)
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        if i % 50 == 49 and float(r @ r) <= target:
            break
        z = r / diagonal
        new = r @ z
        p = z + (new / rz) * p
        rz = new
    return x


def _film(problem, hexes):
    """Lumped film conductance and R T_amb of the two faces, nodal sources, fixed nodes."""

    robin = torch.zeros(hexes.nodes, device=DEVICE, dtype=torch.float64)
    ambient = torch.zeros_like(robin)
    area = (hexes.h[1] * hexes.h[2])[0]
    for face in problem.convection:
        z = -1 if face.side == "top" else 0
        share = float(face.coefficient_w_per_m2_k) * area / 4.0
        for dy in (0, 1):
            for dx in (0, 1):
                rows, cols = area.shape
                robin[z, dy : dy + rows, dx : dx + cols] += share
                ambient[z, dy : dy + rows, dx : dx + cols] += share * float(face.ambient_temperature_k)
    load = torch.zeros_like(robin)
    for source in problem.heat_sources:
        index = torch.tensor(source.nodes, device=DEVICE).T
        value = torch.full((index.shape[1],), source.power_w / len(source.nodes), device=DEVICE, dtype=torch.float64)
        load.index_put_(tuple(index), value, accumulate=True)
    fixed = torch.tensor(np.asarray(problem.fixed_temperature_mask), device=DEVICE).reshape(-1)
    held = torch.tensor(np.asarray(problem.fixed_temperature_k), device=DEVICE, dtype=torch.float64).reshape(-1)
    return robin.reshape(-1), ambient.reshape(-1), load.reshape(-1), fixed, held


def _steady(problem, hexes, capacity=None, previous=None):
    robin, ambient, load, fixed, held = _film(problem, hexes)
    reference = float(problem.convection[0].ambient_temperature_k)
    free = (~fixed).to(torch.float64)
    shift = torch.where(fixed, held - reference, torch.zeros_like(held))
    diagonal = hexes.diagonal() + robin
    b = load + ambient - robin * reference - hexes(shift)
    total = robin
    if capacity is not None:
        diagonal, total = diagonal + capacity, robin + capacity
        b = b + capacity * (previous - reference)
    b = b * free
    diagonal = torch.where(fixed, torch.ones_like(diagonal), diagonal)
    rise = _pcg(lambda v: (hexes(v) + total * v) * free, diagonal, b)
    return rise * free + shift + reference, robin, ambient


def _film_heat(problem, hexes, t):
    out = []
    for face in problem.convection:
        alone = thermal.ThermalConductionProblem(problem.mesh, convection=(face,))
        robin, ambient = _film(alone, hexes)[:2]
        out.append(torch.sum(robin * t - ambient))
    return torch.stack(out)


def _sheets(problem):
    """K v of the bilinear sheets and vias, its diagonal, and the terminal data."""

    f64 = dict(device=DEVICE, dtype=torch.float64)
    mesh = problem.mesh
    active = torch.tensor(np.asarray(mesh.element_active), device=DEVICE)
    thickness = torch.tensor(np.asarray(mesh.layer_thickness_m), **f64)[:, None, None]
    sigma = torch.tensor(np.broadcast_to(np.asarray(mesh.conductivity_s_per_m), mesh.element_active.shape).copy(),
                         **f64)
    hy = torch.tensor(np.asarray(mesh.pitch_y_m), **f64)[None, :, None]
    hx = torch.tensor(np.asarray(mesh.pitch_x_m), **f64)[None, None, :]
    sheet = sigma * thickness * active
    a = [(sheet * hy / hx).reshape(-1), (sheet * hx / hy).reshape(-1)]
    u = [torch.tensor(np.kron(_M, _S), device=DEVICE), torch.tensor(np.kron(_S, _M), device=DEVICE)]
    layers, rows, cols = mesh.element_active.shape
    nodes = (layers, rows + 1, cols + 1)

    def views(grid):
        return [grid[:, i >> 1 : (i >> 1) + rows, i % 2 : i % 2 + cols] for i in range(4)]

    def flat(node):
        return int(np.ravel_multi_index(node, nodes))

    low = torch.tensor([flat(v.lower) for v in problem.vias], device=DEVICE)
    up = torch.tensor([flat(v.upper) for v in problem.vias], device=DEVICE)
    g = torch.tensor([v.conductance_s for v in problem.vias], **f64)

    def apply(v):
        e = torch.stack(views(v.reshape(nodes))).reshape(4, -1)
        f = (a[0] * (u[0] @ e) + a[1] * (u[1] @ e)).reshape((4,) + tuple(active.shape))
        out = torch.zeros(nodes, **f64)
        for view, part in zip(views(out), f):
            view += part
        out = out.reshape(-1)
        drop = g * (v[low] - v[up])
        return out.index_add(0, low, drop).index_add(0, up, -drop)

    diagonal = torch.zeros(nodes, **f64)
    f = (a[0] * u[0][0, 0] + a[1] * u[1][0, 0]).reshape(active.shape)
    for view in views(diagonal):
        view += f
    diagonal = diagonal.reshape(-1).index_add(0, low, g).index_add(0, up, g)
    return apply, diagonal, views, nodes, flat, (low, up, g), sigma * active, (hy, hx), (a, u)


def _dc(problem):
    apply, diagonal, views, nodes, flat, (low, up, g), sigma, (hy, hx), (a, u) = _sheets(problem)
    b = torch.zeros_like(diagonal)
    for terminal in problem.terminals:
        for node in terminal.nodes:
            b[flat(node)] += terminal.current_a / len(terminal.nodes)
    held = torch.zeros_like(diagonal)
    fixed = diagonal == 0.0
    for terminal in problem.voltage_terminals:
        index = torch.tensor([flat(n) for n in terminal.nodes], device=DEVICE)
        held[index] = terminal.voltage_v
        fixed[index] = True
    free = (~fixed).to(torch.float64)
    b = (b - apply(held)) * free
    v = _pcg(lambda w: apply(w) * free, torch.where(fixed, torch.ones_like(diagonal), diagonal), b) * free + held
    c = views(v.reshape(nodes))
    field = torch.stack([-(c[1] + c[3] - c[0] - c[2]) / (2.0 * hx), -(c[2] + c[3] - c[0] - c[1]) / (2.0 * hy)], dim=-1)
    e = torch.stack(c).reshape(4, -1)
    drop = v[low] - v[up]
    loss = float(sum((w * (e * (m @ e)).sum(0)).sum() for w, m in zip(a, u)) + (g * drop * drop).sum())
    return dict(potential_v=v.reshape(nodes), current_density=sigma[..., None] * field, via_current_a=g * drop,
                loss_w=loss)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    if kind == "dc":
        if 4 * case["rows"] * case["cols"] > 4 * EXACT_NODES:
            return None
        return _dc(workloads.dc_power_net(seed, None, case["rows"], case["cols"], case["vias"]))
    nodes = (SLABS[case["rules"]] + 1) * (case["rows"] + 1) * (case["cols"] + 1)
    if kind != "action" and nodes > EXACT_NODES:
        return None
    problem = _board(case, seed)
    if kind == "action":
        hexes = _Hex(problem.mesh)
        robin, _, _, fixed, _ = _film(problem, hexes)
        generator = torch.Generator(device=DEVICE).manual_seed(seed)
        dtype = torch.float32 if case["precision"] == "low" else torch.float64
        x = torch.randn(nodes, generator=generator, device=DEVICE, dtype=dtype).to(torch.float64)
        free = (~fixed).to(torch.float64)
        return torch.where(fixed, x, hexes(x * free) + robin * x)
    if kind == "transient":
        problem = _heat_capacity(problem)
        hexes = _Hex(problem.mesh)
        lump = torch.tensor(problem.mesh.nodal_heat_capacity_j_per_k(), device=DEVICE).reshape(-1)
        t = torch.full((nodes,), float(problem.convection[0].ambient_temperature_k), device=DEVICE,
                       dtype=torch.float64)
        fields = [t]
        for step in _schedule(case).steps_s:
            t, _, _ = _steady(problem, hexes, lump / step, fields[-1])
            fields.append(t)
        stored = float(torch.sum(lump / step * (fields[-1] - fields[-2])))
        return dict(temperature_k=torch.stack(fields).reshape((-1,) + hexes.nodes), stored_w=stored)
    hexes = _Hex(problem.mesh)
    t, _, _ = _steady(problem, hexes)
    if kind == "resident":
        return t
    return dict(temperature_k=t.reshape(hexes.nodes), heat_flux=hexes.flux(t),
                convective_w=_film_heat(problem, hexes, t))

"""The work a program gives this library, as cases that can be timed.

A case names a call that users make (a quasi-steady or dynamic `Simulation.do_step`, a sweep of
conditions through `CompleteSailModel`, the standalone `panel_sweep`, a step of a `Batch`, the
warm-start network's forward pass and an epoch of its training) and its sizes. `prepare` builds what
the program has in hand before the call, `run` makes the call once, `work` says what the call cannot
do without, and `exact` restates the result in 64 bits in plain torch.

Simulations start from a loaded state: a shed wake of seeded shape and strength, so that a pass is a
step in the middle of a run and not the first step of one. Every pass is the next time step: the wind
gusts from step to step (a period of 8 steps), so that the circulation has to be solved for anew.

Outputs are everything the call returns, with one exception: the solver's `residual`, the mean
difference of two lift coefficients that the iteration drives towards 0, whose trailing digits are the
rounding of the two. The circulation and the iteration count beside it say what it says.
"""
from __future__ import annotations

import json
import math
import random

import numpy as np
import torch

SPAN, CHORD, SPACING, DENSITY = 30.0, 10.0, 40.0, 1.225  # the sails of stormbird_gb300.setups
INCIDENCE = math.radians(8.0)                            # local angle of attack of the sails
STALL, STALL_RANGE, CD_MIN, CDI = math.radians(15.0), math.radians(6.0), 0.01, 0.05
PERIOD, GUST = 8, 0.025                                  # steps of a gust and its part of the wind speed
PAIRS_EXACT = 7e9                                        # target-panel pairs that exact() sums up in time


# ---------------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # One sail, quasi-steady, damped iterations to a tight residual: a polar, or the inner call of
        # an optimiser, made one condition after another. The smallest call: latency alone.
        dict(name="qs_wing_iterative", kind="quasi_steady", solver="iterative", sails=1, panels=32, wind=10.0,
             awa=8.0),
        # A ship's whole row, quasi-steady with the default (Linearized) solver at a fine resolution.
        dict(name="qs_row_linearized", kind="quasi_steady", solver="linearized", sails=6, panels=95, wind=11.0,
             awa=50.0),
        # The sails' forces over all wind directions, as a routing or a velocity prediction program asks
        # for: one batched call of a CompleteSailModel, controller included.
        dict(name="csm_wind_directions", kind="csm", sails=3, panels=24, conditions=36, wind=9.0),
        # Co-simulation with a ship: a step of one sail with the reference's default wake (100 rows, not
        # rolled up) and default solver, freestream from the host, next points back to the host.
        dict(name="dynamic_default_wake", kind="dynamic", sails=1, panels=21, rows=100, far_ratio=5.0, rollup=False,
             source="host", wind=10.0, awa=60.0),
        # The benchmark's headline: four sails, 300 rows rolled up with every panel a vortex ring.
        dict(name="dynamic_row_all_near", kind="dynamic", sails=4, panels=64, rows=300, far_ratio=1e30, rollup=True,
             source="host", wind=12.0, awa=45.0),
        # An odd row with the default far field, its wind generated on the GPU.
        dict(name="dynamic_row_far_wind", kind="dynamic", sails=3, panels=61, rows=301, far_ratio=5.0, rollup=True,
             source="wind", wind=11.0, awa=70.0),
        # The large ship: eight sails at 128 panels with 400 rows, freestream already on the GPU.
        dict(name="dynamic_large_far", kind="dynamic", sails=8, panels=128, rows=400, far_ratio=5.0, rollup=True,
             source="device", wind=12.0, awa=45.0),
        # The standalone sum over panels in 64 bits, for a check of the 32-bit one at field points.
        dict(name="panel_sweep_fp64", kind="sweep", sails=2, panels=33, rows=150, targets=1501, far_ratio=5.0,
             precision="fp64", symmetry=0),
        # A parameter study over many uneven cases with short wakes: the solves are most of it.
        dict(name="batch_short_wakes", kind="batch", cases=64, rows_from=8, rows_to=24),
        # The same kind of study with the benchmark's long wakes, rolled up.
        dict(name="batch_long_wakes", kind="batch", cases=24, rows_from=50, rows_to=400),
        # The warm-start network over the panels of some 500 cases.
        dict(name="network_forward", kind="forward", rows=98_307),
        # An epoch of its training (8 steps of 16,384 rows).
        dict(name="network_train_epoch", kind="train", rows=131_072, batch_rows=16_384, lr=5e-4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["quasi_steady", "csm", "dynamic", "dynamic", "sweep", "batch", "forward", "train"])
    wind, awa = rng.uniform(5.0, 20.0), rng.uniform(20.0, 180.0)
    if kind == "quasi_steady":
        return dict(kind=kind, solver=rng.choice(["iterative", "linearized"]), sails=rng.randint(1, 6),
                    panels=rng.randint(16, 96), wind=wind, awa=awa)
    if kind == "csm":
        return dict(kind=kind, sails=rng.randint(1, 6), panels=rng.randint(16, 48), conditions=_log(rng, 5, 72),
                    wind=wind)
    if kind == "dynamic":
        far = rng.choice([5.0, 5.0, 1e30])
        # a wholly near wake of more than the headline's size would cost more than the largest case
        sails, panels, rows = rng.randint(1, 4 if far > 5.0 else 8), _log(rng, 16, 64 if far > 5.0 else 128), _log(
            rng, 20, 300 if far > 5.0 else 400)
        return dict(kind=kind, sails=sails, panels=panels, rows=rows, far_ratio=far, rollup=rng.random() < 0.75,
                    source=rng.choice(["host", "device", "wind"]), wind=wind, awa=awa)
    if kind == "sweep":
        return dict(kind=kind, sails=rng.randint(1, 4), panels=_log(rng, 8, 64), rows=_log(rng, 20, 150),
                    targets=_log(rng, 100, 3000), far_ratio=rng.choice([5.0, 1e30]),
                    precision=rng.choice(["fp64", "fp32", "kahan"]), symmetry=rng.choice([0, 0, 2]))
    if kind == "batch":
        rows_from = _log(rng, 5, 100)
        return dict(kind=kind, cases=_log(rng, 4, 32), rows_from=rows_from, rows_to=rows_from * rng.randint(2, 3))
    if kind == "forward":
        return dict(kind=kind, rows=_log(rng, 500, 131_072))
    n = _log(rng, 16_384, 131_072)
    return dict(kind=kind, rows=n, batch_rows=_log(rng, 2_048, 16_384), lr=5e-4)


# ---------------------------------------------------------------------------------------------------
# Inputs: made from the seed alone, the same for prepare() and exact()
# ---------------------------------------------------------------------------------------------------
class Row:
    """A row of sails, its wind and the state of its wake before the first pass."""

    def __init__(self, seed, sails, panels, rows, wind, awa, time_step=0.05):
        rng = np.random.default_rng(seed)
        panels = math.ceil(SPAN / (SPAN / panels))  # as the reference counts them: one more for some numbers
        self.sails, self.panels, self.rows, self.dt = sails, panels, rows, time_step
        self.N, self.Np = sails * panels, sails * (panels + 1)
        self.wind, self.awa = wind * rng.uniform(0.97, 1.03), math.radians(awa)
        self.phase = rng.uniform(0.0, 2.0 * math.pi)
        self.direction = np.array([math.cos(self.awa), math.sin(self.awa), 0.0])
        self.chord = CHORD * np.array([math.cos(self.awa - INCIDENCE), math.sin(self.awa - INCIDENCE), 0.0])
        z = np.linspace(0.0, SPAN, panels + 1)
        x = np.repeat(SPACING * np.arange(sails), panels + 1)
        self.span_points = np.stack([x, np.zeros(self.Np), np.tile(z, sails)], axis=1)
        mid = (np.arange(panels) + 0.5) / panels
        lift = np.sqrt(1.0 - (2.0 * mid - 1.0) ** 2)
        start = -0.5 * CHORD * wind * 0.6
        self.gamma = start * np.tile(lift, sails) * rng.uniform(0.95, 1.05, self.N)
        self.velocity = [self.speed(k) * self.direction for k in range(PERIOD)]
        u = self.velocity[0]
        self.history = [u + rng.normal(0.0, 0.2, (self.N, 3)) for _ in range(2)]
        self.age = rows + 7  # steps taken: the wake is full
        if rows == 0:
            return
        # the wake: shed along the wind from the trailing edge, rolling up with the distance
        s = np.arange(rows + 1, dtype=np.float64)[:, None, None]
        self.first_length = time_step * wind
        behind = np.where(s > 0, self.first_length * self.chord / CHORD + (s - 1.0) * time_step * u, 0.0)
        along = self.span_points[None, :, 2:3] / SPAN
        a, b, c = rng.uniform(0.5, 1.5, 3)
        roll = 0.01 * np.minimum(s, 150.0)
        side = np.array([-self.direction[1], self.direction[0], 0.0])
        up = np.array([0.0, 0.0, 1.0])
        shape = roll * (np.sin(math.pi * along * b + 0.1 * s * a) * up + np.cos(math.pi * along) * c * side)
        self.points = self.span_points[None] + behind + shape
        self.points_velocity = u + 0.05 * wind * np.sin(0.07 * s * c + 3.0 * along) * (side + 0.3 * up)
        g = start * np.tile(lift, sails) * (1.0 + 0.05 * np.sin(0.2 * np.arange(rows)[:, None] + self.phase))
        self.strengths = g * rng.uniform(0.98, 1.02, (rows, self.N))
        self.strengths[0] = self.gamma

    def speed(self, k):
        return self.wind * (1.0 + GUST * math.sin(2.0 * math.pi * k / PERIOD + self.phase))

    def state(self):
        """As Simulation.set_state takes it."""
        parts = [[self.age if self.rows else 0.0, 1.0, self.age]]
        if self.rows:
            parts += [self.points, self.points_velocity, self.strengths]
        return np.concatenate([np.asarray(p, dtype=np.float64).reshape(-1) for p in parts + [self.gamma] + self.history])

    def corners(self):
        """Vortex rings [rows * N, 4, 3] of the wake."""
        return _ring_corners(self.points, self.sails, self.panels)


def _ring_corners(points, sails, panels):
    a = np.array([i * (panels + 1) + j for i in range(sails) for j in range(panels)])
    p = points
    if isinstance(p, torch.Tensor):
        a = torch.as_tensor(a, device=p.device)
        return torch.stack([p[:-1][:, a], p[:-1][:, a + 1], p[1:][:, a + 1], p[1:][:, a]], dim=2).reshape(-1, 4, 3)
    return np.stack([p[:-1][:, a], p[:-1][:, a + 1], p[1:][:, a + 1], p[1:][:, a]], axis=2).reshape(-1, 4, 3)


def _row(case, seed):
    return Row(seed, case["sails"], case["panels"], case.get("rows", 0), case["wind"], case["awa"])


def _batch_rows(case, seed):
    """Sails, panels, wake length, wind angle and speed of each case drawn as the benchmark's uneven cases are."""
    r, out = random.Random(9_000 + case["cases"]), []
    for i in range(case["cases"]):
        rows = r.randint(case["rows_from"], case["rows_to"])
        out.append(Row(seed * 1_000 + i, r.randint(1, 6), r.randint(16, 96), rows, r.uniform(5.0, 20.0),
                       r.uniform(20.0, 180.0)))
    return out


def _sweep_inputs(case, seed):
    row = Row(seed, case["sails"], case["panels"], case["rows"], 12.0, 45.0)
    rng = np.random.default_rng(seed + 1)
    # field points around and behind the sails
    t = rng.uniform([-20.0, -20.0, 0.0], [SPACING * case["sails"] + 80.0, 120.0, 1.2 * SPAN], (case["targets"], 3))
    return row.corners(), row.strengths.reshape(-1), np.full(row.strengths.size, 0.1 * CHORD), t


def _csm_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["conditions"]
    directions = np.radians(np.linspace(30.0, 330.0, n) + rng.uniform(-2.0, 2.0, n))
    directions[np.abs(directions - math.pi) < 0.3] += 0.4  # sailing into the sails' own wakes is not asked for
    return case["wind"] * rng.uniform(0.9, 1.1, n), directions, rng.uniform(1.0, 3.0, n), rng.uniform(0.5, 1.0, n)


WIDTHS = [(256, 64), (256, 256), (256, 256), (256, 256)]  # the network's layers; 16 of the 64 inputs are used
FEATURES = 16


def _network(seed):
    rng, parts = np.random.default_rng(seed), []
    for i, (o, n) in enumerate(WIDTHS):
        fan = FEATURES if i == 0 else n
        w = rng.uniform(-1.0, 1.0, (o, n)) * math.sqrt(6.0 / fan)
        if i == 0:
            w[:, FEATURES:] = 0.0
        parts += [w.reshape(-1), rng.normal(0.0, 0.02, o)]
    parts.append(rng.uniform(-1.0, 1.0, 257) * math.sqrt(3.0 / 256))
    return np.concatenate(parts).astype(np.float32)


def _features(seed, rows):
    """The features' ranges as a batch makes them: lift coefficients, angles, positions, counts; and targets."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    x = torch.rand((rows, FEATURES), generator=g, device="cuda") * 2.0 - 1.0
    x[:, 8:] = x[:, 8:].abs()
    t = 0.02 * torch.sin(3.0 * x[:, 0] + x[:, 6]) * x[:, 4] + 0.002 * torch.randn(rows, generator=g, device="cuda")
    return x, t


# ---------------------------------------------------------------------------------------------------
# prepare() and run()
# ---------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("quasi_steady", "dynamic"):
        return _prepare_simulation(case, seed)
    if kind == "csm":
        from stormbird_gb300 import CompleteSailModel, setups

        model = CompleteSailModel(setups.complete_sail_model(case["sails"], case["panels"]))
        return {"kind": kind, "model": model, "conditions": _csm_inputs(case, seed)}
    if kind == "sweep":
        return {"kind": kind, "case": dict(case), "inputs": _sweep_inputs(case, seed)}
    if kind == "batch":
        return _prepare_batch(case, seed)
    from stormbird_gb300.warm_start import WarmStartNet

    net = WarmStartNet(FEATURES, seed=0)
    net.set_params(_network(seed))
    x, t = _features(seed, case["rows"])
    return {"kind": kind, "case": dict(case), "net": net, "x": x, "t": t}


def _prepare_simulation(case, seed):
    from stormbird_gb300 import Simulation, setups

    row = _row(case, seed)
    if case["kind"] == "dynamic":
        document = setups.wing_sail_row(case["sails"], case["panels"], case["rows"], time_step=row.dt,
                                        wind_speed=case["wind"], apparent_wind_angle_deg=case["awa"],
                                        far_field_ratio=case["far_ratio"],
                                        ratio_of_wake_affected=1.0 if case["rollup"] else 0.0)
    else:
        d = json.loads(setups.wing_sail_row(case["sails"], case["panels"], 1, apparent_wind_angle_deg=case["awa"]))
        solver = wake = None  # the defaults: Linearized, a core of a tenth of a panel
        if case["solver"] == "iterative":
            solver = setups.simple_iterative(1000, 0.1, 1e-8, 1e-7)
            wake = {"wake_length_factor": 100.0, "viscous_core_length": {"Absolute": 0.05 * CHORD}}
        document = setups.simulation(d["line_force_model"], False, solver, wake)
    sim = Simulation(document)
    sim.set_state(row.state())
    state = {"kind": case["kind"], "sim": sim, "dt": row.dt, "step": 0, "source": case.get("source", "host"),
             "rollup": case.get("rollup", False)}
    n = sim.nr_freestream_points
    if state["source"] == "wind":
        sim.set_wind("{}", json.dumps({
            "direction_coming_from": row.awa, "velocity_variation": {"Constant": row.wind},
            "parallel_gust": {"frequencies": [1.0 / (PERIOD * row.dt)], "amplitudes": [GUST * row.wind],
                              "phases": [row.phase]}}))
    else:
        state["freestream"] = [np.tile(u, (n, 1)) for u in row.velocity]
        if state["source"] == "device":
            state["freestream"] = [torch.from_numpy(f).cuda() for f in state["freestream"]]
    return state


def _prepare_batch(case, seed):
    from stormbird_gb300 import Batch, setups

    rows = _batch_rows(case, seed)
    batch = Batch([setups.wing_sail_row(r.sails, r.panels, r.rows, time_step=r.dt, wind_speed=r.first_length / r.dt,
                                        apparent_wind_angle_deg=math.degrees(r.awa), max_iterations=1000,
                                        residual_tolerance=1e-8, strength_tolerance=0.0) for r in rows])
    for i, r in enumerate(rows):
        batch.set_case_state(i, r.state())
    # two of the gust's steps, in turn: the freestream of all wake points is large
    fs = [np.concatenate([np.tile(r.velocity[k], (c["freestream_points"], 1)) for r, c in zip(rows, batch.cases)])
          for k in (0, 1)]
    largest = max(range(len(rows)), key=lambda i: rows[i].N * rows[i].rows)
    return {"kind": "batch", "batch": batch, "dt": rows[0].dt, "step": 0, "freestream": fs, "largest": largest}


def run(state):
    return _RUN[state["kind"]](state)


def _run_simulation(state):
    sim, k, dt = state["sim"], state["step"], state["dt"]
    state["step"] = k + 1
    if state["source"] == "wind":
        result = sim.do_step_wind(time=k * dt, time_step=dt, ship_velocity=0.0)
    elif state["source"] == "device":
        sim.do_step_device(time=k * dt, time_step=dt, freestream_device_ptr=state["freestream"][k % PERIOD].data_ptr())
        result = sim.read_output(k * dt)
    else:
        result = sim.do_step(time=k * dt, time_step=dt, freestream_velocity=state["freestream"][k % PERIOD])
    out = _result(result)
    if state["kind"] == "dynamic":
        if state["rollup"]:  # what the roll-up computed
            out["points"], out["strengths"], out["points_velocity"] = sim.wake_state()
        else:                # where the next step's freestream is asked for
            out["freestream_points"] = sim.get_freestream_velocity_points()
    return out


def _result(r):
    f, s = r.force_input, r.sectional_forces
    whole = ("circulatory", "viscous_lift", "sectional_drag", "added_mass", "gyroscopic", "total")
    return {
        "circulation": f.circulation_strength, "force_velocity": f.velocity, "angles": f.angles_of_attack,
        "acceleration": f.acceleration, "velocity": r.output_ctrl_points_velocity,
        "input_velocity": r.solver_input_ctrl_points_velocity, "control_points": r.ctrl_points,
        "sections": np.stack([getattr(s, w) for w in whole]),
        "forces": np.stack([[getattr(i, w) for w in whole] for i in r.integrated_forces]),
        "moments": np.stack([[getattr(i, w) for w in whole] for i in r.integrated_moments]),
        "force": r.force_sum, "moment": r.moment_sum, "iterations": r.iterations, "converged": r.converged,
    }


def _run_csm(state):
    return {"sails": state["model"].sweep_steady_state(*state["conditions"])}


def _run_sweep(state):
    from stormbird_gb300.simulation import panel_sweep

    c = state["case"]
    corners, strengths, cores, targets = state["inputs"]
    return {"velocity": panel_sweep(corners, strengths, cores, targets, far_field_ratio=c["far_ratio"],
                                    symmetry=c["symmetry"], precision=c["precision"])}


def _run_batch(state):
    b, k, dt = state["batch"], state["step"], state["dt"]
    state["step"] = k + 1
    b.do_step(time=k * dt, time_step=dt, freestream_velocity=state["freestream"][k % 2])
    s = b.summary()
    return {"circulation": b.circulation(), "forces": s[:, :6], "iterations": s[:, 7].astype(np.int64),
            "converged": s[:, 8].astype(np.int64), "largest_state": b.case_state(state["largest"])}


def _run_forward(state):
    return {"y": state["net"].forward(state["x"])}


def _run_train(state):
    from stormbird_gb300.warm_start import train

    c = state["case"]
    losses = train(state["net"], state["x"], state["t"], epochs=1, batch_rows=c["batch_rows"], lr=c["lr"])
    return {"losses": losses, "parameters": state["net"].get_params()}


_RUN = {"quasi_steady": _run_simulation, "dynamic": _run_simulation, "csm": _run_csm, "sweep": _run_sweep,
        "batch": _run_batch, "forward": _run_forward, "train": _run_train}


# ---------------------------------------------------------------------------------------------------
# work()
# ---------------------------------------------------------------------------------------------------
NEAR, FAR, HORSESHOE = 236, 34, 180  # operations of a pair: vortex ring, point doublet, three lines


def _step_work(N, Np, W, rollup, pair, iterations):
    points = (W + 1) * Np
    flops = N * W * N * pair + iterations * (4.0 * N * N + 300.0 * N)  # two components in a line's plane
    flops += points * W * N * pair if rollup else 0.0
    # wake points, their velocities and the strengths in and out, the freestream in, the result out
    return 8.0 * (points * (6 + 6 + 3) + 2 * W * N + 40 * N), flops


def work(case):
    kind = case["kind"]
    if kind == "dynamic":
        N, Np, W = case["sails"] * case["panels"], case["sails"] * (case["panels"] + 1), case["rows"]
        b, f = _step_work(N, Np, W, case["rollup"], NEAR if case["far_ratio"] > 5.0 else FAR, 17)
    elif kind == "quasi_steady":
        N = case["sails"] * case["panels"]
        f = HORSESHOE * N * N + (2.0 * N**3 / 3.0 if case["solver"] == "linearized" else 100 * (4.0 * N * N + 300.0 * N))
        b = 8.0 * 60 * N
    elif kind == "csm":
        N = case["sails"] * case["panels"]
        f, b = case["conditions"] * (HORSESHOE * N * N + 2.0 * N**3 / 3.0), 8.0 * case["conditions"] * 60 * N
    elif kind == "sweep":
        P = case["sails"] * case["panels"] * case["rows"]
        f = P * case["targets"] * (NEAR if case["far_ratio"] > 5.0 else FAR) * (2 if case["symmetry"] else 1)
        b = 8.0 * (P * 14 + 6 * case["targets"])
    elif kind == "batch":
        b = f = 0.0
        for r in _batch_rows(case, 0):
            x, y = _step_work(r.N, r.Np, r.rows, True, FAR, 90)
            b, f = b + x, f + y
    else:
        weights = sum(o * n for o, n in WIDTHS)
        f, b = 2.0 * case["rows"] * weights, 4.0 * case["rows"] * (FEATURES + 1) + 4.0 * weights
        if kind == "train":
            f, b = 3.0 * f, b + 4.0 * 6 * weights * (case["rows"] // case["batch_rows"])
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------------------
# exact(): the same results in 64 bits
# ---------------------------------------------------------------------------------------------------
def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    n = a.norm(dim=-1, keepdim=True)
    return torch.where(n > 0.0, a / n, torch.zeros_like(a))


def _line(a, b, x, core):
    """Velocity at x of vortex lines a -> b of unit strength with a viscous core [..., 3]."""
    r1, r2 = x - a, x - b
    s1, s2 = _dot(r1, r1), _dot(r2, r2)
    l1, l2 = s1.sqrt(), s2.sqrt()
    den = l1 * l2 * (l1 * l2 + _dot(r1, r2))
    d = b - a
    length = d.norm(dim=-1)
    t = _dot(r1, d) / length
    d2 = torch.where(t < 0.0, s1, torch.where(t > length, s2, s1 - t * t))
    k = d2 / (core**4 + d2 * d2).sqrt() * (l1 + l2) / (den * 4.0 * math.pi)
    k = torch.where(den.abs() > 1e-10, k, torch.zeros_like(k))
    return k[..., None] * torch.linalg.cross(r1, r2)


class Rings:
    """Vortex rings with a far field: point doublets beyond `ratio` panel sizes."""

    def __init__(self, corners, core, ratio):
        self.p, self.core = corners, core
        e = [(self.p[:, (k + 1) % 4] - self.p[:, k]).norm(dim=-1) for k in range(4)]
        s = 0.5 * sum(e)
        area = ((s - e[0]) * (s - e[1]) * (s - e[2]) * (s - e[3])).clamp_min(0.0).sqrt()
        self.centre, self.moment = self.p.mean(dim=1), area / (4.0 * math.pi)
        self.normal = _unit(torch.linalg.cross(self.p[:, 2] - self.p[:, 0], self.p[:, 3] - self.p[:, 1]))
        self.far2 = (ratio * torch.maximum(e[0], e[1])) ** 2

    def unit(self, x, i):
        """Velocity at x [n, 3] of the rings i [n], pair by pair."""
        return sum(_line(self.p[i, k], self.p[i, (k + 1) % 4], x, self.core) for k in range(4))

    def pairs(self, x):
        """Velocity of every ring at every x: [targets, rings, 3]."""
        e = x[:, None] - self.centre[None]
        d2 = _dot(e, e)
        near = d2 <= self.far2[None]
        if bool(near.all()):
            return sum(_line(self.p[None, :, k], self.p[None, :, (k + 1) % 4], x[:, None], self.core) for k in range(4))
        h = _dot(e, self.normal[None])
        u = (self.moment / (d2 * d2 * d2.sqrt()))[..., None] * (3.0 * h[..., None] * e - d2[..., None] * self.normal)
        j, i = near.nonzero(as_tuple=True)
        u[j, i] = self.unit(x[j], i)
        return u

    def velocity(self, x, strength, pairs_at_once=4_000_000):
        out = torch.empty_like(x)
        n = max(1, pairs_at_once // max(1, len(strength)))
        for k in range(0, len(x), n):
            out[k:k + n] = torch.einsum("tpc,p->tc", self.pairs(x[k:k + n]), strength)
        return out


def _stall(a):
    return 1.0 / (1.0 + torch.exp(-4.5951212 / STALL_RANGE * (a.abs() - STALL)))


def _cl_pre(a):
    return 2.0 * math.pi * torch.sin(a) * (1.0 - _stall(a))


def _cl_post(a):
    return torch.sin(2.0 * a) * _stall(a)


def _drag(a):
    s = _stall(a)
    cl = _cl_post(a) + _cl_pre(a)
    return CD_MIN * (1.0 - s) + s * torch.sin(a).abs() ** 1.6 + CDI * cl * cl


def _angle(chord, u):
    """From the chord to u in the horizontal plane (the spans are vertical)."""
    return torch.atan2(chord[..., 0] * u[..., 1] - chord[..., 1] * u[..., 0], _dot(chord[..., :2], u[..., :2]))


def _flat(u):
    return u * torch.tensor([1.0, 1.0, 0.0], dtype=u.dtype, device=u.device)


def _iterate(fs, fixed, matrix, chord, gamma, limit, damping, tolerance, strength_tolerance):
    """The damped iterations: circulation and velocity."""
    converged, n = False, 0
    while n < limit and not converged:
        n += 1
        u = _flat(fs + fixed + torch.einsum("ijc,j->ic", matrix, gamma))
        speed = u.norm(dim=-1)
        cl = _cl_pre(_angle(chord, u))
        estimate = -0.5 * CHORD * speed * cl
        residual = float((-2.0 * gamma / (CHORD * speed) - cl).abs().mean())
        change = estimate - gamma
        gamma = gamma + damping * change
        converged = residual < tolerance or (strength_tolerance > 0.0 and float(change.abs().max()) < strength_tolerance)
    return estimate, u


def _linearized(fs, matrix, chord):
    """The linearized solve with its viscous correction."""
    v = _flat(fs)
    un = _unit(v)
    up = torch.tensor([0.0, 0.0, 1.0], dtype=v.dtype, device=v.device).expand_as(v)
    normal = torch.linalg.cross(un, up)
    ut = _dot(v, un)
    a = -2.0 * math.pi * torch.einsum("ijc,ic->ij", matrix, normal) / ut[:, None]
    a += torch.diag(2.0 / (CHORD * ut))
    gamma = torch.linalg.solve(a, -2.0 * math.pi * torch.sin(_angle(chord, v)))
    velocity = fs + torch.einsum("ijc,j->ic", matrix, gamma)
    angle = _angle_about(chord, velocity)
    gamma = gamma * (_cl_pre(angle) / (2.0 * math.pi * torch.sin(angle)))
    return gamma, fs + torch.einsum("ijc,j->ic", matrix, gamma)


def _angle_about(chord, u):
    """The angle of attack of a velocity that keeps its part along the span: the angle between the two
    vectors, with the sign of the turn about the span."""
    c = (_dot(chord, u) / (_dot(chord, chord) * _dot(u, u)).sqrt()).clamp(-1.0, 1.0)
    a = torch.acos(c)
    turn = chord[..., 0] * u[..., 1] - chord[..., 1] * u[..., 0]
    return torch.where(turn > 0.0, a, -a)


def _forces(row, control, chord, gamma, u, acceleration, fs):
    n, ds = row.N, SPAN / row.panels
    span = torch.tensor([0.0, 0.0, ds], dtype=u.dtype, device=u.device).expand(n, 3)
    angle = _angle_about(chord, u)
    q = 0.5 * CHORD * ds * DENSITY * _dot(u, u)
    circulatory = DENSITY * gamma[:, None] * torch.linalg.cross(u, span)
    viscous = _unit(torch.linalg.cross(span, u)) * (_cl_post(angle) * q)[:, None]
    drag = _unit(u) * (_drag(angle) * q)[:, None]
    zero = torch.zeros_like(drag)
    sections = torch.stack([circulatory, viscous, drag, zero, zero, circulatory + viscous + drag])
    moments = torch.linalg.cross(control[None].expand_as(sections), sections)
    total = [s.reshape(6, row.sails, row.panels, 3).sum(2).transpose(0, 1) for s in (sections, moments)]
    return {"circulation": gamma, "force_velocity": u, "angles": angle, "acceleration": acceleration, "velocity": u,
            "input_velocity": fs, "control_points": control, "sections": sections, "forces": total[0],
            "moments": total[1], "force": total[0][:, 5].sum(0), "moment": total[1][:, 5].sum(0),
            "iterations": None, "converged": None}


def _control(row):
    p = row.span_points.reshape(row.sails, row.panels + 1, 3)
    return _t(0.5 * (p[:, 1:] + p[:, :-1])).reshape(-1, 3)


def _horseshoes(row, fs, control, length, core):
    """Unit velocity of each line with its two trailing vortices at each control point."""
    w = row.panels
    f = fs.reshape(row.sails, w, 3)
    at_points = torch.cat([f[:, :1], 0.5 * (f[:, 1:] + f[:, :-1]), f[:, -1:]], dim=1)
    p = _t(row.span_points).reshape(row.sails, w + 1, 3)
    tail = p + length * _unit(at_points)
    s, e = p[:, :-1].reshape(-1, 3), p[:, 1:].reshape(-1, 3)
    st, et = tail[:, :-1].reshape(-1, 3), tail[:, 1:].reshape(-1, 3)
    x = control[:, None]
    return _line(s[None], e[None], x, core) + _line(st[None], s[None], x, core) + _line(e[None], et[None], x, core)


def _exact_step(row, ratio, solver, rollup, velocities=True):
    """One step of a dynamic row from its loaded state; the velocities at the points only where asked for."""
    control, n, dt = _control(row), row.N, row.dt
    chord = _t(row.chord).expand(n, 3)
    u0 = _t(row.velocity[0])
    fs = u0.expand(n, 3)
    old, v = _t(row.points), _t(row.points_velocity)
    new = torch.empty_like(old)
    new[0] = _t(row.span_points)
    if row.rows > 1:
        new[2:] = old[1:-1] + dt * v[1:-1]
        new[1] = new[0] + row.first_length * chord[0] / CHORD
        new[-1] = new[-2] + 0.25 * CHORD * _unit(new[-2] - new[-3])
    g = _t(row.strengths)
    strengths = torch.cat([g[:1], g[:-1]])
    corners = _ring_corners(new, row.sails, row.panels)
    first, rest = Rings(corners[:n], 0.1 * CHORD, ratio), Rings(corners[n:], 0.1 * CHORD, ratio)
    live = strengths[1:].reshape(-1)
    fixed = rest.velocity(control, live)
    gamma, u = _iterate(fs, fixed, first.pairs(control), chord, _t(row.gamma), *solver)
    strengths[0] = gamma
    h0, h1 = (_t(h) for h in row.history)
    out = _forces(row, control, chord, gamma, u, (3.0 * u - 4.0 * h1 + h0) / (2.0 * dt), fs)
    out["points"], out["strengths"] = new.reshape(-1, 3), strengths.reshape(-1)
    if velocities:
        points = out["points"]
        vel = u0.expand(points.shape).clone()
        if rollup:  # every point but the last (the ratio of the wake that is affected, of its points less one)
            vel[:-1] += Rings(corners, 0.1 * CHORD, ratio).velocity(points[:-1], out["strengths"])
        out["points_velocity"] = vel
    return out, u


def exact(case, seed):
    kind = case["kind"]
    return {"quasi_steady": _exact_quasi_steady, "dynamic": _exact_dynamic, "csm": _exact_csm, "sweep": _exact_sweep,
            "batch": _exact_batch, "forward": _exact_forward, "train": _exact_train}[kind](case, seed)


def _exact_quasi_steady(case, seed):
    row = _row(case, seed)
    control, chord = _control(row), _t(row.chord).expand(row.N, 3)
    fs = _t(row.velocity[0]).expand(row.N, 3)
    core = 0.05 * CHORD if case["solver"] == "iterative" else 0.1 * SPAN / row.panels
    matrix = _horseshoes(row, fs, control, 100.0 * CHORD, core)
    if case["solver"] == "iterative":
        gamma, u = _iterate(fs, 0.0 * fs, matrix, chord, _t(row.gamma), 1000, 0.1, 1e-8, 1e-7)
    else:
        gamma, u = _linearized(fs, matrix, chord)
    h0, h1 = (_t(h) for h in row.history)
    return _forces(row, control, chord, gamma, u, (3.0 * u - 4.0 * h1 + h0) / (2.0 * row.dt), fs)


def _exact_dynamic(case, seed):
    row = _row(case, seed)
    pairs = (row.rows + 1) * row.Np * row.rows * row.N if case["rollup"] else 0
    if case["rows"] < 2 or row.N * row.N * row.rows > PAIRS_EXACT:
        return None
    out, _ = _exact_step(row, case["far_ratio"], (40, 0.05, 1e-4, 1e-6), case["rollup"], pairs <= PAIRS_EXACT)
    if not case["rollup"]:
        out["freestream_points"] = torch.cat([out["control_points"], out["points"]])
        for k in ("points", "strengths", "points_velocity"):
            out.pop(k, None)
    elif pairs > PAIRS_EXACT:
        out["points_velocity"] = None
    return out


def _exact_csm(case, seed):
    row, out = Row(0, case["sails"], case["panels"], 0, 10.0, 0.0), []
    rows, control = row.panels, _control(row)
    for v, d, ship, loading in zip(*_csm_inputs(case, seed)):
        up = (control[:, 2].clamp_min(0.0) / 10.0) ** (1.0 / 9.0)
        fs = v * up[:, None] * _t([math.cos(d), math.sin(d), 0.0]) + _t([ship, 0.0, 0.0])
        directions = torch.atan2(fs[:, 1], fs[:, 0]).reshape(row.sails, rows)
        chords = []
        for s in range(row.sails):  # the set points of a single-element wing sail, the last strip not measured
            a = float(directions[s, :-1].mean())
            deg = [math.radians(x) for x in (-180, -15, -10, 10, 15, 180)]
            top = math.radians(15.0)
            a -= loading * float(np.interp(a, deg, [-top, -top, 0.0, 0.0, top, top]))
            chords.append(_t([CHORD * math.cos(a), CHORD * math.sin(a), 0.0]).expand(rows, 3))
        chord = torch.cat(chords)
        matrix = _horseshoes(row, fs, control, 100.0 * CHORD, 0.1 * SPAN / rows)
        gamma, u = _linearized(fs, matrix, chord)
        f = _forces(row, control, chord, gamma, u, 0.0 * u, fs)
        out.append(torch.cat([f["forces"][:, 5], f["moments"][:, 5], torch.zeros_like(f["forces"][:, 5, :1])], dim=1))
    return {"sails": torch.stack(out)}


def _exact_sweep(case, seed):
    corners, strengths, cores, targets = _sweep_inputs(case, seed)
    rings, x, g = Rings(_t(corners), float(cores[0]), case["far_ratio"]), _t(targets), _t(strengths)
    u = rings.velocity(x, g)
    if case["symmetry"]:  # the mirror image in the plane y = 0
        flip = _t([1.0, -1.0, 1.0])
        u = u + flip * rings.velocity(x * flip, g)
    return {"velocity": u}


def _exact_batch(case, seed):
    rows = _batch_rows(case, seed)
    if sum(r.N * r.N * r.rows for r in rows) > PAIRS_EXACT:
        return None
    solver = (1000, 0.05, 1e-8, 0.0)
    largest = max(range(len(rows)), key=lambda i: rows[i].N * rows[i].rows)
    gamma, forces, state = [], [], None
    for i, row in enumerate(rows):
        follow = i == largest and (row.rows + 1) * row.Np * row.rows * row.N <= PAIRS_EXACT
        o, u = _exact_step(row, 5.0, solver, True, velocities=follow)
        gamma.append(o["circulation"])
        forces.append(torch.cat([o["force"], o["moment"]]))
        if follow:
            head = _t([row.age + 1, 1.0, row.age + 1])
            parts = [o["points"], o["points_velocity"], o["strengths"], o["circulation"], _t(row.history[1]), u]
            state = torch.cat([head] + [p.reshape(-1) for p in parts])
    return {"circulation": torch.cat(gamma), "forces": torch.stack(forces), "iterations": None, "converged": None,
            "largest_state": state}


def _layers(flat):
    out, at = [], 0
    for o, n in WIDTHS:
        out.append([flat[at:at + o * n].reshape(o, n), flat[at + o * n:at + o * n + o]])
        at += o * n + o
    return out, flat[at:at + 256], flat[at + 256]


def _net_forward(flat, x):
    layers, w, b = _layers(flat)
    h = torch.cat([x, x.new_zeros((len(x), 64 - FEATURES))], dim=1)
    for weight, bias in layers:
        h = torch.nn.functional.gelu(h @ weight.T + bias)
    return h @ w + b


def _exact_forward(case, seed):
    x, _ = _features(seed, case["rows"])
    flat = _t(_network(seed))
    return {"y": torch.cat([_net_forward(flat, part) for part in x.double().split(16_384)])}


def _exact_train(case, seed):
    x, t = _features(seed, case["rows"])
    p = _t(_network(seed)).requires_grad_(True)
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    g = torch.Generator(device=x.device)
    g.manual_seed(0)
    perm = torch.randperm(len(x), device=x.device, generator=g)
    x, t, size = x[perm].double(), t[perm].double(), min(case["batch_rows"], len(x))
    for k, s in enumerate(range(0, len(x) - size + 1, size), start=1):
        loss = ((_net_forward(p, x[s:s + size]) - t[s:s + size]) ** 2).mean()
        (grad,) = torch.autograd.grad(loss, p)
        losses.append(float(loss))
        with torch.no_grad():
            m = 0.9 * m + 0.1 * grad
            v = 0.999 * v + 0.001 * grad * grad
            p -= case["lr"] * math.sqrt(1.0 - 0.999**k) / (1.0 - 0.9**k) * m / (v.sqrt() + 1e-8)
    return {"losses": [sum(losses) / len(losses)], "parameters": p.detach()}

"""Performance cases of the beam time step, run through the public Python API.

A pass is what a coupled simulation does once per time step: hand the loads
(and the prescribed root motion or the controls) of this step to the models,
advance them one step, and read back the motion (q and v of every node) with
the Newton outcome of every model.  The load records are periodic in the step
number, so that a run of any length stays in the regime it starts in.

Families (the sizes are those of this repository's workloads, tests and
benchmark, or generic ones between them):

* cantilever -- clamped beams of 5 to 21 nodes, nodes + 2 Gauss points,
  tapered sections with couplings, distributed lateral loads: one model alone,
  or an ensemble of designs under load cases of their own (parameter studies,
  design load cases, a served stream);
* rotor -- three 60 m blades whose roots follow a prescribed rotation, under
  gravity and distributed loads (a blade-resolved rotor on a given shaft);
* drivetrain -- the same blades on a hub that turns on a revolute joint with a
  generator torque;
* platform -- a floating platform with three mooring lines, no beams;
* turbine -- tower, nacelle, drive train, hub and three pitched blades in one
  coupled system (aero-elastic simulation of a whole machine).

The FP32 form takes one FP64-residual correction after convergence and gives
positions only, as in the benchmark's end-to-end leg: the Newton iterates of
that form are its own, so it is judged on the state it ends in.

``transfer`` says where the caller's arrays live: "host" (a CPU aerodynamics
code, pinned buffers), "device" (a GPU flow solver), or "single" (the
per-model calls, the way a script steps one model).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from openturbine_b200.model import (BeamSection, CreateTrapezoidalQuadrature, GaussLegendreQuadrature,
                                    GenerateGLLPoints, Model, QuaternionCompose, RotateVectorByQuaternion,
                                    RotationVectorToQuaternion, StepParameters)
from openturbine_b200.runtime import LOAD_NODE_FX, LOAD_STATE_F, Context

STEP = 0.01          # time step of every case, s
RECORD = 50          # steps after which the load record repeats
TURN = 786           # steps of one rotor revolution (0.8 rad/s)
DESIGNS = 48         # most distinct designs of an ensemble; its models share them
STIFFNESS = np.array([1e9, 4e8, 4e8, 1e7, 2e7, 2e7])
MASS = np.array([10., 10., 10., 2., 1., 1.])
ITERATIONS = 4       # Newton iterations of an ordinary step, for work()


# ---- the cases ---------------------------------------------------------------------
def listed():
    return [
        # a script stepping one small beam: latency of the calls and of one step
        {"name": "cantilever_1", "family": "cantilever", "models": 1, "nodes_lo": 5, "nodes_hi": 5,
         "points_extra": 2, "fp32": False, "transfer": "single"},
        # a rotor on a prescribed shaft, alone: three blades that share a Newton loop
        {"name": "rotor_1", "family": "rotor", "models": 1, "nodes": 11, "stations": 21, "transfer": "host"},
        # a moored floater, alone: the smallest coupled system
        {"name": "platform_1", "family": "platform", "models": 1, "transfer": "single"},
        # one whole turbine, alone: an aero-elastic simulation that wants real time
        {"name": "turbine_1", "family": "turbine", "models": 1, "blade_nodes": 11, "tower_nodes": 11,
         "transfer": "single"},
        # a small study that leaves most of the GPU idle
        {"name": "beams_64", "family": "cantilever", "models": 64, "nodes_lo": 5, "nodes_hi": 21,
         "points_extra": 2, "fp32": False, "transfer": "host"},
        # the benchmark's ensemble of uneven beams, loads from a host code
        {"name": "beams_4096", "family": "cantilever", "models": 4096, "nodes_lo": 5, "nodes_hi": 21,
         "points_extra": 2, "fp32": False, "transfer": "host"},
        # the same in the FP32 form with one FP64-residual correction after convergence
        {"name": "beams_4096_fp32", "family": "cantilever", "models": 4096, "nodes_lo": 5, "nodes_hi": 21,
         "points_extra": 2, "fp32": True, "transfer": "host"},
        # many short beams (the order-4 element of the tests), loads from a GPU code
        {"name": "short_8192", "family": "cantilever", "models": 8192, "nodes_lo": 5, "nodes_hi": 8,
         "points_extra": 2, "fp32": False, "transfer": "device"},
        # the finest beams: one fills an SM's shared memory
        {"name": "long_1184", "family": "cantilever", "models": 1184, "nodes_lo": 19, "nodes_hi": 21,
         "points_extra": 2, "fp32": False, "transfer": "device"},
        # rotors of a design study, all on prescribed shafts
        {"name": "rotors_256", "family": "rotor", "models": 256, "nodes": 11, "stations": 21,
         "transfer": "host"},
        # rotors that turn freely against a generator torque
        {"name": "drivetrains_100", "family": "drivetrain", "models": 100, "nodes": 9, "stations": 13,
         "transfer": "host"},
        # a farm or a design-load-case table of whole turbines
        {"name": "turbines_148", "family": "turbine", "models": 148, "blade_nodes": 11, "tower_nodes": 11,
         "transfer": "host"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["cantilever"] * 5 + ["rotor", "rotor", "drivetrain", "platform", "turbine"])
    if family == "cantilever":
        lo = rng.randint(5, 21)
        hi = rng.choice([lo, rng.randint(lo, 21), 21])
        cap = 1184 if hi + lo > 36 else 2048 if hi + lo > 28 else 4096
        models = _log_int(rng, 1, cap)
        return {"family": family, "models": models, "nodes_lo": lo, "nodes_hi": hi,
                "points_extra": rng.randint(1, 4), "fp32": rng.random() < 0.25,
                "transfer": "single" if models == 1 else rng.choice(["host", "device"])}
    if family == "platform":
        return {"family": family, "models": _log_int(rng, 1, 2000), "transfer": "host"}
    if family == "turbine":
        return {"family": family, "models": _log_int(rng, 1, 148), "blade_nodes": rng.randint(7, 11),
                "tower_nodes": rng.randint(6, 11), "transfer": rng.choice(["host", "device"])}
    return {"family": family, "models": _log_int(rng, 1, 256 if family == "rotor" else 100),
            "nodes": rng.randint(6, 13 if family == "rotor" else 11), "stations": rng.randint(9, 23),
            "transfer": rng.choice(["host", "device"])}


# ---- inputs ------------------------------------------------------------------------
def _params(case):
    if case["family"] == "cantilever":
        if case["fp32"]:
            return StepParameters(True, 10, STEP, 0.9, a_tol=1e-7, r_tol=1e-3, precision=1, refine_iters=1)
        return StepParameters(True, 10, STEP, 0.9, a_tol=1e-7, r_tol=1e-3)
    if case["family"] == "turbine":
        return StepParameters(True, 6, STEP, 0.0, a_tol=1e-6, r_tol=1e-4)
    if case["family"] == "platform":
        return StepParameters(True, 5, STEP, 0.0)
    return StepParameters(True, 10, STEP, 0.9)


def _coupled_matrices(rng, diagonals):
    """Symmetric positive definite 6x6 matrices with the given diagonals times
    (1 + U(-0.05, 0.05)) and couplings of at most 5 % (diagonally dominant)."""
    d = diagonals * (1. + rng.uniform(-0.05, 0.05, diagonals.shape))
    r = np.sqrt(d)
    c = rng.uniform(-0.05, 0.05, d.shape + (6,))
    c = np.triu(c, 1)
    c = c + np.swapaxes(c, -1, -2) + np.eye(6)
    return c * r[..., :, None] * r[..., None, :]


def _blade_design(rng, nodes, points_or_grid, length, gauss, stations=21):
    """Geometry and sections of one straight tapered beam along x."""
    grid = np.linspace(0., 1., stations)
    taper = 1. - 0.9 * grid
    return {"nodes": nodes, "length": length, "s": (np.array(GenerateGLLPoints(nodes - 1)) + 1.) / 2.,
            "grid": grid, "mass": _coupled_matrices(rng, taper[:, None] * MASS),
            "stiffness": _coupled_matrices(rng, taper[:, None] * STIFFNESS),
            "quadrature": (GaussLegendreQuadrature(points_or_grid) if gauss
                           else CreateTrapezoidalQuadrature(list(points_or_grid)))}


def _add_blade(m, b, offset=0.):
    ids = [m.AddNode().SetElemLocation(float(s)).SetPosition(offset + b["length"] * float(s), 0., 0., 1., 0., 0., 0.)
           .Build() for s in b["s"]]
    e = m.AddBeamElement(ids, [BeamSection(float(g), M, K) for g, M, K in
                               zip(b["grid"], b["mass"], b["stiffness"])], b["quadrature"])
    return ids, e


def _load_shape(rng, b, count):
    """Nodal load amplitudes [count][nodes][6] of `count` load cases of one
    beam: lateral forces growing towards the tip and a little torsion, sized
    so that held statically they would bend the tip by 0.2 to 2 % of the
    length."""
    n, length = b["nodes"], b["length"]
    w = b["s"] * np.gradient(b["s"])
    w = w / w.sum()
    total = rng.uniform(0.002, 0.02, count) * 3. * 2e7 * 0.5 / length ** 2
    angle = rng.uniform(0., 2. * math.pi, count)
    amp = np.zeros((count, n, 6))
    amp[:, :, 1] = (total * np.cos(angle))[:, None] * w
    amp[:, :, 2] = (total * np.sin(angle))[:, None] * w
    amp[:, :, 3] = 0.01 * length * total[:, None] * w
    return amp


def _cantilevers(case, seed):
    """Designs and load cases of an ensemble: node counts, arrays and the
    design of each model."""
    rng = np.random.default_rng([seed, 1])
    count = case["models"]
    lo, hi = case["nodes_lo"], case["nodes_hi"]
    designs = []
    nd = min(count, DESIGNS)
    for i in range(nd):
        n = lo + i % (hi - lo + 1) if nd > hi - lo else int(rng.integers(lo, hi + 1))
        length = float(rng.uniform(5., 100.)) if count > 1 else 10.
        designs.append(_blade_design(rng, n, n + case["points_extra"], length, True))
    which = rng.permutation(np.arange(count) % nd)
    amps = [_load_shape(rng, d, int((which == i).sum())) for i, d in enumerate(designs)]
    at = np.zeros(nd, dtype=int)
    amp = []
    for w in which:
        amp.append(amps[w][at[w]])
        at[w] += 1
    return designs, which, amp, rng.integers(1, 3, count), rng.uniform(-0.6, 0.6, count)


def _rotor_model(case, design, torque):
    """Three blades about z, spinning; their roots prescribed, or jointed to a
    hub on a revolute joint (torque in N m) from a fixed shaft base."""
    omega = 2. * math.pi / (TURN * STEP)
    m = Model()
    m.SetGravity(0., 0., -9.81)
    roots = []
    for k, b in enumerate(design):
        ids, e = _add_blade(m, b, 2.)
        m.RotateBeamAboutPoint(e, RotationVectorToQuaternion([0., 0., 2. * math.pi * k / 3.]), [0., 0., 0.])
        m.SetBeamVelocityAboutPoint(e, [0., 0., 0., 0., 0., omega], [0., 0., 0.])
        roots.append(ids[0])
    if torque is None:
        for r in roots:
            m.AddPrescribedBC(r)
    else:
        spin = [0., 0., 0., 0., 0., omega]
        hub = m.AddNode().SetPosition(0., 0., 0., 1., 0., 0., 0.).SetVelocity(*spin).Build()
        ground = m.AddNode().SetPosition(0., 0., -1., 1., 0., 0., 0.).Build()
        m.AddFixedBC(ground)
        m.AddRevoluteJointConstraint([ground, hub], [0., 0., 1.], np.zeros(1))
        for r in roots:
            m.AddRigidJointConstraint([hub, r])
    return m


def _rotors(case, seed):
    rng = np.random.default_rng([seed, 2])
    nd = min(case["models"], 8)
    grid = np.linspace(0., 1., case["stations"])
    designs = [[_blade_design(rng, case["nodes"], grid, 60., False, case["stations"]) for _ in range(3)]
               for _ in range(nd)]
    which = np.arange(case["models"]) % nd
    amp = [np.concatenate([_load_shape(rng, b, 1)[0] for b in designs[w]]) for w in which]
    return designs, which, amp, rng.integers(1, 3, case["models"]), rng.uniform(-0.6, 0.6, case["models"])


def _root_motion(model, step):
    """Prescribed displacement of every blade root at the end of step `step`."""
    q = RotationVectorToQuaternion([0., 0., 2. * math.pi * (step + 1) / TURN])
    out = []
    for c in model.constraints_:
        x0 = model.GetNode(c.node_ids[1]).x0[:3]
        xr = RotateVectorByQuaternion(q, x0)
        out.append([xr[0] - x0[0], xr[1] - x0[1], xr[2] - x0[2], *q])
    return out


def _platform_model(rng):
    m = Model()
    m.SetGravity(0., 0., -9.8124)
    mass = 1.419625e7 * rng.uniform(0.95, 1.05)
    node = m.AddNode().SetPosition(0., 0., -7.53, 1., 0., 0., 0.).Build()
    m.AddMassElement(node, np.diag([mass] * 3 + [1.2898e10, 1.2851e10, 1.4189e10]))
    spring = 48.9e3 * rng.uniform(0.95, 1.05)
    for k in range(3):
        c, s = math.cos(math.pi + 2. * math.pi * k / 3.), math.sin(math.pi + 2. * math.pi * k / 3.)
        fair = m.AddNode().SetPosition(40.87 * c, 40.87 * s, -14., 1., 0., 0., 0.).Build()
        anchor = m.AddNode().SetPosition(105.47 * c, 105.47 * s, -58.4, 1., 0., 0., 0.).Build()
        m.AddFixedBC3DOFs(anchor)
        m.AddRigidJoint6DOFsTo3DOFs([node, fair])
        m.AddSpringElement(fair, anchor, spring, 55.432)
    stretch = math.hypot(105.47 - 40.87, 58.4 - 14.)
    hold = 9.8124 * mass + 3. * spring * (1. - 55.432 / stretch) * (58.4 - 14.)
    return m, hold


def _tube(diameter, wall):
    E, G, rho = 200e9, 79.3e9, 7850.
    ro, ri = diameter / 2., diameter / 2. - wall
    A, I = math.pi * (ro ** 2 - ri ** 2), math.pi * (ro ** 4 - ri ** 4) / 4.
    return (np.diag([rho * A] * 3 + [rho * 2. * I, rho * I, rho * I]),
            np.diag([E * A, 0.53 * G * A, 0.53 * G * A, G * 2. * I, E * I, E * I]))


def _turbine_model(case, rng):
    """A three-bladed machine of the 15 MW class: tower along z, yaw bearing,
    shaft base, azimuth, hub and apex nodes; yaw and pitch as rotation
    controls, the shaft as a revolute joint.  Returns the model, its blade
    element ids and the constraint ids (base, yaw, torque, pitches)."""
    m = Model()
    m.SetGravity(0., 0., -9.81)
    speed, tilt, hub_radius, overhang, rise = 0.6, math.radians(6.), 4., 12., 5.6
    to_z = RotationVectorToQuaternion([0., -math.pi / 2., 0.])
    q_tilt = RotationVectorToQuaternion([0., tilt, 0.])
    grid = list(np.linspace(0., 1., 26))
    quad = CreateTrapezoidalQuadrature(grid)

    def beam(nodes, length, mass, stiffness, g):
        ids = [m.AddNode().SetElemLocation((x + 1.) / 2.)
               .SetPosition(length * (x + 1.) / 2., 0., 0., 1., 0., 0., 0.).Build()
               for x in GenerateGLLPoints(nodes - 1)]
        return ids, m.AddBeamElement(ids, [BeamSection(s, M, K) for s, M, K in zip(g, mass, stiffness)],
                                     CreateTrapezoidalQuadrature(g))

    blades = []
    for _ in range(3):
        t = np.array(grid)
        scale = (1. - 0.95 * t) ** 2
        K = scale[:, None] * np.array([1.5e10, 8e8, 8e8, 1e10, 3e10, 4e10])
        M = (1. - 0.95 * t)[:, None] * np.array([900., 900., 900., 3000., 1200., 1800.])
        blades.append(beam(case["blade_nodes"], 117., _coupled_matrices(rng, M), _coupled_matrices(rng, K), grid))
    tgrid = list(np.linspace(0., 1., 20))
    tubes = [_tube(10. - 3.5 * s, 0.045 - 0.02 * s) for s in tgrid]
    tower_ids, tower = beam(case["tower_nodes"], 130., [a for a, _ in tubes], [k for _, k in tubes], tgrid)
    m.RotateBeamAboutPoint(tower, to_z, [0., 0., 0.])
    top = m.GetNode(tower_ids[-1]).x0[:3]
    apex = [top[0] - overhang, top[1], top[2] + rise]
    shaft = overhang / math.cos(tilt)
    hub = m.AddNode().SetPosition(0., 0., 0., 1., 0., 0., 0.).Build()
    azimuth = m.AddNode().SetPosition(shaft, 0., 0., 1., 0., 0., 0.).Build()
    base = m.AddNode().SetPosition(shaft, 0., 0., 1., 0., 0., 0.).Build()
    yaw = m.AddNode().SetPosition(*top, 1., 0., 0., 0.).Build()
    tips = [m.AddNode().SetPosition(0., 0., 0., 1., 0., 0., 0.).Build() for _ in blades]
    rotor = [hub, azimuth, base]
    for k, (ids, _) in enumerate(blades):
        for n in ids:
            m.GetNode(n).RotateAboutPoint(to_z, [0., 0., 0.])
            m.GetNode(n).Translate([0., 0., hub_radius])
        for n in ids + [tips[k]]:
            m.GetNode(n).RotateAboutPoint(RotationVectorToQuaternion([2. * math.pi * k / 3., 0., 0.]), [0., 0., 0.])
        rotor += ids + [tips[k]]
    for n in rotor:
        m.GetNode(n).RotateAboutPoint(q_tilt, [0., 0., 0.])
        m.GetNode(n).Translate(apex)
    m.AddMassElement(yaw, np.diag([6.5e5, 6.5e5, 6.5e5, 1.2e7, 1.0e7, 1.0e7]))
    m.AddMassElement(hub, np.diag([1.9e5, 1.9e5, 1.9e5, 1.4e6, 9.7e5, 9.7e5]))
    pitch = []
    for k, (ids, _) in enumerate(blades):
        a, r = m.GetNode(tips[k]).x0, m.GetNode(ids[0]).x0
        pitch.append(m.AddRotationControl([ids[0], tips[k]], [r[i] - a[i] for i in range(3)], np.zeros(1)))
        m.AddRigidJointConstraint([hub, tips[k]])
    m.AddRigidJointConstraint([azimuth, hub])
    torque = m.AddRevoluteJointConstraint([base, azimuth], [-math.cos(tilt), 0., math.sin(tilt)], np.zeros(1))
    m.AddRigidJointConstraint([yaw, base])
    yaw_c = m.AddRotationControl([tower_ids[-1], yaw], [0., 0., 1.], np.zeros(1))
    ground = m.AddPrescribedBC(tower_ids[0])
    h, s = np.array(m.GetNode(hub).x0[:3]), np.array(m.GetNode(base).x0[:3])
    axis = (h - s) / np.linalg.norm(h - s)
    for n in [hub, azimuth] + [x for k, (ids, _) in enumerate(blades) for x in ids + [tips[k]]]:
        m.GetNode(n).SetVelocityAboutPoint([0., 0., 0., *(speed * axis)], list(h))
    return m, blades, {"base": ground, "yaw": yaw_c, "torque": torque, "pitch": pitch}


# ---- a state: the models and the caller's arrays -------------------------------------
def _record(amp, freq, phase):
    """Load record [RECORD][rows][6]: amplitude times cos of the model's own
    frequency (2 or 4 Hz) and phase; amp: one [rows][6] array per model."""
    k = np.arange(RECORD)
    wave = np.cos(2. * math.pi * np.outer(k, freq) / RECORD + phase)          # [RECORD][models]
    rows = torch.from_numpy(np.repeat(wave, [a.shape[0] for a in amp], axis=1))
    return rows[:, :, None] * torch.from_numpy(np.concatenate(amp))[None]


def _place(case, t):
    t = t.contiguous()
    return t.cuda() if case["transfer"] == "device" else t.pin_memory()


def prepare(case, seed):
    ctx = Context(0)
    ctx.set_cuda_graph(case["transfer"] != "single")
    st = {"case": case, "ctx": ctx, "params": _params(case), "step": 0, "motion": None,
          "load_kind": LOAD_NODE_FX}
    family = case["family"]
    if family == "cantilever":
        designs, which, amp, freq, phase = _cantilevers(case, seed)
        templates = []
        for d in designs:
            m = Model()
            ids, _ = _add_blade(m, d)
            m.AddFixedBC(ids[0])
            templates.append(m)
    elif family in ("rotor", "drivetrain"):
        designs, which, amp, freq, phase = _rotors(case, seed)
        templates = [_rotor_model(case, d, None if family == "rotor" else 0.) for d in designs]
        if family == "rotor":
            turn = torch.tensor([_root_motion(templates[0], k) for k in range(TURN)], dtype=torch.float64)
            st["motion"] = _place(case, turn.repeat(1, case["models"], 1))
        else:  # constraint order: shaft base, revolute joint (torque), rigid joints
            u = torch.zeros(RECORD, case["models"], 5, 7, dtype=torch.float64)
            u[..., 3] = 1.
            t = torch.from_numpy(1e4 * np.cos(2. * math.pi * np.outer(np.arange(RECORD), freq) / RECORD + phase))
            u[:, :, 1, 0] = t
            st["motion"] = _place(case, u.reshape(RECORD, -1, 7))
    else:
        rng = np.random.default_rng([seed, 3])
        count = case["models"]
        nd = min(count, 4)
        which = np.arange(count) % nd
        freq, phase = rng.integers(1, 3, count), rng.uniform(-0.6, 0.6, count)
        st["load_kind"] = LOAD_STATE_F
        if family == "platform":
            built = [_platform_model(rng) for _ in range(nd)]
            templates = [m for m, _ in built]
            amp, mean = [], []
            for w in which:
                a, b = np.zeros((templates[0].NumNodes(), 6)), np.zeros((templates[0].NumNodes(), 6))
                a[0] = rng.uniform(0.5, 1., 6) * [1e6, 1e6, 9e5, 5e5, 1e6, 2e7]
                b[0, 2] = built[w][1]
                amp.append(a)
                mean.append(b)
        else:
            built = [_turbine_model(case, rng) for _ in range(nd)]
            templates = [m for m, _, _ in built]
            amp, mean = [], []
            for w in which:
                nn = templates[w].NumNodes()
                a, b = np.zeros((nn, 6)), np.zeros((nn, 6))
                for ids, _ in built[w][1]:
                    force = rng.uniform(0.7, 1.)
                    for n in ids:  # thrust and drive along the blades, pulsating
                        b[n, 0] = 6e4 * force
                        a[n, 0:3] = 6e3 * rng.uniform(0.5, 1., 3)
                amp.append(a)
                mean.append(b)
            con = built[0][2]
            u = torch.zeros(RECORD, count, templates[0].NumConstraints(), 7, dtype=torch.float64)
            u[..., 3] = 1.
            k = np.outer(np.arange(RECORD), np.ones(count))
            wave = torch.from_numpy(np.cos(2. * math.pi * k * freq / RECORD + phase))
            for c in con["pitch"]:
                u[:, :, c, 0] = 2e-4 * (wave - wave[0])
                u[:, :, c, 3] = 0.
            u[:, :, con["yaw"], 3] = 0.
            u[:, :, con["torque"], 0] = 1e6 * wave
            u[:, :, con["torque"], 3] = 0.
            st["motion"] = _place(case, u.reshape(RECORD, -1, 7))
            st["controls"] = [con["torque"], *con["pitch"]]
    made = [ctx.create_model(m) for m in templates]
    ids, used = [], set()
    for w in which:
        ids.append(made[w] if w not in used else ctx.clone_model(made[w]))
        used.add(w)
    st["ids"] = ctx.batch_ids(ids)
    loads = _record(amp, freq, phase)
    if st["load_kind"] == LOAD_STATE_F:
        loads = loads + torch.from_numpy(np.concatenate(mean))[None]
    rows = sum(ctx.info(i).num_nodes for i in ids)
    if case["transfer"] == "single":
        st["loads"] = loads.numpy()
    else:
        st["loads"] = _place(case, loads)
        st["q"] = _place(case, torch.zeros(rows, 7, dtype=torch.float64))
        st["v"] = _place(case, torch.zeros(rows, 6, dtype=torch.float64))
    return st


def run(st):
    """One time step of every model."""
    ctx, ids, k = st["ctx"], st["ids"], st["step"]
    st["step"] = k + 1
    loads = st["loads"][k % RECORD]
    motion = st["motion"]
    if motion is not None:
        motion = motion[k % motion.shape[0]]
    if st["case"]["transfer"] == "single":
        i = int(ids[0])
        if st["load_kind"] == LOAD_NODE_FX:
            ctx.set_node_fx(i, loads)
        else:
            ctx.set_state_f(i, loads)
        for c in st.get("controls", ()):
            ctx.set_control(i, c, float(motion[c, 0]))
        status, iters = ctx.step(ids, st["params"])
        if st["params"].precision:
            return {"q": ctx.state(i, "q"), "status": status}
        return {"q": ctx.state(i, "q"), "v": ctx.state(i, "v"), "status": status, "iters": iters}
    on_device = st["case"]["transfer"] == "device"
    ctx.set_loads_batch(ids, st["load_kind"], loads.data_ptr(), on_device)
    if motion is not None:
        ctx.set_prescribed_batch(ids, motion.data_ptr(), on_device)
    status, iters = ctx.step(ids, st["params"])
    ctx.get_state_batch(ids, "q", st["q"].data_ptr(), on_device)
    if st["params"].precision:
        return {"q": st["q"], "status": status}
    ctx.get_state_batch(ids, "v", st["v"].data_ptr(), on_device)
    return {"q": st["q"], "v": st["v"], "status": status, "iters": iters}


def _beam_work(n, q, models):
    """Bytes and operations of one beam's step: its constants and state read
    once, its state written once; quadrature physics, the two-stage integration
    of the node-pair blocks, assembly and the LU of the free block, per Newton
    iteration."""
    consts = 3 * q * n + 4 * q + 79 * q + 7 * n + 6 * n
    state = (7 + 6 * 3) * n
    dof = 6 * (n - 1)
    flops = q * (3112 + 55 * n) + 144 * n * n * q + 200 * n * q + 2. * dof ** 3 / 3. + 2. * dof ** 2
    return models * 8. * (consts + 2 * state + 13 * n), models * ITERATIONS * flops


def work(case):
    count = case["models"]
    if case["family"] == "cantilever":
        lo, hi = case["nodes_lo"], case["nodes_hi"]
        each = [_beam_work(n, n + case["points_extra"], count / (hi - lo + 1)) for n in range(lo, hi + 1)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    if case["family"] == "platform":
        dof = 6 + 18 + 18
        return {"bytes": count * 8. * 7 * 45, "flops": count * ITERATIONS * (2. * dof ** 3 / 3. + 500.)}
    if case["family"] in ("rotor", "drivetrain"):
        b, f = _beam_work(case["nodes"], case["stations"], 3 * count)
        return {"bytes": b, "flops": f}
    b1, f1 = _beam_work(case["blade_nodes"], 26, 3 * count)
    b2, f2 = _beam_work(case["tower_nodes"], 20, count)
    return {"bytes": b1 + b2, "flops": f1 + f2 + count * ITERATIONS * 2. * 137. ** 3 / 3.}


# ---- the same step in plain torch, 64 bits -------------------------------------------
def _tilde(v):
    z = torch.zeros_like(v[..., 0])
    return torch.stack([z, -v[..., 2], v[..., 1], v[..., 2], z, -v[..., 0], -v[..., 1], v[..., 0], z],
                       -1).reshape(*v.shape[:-1], 3, 3)


def _rot(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), w * w - x * x + y * y - z * z, 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), w * w - x * x - y * y + z * z],
                       -1).reshape(*q.shape[:-1], 3, 3)


def _qmul(a, b):
    return torch.stack([a[..., 0] * b[..., 0] - (a[..., 1:] * b[..., 1:]).sum(-1),
                        a[..., 0] * b[..., 1] + a[..., 1] * b[..., 0] + a[..., 2] * b[..., 3] - a[..., 3] * b[..., 2],
                        a[..., 0] * b[..., 2] - a[..., 1] * b[..., 3] + a[..., 2] * b[..., 0] + a[..., 3] * b[..., 1],
                        a[..., 0] * b[..., 3] + a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1] + a[..., 3] * b[..., 0]],
                       -1)


def _expmap(r):
    a = r.norm(dim=-1, keepdim=True)
    f = torch.where(a < 1e-12, torch.zeros_like(a), torch.sin(a / 2) / a.clamp_min(1e-300))
    return torch.cat([torch.cos(a / 2), r * f], -1)


def _shapes(s_nodes, xi):
    """Lagrange values and derivatives [Q][N] of the nodes 2 s - 1 at xi."""
    x = 2. * np.asarray(s_nodes) - 1.
    n = len(x)
    val, der = np.zeros((len(xi), n)), np.zeros((len(xi), n))
    for a in range(n):
        others = [j for j in range(n) if j != a]
        den = np.prod([x[a] - x[j] for j in others])
        for q, t in enumerate(xi):
            val[q, a] = np.prod([t - x[j] for j in others]) / den
            der[q, a] = sum(np.prod([t - x[j] for j in others if j != k]) for k in others) / den
    return val, der


def _exact_step(nodes_x0, s, design, gravity, v0, fx, motion, p, per_model, device):
    """One step of beams of one shape, [B] beams, `per_model` of them in each
    model (they share the convergence test).  design: mass and stiffness
    [B][stations][6][6], grid, quadrature; motion: prescribed root motion
    [B][7] (identity for a clamped root).  Returns q, v."""
    T = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=device)  # noqa: E731
    xi, w = (np.array(c) for c in zip(*design["quadrature"]))
    val, der = _shapes(s, xi)
    phi, dphi, wq = T(val), T(der), T(w)
    at = np.clip((xi + 1.) / 2., 0., 1.)
    grid = design["grid"]
    k = np.clip(np.searchsorted(grid, at, side="right") - 1, 0, len(grid) - 2)
    f = T((at - grid[k]) / (grid[k + 1] - grid[k]))[:, None, None]
    k = torch.as_tensor(k, device=device)
    Ms, Cs = ((1. - f) * m[:, k] + f * m[:, k + 1] for m in (T(design["mass"]), T(design["stiffness"])))
    x0, v, F, g, u0 = T(nodes_x0), T(v0), T(fx), T(gravity), T(motion)
    B, N, Q = x0.shape[0], x0.shape[1], len(xi)
    xp = torch.einsum("qn,bnc->bqc", dphi, x0[..., :3])
    J = xp.norm(dim=-1)
    xp = xp / J[..., None]
    r0 = torch.einsum("qn,bnc->bqc", phi, x0[..., 3:])
    r0 = r0 / r0.norm(dim=-1, keepdim=True)
    dphiJ = dphi[None] / J[..., None]
    h, tp = p.h, torch.float64
    ident = torch.tensor([0., 0., 0., 1., 0., 0., 0.], dtype=tp, device=device)
    q_prev = ident.expand(B, N, 7)
    vd = torch.zeros_like(v)
    an = torch.zeros_like(v)
    qd = v + (0.5 - p.beta) * h * an + p.beta * h * an
    v = v.clone()
    lam = torch.zeros(B, 6, dtype=tp, device=device)
    active = torch.ones(B // per_model, dtype=torch.bool, device=device)
    eye3, eye6 = torch.eye(3, dtype=tp, device=device), torch.eye(6, dtype=tp, device=device)
    X0 = torch.zeros(3, dtype=tp, device=device)

    def displaced(qd):
        return torch.cat([q_prev[..., :3] + h * qd[..., :3], _qmul(_expmap(h * qd[..., 3:]), q_prev[..., 3:])], -1)

    extra = torch.full_like(active, p.refine_iters, dtype=torch.int64)
    for _ in range(p.max_iter + p.refine_iters):
        q = displaced(qd)
        rv = h * qd[..., 3:]
        ph = rv.norm(dim=-1)[..., None, None]
        safe = ph.clamp_min(1e-300)
        big = ph > 1e-16
        t1 = torch.where(big, (torch.cos(ph) - 1.) / safe ** 2, torch.zeros_like(ph))
        t2 = torch.where(big, (1. - torch.sin(ph) / safe) / safe ** 2, torch.zeros_like(ph))
        rt = _tilde(rv)
        tan = eye3 + (t1 * rt + t2 * (rt @ rt)).transpose(-1, -2)
        at_q = lambda a: torch.einsum("qn,bnc->bqc", phi, a)           # noqa: E731
        slope = lambda a: torch.einsum("bqn,bnc->bqc", dphiJ, a)       # noqa: E731
        r = at_q(q[..., 3:])
        r = r / r.norm(dim=-1, keepdim=True)
        ud, om, omd = at_q(vd[..., :3]), at_q(v[..., 3:]), at_q(vd[..., 3:])
        up, rp = slope(q[..., :3]), slope(q[..., 3:])
        R6 = torch.zeros(B, Q, 6, 6, dtype=tp, device=device)
        R6[..., :3, :3] = R6[..., 3:, 3:] = _rot(_qmul(r, r0))
        Mu, Cu = (R6 @ m @ R6.transpose(-1, -2) for m in (Ms, Cs))
        conj = torch.cat([r[..., :1], -r[..., 1:]], -1)
        strain = torch.cat([xp + up - (_rot(r) @ xp[..., None])[..., 0], 2. * _qmul(rp, conj)[..., 1:]], -1)
        fc = (Cu @ strain[..., None])[..., 0]
        xs = xp + up
        S, Nt, Mt = _tilde(xs), _tilde(fc[..., :3]), _tilde(fc[..., 3:])
        C11, C21 = Cu[..., :3, :3], Cu[..., 3:, :3]
        O = torch.zeros_like(Cu)
        O[..., :3, 3:] = C11 @ S - Nt
        O[..., 3:, 3:] = C21 @ S - Mt
        P = torch.zeros_like(Cu)
        P[..., 3:, :3] = S.transpose(-1, -2) @ C11 + Nt
        P[..., 3:, 3:] = S.transpose(-1, -2) @ Cu[..., :3, 3:]
        Qm = torch.zeros_like(Cu)
        Qm[..., 3:, 3:] = S.transpose(-1, -2) @ O[..., :3, 3:]
        fd = torch.cat([torch.zeros_like(xs), (S.transpose(-1, -2) @ fc[..., :3, None])[..., 0]], -1)
        m = Mu[..., 0, 0]
        me = torch.stack([Mu[..., 5, 1], -Mu[..., 5, 0], Mu[..., 4, 0]], -1)     # mass times eta
        rho, om_t, omd_t, me_t = Mu[..., 3:, 3:], _tilde(om), _tilde(omd), _tilde(me)
        vec = lambda A, x: (A @ x[..., None])[..., 0]                    # noqa: E731
        cr = lambda a, b: torch.linalg.cross(a, b, dim=-1)               # noqa: E731
        fi = torch.cat([m[..., None] * ud + cr(om, cr(om, me)) + cr(omd, me),
                        cr(me, ud) + vec(rho, omd) + cr(om, vec(rho, om))], -1)
        gq = g.expand_as(ud)
        fg = torch.cat([m[..., None] * gq, cr(me, gq)], -1)
        Gy = torch.zeros_like(Cu)
        Gy[..., :3, 3:] = -_tilde(cr(om, me)) - om_t @ me_t
        Gy[..., 3:, 3:] = om_t @ rho - _tilde(vec(rho, om))
        Ki = torch.zeros_like(Cu)
        Ki[..., :3, 3:] = -(omd_t + om_t @ om_t) @ me_t
        Ki[..., 3:, 3:] = (_tilde(ud) @ me_t + rho @ omd_t - _tilde(vec(rho, omd))
                           + om_t @ (rho @ om_t - _tilde(vec(rho, om))))
        res = (torch.einsum("q,qn,bqc->bnc", wq, dphi, fc)
               + torch.einsum("q,bq,qn,bqc->bnc", wq, J, phi, fd + fi - fg)) - F

        def pairs(a, b, wt, A):
            return torch.einsum("qi,qj,bq,bqrc->bijrc", a, b, wt, A)

        wJ, wd = wq * J, wq / J
        Sm = (pairs(phi, phi, wJ, Ki + Qm) + pairs(phi, dphi, wq.expand(B, Q), P)
              + pairs(dphi, dphi, wd, Cu) + pairs(dphi, phi, wq.expand(B, Q), O))
        T6 = eye6.repeat(B, N, 1, 1)
        T6[..., 3:, 3:] = tan
        A = torch.einsum("bijrk,bjkc->bijrc", Sm, T6) + pairs(phi, phi, wJ, p.beta_prime * Mu + p.gamma_prime * Gy)
        A = p.conditioner * A.permute(0, 1, 3, 2, 4).reshape(B, 6 * N, 6 * N)
        # root constraint: residual, B = grad T, grad^T
        R1 = u0[..., 3:]
        c1 = torch.cat([R1[..., :1], -R1[..., 1:]], -1) / R1.norm(dim=-1, keepdim=True)
        Cm = _rot(_qmul(q[:, 0, 3:], c1))
        res_c = torch.cat([q[:, 0, :3] + X0 - u0[:, :3],
                           torch.stack([Cm[:, 2, 1] - Cm[:, 1, 2], Cm[:, 0, 2] - Cm[:, 2, 0],
                                        Cm[:, 1, 0] - Cm[:, 0, 1]], -1) / 2.], -1)
        AX = torch.diagonal(Cm, dim1=-2, dim2=-1).sum(-1)[:, None, None] / 2. * eye3 - Cm / 2.
        n6 = 6 * N
        full = torch.zeros(B, n6 + 6, n6 + 6, dtype=tp, device=device)
        full[:, :n6, :n6] = A
        full[:, n6:n6 + 3, :3] = eye3
        full[:, :3, n6:n6 + 3] = eye3
        full[:, n6 + 3:, 3:6] = AX.transpose(-1, -2) @ tan[:, 0]
        full[:, 3:6, n6 + 3:] = AX
        gl = torch.cat([lam[:, :3], vec(AX, lam[:, 3:])], -1)
        rhs = res.clone()
        rhs[:, 0] += gl
        rhs = torch.cat([-p.conditioner * rhs.reshape(B, n6), -res_c], -1)
        x = torch.linalg.solve(full, rhs)
        dx, dl = x[:, :n6].reshape(B, N, 6), x[:, n6:] / p.conditioner
        a_tol, r_tol = p.absolute_convergence_tol, p.relative_convergence_tol
        e2 = (((dx / (a_tol + r_tol * (h * qd).abs())) ** 2).sum((1, 2))
              + ((dl / (a_tol + r_tol * lam.abs())) ** 2).sum(1))
        err = (e2.reshape(-1, per_model).sum(1) / (per_model * (n6 + 6))).sqrt()
        on = active.repeat_interleave(per_model)[:, None, None].to(tp)
        qd = qd + on * dx / h
        v = v + on * p.gamma_prime * dx
        vd = vd + on * p.beta_prime * dx
        lam = lam + on[:, 0] * dl
        done = err <= 1.
        active = active & ~(done & (extra <= 0))
        extra = extra - done.to(extra.dtype)
        if not bool(active.any()):
            break
    return displaced(qd), v


def exact(case, seed):
    """q and v after the first pass, for the families whose beams carry only
    boundary conditions (the jointed systems have none here)."""
    if case["family"] not in ("cantilever", "rotor"):
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    p = _params(case)
    none = {"status": None, "iters": None}
    if p.precision:
        none = {"status": None}
    if case["family"] == "rotor":
        designs, which, amp, _, phase = _rotors(case, seed)
        models = [_rotor_model(case, d, None) for d in designs]
        x0 = np.stack([[n.x0 for n in models[w].nodes_] for w in which]).reshape(-1, case["nodes"], 7)
        v0 = np.stack([[n.v for n in models[w].nodes_] for w in which]).reshape(-1, case["nodes"], 6)
        fx = np.stack([a * math.cos(f) for a, f in zip(amp, phase)]).reshape(-1, case["nodes"], 6)
        u = np.tile(np.array(_root_motion(models[0], 0)), (case["models"], 1))
        d = {**designs[0][0], "mass": np.stack([b["mass"] for w in which for b in designs[w]]),
             "stiffness": np.stack([b["stiffness"] for w in which for b in designs[w]])}
        q, v = _exact_step(x0, d["s"], d, [0., 0., -9.81], v0, fx, u, p, 3, device)
        return {"q": q.reshape(-1, 7), "v": v.reshape(-1, 6), **none}
    designs, which, amp, _, phase = _cantilevers(case, seed)
    q_of, v_of = [None] * case["models"], [None] * case["models"]
    sizes = sorted({d["nodes"] for d in designs})
    for n in sizes:
        group = [i for i, w in enumerate(which) if designs[w]["nodes"] == n]
        ds = [designs[which[i]] for i in group]
        x0 = np.zeros((len(group), n, 7))
        x0[:, :, 3] = 1.
        x0[:, :, 0] = np.stack([d["length"] * d["s"] for d in ds])
        d = {**ds[0], "mass": np.stack([b["mass"] for b in ds]), "stiffness": np.stack([b["stiffness"] for b in ds])}
        clamp = np.tile([0., 0., 0., 1., 0., 0., 0.], (len(group), 1))
        q, v = _exact_step(x0, ds[0]["s"], d, [0., 0., 0.], np.zeros((len(group), n, 6)),
                           np.stack([amp[i] * math.cos(phase[i]) for i in group]), clamp, p, 1, device)
        for j, i in enumerate(group):
            q_of[i], v_of[i] = q[j], v[j]
    out = {"q": torch.cat(q_of), **none}
    return out if p.precision else {**out, "v": torch.cat(v_of)}

"""The rod steps a user of this framework runs, as cases that can be timed and compared.

Every case is one pass of a simulation that is under way: the batch (or server)
with its rods, material draws, drives and launch settings is in hand, and a
pass steps it through the public API and brings the centre lines, frames and
contact states back to pinned host memory, as a program that draws or scores
each step does. The state moves on from pass to pass.

kind      what it stands for
hanging   rods of one shape hanging from a pinned, driven top over a floor, or
          one clamped cantilever with a tip load: parameter studies and the
          single interactive cable. Sizes from one rod to the 4096 x 64 grid,
          both strategies, every precision, one and several sweeps
uneven    rods of mixed lengths, coiled, each with its own primitives,
          self-collision on, some steps after the start so that contacts
          are live: the framework's batching workload (rods in free fall) and,
          with a floor under each rod, scenes of cables that come to rest
hook      cables draped over a bar, hold/slide observer armed, compensated
          positions with FP64 friction cones: the mixed-precision sweep
harness   cables on a board following gripper schedules, 4 substeps x 4
          sweeps of 1 ms: the inner loop of the harness learner
served    one request of rods submitted to the continuous-batching server and
          waited for: a rollout service seen by its client
"""
import math

import numpy as np
import torch

from ropephysics_b200 import (Batch, Drive, Precision, Primitive, Rod, Server, StepParams, Strategy, World,
                              harness, synth, workloads)

MIXED = int(Precision.COMPENSATED | Precision.FP64_CONE | Precision.FP64_VERDICT)
PRECISION = {"reference": 0, "compensated": int(Precision.COMPENSATED), "mixed": MIXED,
             "coloured": int(Precision.COLORED_SELF)}

# FP32 operations of the reference step per segment-substep, as counted by the
# repository's oracle on these shapes
FLOPS = {"hanging": 890.5, "uneven": 1696.2, "hook": 1463.8, "harness": 1463.8, "served": 890.5}


def hanging(name, rods, segments, substeps=20, steps=1, iterations=1, interval=1, strategy="batched",
            precision="reference", clamped=False):
    return {"name": name, "kind": "hanging", "rods": rods, "segments": segments, "substeps": substeps,
            "steps": steps, "iterations": iterations, "interval": interval, "strategy": strategy,
            "precision": precision, "clamped": clamped}


def uneven(name, rods, low, high, substeps=50, precision="reference", interval=1, lead=20, floor=True):
    return {"name": name, "kind": "uneven", "rods": rods, "low": low, "high": high, "substeps": substeps,
            "precision": precision, "interval": interval, "lead": lead, "floor": floor}


def listed():
    return [
        # one interactive cable: the smallest call, bound by latency
        hanging("cantilever-1x64", 1, 64, clamped=True),
        # the parameter-study grid, four graph-replayed steps per look at the state
        hanging("grid-4096x64", 4096, 64, steps=4),
        # the same study in the API's default strategy (one rod per block)
        hanging("grid-fused-512x64", 512, 64, strategy="fused"),
        # an odd shape with several sweeps, kept contacts and compensation
        hanging("sweeps-777x97", 777, 97, substeps=8, iterations=3, interval=2, precision="compensated"),
        # a scene of a few cables of any length
        uneven("scene-8x[40,200]", 8, 40, 200, substeps=20),
        # very long cables, fewer than the GPU has SMs
        uneven("long-32x[1500,2200]", 32, 1500, 2200, substeps=20, lead=10),
        # a small mixed-length batch and the headline shape
        uneven("uneven-256x[16,512]", 256, 16, 512),
        uneven("uneven-4096x[16,512]", 4096, 16, 512, floor=False),
        # the mixed-precision sweep of 3600 placements
        {"name": "hook-3600x120", "kind": "hook", "ratios": 60, "frictions": 30, "stiffnesses": 2, "substeps": 20},
        # the learner's population, one control tick of every attempt
        {"name": "harness-1024x120", "kind": "harness", "rods": 1024, "steps": 10},
        # one client's request
        {"name": "served-64x256", "kind": "served", "rods": 64, "segments": 256, "steps": 20, "substeps": 20},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["hanging", "hanging", "uneven", "uneven", "hook", "harness", "served"])
    if kind == "hanging":
        segments = _log(rng, 16, 256)
        strategy = rng.choice(["batched", "batched", "fused"])
        rods = _log(rng, 1, 512 if strategy == "fused" else min(4096, 262144 // segments))
        case = hanging("", rods, segments, rng.choice([8, 20, 20]), rng.randint(1, 4), rng.choice([1, 1, 2, 4]),
                       rng.choice([1, 1, 2]), strategy, rng.choice(["reference", "reference", "compensated", "mixed"]))
    elif kind == "uneven":
        low = _log(rng, 16, 512)
        high = rng.randint(low + 1, min(1600, 8 * low + 16))
        rods = _log(rng, 4, min(4096, 1_000_000 // (low + high)))
        # without a floor a long run of a small batch would be a long fall
        case = uneven("", rods, low, high, rng.choice([20, 50]),
                      rng.choice(["reference", "reference", "mixed", "coloured"]), rng.choice([1, 1, 4]), 10,
                      rods < 1024 or rng.random() < 0.5)
    elif kind == "hook":
        case = {"kind": "hook", "ratios": rng.randint(2, 60), "frictions": rng.randint(1, 30),
                "stiffnesses": rng.choice([1, 2]), "substeps": rng.choice([12, 20])}
    elif kind == "harness":
        case = {"kind": "harness", "rods": _log(rng, 16, 1024), "steps": rng.choice([5, 10, 20])}
    else:
        case = {"kind": "served", "rods": _log(rng, 1, 256), "segments": rng.randint(32, 512),
                "steps": rng.randint(5, 40), "substeps": 20}
    case.pop("name", None)
    return case


def _hanging_inputs(case, seed):
    """Prototype, world, material scales and drives of a hanging case."""
    rng = np.random.default_rng(seed)
    n, count = case["segments"], case["rods"]
    length = n / 64.0
    if case.get("clamped"):
        rod = Rod.straight(n, length, workloads.GRID_MATERIAL)
        rod.clamp_end(tip=False)
        rod.ext_force[-1] = (0.0, 0.0, -float(rng.uniform(0.02, 0.08)))
        return rod, None, None, None, None
    rod = Rod.straight(n, length, workloads.GRID_MATERIAL, origin=(0.0, 0.0, 0.0), direction=(0.0, 0.0, -1.0))
    rod.pin_particle(0)
    world = World([Primitive.plane((0.0, 0.0, -length - 0.02), (0.0, 0.0, 1.0), 0.5)],
                  self_collision=case["kind"] == "served", self_friction=0.5,
                  hash_table_size=workloads.table_for(n))
    youngs = rng.uniform(0.4, 4.0, count).astype(np.float32)
    friction = rng.uniform(0.6, 1.4, count).astype(np.float32)
    axes = rng.normal(size=(count, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    amplitude, frequency = rng.uniform(0.0, 0.1, count), rng.uniform(0.5, 2.0, count)
    phase = rng.uniform(0.0, 2.0 * math.pi, count)
    drives = [Drive(0, tuple(map(float, a)), float(m), float(f), float(p))
              for a, m, f, p in zip(axes, amplitude, frequency, phase)]
    return rod, world, youngs, friction, drives


def _uneven_inputs(case, seed):
    """Coiled rods with a straight rest shape and their worlds. How many
    segments and primitives each has is part of the case, the rest is drawn."""
    shape = np.random.default_rng([case["rods"], case["low"], case["high"]])
    rng = np.random.default_rng(seed)
    rods, worlds = [], []
    for _ in range(case["rods"]):
        n, obstacles = int(shape.integers(case["low"], case["high"] + 1)), int(shape.integers(1, 5))
        points = workloads.helix(n, 0.2 * n / 32.0, float(rng.uniform(0.05, 0.2)), pitch=0.02)
        mu, low, high = float(rng.uniform(0.2, 1.0)), points.min(axis=0), points.max(axis=0)
        rod = Rod.centerline(points, workloads.GRID_MATERIAL, frame_seed=(0.0, 0.0, 1.0))
        rod.b_rest_darboux[:] = 0.0
        prims = [workloads.primitive(synth.random_primitive(rng, points.mean(axis=0), mu, low, high))
                 for _ in range(obstacles)]
        if case["floor"]:
            prims.append(Primitive.plane((0.0, 0.0, float(low[2]) - 0.02), (0.0, 0.0, 1.0), mu))
        rods.append(rod)
        worlds.append(World(prims, self_collision=True, self_friction=mu, hash_table_size=workloads.table_for(n)))
    return rods, worlds


def _hook_inputs(case, seed):
    """The sweep's rods (one per leg ratio and stiffness), its worlds, and
    which rod and world each placement has."""
    rng = np.random.default_rng(seed)
    mus = np.linspace(0.05, 0.6, case["frictions"]) + rng.uniform(0.0, 0.02)
    ratios = np.linspace(1.0, 4.0, case["ratios"]) + rng.uniform(0.0, 0.05, case["ratios"])
    worlds = [World([Primitive.capsule((0.0, -0.3, 0.8), (0.0, 0.3, 0.8), 0.02, float(mu)),
                     Primitive.plane((0.0, 0.0, workloads.HOOK_FLOOR_Z), (0.0, 0.0, 1.0), float(mu))],
                    self_collision=True, self_friction=float(mu), hash_table_size=256) for mu in mus]
    shapes = []
    for stiffness in (1e8, 3e8)[:case["stiffnesses"]]:
        material = workloads.Material(youngs=stiffness, **workloads.HOOK_MATERIAL)
        for ratio in ratios:
            rod = Rod.centerline(workloads.hanging_cable_points(float(ratio)), material, frame_seed=(0.0, 1.0, 0.0))
            rod.b_rest_darboux[:] = 0.0
            shapes.append(rod)
    shape_of = [s for s in range(len(shapes)) for _ in mus]
    world_of = [w for _ in shapes for w in range(len(worlds))]
    return shapes, worlds, shape_of, world_of


def _harness_inputs(case, seed):
    """The task, and one cable and motion per attempt."""
    task, rng, count = harness.HarnessTask(), np.random.default_rng(seed), case["rods"]
    youngs, friction = harness.random_cables(rng, count)
    mean = task.hand_written_policy().reshape(-1)
    drives = [task.drive(task.to_policy(mean + 0.08 * rng.standard_normal(mean.shape))) for _ in range(count)]
    return task, youngs, friction, drives


def _params(case):
    return StepParams(dt=1.0 / 60, substeps=case["substeps"], iterations=case.get("iterations", 1),
                      contact_interval=case.get("interval", 1))


def _pinned(batch, contacts):
    """Pinned host buffers for what a pass reads back."""
    def buffer(what, dtype, columns):
        t = torch.empty(batch.state_bytes(what) // dtype.itemsize, dtype=dtype, pin_memory=True)
        return t.view(-1, columns) if columns else t
    out = {"positions": buffer(Batch.POSITIONS, torch.float32, 4), "frames": buffer(Batch.FRAMES, torch.float32, 4)}
    if contacts:
        out["contacts"] = buffer(Batch.CONTACTS, torch.uint8, 0)
    return out


def prepare(case, seed):
    kind, contacts, steps = case["kind"], True, case.get("steps", 1)
    if kind == "served":
        rod, world, youngs, friction, drives = _hanging_inputs(case, seed)
        request = dict(rods=[rod] * case["rods"], steps=steps, worlds=[world], drives=drives, youngs_scale=youngs,
                       friction_scale=friction)
        return {"server": Server(2 << 30, _params(case)), "request": request}
    if kind == "hanging":
        rod, world, youngs, friction, drives = _hanging_inputs(case, seed)
        strategy = Strategy.FUSED if case["strategy"] == "fused" else Strategy.BATCHED
        batch = Batch.create(rod, case["rods"], strategy, world)
        if drives is not None:
            batch.set_material_scales(youngs, friction)
            batch.set_drives(drives)
        contacts, params = world is not None, _params(case)
        batch.set_precision(PRECISION[case["precision"]])
        batch.upload(rod)
    elif kind == "uneven":
        rods, worlds = _uneven_inputs(case, seed)
        batch, params = Batch.create_mixed(rods, worlds, range(len(rods))), _params(case)
        batch.set_precision(PRECISION[case["precision"]])
        batch.step_many(params, case["lead"])
    elif kind == "hook":
        shapes, worlds, shape_of, world_of = _hook_inputs(case, seed)
        rods = [shapes[s] for s in shape_of]
        batch = Batch.create_mixed(rods, worlds, world_of)
        batch.set_precision(MIXED)
        batch.arm_hold_observer([0] * len(rods), interval=50)
        params = _params(case)
    else:
        task, youngs, friction, drives = _harness_inputs(case, seed)
        batch = Batch.create(task.build(), case["rods"], Strategy.BATCHED, task.world())
        batch.set_material_scales(youngs, friction)
        batch.set_waypoint_drives(drives)
        params = task.params()
    batch.set_graph(steps > 1)
    batch.synchronize()
    return {"batch": batch, "params": params, "steps": steps, "out": _pinned(batch, contacts)}


def run(state):
    if "server" in state:
        server = state["server"]
        request = server.submit(**state["request"])
        server.wait(request)
        positions = server.result(request)
        server.release(request)
        return {"positions": positions}
    batch, out = state["batch"], state["out"]
    if state["steps"] > 1:
        batch.step_many(state["params"], state["steps"])
    else:
        batch.step(state["params"])
    for name, what in (("positions", Batch.POSITIONS), ("frames", Batch.FRAMES), ("contacts", Batch.CONTACTS)):
        if name in out:
            batch.read_state_async(what, out[name].data_ptr(), out[name].nbytes)
    return out


def _sizes(case):
    """Segments, segment-substeps and sweeps per substep of one pass."""
    kind = case["kind"]
    if kind == "uneven":  # the draws' expected total
        segments = case["rods"] * (case["low"] + case["high"]) // 2
    elif kind == "hook":
        segments = case["ratios"] * case["frictions"] * case["stiffnesses"] * 120
    elif kind == "harness":
        return case["rods"] * 120, case["rods"] * 120 * 4 * case["steps"], 4
    else:
        segments = case["rods"] * case["segments"]
    return segments, segments * case["substeps"] * case.get("steps", 1), case.get("iterations", 1)


def work(case):
    """Each state row read once and written once per pass, positions and
    frames copied out; the reference step's operations."""
    segments, substeps, sweeps = _sizes(case)
    copies = 12 if case["kind"] == "served" else 32
    return {"bytes": segments * (11 * 16 + copies), "flops": substeps * FLOPS[case["kind"]] * (0.4 + 0.6 * sweeps)}


# ---- the same pass in 64 bits ----

def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _rotate(q, v):
    u = q[..., 1:]
    t = 2.0 * _cross(u, v)
    return v + q[..., :1] * t + _cross(u, t)


def _conjugate(q):
    return torch.cat([q[..., :1], -q[..., 1:]], -1)


def _multiply(a, b):
    w = a[..., :1] * b[..., :1] - (a[..., 1:] * b[..., 1:]).sum(-1, keepdim=True)
    return torch.cat([w, a[..., :1] * b[..., 1:] + b[..., :1] * a[..., 1:] + _cross(a[..., 1:], b[..., 1:])], -1)


def _turn(q, theta):
    p = _multiply(q, torch.cat([torch.ones_like(theta[..., :1]), 0.5 * theta], -1))
    return p / p.norm(dim=-1, keepdim=True)


def _skew(v):
    x, y, z = v.unbind(-1)
    o = torch.zeros_like(x)
    return torch.stack([torch.stack([o, -z, y], -1), torch.stack([z, o, -x], -1), torch.stack([-y, x, o], -1)], -2)


class _Chains:
    """XPBD Cosserat steps of chains of one segment count, in float64: the
    order of the framework's step (contacts, prediction, even then odd stretch
    constraints, even then odd bends, world contacts with friction, velocity
    recovery). Arrays are (rods, elements, ...)."""

    def __init__(self, shapes, shape_of, scale, friction):
        def column(name):
            a = np.stack([np.asarray(getattr(r, name), np.float64) for r in shapes])
            return torch.from_numpy(a)[torch.as_tensor(shape_of)].cuda()
        self.x, self.v, self.q, self.w = column("x"), column("v"), column("q"), column("omega")
        self.mass, self.force, self.kin = column("inv_mass")[..., None], column("ext_force"), column("kin_velocity")
        self.inertia, self.inv_inertia, self.torque = column("inertia"), column("inv_inertia"), column("ext_torque")
        self.s_rest, self.b_rest = column("s_rest")[..., None], column("b_rest")[..., None]
        self.s_soft = column("s_compliance") * scale[:, None, None]
        self.b_soft = column("b_compliance") * scale[:, None, None]
        self.darboux = column("b_rest_darboux")
        self.b_a, self.b_b = (torch.from_numpy(np.array(getattr(shapes[0], k), np.int64)).cuda() for k in ("b_a", "b_b"))
        self.radius = shapes[0].material.radius
        self.friction = friction

    def stretch(self, k, stiff):
        w0, w1, inv, rest = self.mass[:, k], self.mass[:, k + 1], self.inv_inertia[:, k], self.s_rest[:, k]
        q = self.q[:, k]
        u = _rotate(_conjugate(q), self.x[:, k + 1] - self.x[:, k]) / rest
        c = u - torch.tensor([0.0, 0.0, 1.0], dtype=u.dtype, device=u.device)
        s, alpha = _skew(u), self.s_soft[:, k] * stiff
        a = torch.diag_embed((w0 + w1) / rest ** 2 + alpha) + (s * inv[..., None, :]) @ s.transpose(-1, -2)
        lam = self.lam_s[:, k]
        step = torch.linalg.solve(a, -(c + alpha * lam))
        self.lam_s[:, k] = lam + step
        world = _rotate(q, step)
        self.x[:, k] -= world * (w0 / rest)
        self.x[:, k + 1] += world * (w1 / rest)
        self.q[:, k] = _turn(q, inv * _cross(step, u))

    def bend(self, k, stiff):
        a, b = self.b_a[k], self.b_b[k]
        qa, qb, ia, ib, rest = self.q[:, a], self.q[:, b], self.inv_inertia[:, a], self.inv_inertia[:, b], self.b_rest[:, k]
        p = _multiply(_conjugate(qa), qb)
        p = torch.where(p[..., :1] < 0.0, -p, p)
        w, v = p[..., :1], p[..., 1:]
        eye = torch.eye(3, dtype=p.dtype, device=p.device)
        ja, jb = ((eye * m[..., None] + _skew(v)) / rest[..., None] for m in (-w, w))
        alpha = self.b_soft[:, k] * stiff
        m = torch.diag_embed(alpha) + (ja * ia[..., None, :]) @ ja.transpose(-1, -2) + \
            (jb * ib[..., None, :]) @ jb.transpose(-1, -2)
        lam = self.lam_b[:, k]
        step = torch.linalg.solve(m, -(2.0 / rest * v - self.darboux[:, k] + alpha * lam))
        self.lam_b[:, k] = lam + step
        side = _cross(v, step)
        self.q[:, a] = _turn(qa, ia * (-w * step - side) / rest)
        self.q[:, b] = _turn(qb, ib * (w * step - side) / rest)

    def contacts(self, worlds, margin=0.25):
        """Normals, offsets and whether a contact is generated, per primitive."""
        found = []
        for prims in zip(*worlds):
            a = torch.tensor([p.a for p in prims], dtype=self.x.dtype, device=self.x.device)[:, None]
            mu = torch.tensor([p.friction for p in prims], dtype=self.x.dtype, device=self.x.device) * self.friction
            if prims[0].type == 0:
                n = torch.tensor([p.normal for p in prims], dtype=a.dtype, device=a.device)[:, None].expand_as(self.x)
                gap = ((self.x - a) * n).sum(-1) - self.radius
            else:
                d = torch.tensor([p.b for p in prims], dtype=a.dtype, device=a.device)[:, None] - a
                t = (((self.x - a) * d).sum(-1, keepdim=True) / (d * d).sum(-1, keepdim=True)).clamp(0.0, 1.0)
                n = self.x - (a + d * t)
                length = n.norm(dim=-1)
                n = n / length[..., None]
                gap = length - prims[0].radius - self.radius
            live = (gap < margin * self.radius) & (self.mass[..., 0] > 0.0)
            zero = torch.zeros_like(gap)
            found.append([n, (self.x * n).sum(-1) - gap, live, mu[:, None], zero, zero.clone(), zero.to(torch.uint8)])
        return found

    def project(self, found, prev):
        w = self.mass[..., 0].clamp_min(1e-300)
        for c in found:
            n, offset, live, mu, lam, applied, _ = c
            gap = (self.x * n).sum(-1) - offset
            total = (lam - gap / w).clamp_min(0.0)
            push = torch.where(live, total - lam, torch.zeros_like(total))
            lam += push
            self.x += n * (w * push)[..., None]
            d = self.x - prev
            side = d - n * (d * n).sum(-1, keepdim=True)
            slide = side.norm(dim=-1)
            budget = mu * lam * w - applied
            rub = live & (mu > 0.0) & (lam > 0.0) & (slide >= 1e-15)
            capped = torch.where(rub & (budget > 0.0), torch.minimum(slide, budget), torch.zeros_like(slide))
            applied += capped
            self.x -= side * (capped / slide.clamp_min(1e-300))[..., None]

    def step(self, params, worlds):
        h = params.dt / params.substeps
        stiff, g = 1.0 / (h * h), torch.tensor(params.gravity, dtype=self.x.dtype, device=self.x.device)
        pairs = [torch.arange(c, n, 2, device=self.x.device) for n in (self.s_rest.shape[1], self.b_rest.shape[1])
                 for c in (0, 1)]
        found = []
        for sub in range(params.substeps):
            self.lam_s, self.lam_b = torch.zeros_like(self.s_soft), torch.zeros_like(self.b_soft)
            if worlds and sub % params.contact_interval == 0:
                found = self.contacts(worlds)
            for c in found:
                c[4], c[5] = torch.zeros_like(c[4]), torch.zeros_like(c[5])
            x0, q0 = self.x.clone(), self.q.clone()
            free = self.mass > 0.0
            self.v = torch.where(free, self.v + h * (g + self.force * self.mass), self.kin)
            self.x = self.x + h * self.v
            turns = (self.inv_inertia ** 2).sum(-1, keepdim=True) > 0.0
            spin = self.inv_inertia * (_rotate(_conjugate(self.q), self.torque) - _cross(self.w, self.inertia * self.w))
            self.w = self.w + h * spin
            q = self.q + 0.5 * h * _multiply(self.q, torch.cat([torch.zeros_like(self.w[..., :1]), self.w], -1))
            self.q = torch.where(turns, q / q.norm(dim=-1, keepdim=True), self.q)
            for _ in range(params.iterations):
                for k in pairs[:2]:
                    self.stretch(k, stiff)
                for k in pairs[2:]:
                    if len(k):
                        self.bend(k, stiff)
                self.project(found, x0)
            self.v = torch.where(free, (self.x - x0) / h, self.kin)
            dq = _multiply(_conjugate(q0), self.q)
            dq = torch.where(dq[..., :1] < 0.0, -dq, dq)
            self.w = torch.where(turns, 2.0 / h * dq[..., 1:], torch.zeros_like(self.w))


def _gripper(drive, t):
    """Where a waypoint schedule's gripper is at time t."""
    at, begun = np.asarray(drive.start, np.float64), 0.0
    for goal, leg in zip(drive.waypoints, drive.legs):
        if t < begun + leg:
            u = (t - begun) / leg
            return at + (np.asarray(goal) - at) * (u * u * (3.0 - 2.0 * u))
        at, begun = np.asarray(goal, np.float64), begun + leg
    return at


def exact(case, seed):
    """Positions and frames of the first pass in float64, for the cases whose
    rods meet no self contact in it. Contact states have no value in 64 bits
    (a gap within rounding of the margin is a contact or is none)."""
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "uneven" or _sizes(case)[1] * _sizes(case)[2] > 3e7:
        return None

    def per_rod(values):
        return torch.as_tensor(values, dtype=torch.float64, device="cuda")

    if kind == "hook":
        shapes, worlds, shape_of, world_of = _hook_inputs(case, seed)
        params, prims, tops = _params(case), [worlds[w].primitives for w in world_of], None
        one = torch.ones(len(shape_of), dtype=torch.float64, device="cuda")
        rods = _Chains(shapes, shape_of, one, one)
    elif kind == "harness":
        task, youngs, friction, drives = _harness_inputs(case, seed)
        params, prims = task.params(), [task.world().primitives] * case["rods"]
        rods = _Chains([task.build()], [0] * case["rods"], 1.0 / per_rod(youngs), per_rod(friction))
        tick = task.steps_per_control * params.dt

        def tops(k):
            k //= task.steps_per_control
            v = np.stack([(_gripper(d, (k + 1) * tick) - _gripper(d, k * tick)) / tick for d in drives])
            rods.kin[:, -1] = per_rod(np.concatenate([v, 0.0 * v[:, :1]], 1))
    else:
        rod, world, youngs, friction, drives = _hanging_inputs(case, seed)
        params, count, tops = _params(case), case["rods"], None
        youngs, friction = (np.ones(count) if a is None else a for a in (youngs, friction))
        prims = [world.primitives] * count if world else []
        rods = _Chains([rod], [0] * count, 1.0 / per_rod(youngs), per_rod(friction))
        if drives:
            axis, omega = per_rod([d.axis for d in drives]), per_rod([2.0 * math.pi * d.frequency for d in drives])
            speed, phase = per_rod([d.amplitude for d in drives]) * omega, per_rod([d.phase for d in drives])

            def tops(k):
                rods.kin[:, 0] = axis * (speed * torch.cos(omega * k * params.dt + phase))[:, None]
    for k in range(steps):
        if tops:
            tops(k)
        rods.step(params, prims)
    if kind == "served":
        return {"positions": rods.x.reshape(-1, 3).cpu()}

    def rows(a):
        pad = a if a.shape[-1] == 4 else torch.cat([a, torch.zeros_like(a[..., :1])], -1)
        return pad.reshape(-1, 4).cpu()
    out = {"positions": rows(rods.x), "frames": rows(rods.q)}
    if prims:
        out["contacts"] = None
    return out

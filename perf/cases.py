"""Timed cases of the AVBD world step: what a program that uses this framework
has it do, through `GpuBackend` (pack once, then frames), from a ten-cube
stack to a batch of piles and the 53-layer pyramid.

A pass of a scene case is a host-authoritative stretch of frames, the calls
the end-to-end benchmark makes: hand the body (and joint, spring) state over
(`write_state`), step, read the state back (`sync_to_cpu`). The contacts stay
on the device between passes, as they do between a program's frames. Its
outputs are the whole state that comes back. `prepare` builds the scene,
packs it and steps it to where the case begins; the seed moves the bodies.
"""
import importlib
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
_PKG = "avbd-sandbox_gb300"


def _mod(name):
    return importlib.import_module(_PKG + "." + name)


def listed():
    return [
        # The smallest scene a sandbox opens with, one frame at a time: ten cubes on
        # the ground, launches and latency.
        {"name": "stack_frame", "kind": "stack", "n": 10, "steps": 1, "graph": 0},
        # Joints and springs without contacts, 20 iterations, the FP64 bodies of a
        # 26,000:1 mass ratio: a hanging chain and a spring chain, one frame.
        {"name": "chain_frame", "kind": "chain", "n": 50, "springs": 100, "steps": 1, "graph": 0},
        # Destruction: a bonded 16 x 16 brick wall while the sphere strikes it, four
        # steps between two looks at the state.
        {"name": "wall_strike", "kind": "wall", "n": 16, "steps": 4, "graph": 0},
        # A small pile of mixed boxes, each step replayed as a CUDA graph: a training
        # environment with an action repeat of four.
        {"name": "pile_small", "kind": "pile", "n": 200, "spheres": 0, "steps": 4, "graph": 1},
        # An odd mid-sized pile with spheres among the boxes, one frame.
        {"name": "pile_spheres", "kind": "pile", "n": 1777, "spheres": 1, "steps": 1, "graph": 0},
        # The largest single pile of the batched workload.
        {"name": "pile_large", "kind": "pile", "n": 8192, "spheres": 0, "steps": 2, "graph": 0},
        # The contact extensions (materials model): speculative contacts, restitution,
        # two friction coefficients.
        {"name": "materials", "kind": "materials", "n": 1000, "steps": 2, "graph": 0},
        # The headline scene: 51,039 cubes standing (the middle of the benchmark's 20
        # steps: the layers have met), each step one CUDA graph, a frame.
        {"name": "pyramid", "kind": "pyramid", "n": 53, "settle": 12, "steps": 1, "graph": 1},
        # The same kind of scene after it has been crushed into a dense pile.
        {"name": "crushed", "kind": "pyramid", "n": 36, "settle": 150, "steps": 1, "graph": 0},
        # Many independent piles in one context (a batch of environments).
        {"name": "batch", "kind": "batch", "n": 96, "steps": 2, "graph": 1},
        # The differentiable step: the wall of 256 bricks, forward with five
        # directions, readback and the backward.
        {"name": "adjoint_wall", "kind": "adjoint", "n": 16, "steps": 6},
        # The broad phase alone, on a program's own device buffers.
        {"name": "pairs", "kind": "pairs", "n": 20011},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stack", "chain", "wall", "pile", "pile", "materials", "pyramid", "pyramid", "batch",
                       "adjoint", "pairs"])
    graph = rng.randint(0, 1)
    if kind == "stack":
        return {"kind": kind, "n": 2 * rng.randint(1, 20) + 1, "steps": rng.randint(1, 4), "graph": graph}
    if kind == "chain":
        return {"kind": kind, "n": _log(rng, 8, 100), "springs": _log(rng, 4, 200), "steps": rng.randint(1, 2),
                "graph": graph}
    if kind == "wall":
        return {"kind": kind, "n": 2 * rng.randint(2, 11) + 1, "steps": rng.randint(1, 4), "graph": graph}
    if kind == "pile":
        return {"kind": kind, "n": _log(rng, 64, 8192), "spheres": rng.randint(0, 1), "steps": rng.randint(1, 4),
                "graph": graph}
    if kind == "materials":
        return {"kind": kind, "n": _log(rng, 60, 2000), "steps": rng.randint(1, 3), "graph": graph}
    if kind == "pyramid":
        if rng.random() < 0.5:
            return {"kind": kind, "n": rng.randint(10, 53), "settle": rng.randint(0, 20), "steps": rng.randint(1, 2),
                    "graph": graph}
        return {"kind": kind, "n": rng.randint(10, 36), "settle": rng.randint(100, 149), "steps": 1, "graph": graph}
    if kind == "batch":
        return {"kind": kind, "n": rng.randint(8, 95), "steps": rng.randint(1, 2), "graph": graph}
    if kind == "adjoint":
        return {"kind": kind, "n": rng.randint(4, 15), "steps": rng.randint(2, 7)}
    return {"kind": kind, "n": _log(rng, 1000, 65000)}


# --- scenes ------------------------------------------------------------------
def _pile(n, rng, spheres=False):
    """One scene of the batched workload (random_pile's ranges) from `rng`:
    boxes on a contact-free lattice above the ground, every third body a
    sphere when asked. Built in arrays: a batch has 100,000 bodies and more."""
    abi, sc = _mod("abi"), _mod("scene")
    g = sc.Scene("ground")
    sc.add_ground(g, 0.5)
    gw = g.world()
    w = abi.World(n + 1)
    for f in ("shape",) + abi.World.BODY_F:
        getattr(w, f)[0] = getattr(gw, f)[0]
    i = np.arange(n)
    side = max(1, int(math.ceil(n ** (1.0 / 3.0))))
    size = rng.uniform(0.3, 2.0, (n, 3))
    ball = (i % 3 == 2) if spheres else np.zeros(n, bool)
    size[ball] = size[ball, :1]
    density = np.exp(rng.uniform(math.log(100.0), math.log(1e4), n))
    vol = np.where(ball, math.pi / 6, 1.0) * size.prod(axis=1)
    sq = size * size
    w.shape[1:] = np.where(ball, abi.SHAPE_SPHERE, abi.SHAPE_BOX)
    w.size[1:] = size
    w.mass[1:] = vol * density
    cube = (sq.sum(axis=1, keepdims=True) - sq) / 12.0
    w.moment[1:] = np.where(ball[:, None], sq / 10.0, cube) * (vol * density)[:, None]
    w.radius[1:] = np.where(ball, size[:, 0] * 0.5, 0.5 * np.sqrt(sq.sum(axis=1)))
    w.friction[1:] = rng.uniform(0.2, 0.9, n)
    half = (side - 1) / 2
    w.pos[1:] = np.stack([(i % side - half) * 3.5, (i // side % side - half) * 3.5, 2.0 + i // (side * side) * 3.5], 1)
    w.vel[1:] = rng.normal(0.0, 0.2, (n, 3))
    w.prev_vel[1:] = w.vel[1:]
    return w


def _world(case, seed):
    """The scene of a case before any step, and its solver parameters."""
    sc = _mod("scene")
    rng = np.random.default_rng([seed, 17])
    kind, n = case["kind"], case["n"]
    params = dict(gravity=-9.81, iterations=10)
    if kind == "stack":
        w = sc.cube_stack(n=n, seed=1 + seed % 100000, beta=None).world()
    elif kind == "chain":
        s = sc.heavy_chain(links=n, springs=case["springs"])
        w, params = s.world(), dict(s.params)
        dyn = w.mass > 0
        w.vel[dyn] = rng.normal(0.0, 0.05, (int(dyn.sum()), 3))
        w.omega[dyn] = rng.normal(0.0, 0.05, (int(dyn.sum()), 3))
        w.prev_vel[:] = w.vel
    elif kind in ("wall", "adjoint"):
        speed = 8.0 + rng.uniform(-1.0, 1.0)
        build = sc.brick_wall if kind == "wall" else sc.brick_wall_c5
        s = build(cols=n, rows=n, sphere_speed=speed) if kind == "wall" else \
            build(cols=n, rows=n, mu=rng.uniform(0.4, 0.8), sphere_velocity=(rng.normal(0, 0.1), speed, 0.0))
        w = s.world()
        w.pos[-1, 1] = -0.75  # in front of the wall: the strike falls within the first steps
    elif kind in ("pile", "materials"):
        w = _pile(n, rng, bool(case.get("spheres")))
        if kind == "materials":
            sf = rng.uniform(0.3, 0.9, n + 1)
            e, ro = rng.uniform(0.0, 0.8, n + 1), rng.uniform(-0.02, -0.005, n + 1)
            e[0], ro[0] = 0.0, -0.005
            w.set_materials(static_friction=sf, dynamic_friction=sf * rng.uniform(0.3, 1.0, n + 1), restitution=e,
                            rest_offset=ro)
            params["contact_model"] = _mod("abi").CONTACT_MATERIALS
    elif kind == "pyramid":
        w = sc.pyramid(layers=n, sphere_speed=10.0 + rng.uniform(-2.0, 2.0)).world()
        w.vel[1:-1] += rng.normal(0.0, 0.01, (w.n_bodies - 2, 3))
        w.prev_vel[:] = w.vel
    elif kind == "batch":
        counts = np.exp(rng.uniform(math.log(64), math.log(8192), n)).round().astype(int)
        # log-uniform draws, scaled to one total so that the case is the same size for every seed
        counts = np.maximum(64, (counts * (1700.0 * n / counts.sum())).astype(int))
        counts[np.argmax(counts)] += 1700 * n - counts.sum()
        w = sc.batch_worlds([_pile(int(c), rng) for c in counts])
    else:
        raise KeyError(kind)
    return w.round_to_device(), params


def _settle(case):
    """Steps before the case begins: a random pile's bodies have landed."""
    return {"pile": 150, "materials": 120, "batch": 150, "stack": 10}.get(case["kind"], case.get("settle", 0))


def prepare(case, seed):
    abi, be = _mod("abi"), _mod("backend")
    if case["kind"] == "pairs":
        return _prepare_pairs(case, seed)
    w, p = _world(case, seed)
    params = abi.default_params(**p, body_order=abi.ORDER_PRIORITY, graph=case.get("graph", 0))
    gpu = be.GpuBackend(params)
    if case["kind"] == "adjoint":
        n = case["n"]
        ball = w.n_bodies - 1
        seeds = [(abi.SEED_VELOCITY, ball, k, k) for k in range(3)]
        seeds += [(abi.SEED_FRICTION, b, 0, 3) for b in range(1, 1 + n * n)] + [(abi.SEED_PENALTY_MAX, 0, 0, 4)]
        up = np.random.default_rng([seed, 5]).normal(size=(w.n_bodies, 3))
        return {"kind": "adjoint", "gpu": gpu, "world": w, "seeds": seeds, "steps": case["steps"], "up": up}
    gpu.pack(w)
    if _settle(case):
        gpu.step(_settle(case))
        gpu.idle()
        w = gpu.read_state()
    return {"kind": "frame", "gpu": gpu, "world": w, "out": w.copy(), "steps": case["steps"]}


def run(state):
    if state["kind"] == "pairs":
        s = state
        _mod("backend").overlap_pairs_static(s["n"], s["pos"].data_ptr(), s["radius"].data_ptr(),
                                             s["dynamic"].data_ptr(), s["cell"], s["keys"].data_ptr(),
                                             s["keys"].numel(), s["count"].data_ptr(),
                                             torch.cuda.current_stream().cuda_stream)
        return {"keys": s["keys"], "count": s["count"]}
    gpu, w = state["gpu"], state["world"]
    if state["kind"] == "adjoint":
        gpu.adjoint_forward(w, state["steps"], state["seeds"])
        pos, dpos, quat = gpu.adjoint_read()
        return {"pos": pos, "dpos": dpos, "quat": quat, "grad": gpu.adjoint_backward(state["up"])}
    gpu.write_state(w)
    gpu.step(state["steps"])
    o = state["out"]
    gpu.sync_to_cpu(o)
    got = {"pos": o.pos, "quat": o.quat, "vel": o.vel, "omega": o.omega, "prev_vel": o.prev_vel}
    if o.n_joints:
        got.update(penalty_lin=o.j_penalty_lin, lambda_lin=o.j_lambda_lin, lambda_ang=o.j_lambda_ang,
                   broken=o.j_broken)
    if o.n_springs:
        got.update(peak=o.s_peak_strain, torn=o.s_broken)
    return got


def _prepare_pairs(case, seed):
    """A cloud of boxes with edges U[0.3, 2] m, a few overlaps a body."""
    n = case["n"]
    rng = np.random.default_rng([seed, 23])
    side = int(math.ceil(n ** (1.0 / 3.0)))
    i = np.arange(n)
    pos = np.stack([i % side, i // side % side, i // (side * side)], 1) * 1.6 + rng.uniform(-0.5, 0.5, (n, 3))
    r = 0.5 * np.sqrt((rng.uniform(0.3, 2.0, (n, 3)) ** 2).sum(axis=1))
    dev = torch.device("cuda", torch.cuda.current_device())
    return {"kind": "pairs", "n": n, "pos": torch.from_numpy(pos).to(dev), "radius": torch.from_numpy(r).to(dev),
            "dynamic": torch.from_numpy((rng.random(n) < 0.95).astype(np.int32)).to(dev),
            "cell": 2.0 * float(r.max()) * (1 + 1e-6) + 1e-9,
            "keys": torch.full((32 * n,), -1, dtype=torch.int64, device=dev),
            "count": torch.zeros(1, dtype=torch.int32, device=dev)}


# --- what a pass cannot do without -------------------------------------------
def work(case):
    """Bytes: the caller's state in and out (128 B a body each way), the shapes
    (80 B a body) and, once a step, the contacts' warm-start records (60 B
    read, 80 B written) and manifold headers; flops: per iteration a body's
    6x6 system and solve and each constraint's two primal stamps and dual.
    Constraints per body are what these scenes hold (a standing cube rests on
    four others; a crushed one touches tens)."""
    kind, n = case["kind"], case["n"]
    if kind == "pairs":
        return {"bytes": n * 36 + 8 * n * 8, "flops": n * 27 * 8}
    steps, iters, joints = case["steps"], 10, 0
    bodies = {"stack": n + 1, "wall": n * n + 2, "adjoint": n * n + 2, "pile": n + 1, "materials": n + 1,
              "pyramid": n * (n + 1) * (2 * n + 1) // 6 + 2, "batch": 1701 * n,
              "chain": n + case.get("springs", 0) + 3}[kind]
    contacts = {"stack": 4, "wall": 4, "adjoint": 4, "pile": 6, "materials": 6, "batch": 6, "chain": 0}.get(
        kind, 40 if case.get("settle", 0) > 60 else 16) * bodies
    if kind == "chain":
        joints, iters = bodies, 20
    elif kind in ("wall", "adjoint"):
        joints = 2 * bodies
    dirs = 6 if kind == "adjoint" else 1
    step_bytes = contacts * 140 + contacts // 4 * 132 + joints * 200
    step_flops = iters * (bodies * 500 + contacts * 900 + joints * 900) * dirs
    return {"bytes": bodies * (256 + 80) * (dirs if dirs > 1 else 1) + steps * step_bytes, "flops": steps * step_flops}


# --- the same step in 64 bits --------------------------------------------------
def exact(case, seed):
    """The hanging and the spring chain stepped in f64, constraint by
    constraint; None for the scenes with contacts (an f64 collider in numpy
    takes longer than these calls may)."""
    if case["kind"] != "chain":
        return None
    w, p = _world(case, seed)
    got = {k: getattr(w, k).copy() for k in ("pos", "quat", "vel", "omega", "prev_vel")}
    got.update(k_lin=w.j_penalty_lin.copy(), lam_lin=w.j_lambda_lin.copy(), peak=w.s_peak_strain.copy())
    for _ in range(case["steps"]):
        _chain_step(w, got, p["gravity"], p["iterations"])
    return {"pos": got["pos"], "quat": got["quat"], "vel": got["vel"], "omega": got["omega"],
            "prev_vel": got["prev_vel"], "penalty_lin": got["k_lin"], "lambda_lin": got["lam_lin"],
            "lambda_ang": np.zeros_like(got["lam_lin"]), "broken": None, "peak": None, "torn": None}


def _rot(q, v):
    t = 2.0 * np.cross(q[:3], v)
    return v + q[3] * t + np.cross(q[:3], t)


def _qmul(a, b):
    return np.concatenate([a[3] * b[:3] + b[3] * a[:3] + np.cross(a[:3], b[:3]), [a[3] * b[3] - a[:3] @ b[:3]]])


def _qsub(a, b):
    return 2.0 * _qmul(a, np.concatenate([-b[:3], b[3:]]) / (b @ b))[:3]


def _qint(q, dw):
    r = q + 0.5 * _qmul(np.concatenate([dw, [0.0]]), q)
    return r / np.sqrt(r @ r)


def _skew(r):
    return np.array([[0, -r[2], r[1]], [r[2], 0, -r[0]], [-r[1], r[0], 0]])


def _matrix(q):
    return np.stack([_rot(q, e) for e in np.eye(3)], axis=1)


def _chain_order(w):
    """Bodies by (colour, index): each takes the smallest colour that none of
    its neighbours earlier in hash order has."""
    n = w.n_bodies

    def h(x):
        x ^= x >> 16
        x = x * 0x7FEB352D & 0xFFFFFFFF
        x ^= x >> 15
        x = x * 0x846CA68B & 0xFFFFFFFF
        return x ^ x >> 16

    near = [set() for _ in range(n)]
    for a, b in list(zip(w.j_body_a, w.j_body_b)) + list(zip(w.s_body_a, w.s_body_b)):
        if a >= 0 and w.mass[a] > 0 and w.mass[b] > 0:
            near[a].add(b)
            near[b].add(a)
    colour = {}
    for i in sorted(np.nonzero(w.mass > 0)[0], key=lambda i: (h(int(i)), i)):
        taken = {colour[j] for j in near[i] if j in colour}
        colour[i] = next(c for c in range(n) if c not in taken)
    return sorted(colour, key=lambda i: (colour[i], i))


def _chain_step(w, s, gravity, iterations):
    """One step of hard ball sockets and plain springs, no contacts."""
    dt, alpha, gamma, beta, kmin, kmax = 1.0 / 60.0, 0.95, 0.999, 1e4, 1.0, 1e10
    g = np.array([0.0, 0.0, gravity])
    pos, quat, vel, omega = s["pos"], s["quat"], s["vel"], s["omega"]
    n, nj = w.n_bodies, w.n_joints
    dyn = w.mass > 0
    of = [[] for _ in range(n)]
    for j in range(nj):
        for side, b in enumerate((w.j_body_a[j], w.j_body_b[j])):
            if b >= 0:
                of[b].append((True, j, side))
    for k in range(w.n_springs):
        of[w.s_body_a[k]].append((False, k, 0))
        of[w.s_body_b[k]].append((False, k, 1))

    def lin(j):
        a, b = w.j_body_a[j], w.j_body_b[j]
        pa = w.j_r_a[j] if a < 0 else pos[a] + _rot(quat[a], w.j_r_a[j])
        return pa - (pos[b] + _rot(quat[b], w.j_r_b[j]))

    c0 = np.array([lin(j) for j in range(nj)]).reshape(nj, 3)
    s["lam_lin"] *= alpha * gamma
    s["k_lin"][:] = np.clip(s["k_lin"] * gamma, kmin, kmax)
    y, yq = pos + vel * dt + np.where(dyn[:, None], g * dt * dt, 0.0), quat.copy()
    start, startq = pos.copy(), quat.copy()
    for i in np.nonzero(dyn)[0]:
        yq[i] = _qint(quat[i], omega[i] * dt)
        weight = min(max((vel[i, 2] - s["prev_vel"][i, 2]) / dt * np.sign(gravity) / abs(gravity), 0.0), 1.0)
        pos[i] = pos[i] + vel[i] * dt + g * weight * dt * dt
    quat[dyn] = yq[dyn]
    order = _chain_order(w)
    for _ in range(iterations):
        for i in order:
            R = _matrix(quat[i])
            A = np.zeros((6, 6))
            A[:3, :3] = np.eye(3) * w.mass[i] / dt ** 2
            A[3:, 3:] = R @ np.diag(w.moment[i]) @ R.T / dt ** 2
            f = np.concatenate([A[:3, :3] @ (pos[i] - y[i]), A[3:, 3:] @ _qsub(quat[i], yq[i])])
            for joint, k, side in of[i]:
                sign = 1.0 if side == 0 else -1.0
                if joint:
                    K = np.diag(s["k_lin"][k])
                    F = K @ (lin(k) - alpha * c0[k]) + s["lam_lin"][k]
                    r = sign * _rot(quat[i], w.j_r_a[k] if side == 0 else w.j_r_b[k])
                    J = np.hstack([sign * np.eye(3), _skew(-r)])
                    A += J.T @ K @ J
                    f += J.T @ F
                    H = np.outer(r, F) - np.eye(3) * (r @ F)
                    A[3:, 3:] += np.diag(np.sqrt((H * H).sum(axis=0)))
                else:
                    a, b = w.s_body_a[k], w.s_body_b[k]
                    ra, rb = _rot(quat[a], w.s_r_a[k]), _rot(quat[b], w.s_r_b[k])
                    d = pos[a] + ra - pos[b] - rb
                    length = np.sqrt(d @ d)
                    nrm, rw = d / length, ra if side == 0 else rb
                    F = w.s_stiffness[k] * (length - w.s_rest[k])
                    J = sign * np.concatenate([nrm, np.cross(rw, nrm)])
                    A += w.s_stiffness[k] * np.outer(J, J)
                    f += F * J
                    P, S = (np.eye(3) - np.outer(nrm, nrm)) / length, _skew(rw)
                    aa = -S @ P @ S + sign * (np.outer(rw, nrm) - np.eye(3) * (nrm @ rw))
                    G = np.block([[P, -P @ S], [S @ P, aa]])
                    A += np.diag(np.sqrt((G * G).sum(axis=0)) * abs(F))
            x = np.linalg.solve(A, -f)
            pos[i] = pos[i] + x[:3]
            quat[i] = _qint(quat[i], x[3:])
        for j in range(nj):
            C = lin(j) - alpha * c0[j]
            s["lam_lin"][j] += s["k_lin"][j] * C
            s["k_lin"][j] = np.minimum(s["k_lin"][j] + beta * np.abs(C), kmax)
    s["prev_vel"][:] = vel
    for i in np.nonzero(dyn)[0]:
        vel[i] = (pos[i] - start[i]) / dt
        omega[i] = _qsub(quat[i], startq[i]) / dt

"""The work that users of this package have it do, as cases to be timed.

Kinds of case, each through the package's public entry points:

  sim       a run of the device-resident simulator from a saved state (a restart, or one member of a
            parameter sweep): the state copied back, then `steps` steps, in graph replays or plain calls
  host      one step of a simulation whose state lives in host memory (copied in and back every step)
  narrow    the narrow phase and contact force over independent random pairs
  contact   the drop-in Contact_detection_GPU over a reference-style candidate list, arrays on the GPU
            or in host memory
  verlet    the drop-in Verlet_GPU (FP64 leapfrog), arrays on the GPU
  broad     the drop-in broad phase: cell keys, wall candidates, Linked_cell_hash pairs
  diff      a differentiable rollout: forward, then the gradient of a loss on the centre of mass and
            the final state

The scenes are the package's own configurations (the settling cubes, the hull pour, the batch of boxes
with mixed shapes, packed hulls), at sizes from tens of particles to a batch of two million.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mwdiem_gb300 import LIBRARY_Coarse_contact_detection as coarse
from mwdiem_gb300 import autotune, gpu_fine_contact_detection, gpu_Verlet, scene, shapes
from mwdiem_gb300.diff import DiffEngine, rollout
from mwdiem_gb300.pairbench import PairScene
from mwdiem_gb300.sim import Simulator

DT = 5e-5
LARGE_LANES = 1 | (16 << 8) | autotune.EPA_IN_PLACE  # what the autotuner settles on for many pairs
SMALL_LANES = 8 | (32 << 8) | autotune.EPA_IN_PLACE  # and for a scene of some ten thousand hulls
LANES = {"default": 8, "large": LARGE_LANES, "small": SMALL_LANES}
OUT = ("pos", "dx_all", "vel", "vel_half", "w_half_bf", "w_bf", "w", "q", "q_half", "q_all", "q_acc")


def listed():
    return [
        # the settling cubes: the smallest scene, plain step calls (launches and latency)
        dict(name="settle125", kind="sim", scene="cubes", n=125, steps=10, graph=0, lanes="default"),
        # the headline pour of 20,000 hulls, one step per graph replay as the benchmark steps it
        dict(name="pour20k", kind="sim", scene="pour", n=20000, steps=8, graph=1, lanes="small"),
        # a packed bed of hulls touching their neighbours: contact-rich steps, ragged count
        dict(name="packed30k", kind="sim", scene="packed", n=30011, steps=4, graph=1, lanes="small"),
        # the same with the options of a production run: reproducible sums, persistent history and the
        # physical law, default lanes
        dict(name="packed5k_options", kind="sim", scene="packed", n=5003, steps=4, graph=1, lanes="default",
             deterministic=True, history=True, law="physical"),
        # the batch of boxes with mixed shapes: throughput, several steps per graph
        dict(name="batch2M", kind="sim", scene="batch", n=2000000, scenes=256, steps=8, graph=4, lanes="large"),
        # a pour whose state the caller keeps in host memory
        dict(name="host20k", kind="host", n=20000),
        # independent pairs: a small set and the narrow-phase benchmark's kind of list
        dict(name="narrow3k", kind="narrow", n=3001, lanes="default"),
        dict(name="narrow2M", kind="narrow", n=2000000, lanes="large"),
        # the drop-in contact kernel, arrays kept on the GPU / passed from host memory
        dict(name="contact130k", kind="contact", n=10000, host=False),
        # the drop-in integrator: the pour's rows, vertices padded to 32
        dict(name="verlet20k", kind="verlet", n=20005, vmax=32),
        # the drop-in broad phase on the pour's centres
        dict(name="broad20k", kind="broad", n=20000),
        # calibration: 1,000 hulls, 40 steps forward and back
        dict(name="diff1k", kind="diff", n=1000, steps=40, ckpt=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sim", "sim", "sim", "host", "narrow", "narrow", "contact", "verlet", "broad", "diff"])
    if kind == "sim":
        sc = rng.choice(["cubes", "pour", "packed", "packed", "batch"])
        if sc == "cubes":
            return dict(kind=kind, scene=sc, n=rng.randint(3, 9) ** 3, steps=10, graph=rng.choice([0, 1]),
                        lanes=rng.choice(["default", "small"]))
        if sc == "batch":
            s = _log(rng, 8, 250)
            return dict(kind=kind, scene=sc, n=s * rng.randint(2000, 7800), scenes=s, steps=4,
                        graph=rng.choice([1, 4]), lanes=rng.choice(["default", "large"]))
        c = dict(kind=kind, scene=sc, n=_log(rng, 50, 60000), steps=4, graph=rng.choice([0, 1, 4]),
                 lanes=rng.choice(["default", "small", "large"]))
        if rng.random() < 0.4:
            c.update(deterministic=rng.random() < 0.5, history=rng.random() < 0.5,
                     law=rng.choice(["reference", "physical"]))
        return c
    if kind == "host":
        return dict(kind=kind, n=_log(rng, 500, 60000))
    if kind == "narrow":
        return dict(kind=kind, n=_log(rng, 100, 1900000), lanes=rng.choice(["default", "small", "large"]))
    if kind == "contact":
        host = rng.random() < 0.3
        return dict(kind=kind, n=_log(rng, 50, 2000 if host else 20000), host=host)
    if kind == "verlet":
        return dict(kind=kind, n=_log(rng, 100, 100000), vmax=rng.choice([8, 20, 32, 47, 64]))
    if kind == "broad":
        return dict(kind=kind, n=_log(rng, 100, 400000))
    return dict(kind=kind, n=_log(rng, 16, 2000), steps=rng.randint(5, 40), ckpt=rng.choice([5, 10]))


# ------------------------------------------------------------------ scenes
# (how many vertices a scene has does not depend on the seed, only which particle has how many)
def _hulls(rng, pool, n_min=12, n_max=32):
    counts = [n_min + k % (n_max - n_min + 1) for k in range(pool)]
    return [scene.fast_hull_body(rng, m, m, 0.8, 1.2) for m in counts]


def _mixed(rng, pool):
    """One third cubes, one third tetrahedra, one third hulls, of the hulls' radii."""
    out = []
    for k in range(pool):
        r = rng.uniform(0.8, 1.2)
        if k % 3 == 0:
            out.append(scene.body_from_shape(shapes.cube(2 * r / math.sqrt(3))))
        elif k % 3 == 1:
            out.append(scene.body_from_shape(shapes.tetrahedron(r * math.sqrt(8 / 3))))
        else:
            out += [scene.fast_hull_body(rng, 12 + k // 3 % 21, 12 + k // 3 % 21, 0.8, 1.2)]
    return out


def _compact(rng, base, n):
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    return scene.CompactBodies(pool=base, pick=rng.permutation(n) % len(base), quats=q)


def _batch(n, scenes, seed):
    """`scenes` boxes of 100 to 50,000 particles (log-uniform; n in all) with mixed shapes, as scene.batched_scenes
    builds them."""
    sizes = np.exp(np.random.default_rng(scenes).uniform(math.log(100), math.log(50000), size=scenes))
    sizes = np.clip(np.round(sizes * n / sizes.sum()), 100, 50000).astype(int)
    rng = np.random.default_rng(seed)
    base = _mixed(rng, 192)
    en = scene.restitution_from_damping(0.3)
    out = []
    for m in sizes:
        side = max(8.0, 2.6 * math.ceil(math.sqrt(m / 40.0)))
        centres, _ = scene.lattice(int(m), side, side, 2.6, 0.1, rng)
        walls = scene.box_walls(side, side, 2.6 * math.ceil(m / int(side // 2.6) ** 2) + 7.4, 24.0)
        out.append(scene.SceneSpec(walls=walls, bodies=_compact(rng, base, int(m)), centres=centres, en=en, et=en,
                                   en_wall=en, et_wall=en, dt=DT))
    return out


def _hull_scene(n, seed, spacing, jitter, speed, law="reference"):
    """n hulls of 12-32 points in a box, on a jittered lattice: spacing 2.6 is the pour (apart), 2.1 a
    packed bed (touching), speed the spread of the initial velocities."""
    rng = np.random.default_rng(seed)
    box = 40.0 if n >= 4000 else max(8.0, spacing * math.ceil(math.sqrt(n / 10.0)))
    centres, _ = scene.lattice(n, box, box, spacing, jitter, rng)
    en = scene.restitution_from_damping(0.3)
    return scene.SceneSpec(walls=scene.pour_walls(n, box, spacing, 1.2), bodies=_compact(rng, _hulls(rng, 96), n),
                           centres=centres, velocities=rng.normal(size=(n, 3)) * speed, en=en, et=en, en_wall=en,
                           et_wall=en, dt=DT, law=law)


def _scenes(case, seed):
    if case["scene"] == "cubes":
        return scene.settling_scene(seed=seed, n_side=round(case["n"] ** (1 / 3)))
    if case["scene"] == "batch":
        return _batch(case["n"], case["scenes"], seed)
    packed = case["scene"] == "packed"
    return _hull_scene(case["n"], seed, 2.1 if packed else 2.6, 0.05 if packed else 0.1, 0.3 if packed else 0.0,
                       case.get("law", "reference"))


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_sim(case, seed):
    sim = Simulator(_scenes(case, seed), lanes=LANES[case["lanes"]],
                    deterministic=bool(case.get("deterministic")), persistent_history=bool(case.get("history")))
    saved = {k: sim.t[k].clone() for k in ("world_verts", "force", "torque")}
    saved["mutable"] = sim.mutable.clone()
    hist = sim.w["hist_keys"].clone() if case.get("history") else None
    if case["graph"]:
        sim.capture(case["graph"])
    return dict(kind="sim", sim=sim, saved=saved, hist=hist, steps=case["steps"], graph=case["graph"])


def _prepare_host(case, seed):
    sim = Simulator(_hull_scene(case["n"], seed, 2.6, 0.1, 0.0, "physical"), lanes=SMALL_LANES)
    host = sim.host_state()
    sim.capture_host(host)
    return dict(kind="host", sim=sim, host=host)


def _prepare_narrow(case, seed):
    return dict(kind="narrow", ps=PairScene(case["n"], seed=seed, pool=256, lanes=LANES[case["lanes"]]))


def _rows(n, seed, V=32):
    """n random hulls (from a pool, turned at random) on a packed lattice: centres (n, 3) float64,
    body-frame vertices (n, V, 3) float64 padded with zeros, their counts, and the pool's inertia."""
    rng = np.random.default_rng(seed)
    base = _hulls(rng, 64, min(8, V), V)
    centres, _ = scene.lattice(n, 40.0, 40.0, 2.1, 0.05, rng)
    pool = np.zeros((len(base), V, 3))
    for k, b in enumerate(base):
        pool[k, :len(b.vertices)] = b.vertices
    pick = rng.permutation(n) % len(base)
    q = torch.from_numpy(rng.normal(size=(n, 4))).cuda()
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).view(n, 3, 3)
    pick_t = torch.from_numpy(pick).cuda()
    verts = torch.einsum("nij,nvj->nvi", R, torch.from_numpy(pool).cuda()[pick_t])
    counts = torch.tensor([len(b.vertices) for b in base], dtype=torch.int32).cuda()[pick_t]
    inertia = torch.tensor(np.array([b.inertia_bf for b in base])).cuda()[pick_t]
    size = torch.tensor([b.inertia_size for b in base], dtype=torch.float64).cuda()[pick_t]
    mass = torch.tensor([b.mass for b in base], dtype=torch.float64).cuda()[pick_t]
    return torch.from_numpy(centres).cuda(), verts, counts, inertia, size, mass


def _prepare_contact(case, seed):
    """A packed bed's candidate list as the reference's gather leaves it: every particle with its 13
    forward neighbours on the lattice, float32 arrays padded to 32 vertices."""
    n, V = case["n"], 32
    c, bv, nv, _, size, _ = _rows(n, seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    nx = int(40.0 // 2.1)
    ids = torch.arange(n, device="cuda")
    pairs = []
    ahead = [(0, 0, 1), (0, 1, -1), (0, 1, 0), (0, 1, 1)] + [(1, j, i) for j in (-1, 0, 1) for i in (-1, 0, 1)]
    for dz, dy, dx in ahead:
        i, j = ids % nx + dx, ids // nx % nx + dy
        b = ids + dx + dy * nx + dz * nx * nx
        ok = (i >= 0) & (i < nx) & (j >= 0) & (j < nx) & (b < n)
        pairs.append(torch.stack([ids[ok], b[ok]], 1))
    A, B = torch.cat(pairs).unbind(1)
    f32 = torch.float32
    vel = torch.randn((n, 3), generator=g, device="cuda") * 0.3
    w = torch.randn((n, 3), generator=g, device="cuda")
    q = torch.zeros((n, 4), device="cuda")
    q[:, 0] = 1.0
    world = (bv + c[:, None]).to(f32)
    P = len(A)
    t = [c[A].to(f32), c[B].to(f32), world[A], world[B], vel[A], vel[B], w[A], w[B], nv[A], nv[B], A.int(), B.int(),
         torch.zeros((P, 4), device="cuda"), torch.zeros((n, 3), device="cuda"), torch.zeros((n, 3), device="cuda"),
         q[A], q[B], size[A].to(f32), size[B].to(f32)]
    t = [x.contiguous() for x in t]
    if case["host"]:
        t = [x.cpu().numpy() for x in t]
    return dict(kind="contact", t=t, V=V)


def _prepare_verlet(case, seed):
    n, V = case["n"], case["vmax"]
    c, bv, _, inertia, _, mass = _rows(n, seed, V)
    g = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")

    def rnd(cols, scale):
        return torch.randn((n, cols), generator=g, **f64) * scale

    q = rnd(4, 1.0)
    q /= q.norm(dim=1, keepdim=True)
    v = rnd(3, 0.3)
    s = dict(v=v, v12=v.clone(), w12bf=rnd(3, 1.0), q12=q.clone(), q=q, qall=q.clone(), wbf=rnd(3, 1.0), w=rnd(3, 1.0),
             F=rnd(3, 2.0), T=rnd(3, 0.2), verts=(bv + c[:, None]).contiguous(), com=c, mass=mass,
             Iinv=torch.diag_embed(1.0 / inertia).contiguous(), I=torch.diag_embed(inertia).contiguous(),
             dxall=torch.zeros((n, 3), **f64))
    box = (30.0, -30.0, 30.0, -30.0, float(c[:, 2].max()) + 10.0, -10.0)
    k = gpu_Verlet.gpu_Verlet_init(timestep_size=DT, num_particles=n, num_vertices_max=V, syssize_x_max=box[0],
                                   syssize_x_min=box[1], syssize_y_max=box[2], syssize_y_min=box[3],
                                   syssize_z_max=box[4], syssize_z_min=box[5], num_part_min=5, num_part_max=n)
    return dict(kind="verlet", kernel=k, s=s)


def _prepare_broad(case, seed):
    sp = _hull_scene(case["n"], seed, 2.6, 0.1, 0.0)
    ncell, cs = sp.grid()
    W = sp.n_walls
    walls = np.array([c for _, c, _ in sp.walls])
    com = torch.from_numpy(np.concatenate([walls, sp.centres])).cuda()
    return dict(kind="broad", com=com, wn=torch.tensor(np.array([n for _, _, n in sp.walls])).cuda(),
                wc=torch.from_numpy(walls).cuda(), cs=[float(x) for x in cs], nx=int(ncell[0]), ny=int(ncell[1]), W=W,
                n=len(com), reach=6 * sp.max_particlesize,
                pairs=torch.empty((14 * len(com), 2), dtype=torch.int32, device="cuda"))


def _prepare_diff(case, seed):
    sp = _hull_scene(case["n"], seed, 2.1, 0.05, 0.3)
    eng = DiffEngine(sp, case["steps"], ckpt_every=case["ckpt"], contact_point="midpoint")
    g = torch.Generator(device="cuda").manual_seed(seed)
    target = torch.randn((case["steps"], 3), generator=g, dtype=torch.float64, device="cuda")
    return dict(kind="diff", eng=eng, x0=eng.initial_state(), law=eng.default_law(), steps=case["steps"], target=target)


# ------------------------------------------------------------------ run
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_sim(s):
    sim, saved = s["sim"], s["saved"]
    sim.mutable.copy_(saved["mutable"])
    sim.t["world_verts"].copy_(saved["world_verts"])
    if s["hist"] is not None:
        sim.w["hist_keys"].copy_(s["hist"])
    if s["graph"]:
        sim.replay(s["steps"] // s["graph"])
    else:
        sim.step(s["steps"])
    out = {k: sim.t[k] for k in OUT}
    out["world_verts"] = sim.t["world_verts"]
    return out


def _run_host(s):
    host = s["sim"].step_host(s["host"], 1)
    return {k: host[k] for k in OUT}


def _run_narrow(s):
    ps = s["ps"]
    ps.narrow()
    return {"force": ps.t["force"], "torque": ps.t["torque"], "collision": ps.w["collision"]}


def _run_contact(s):
    t = s["t"]
    for k in (12, 13, 14):  # the reference zeroes history, forces and torques every step
        t[k][...] = 0
    F, T, hist, coll = gpu_fine_contact_detection.Contact_detection_GPU(
        *t[:13], 1e5, 0.372, 0.372, 0.5, 1e5, 0.372, 0.372, 0.5, 0, t[13], t[14], s["V"], t[15], t[16], DT, *t[17:])
    return {"force": F, "torque": T, "history": hist, "collision": coll}


def _run_verlet(s):
    d = s["s"]
    r = gpu_Verlet.gpu_Verlett(s["kernel"], d["v"], d["v12"], d["w12bf"], d["q12"], d["q"], d["qall"], d["wbf"], d["w"],
                               d["F"], d["T"], d["verts"], d["com"], d["mass"], d["Iinv"], d["I"], d["dxall"])
    return list(r)


def _run_broad(s):
    keys = coarse.cell_keys(s["com"], *s["cs"], s["nx"], s["ny"])
    walls = coarse.wall_pairs(s["com"], s["wn"], s["wc"], s["W"], s["W"], s["n"], s["reach"])
    cells = coarse.linked_cell_pairs(keys, s["W"], s["n"], s["nx"], s["ny"])
    buf = s["pairs"]  # the candidate list, in the buffer that the caller's gather reads
    m = len(walls) + len(cells)
    buf[:len(walls)] = walls
    buf[len(walls):m] = cells
    buf[m:] = -1
    return {"keys": keys, "pairs": buf}


def _run_diff(s):
    x0 = s["x0"].clone().requires_grad_(True)
    law = s["law"].clone().requires_grad_(True)
    com, xT = rollout(s["eng"], x0, law, s["steps"])
    loss = ((com - s["target"]) ** 2).mean() + (xT[:, 3:6] ** 2).mean()
    loss.backward()
    return {"com": com, "final": xT, "grad_state": x0.grad, "grad_law": law.grad}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes and operations of one pass that the path cannot do without: state, vertices and lists read
    or written once per step, the dot products of about five support queries per near pair and ten per
    contact, the FP64 arithmetic of the integrators."""
    n = case["n"]
    k = case["kind"]
    if k in ("sim", "host"):
        steps = case.get("steps", 1)
        sc = case.get("scene", "pour")
        verts = {"cubes": 8, "batch": 11}.get(sc, 22)
        near, touch = {"cubes": (3, 1), "packed": (3, 1)}.get(sc, (0.7, 0.05))
        step_b = n * (536 + 32 * verts + 56 + 8 * near)
        step_f = n * (near * 5 * 2 * verts * 5 + touch * (10 * 2 * verts * 5 + 4000) + 400 + 18 * verts)
        link = n * 416 if k == "host" else 0
        return {"bytes": steps * step_b + link, "flops": steps * step_f}
    if k == "narrow":
        return {"bytes": n * (2 * 36 * 16 + 2 * 180 + 12), "flops": n * (5 * 72 * 5 + 0.6 * (11 * 72 * 5 + 8000))}
    if k == "contact":
        P = 13 * n
        return {"bytes": P * (2 * 20 * 12 + 2 * 56 + 20), "flops": P * (2 * 40 * 5 + 0.1 * 8000)}
    if k == "verlet":
        return {"bytes": n * (48 * case["vmax"] + 8 * (16 * 3 * 2 + 12)), "flops": n * (21 * case["vmax"] + 450)}
    if k == "broad":
        return {"bytes": n * (24 + 8 + 8 + 8 * 8 + 8), "flops": n * 60}
    return {"bytes": case["steps"] * n * (256 * 6 + 32 * 3), "flops": case["steps"] * n * (1600 + 1400 * 1.5)}


# ------------------------------------------------------------------ exact
def _qmul(a, b):
    aw, av, bw, bv = a[:, :1], a[:, 1:], b[:, :1], b[:, 1:]
    return torch.cat([aw * bw - (av * bv).sum(1, keepdim=True), bv * aw + av * bw + torch.linalg.cross(av, bv)], 1)


def _conj(q):
    return q * torch.tensor([1.0, -1.0, -1.0, -1.0], dtype=q.dtype, device=q.device)


def _turn(q, v):
    zero = torch.zeros_like(v[:, :1])
    return _qmul(q, _qmul(torch.cat([zero, v], 1), _conj(q)))[:, 1:]


def _increment(w, s):
    a = w.norm(dim=1, keepdim=True)
    return torch.cat([torch.cos(a * s), w / torch.where(a > 0, a, torch.ones_like(a)) * torch.sin(a * s)], 1)


def exact(case, seed):
    """The integrator's step in plain float64.  The other kinds end in a contact search (which face of a
    polytope, which pairs) or return whole numbers: no value in closed form."""
    if case["kind"] != "verlet":
        return None
    d = prepare(case, seed)["s"]
    d = {k: x.clone() for k, x in d.items()}
    lo, m, n, V = 5, d["mass"][5:, None], case["n"], case["vmax"]
    o = {k: d[k][lo:] for k in ("v", "v12", "w12bf", "q12", "q", "qall", "wbf", "w", "F", "T", "com", "dxall")}
    I = torch.diagonal(d["I"][lo:], dim1=1, dim2=2)
    Ii = torch.diagonal(d["Iinv"][lo:], dim1=1, dim2=2)
    v12 = o["v12"] + o["F"] / m * DT
    alpha = Ii * (_turn(_conj(o["q"]), o["T"]) - torch.linalg.cross(o["wbf"], I * o["wbf"]))
    w12 = o["w12bf"] + alpha * DT
    q12 = _qmul(_increment(o["w"], DT / 2), o["q12"])
    dx = v12 * DT
    q = _qmul(_increment(_turn(q12, w12 + alpha * DT / 4), DT / 4), q12)
    wbf = w12 + alpha * DT / 2
    new = dict(v12=v12, q=q, wbf=wbf, w12bf=w12, w=_turn(q, wbf), q12=q12, v=v12 + o["F"] * DT / m, com=o["com"] + dx,
               qall=_qmul(q, o["q"]), dxall=o["dxall"] + dx)
    rel = (d["verts"][lo:] - o["com"][:, None]).reshape(-1, 3)
    turned = _turn(q.repeat_interleave(V, 0), rel).view(n - lo, V, 3) + o["com"][:, None] + dx[:, None]
    for k, x in new.items():
        d[k][lo:] = x
    d["verts"][lo:] = turned
    return [d[k] for k in ("v12", "q", "wbf", "w12bf", "w", "q12", "v", "com", "verts", "qall", "dxall")]

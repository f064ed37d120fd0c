"""Timed workloads of the cloth step and the calls around it.

Each case is one pass through the public entry points with the arguments a
program has in hand: a frame of one cloth or of a batch (state up, scStepCloth,
state back), the mesh update a renderer follows it with, the warm-start
network's forward and training step, and vertex normals on caller-owned buffers.
Sizes, materials and colliders are those of solidcloth_b200.scenes and of the
tests; the ranges drawn from lie around them.
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from solidcloth_b200 import api, learned, scenes


def listed():
    return [
        # smallest frame: the 32 x 32 two-pin cloth without colliders, drawn after
        # every step (step, mesh update, vertex and normal buffers)
        {"name": "drop_32", "kind": "frame", "n": 32, "scene": "drop", "fast": False, "mesh": True, "warm": 5},
        # the reference's default solver: mass-spring links with its exit test, as the
        # demo runs it, on an odd size
        {"name": "links_45", "kind": "frame", "n": 45, "scene": "links", "fast": False, "mesh": False, "warm": 5},
        # the live self-proximity path: a cloth folded in half on the floor
        {"name": "fold_48", "kind": "frame", "n": 48, "scene": "fold", "fast": False, "mesh": False, "warm": 4},
        # an ordinary single cloth: draped on a sphere SDF, continuous self-collision
        {"name": "sdf_128", "kind": "frame", "n": 128, "scene": "sdf", "fast": False, "mesh": False, "warm": 12},
        # the same drape at an odd size in the fast solver build, on one fixed solver
        # kernel as the learned comparison runs it (the fast build's bits depend on the kernel)
        {"name": "sdf_91_fast", "kind": "frame", "n": 91, "scene": "sdf", "fast": True, "mesh": False, "warm": 12},
        # the benchmark's default: 256 x 256 on an icosphere mesh over a ground plane,
        # vertex, triangle and edge contacts, continuous self-collision
        {"name": "mesh_256", "kind": "frame", "n": 256, "scene": "mesh", "fast": False, "mesh": False, "warm": 12},
        # uneven cloths stepped as one batch (the batch configuration's distribution)
        {"name": "batch_12", "kind": "batch", "count": 12, "lo": 16, "hi": 128, "warm": 8},
        # the warm-start network over a 256 x 256 cloth's particles
        {"name": "network_forward", "kind": "network", "rows": 65536, "train": False},
        # one training step at the trainer's batch size: gradients, then Adam
        {"name": "network_train", "kind": "network", "rows": 65536, "train": True},
        # normals of a 256 x 256 mesh in a program that must not allocate
        {"name": "normals_256", "kind": "normals", "n": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.randrange(10)
    if k < 6:
        scene = ("drop", "links", "fold", "sdf", "sdf", "mesh")[k]
        lo, hi = {"drop": (16, 160), "links": (16, 128), "fold": (16, 64), "sdf": (24, 220), "mesh": (48, 240)}[scene]
        return {"kind": "frame", "n": _log_int(rng, lo, hi), "scene": scene,
                "fast": scene == "sdf" and rng.random() < 0.5, "mesh": scene == "drop" and rng.random() < 0.5,
                "warm": 4 if scene == "fold" else rng.randint(4, 12)}
    if k == 6:
        return {"kind": "batch", "count": rng.randint(2, 12), "lo": 16, "hi": rng.randint(40, 120), "warm": rng.randint(4, 8)}
    if k < 9:
        return {"kind": "network", "rows": _log_int(rng, 1000, 120000), "train": k == 8}
    return {"kind": "normals", "n": _log_int(rng, 12, 255)}


# ------------------------------------------------------------------ scenes
def _scene(case, seed):
    """(scene, state or None) of a frame case"""
    n, kind = case["n"], case["scene"]
    if kind in ("drop", "links"):
        p = scenes.Params(iterations=10, substeps=4)
        if kind == "links":
            p = scenes.Params(iterations=50, substeps=4, fem=False, dihedral=False, fixed_iterations=False,
                              stretch=1e3, shear=5e2, bend=2.0)
        return scenes.make_grid_scene(f"{kind}_{n}", n, 1.0, 0.0, p, pinned_corners=(1, 3), seed=seed), None
    if kind == "fold":
        # the lower layer rests on the floor, the upper one starts a grid step above it
        # (the crease keeps its length) and settles onto it
        p = scenes.Params(thickness=0.005, tolerance=0.005, friction=0.3, iterations=15, substeps=8,
                          flags=scenes.CF_SELF | scenes.CF_WALLS)
        s = scenes.make_grid_scene(f"fold_{n}", n, 1.0, p.thickness, p, seed=seed)
        s.walls = np.array([-20.0, 0.0, -20.0, 20.0, 20.0, 20.0], dtype=np.float32)
        return s, scenes.folded(s, gap=s.inc)
    # drapes: released two centimetres above the collider, so that a few frames bring contact
    rng = np.random.default_rng(seed)
    drop = float(rng.uniform(0.015, 0.025))
    if kind == "sdf":
        s = scenes.cfg1(seed=seed, n=n)
        lift = np.float32(0.3 + drop - 0.7)
    else:
        s = scenes.cfg2(seed=seed, n=n)
        lift = np.float32(0.5 + drop - 1.0)
    s.offset = (s.offset + np.array([0, lift, 0], np.float32)).astype(np.float32)
    s.positions = (s.positions + np.array([0, lift, 0], np.float32)).astype(np.float32)
    return s, None


def _batch_scenes(case, seed):
    out = scenes.cfg3_instances(count=case["count"], seed=3, lo=case["lo"], hi=case["hi"])
    rng = np.random.default_rng(seed)
    for s in out:
        # the instances' sizes and colliders stay, the seed moves every particle;
        # lowered to just above the colliders' tops
        s.positions = (s.positions + rng.uniform(-5e-4, 5e-4, s.positions.shape)).astype(np.float32)
        s.positions[:, 1] -= np.float32(0.38)
    return out


def _stepped(patch, dt, frames, state):
    """the state (positions, previous positions, velocities) after `frames` frames"""
    if state is not None:
        patch.model.set_state(*state)
    for _ in range(frames):
        patch.step(dt)
    m = patch.model
    return m.positions(), m.prev_positions(), m.velocities()


def _free(world, patch):
    patch.free()
    world.free()


class _Handle:
    """a patch and its world, freed with it"""

    def __init__(self, world, patch):
        self.patch = patch
        weakref.finalize(self, _free, world, patch)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        sc, state = _scene(case, seed)
        h = _Handle(*api.load_scene(sc))
        p = h.patch
        now = _stepped(p, sc.dt, case["warm"], state)
        if case["fast"]:
            p.model.set_fast_math(True)
            p.model.set_cluster_variant(0)
        p.step(sc.dt)           # the handle of a running program: its frame graph exists
        p.synchronize()
        return {"kind": kind, "handle": h, "dt": sc.dt, "state": now, "mesh": case["mesh"]}
    if kind == "batch":
        b = api.load_batch(_batch_scenes(case, seed))
        h = _Handle(b.world, b)
        now = _stepped(b, 1.0 / 60.0, case["warm"], None)
        b.step(1.0 / 60.0)
        b.synchronize()
        return {"kind": "frame", "handle": h, "dt": 1.0 / 60.0, "state": now, "mesh": False}
    if kind == "network":
        return _network(case, seed)
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    pos = torch.from_numpy(scenes.grid_positions(n, 1.0 / (n - 1), (0, 0, 0))).cuda()
    pos[:, 1] = 0.1 * torch.sin(7 * pos[:, 0]) * torch.cos(5 * pos[:, 2]) + 1e-3 * torch.rand(n * n, device="cuda", generator=g)
    tri = torch.from_numpy(scenes.grid_triangles(n).astype(np.int32)).cuda()
    return {"kind": kind, "pos": pos.contiguous(), "tri": tri, "out": torch.empty_like(pos)}


def _network(case, seed):
    """Rows with the features' magnitudes on a drape, weights with a non-zero output
    layer, and (training) the moments of a run under way"""
    S = case["rows"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    scale = torch.tensor([5e-3, 5e-3, 5e-3, 1.0, 1.0, 1.0, 0.05, 0.6, 0.6, 0.6, 0.3, 1e-3], device="cuda")
    X = torch.randn((S, learned.IN), device="cuda", generator=g) * scale
    T = torch.randn((S, learned.OUT), device="cuda", generator=g) * 1e-3 + 0.02 * X[:, :3]
    prm = torch.from_numpy(learned.init_params(seed)).cuda()
    prm += 0.02 * torch.randn(prm.shape, device="cuda", generator=g)
    norm = torch.cat([torch.zeros(learned.IN, device="cuda"), 1.0 / scale, torch.full((learned.OUT,), 1e-3, device="cuda")])
    st = {"kind": "network", "train": case["train"], "X": X, "T": T, "prm": prm, "norm": norm,
          "Y": torch.empty((S, learned.OUT), device="cuda")}
    if case["train"]:
        st["m"] = 1e-3 * torch.randn(prm.shape, device="cuda", generator=g)
        st["v"] = 1e-5 + 1e-5 * torch.rand(prm.shape, device="cuda", generator=g)
        st["grad"] = torch.zeros_like(prm)
        st["loss"] = torch.zeros(1, device="cuda")
        st["step"] = 200
    return st


def run(state):
    kind = state["kind"]
    if kind == "frame":
        p = state["handle"].patch
        p.model.set_state(*state["state"])
        p.step(state["dt"])
        if state["mesh"]:
            p.update_mesh()
            verts, normals, _ = p.mesh_buffers()
            return {"vertices": verts, "normals": normals}
        return {"positions": p.model.positions(), "velocities": p.model.velocities()}
    lib = api.lib()
    s = torch.cuda.current_stream().cuda_stream
    if kind == "network":
        X, prm, norm = state["X"], state["prm"], state["norm"]
        if not state["train"]:
            lib.scMlpForward(X.data_ptr(), X.shape[0], prm.data_ptr(), norm.data_ptr(), state["Y"].data_ptr(), s)
            return state["Y"]
        lib.scMlpGradients(X.data_ptr(), state["T"].data_ptr(), X.shape[0], prm.data_ptr(), norm.data_ptr(),
                           state["grad"].data_ptr(), state["loss"].data_ptr(), s)
        lib.scMlpAdamStep(prm.data_ptr(), state["grad"].data_ptr(), state["m"].data_ptr(), state["v"].data_ptr(),
                          state["step"], 1e-4, s)
        state["step"] += 1
        return {k: state[k] for k in ("grad", "loss", "prm", "m", "v")}
    lib.scComputeVertexNormalsNoAlloc(state["pos"].data_ptr(), state["pos"].shape[0], state["tri"].data_ptr(),
                                      state["tri"].shape[0], state["out"].data_ptr(), s)
    return state["out"]


# ---------------------------------------------------------------- work, exact
def work(case):
    kind = case["kind"]
    if kind == "network":
        S, P = case["rows"], learned.NPARAM
        macs = 12 * 64 + 64 * 64 * 2 + 64 * 3
        if case["train"]:
            return {"bytes": S * 4 * 15 + P * 4 * 8, "flops": 2.0 * S * (3 * macs - 12 * 64)}
        return {"bytes": S * 4 * 15 + P * 4, "flops": 2.0 * S * macs}
    if kind == "normals":
        n = case["n"]
        tris = 2 * (n - 1) ** 2
        return {"bytes": 24 * n * n + 12 * tris, "flops": 150.0 * tris}
    if kind == "batch":
        sides = [s.n for s in scenes.cfg3_instances(count=case["count"], seed=3, lo=case["lo"], hi=case["hi"])]
        p = scenes.Params(iterations=15, substeps=8)
    else:
        sides = [case["n"]]
        p = _scene({**case, "n": 4}, 0)[0].params
    N = sum(n * n for n in sides)
    T = sum(2 * (n - 1) ** 2 for n in sides)
    B = sum(3 * n * n - 8 * n + 5 for n in sides)            # interior edges
    E = sum((n - 1) * (3 * n - 1) for n in sides)
    L = 6 * N if not p.fem else 0
    # state up and back, every constraint's constants, the mesh's triangles and edges
    data = (36 + 24) * N + (48 * T if p.fem else 16 * L) + (16 * B if p.dihedral else 0) + 12 * T + 8 * E
    it = p.iterations if p.fixed_iterations else 1           # the exit test needs one iteration at least
    proj = it * (T * 250.0 if p.fem else L * 40.0) + ((it + 1) // 2 * B * 300.0 if p.dihedral else 0.0)
    return {"bytes": float(data), "flops": p.substeps * proj}


def _mlp(prm, X, norm):
    sizes = [(64, 12), (64,), (64, 64), (64,), (64, 64), (64,), (3, 64), (3,)]
    parts, at = [], 0
    for s in sizes:
        k = math.prod(s)
        parts.append(prm[at:at + k].reshape(s))
        at += k
    h = (X - norm[:12]) * norm[12:24]
    for l in range(3):
        h = torch.nn.functional.gelu(h @ parts[2 * l].T + parts[2 * l + 1], approximate="tanh")
    return h @ parts[6].T + parts[7]


def exact(case, seed):
    kind = case["kind"]
    if kind == "network":
        st = _network(case, seed)
        X, T, norm = st["X"].double(), st["T"].double(), st["norm"].double()
        prm = st["prm"].double().requires_grad_(case["train"])
        y = _mlp(prm, X, norm)
        if not case["train"]:
            return y * norm[24:]
        loss = ((y - T / norm[24:]) ** 2).mean()
        loss.backward()
        g = prm.grad
        m = 0.9 * st["m"].double() + 0.1 * g
        v = 0.999 * st["v"].double() + 0.001 * g * g
        t = st["step"]
        new = prm.detach() - 1e-4 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
        return {"grad": g, "loss": loss.detach().reshape(1), "prm": new, "m": m, "v": v}
    if kind == "normals":
        st = prepare(case, seed)
        p, t = st["pos"].double(), st["tri"].long()
        a, b, c = (p[t[:, k]] for k in range(3))
        nt = torch.nn.functional.normalize(torch.linalg.cross(b - a, c - a), dim=1)
        unit = [torch.nn.functional.normalize(e, dim=1) for e in (b - a, c - b, a - c)]
        out = torch.zeros_like(p)
        for k in range(3):
            w = torch.acos((-(unit[k] * unit[k - 1]).sum(1)).clamp(-1, 1))
            out.index_add_(0, t[:, k], w[:, None] * nt)
        return torch.nn.functional.normalize(out, dim=1)
    # frames: a Gauss-Seidel sweep's result depends on the order of the constraints and
    # on decisions at thresholds (contacts, skipped bends, the exit test): no such value
    return None

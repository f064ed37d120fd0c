"""The tile solver (the automatic mode's kernel) against the one-kernel-per-colour
path: the same projections in the same order, so bit-identical states, at the
sizes where its tiling changes; and the projections' branch-free division and
square root against the oracle on states that leave their range."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu

TILE = 5


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a, np.float32).view(np.uint32),
                          np.ascontiguousarray(b, np.float32).view(np.uint32))


def _states(build, frames, dt, mode):
    out = []
    p = build()
    if mode:
        p.model.set_solver_mode(mode)
    for _ in range(frames):
        p.step(dt)
        out.append((p.model.positions(), p.model.velocities(), p.model.solver_iterations()))
    kind = p.model.solver_choice()[0][0]
    status = p.status()
    p.free()
    return out, kind, status


def _compare(build, frames, dt=1.0 / 60.0, tile=True):
    got, kind, status = _states(build, frames, dt, 0)
    want, _, same = _states(build, frames, dt, 3)
    assert (kind == TILE) == tile
    assert status == same and status & 256 == 0      # 256: an exchange wait gave up
    for f, (a, b) in enumerate(zip(got, want)):
        assert _same(a[0], b[0]) and _same(a[1], b[1]), f
        assert a[2] == b[2], (f, a[2], b[2])


# 2 x 2 and 3 x 50: a handful of records a colour; 27 x 25 / 28 x 25: the last size in
# one closed tile (below 700 particles) and the first split one; 151: ragged tiles
@pytest.mark.parametrize("shape", [(2, 2), (3, 50), (27, 25), (28, 25), (38, 39), (39, 39), (151, 20), (100, 100)])
@pytest.mark.parametrize("kind", ["fem", "bends", "links", "exit", "residual"])
def test_grids(shape, kind):
    from solidcloth_b200 import api
    nx, ny = shape
    rng = np.random.default_rng(nx * 1000 + ny)
    noise = rng.uniform(-2e-3, 2e-3, (nx * ny, 3)).astype(np.float32)

    def build():
        w = api.CollisionWorld()
        w.add_sphere((0.0, -0.05, 0.0), 0.04)
        p = api.ClothPatch(w)
        prm = scenes.Params(iterations=6, substeps=2, thickness=0.005, tolerance=0.005, flags=scenes.CF_VERTICES,
                            dihedral=kind != "fem", fem=kind not in ("links", "exit"), fixed_iterations=kind != "exit",
                            stretch=1e3, shear=5e2, bend=2.0)
        p.model.set_params(prm)
        p.set_num_steps(prm.substeps)
        p.init_grid(nx, ny, 0.02, (0.01 * nx, 0.0, 0.01 * nx), True, True)
        p.model.set_masses(np.where(np.arange(nx * ny) % 37 == 0, 0.0, 1e-3 + 1e-5 * (np.arange(nx * ny) % 11)))
        p.model.set_positions(p.model.positions() + noise)
        if kind == "residual":
            p.model.set_residual_target(5e-4, 40, metres=True)
        return p
    _compare(build, 3)


@pytest.mark.parametrize("count,lo,hi", [(3, 16, 24), (4, 30, 90), (2, 128, 128)])
def test_batches(count, lo, hi):
    """closed tiles, several per CTA or one; instances split over tiles beside them"""
    from solidcloth_b200 import api
    insts = scenes.cfg3_instances(count=count, seed=7, lo=lo, hi=hi)
    for s in insts:
        s.positions[:, 1] -= np.float32(0.38)
    _compare(lambda: api.load_batch(insts), 2)


def test_contacts_take_the_guarded_launch():
    """continuous contacts across a split cloth: the tile launch steps aside for the
    solver that reaches any particle; without contacts it does not"""
    from solidcloth_b200 import api
    sc, state = scenes.ccd_scene(44)

    def build():
        _, p = api.load_scene(sc)
        p.model.set_state(*state)
        return p
    sc.params.flags &= ~scenes.CF_SELF
    _compare(build, 2, sc.dt)


@pytest.mark.parametrize("case", ["flat", "coincident", "huge", "tiny", "pinned"])
def test_projection_range(case):
    """Operands outside the branch-free forms' range (met constraints, zero-length
    edges, huge and tiny cloths, fully pinned triangles) take the plain operators:
    bit-identical to the oracle, NaNs in the same places."""
    from solidcloth_b200 import api
    from oracle.bridge import PortCloth
    PortCloth.set_portable_math(True)
    sc = scenes.cfg0()
    n = sc.n
    pos = scenes.grid_positions(n, sc.inc, sc.offset)
    if case == "coincident":
        pos[40:44] = pos[40]
        pos[300] = pos[301]
    if case == "huge":
        pos = pos * np.float32(3e9)
    if case == "tiny":
        pos = pos * np.float32(1e-9)
    if case == "pinned":
        sc.masses = sc.masses.copy()
        sc.masses[:4 * n] = 0.0
        pos = sc.positions
    vel = np.zeros_like(pos)
    w, p = api.load_scene(sc)
    o = PortCloth.from_scene(sc)
    o.set_tri_order(p.model.constraint_order(0)[0])
    o.set_bend_order(p.model.constraint_order(1)[0])
    p.model.set_state(pos, pos, vel)
    o.set_state(pos, pos, vel)
    for f in range(2):
        p.step(sc.dt)
        o.step(sc.dt)
        g, c = p.model.positions(), o.positions()
        assert np.array_equal(np.isnan(g), np.isnan(c)), f
        assert _same(np.nan_to_num(g), np.nan_to_num(c)), f


@pytest.mark.parametrize("n,colliders", [(24, 1), (45, 1), (60, 3)])
@pytest.mark.parametrize("fixed", [True, False])
def test_triangle_and_edge_contacts(n, colliders, fixed):
    """collider contacts on triangles and edges in one closed tile (24 x 24) and across
    tiles, with one collider and with three (a mesh, a sphere, an SDF): states and
    the reported contact lists equal the per-colour path's"""
    from solidcloth_b200 import api
    sc = scenes.cfg2(n=n, level=3)
    sc.positions = (sc.positions + np.array([0, -0.485, 0], np.float32)).astype(np.float32)
    sc.params.iterations, sc.params.substeps = 6, 4
    sc.params.fixed_iterations = fixed
    if colliders == 3:
        sc.spheres.append(((0.15, 0.3, 0.1), 0.2))
        sc.sdfs.append(scenes.sphere_sdf((-0.15, 0.3, -0.1), 0.2, 31, 0.1))
    runs = []
    for mode in (0, 3):
        w, p = api.load_scene(sc)
        if mode:
            p.model.set_solver_mode(mode)
        for _ in range(4):
            p.step(sc.dt)
        if not mode:
            assert p.model.solver_choice()[0][0] == TILE
        runs.append([p.model.positions(), p.model.velocities(), p.model.solver_iterations(), p.status()] +
                    [x for k in range(3) for x in p.model.contacts(k)])
        p.free()
        w.free()
    assert len(runs[0][6]) > 0 and len(runs[0][8]) > 0
    for k, (a, b) in enumerate(zip(*runs)):
        assert _same(a, b) if isinstance(a, np.ndarray) and a.dtype == np.float32 else np.array_equal(a, b), k

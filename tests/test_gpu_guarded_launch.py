"""Clothes split into tiles that do meet self contacts: the launches behind the tile
launch (one closed tile, the cluster and the grid solver, by size and by the number
of contact colours) against the per-colour path, bit for bit."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu

TILE, CLUSTER, GRID, KERNELS = 5, 1, 2, 3


def _flap(n, rows, iterations=3, substeps=2):
    """a cloth on the floor, its last rows folded over: rows == n // 2 folds it in half"""
    inc = 1.0 / (n - 1)
    t = min(0.005, 0.35 * inc)
    p = scenes.Params(thickness=t, tolerance=t, friction=0.3, iterations=iterations, substeps=substeps, flags=scenes.CF_SELF | scenes.CF_WALLS)
    sc = scenes.make_grid_scene("flap", n, 1.0, p.thickness, p, seed=1)
    noise = np.random.default_rng(1).uniform(-0.1 * inc, 0.1 * inc, (n * n, 3))
    sc.positions = (scenes.grid_positions(n, sc.inc, sc.offset) + noise).astype(np.float32)
    sc.walls = np.array([-20.0, 0.0, -20.0, 20.0, 20.0, 20.0], dtype=np.float32)
    pos = sc.positions.copy().reshape(n, n, 3)
    for k in range(rows):
        pos[:, n - 1 - k, 2] = pos[:, n - 1 - 2 * rows + k, 2]
        pos[:, n - 1 - k, 1] += np.float32(sc.inc)
    pos = pos.reshape(-1, 3).astype(np.float32)
    return sc, (pos, pos.copy(), np.zeros_like(pos))


def _colours(p):
    return sum(int(np.count_nonzero(p.model.contact_colours(k))) for k in (2, 3))


def _run(build, frames, dt, mode, faults=()):
    """states after each frame, the contact colours of each frame's last substep, the solver kind"""
    p = build()
    p.model.set_solver_mode(mode)
    p.model.set_launch_fault(*faults)
    out, colours = [], []
    for _ in range(frames):
        p.step(dt)
        out.append([np.ascontiguousarray(a, np.float32).view(np.uint32) for a in (p.model.positions(), p.model.velocities())])
        colours.append(_colours(p))
    kind, status = p.model.solver_choice()[0][0], p.status()
    p.free()
    return out, colours, kind, status


def _compare(build, frames, dt, faults=()):
    got, c0, kind, s0 = _run(build, frames, dt, 0, faults)
    want, c1, _, s1 = _run(build, frames, dt, KERNELS)
    assert kind == TILE and c0 == c1 and s0 == s1 and s0 & 256 == 0
    for f, (a, b) in enumerate(zip(got, want)):
        for x, y in zip(a, b):
            assert np.array_equal(x, y), f
    return c0


# 40: the last size in one tile; 41: split, with one closed tile behind; 96 and 97: the
# last size with one and the first without. Few and many colours: both launches of a guard.
@pytest.mark.parametrize("n,rows", [(40, 4), (41, 2), (41, 4), (48, 24), (64, 4), (96, 3), (96, 6), (97, 4)])
def test_live_proximity(n, rows):
    from solidcloth_b200 import api
    sc, state = _flap(n, rows)

    def build():
        p = api.load_scene(sc)[1]
        p.model.set_state(*state)
        return p
    assert max(_compare(build, 4, sc.dt)) > 0


def test_both_sides_of_the_colour_rule():
    """fewer contact colours than one in 120 particles, and more"""
    from solidcloth_b200 import api
    seen = []
    for n, rows in ((80, 2), (96, 2), (64, 4)):
        sc, state = _flap(n, rows, 15, 8)

        def build():
            p = api.load_scene(sc)[1]
            p.model.set_state(*state)
            return p
        seen += [c / (n * n // 120) for c in _compare(build, 4, sc.dt)]
    assert any(0 < c < 1 for c in seen) and any(c >= 1 for c in seen), seen


def test_with_collider_contacts():
    """triangle and edge contacts of a collider beside the self contacts, in the closed tile behind"""
    from solidcloth_b200 import api
    sc, state = _flap(48, 4)
    sc.params.flags |= scenes.CF_VERTICES | scenes.CF_TRIANGLES | scenes.CF_EDGES
    sc.masses = np.ones(sc.num_vertices, np.float32)
    sc.meshes.append(scenes.icosphere(3, 0.2, (0.0, -0.195, 0.0)))
    found = []

    def build():
        p = api.load_scene(sc)[1]
        p.model.set_state(*state)
        step = p.step
        def stepped(dt):
            step(dt)
            found.append([len(p.model.contacts(k)[0]) for k in (1, 2)])
        p.step = stepped
        return p
    assert max(_compare(build, 3, sc.dt)) > 0
    assert min(max(f[k] for f in found) for k in (0, 1)) > 0


@pytest.mark.parametrize("n,faults", [(44, ()), (44, (CLUSTER,))])
def test_continuous_contacts(n, faults):
    """behind a split cloth: the cluster solver, and the grid solver where that one is not launched"""
    from solidcloth_b200 import api
    sc, state = scenes.ccd_scene(n)
    sc.params.flags &= ~scenes.CF_SELF

    def build():
        p = api.load_scene(sc)[1]
        p.model.set_state(*state)
        return p
    assert max(_compare(build, 2, sc.dt, faults)) > 0


@pytest.mark.parametrize("count,n", [(3, 40), (60, 30)])
def test_batch_with_one_instance_in_contact(count, n):
    """the cluster solver behind a small batch, the grid solver behind one of 54,000 particles;
    an instance out of contact moves as in a batch of its own"""
    from solidcloth_b200 import api
    sc, state = scenes.ccd_scene(n)
    sc.params.flags &= ~scenes.CF_SELF
    calm = (sc.positions, sc.positions, np.zeros_like(sc.positions))
    every = [state] + [calm] * (count - 1)
    whole = tuple(np.concatenate([s[k] for s in every]).astype(np.float32) for k in range(3))

    def build():
        b = api.load_batch([sc] * count)
        b.model.set_state(*whole)
        return b
    assert max(_compare(build, 2, sc.dt)) > 0
    got = _run(build, 2, sc.dt, 0)[0]

    def alone():
        p = api.load_scene(sc)[1]
        p.model.set_state(*calm)
        return p
    one = _run(alone, 2, sc.dt, 0)[0]
    for a, b in zip(got, one):
        assert np.array_equal(a[0][n * n:2 * n * n], b[0])

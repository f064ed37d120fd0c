"""Solver launches that fail (refused on the host): the step either is solved by the
per-colour kernels or reports an error; never a frame without a solve."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu

CLUSTER, GRID, KERNELS, TILE = 1, 2, 3, 5


def _bits(p):
    return [np.ascontiguousarray(a, np.float32).view(np.uint32) for a in (p.model.positions(), p.model.velocities())]


def _drape():
    from solidcloth_b200 import api
    sc = scenes.cfg1(n=40)
    sc.positions[:, 1] -= np.float32(0.39)
    return api.load_scene(sc)[1], sc.dt


def _run(faults, mode, direct=False):
    p, dt = _drape()
    p.model.set_solver_mode(mode)
    p.model.set_launch_fault(*faults)
    if direct:
        p.set_direct_launch(True)
    for _ in range(3):
        p.step(dt)
    out = _bits(p)
    p.free()
    return out


@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("faults,mode", [((TILE,), 0), ((CLUSTER,), CLUSTER), ((GRID,), GRID)])
def test_per_colour_kernels_take_over(faults, mode, direct):
    got, want = _run(faults, mode, direct), _run((), KERNELS)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("direct", [False, True])
def test_error_where_nothing_takes_over(direct):
    """a split cloth with continuous collision: the tile launch is made, the one behind it is not"""
    p, dt = _drape()
    p.set_direct_launch(direct)
    p.step(dt)
    p.model.set_launch_fault(CLUSTER, GRID)
    assert p.model.solver_choice()[0][0] == TILE
    with pytest.raises(RuntimeError, match="solver launch failed"):
        p.step(dt)
    p.model.set_launch_fault()
    state = p.model.positions(), p.model.prev_positions(), p.model.velocities()
    p.step(dt)                                      # and it goes on
    q, _ = _drape()
    q.model.set_state(*state)
    q.step(dt)
    for a, b in zip(_bits(p), _bits(q)):
        assert np.array_equal(a, b)
    p.free()
    q.free()

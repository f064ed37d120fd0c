"""Self contacts of a cloth in one closed tile, solved from records in colour order:
the states and the contacts (weights, side, normal, multiplier) of the per-colour
path, bit for bit."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _run(n, kind, fixed, mode):
    from solidcloth_b200 import api
    if kind == "fold":
        p = scenes.Params(thickness=0.005, tolerance=0.005, friction=0.3, iterations=6, substeps=3,
                          flags=scenes.CF_SELF | scenes.CF_WALLS, fixed_iterations=fixed)
        sc = scenes.make_grid_scene("fold", n, 1.0, p.thickness, p, seed=3)
        sc.walls = np.array([-20.0, 0.0, -20.0, 20.0, 20.0, 20.0], dtype=np.float32)
        state = scenes.folded(sc, gap=0.006)
    else:
        sc, state = scenes.ccd_scene(n)
        sc.params.fixed_iterations = fixed
        if kind == "ccd":
            sc.params.flags &= ~scenes.CF_SELF
    _, q = api.load_scene(sc)
    q.model.set_solver_mode(mode)
    q.model.set_state(*state)
    out = []
    for _ in range(3):
        q.step(sc.dt)
        out.append((_bits(q.model.positions()), _bits(q.model.velocities()),
                    *(np.ascontiguousarray(a) for k in (3, 4) for a in q.model.contacts(k))))
    found = sum(len(q.model.contacts(k)[0]) for k in (3, 4))
    kind_of = q.model.solver_choice()[0][0]
    status = q.status()
    q.free()
    return out, kind_of, status, found


# fold: 9: less than a warp a colour; 40: colours of more records than threads; ccd_scene:
# continuous hits alone, and behind the proximity contacts
@pytest.mark.parametrize("n,kind", [(9, "fold"), (24, "fold"), (40, "fold"), (12, "ccd"), (16, "both")])
@pytest.mark.parametrize("fixed", [True, False])
def test_records_against_per_colour(n, kind, fixed):
    got, tile, s0, found = _run(n, kind, fixed, 0)
    want, _, s1, same = _run(n, kind, fixed, 3)
    assert tile == 5 and s0 == s1 and found == same
    if kind == "fold":
        assert found > 0
    for f, (a, b) in enumerate(zip(got, want)):
        for x, y in zip(a, b):
            assert np.array_equal(x.view(np.uint32) if x.dtype == np.float32 else x,
                                  y.view(np.uint32) if y.dtype == np.float32 else y), f

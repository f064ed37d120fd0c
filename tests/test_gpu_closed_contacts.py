"""Continuous contacts of a cloth in one closed tile, alone and behind live proximity
contacts, in parallel colours and in the serial one: there are some, and the states
are the per-colour path's, bit for bit."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu


def _run(n, both, mode):
    from solidcloth_b200 import api
    sc, state = scenes.ccd_scene(n)
    if not both:
        sc.params.flags &= ~scenes.CF_SELF
    _, p = api.load_scene(sc)
    p.model.set_solver_mode(mode)
    p.model.set_state(*state)
    p.step(sc.dt)
    out = [np.ascontiguousarray(a, np.float32).view(np.uint32) for a in (p.model.positions(), p.model.velocities())]
    found = [len(p.model.contacts(k)[0]) for k in (3, 4)]
    out += [np.ascontiguousarray(a).view(np.uint32) for k in (3, 4) for a in p.model.contacts(k)]
    kind, status = p.model.solver_choice()[0][0], p.status()
    p.free()
    return out, found, kind, status


@pytest.mark.parametrize("n", [12, 24])
@pytest.mark.parametrize("both", [False, True])
def test_continuous_contacts(n, both):
    got, found, kind, s0 = _run(n, both, 0)
    want, same, _, s1 = _run(n, both, 3)
    assert kind == 5 and s0 == s1 and found == same and min(found) > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)

"""More continuous contacts than a contact list holds: the list keeps the first of them
in (query, candidate) order, as the all-pairs sweep finds them, and the status says so."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu

CCD_OVERFLOW = 4
EE_HITS = 16            # continuous contacts the list holds per edge


def _tangle(n):
    """particles strewn over a small box, moving through one another: about 25 edge-edge
    hits an edge, fewer candidate pairs than the pair lists hold"""
    sc, _ = scenes.ccd_scene(n)
    sc.params.flags &= ~scenes.CF_SELF
    sc.params.iterations = 1
    rng = np.random.default_rng(1)
    pos = rng.uniform(0.0, 1.0, (n * n, 3)).astype(np.float32)
    vel = (60.0 * rng.uniform(-2.0, 2.0, (n * n, 3))).astype(np.float32)
    return sc, (pos, pos.copy(), vel)


@pytest.mark.parametrize("n,full", [(8, True), (5, False)])
def test_first_hits_stay(n, full):
    from solidcloth_b200 import api
    from oracle.bridge import PortCloth
    PortCloth.set_portable_math(True)
    sc, state = _tangle(n)
    o = PortCloth.from_scene(sc)
    o._fn("set_ccd")(o.h, 1)
    o.set_state(*state)
    o.step(sc.dt)
    edges = (n - 1) * (3 * n - 1)
    oi, of = o.contacts(4)
    cap = 1 + EE_HITS * edges
    assert (len(oi) > cap) == full and len(oi) > 0
    runs = []
    for _ in range(2):
        w, p = api.load_scene(sc)
        p.model.set_state(*state)
        p.step(sc.dt)
        runs.append((*p.model.contacts(4), p.status()))
        p.free()
        w.free()
    for gi, gf, status in runs:
        assert np.array_equal(gi, oi[:cap])
        assert np.array_equal(gf[:, [0, 1, 2, 6]].view(np.uint32), of[:cap][:, [0, 1, 2, 6]].view(np.uint32))
        assert bool(status & CCD_OVERFLOW) == full

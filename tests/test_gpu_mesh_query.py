"""Cloth against collider meshes (one warp per query) against the CPU oracle: trees
from a single leaf (20 triangles) to several levels, leaves of more than 32
primitives included; contacts and positions bit for bit."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a, np.float32).view(np.uint32),
                          np.ascontiguousarray(b, np.float32).view(np.uint32))


# level 0: 20 triangles, 30 edges, 12 vertices in the root; level 1: 80 / 120 / 42,
# two or three leaves of up to 40; levels 2 and 4: deeper trees
@pytest.mark.parametrize("level", [0, 1, 2, 4])
@pytest.mark.parametrize("n", [7, 34])
def test_contacts_match_oracle(level, n):
    from solidcloth_b200 import api
    from oracle.bridge import PortCloth
    PortCloth.set_portable_math(True)
    sc = scenes.cfg2(n=n, level=level)
    sc.ccd = False
    sc.params.iterations, sc.params.substeps = 4, 2
    sc.params.tolerance = 0.05
    # the top of the coarsest sphere is a vertex or an edge a little below 0.5
    top = float(sc.meshes[0].vertices[:, 1].max())
    sc.positions = (sc.positions + np.array([0, top + 0.01 - 1.0, 0], np.float32)).astype(np.float32)
    w, p = api.load_scene(sc)
    o = PortCloth.from_scene(sc)
    o.set_tri_order(p.model.constraint_order(0)[0])
    o.set_bend_order(p.model.constraint_order(1)[0])
    o.set_contact_order(1)
    o.set_static_colours(*p.model.static_colours())
    seen = 0
    for f in range(3):
        p.step(sc.dt)
        o.step(sc.dt)
        assert _same(p.model.positions(), o.positions()), f
        for kind in range(3):
            gi, gf = p.model.contacts(kind)
            oi, of = o.contacts(kind)
            assert np.array_equal(gi[:, :2], oi[:, :2]) and len(gi) == len(oi), (f, kind)
            seen += len(gi)
    assert seen > 0
    assert p.status() == 0

"""The continuous broad phase (blocks of 32, groups of 1,024) against the oracle's
all-pairs sweep, at the sizes where a block or a group begins or ends, for one
cloth and for a batch; and the hit lists that follow from it."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu


def _oracle(sc, state, p):
    from oracle.bridge import PortCloth
    PortCloth.set_portable_math(True)
    o = PortCloth.from_scene(sc)
    o._fn("set_ccd")(o.h, 1)
    o.set_state(*state)
    o.set_tri_order(p.model.constraint_order(0)[0])
    o.set_bend_order(p.model.constraint_order(1)[0])
    o.set_contact_order(1)
    o.set_static_colours(*p.model.static_colours())
    return o


# edges: 16 (3 x 3), 56 and 85 (5 x 5, 6 x 6: one vertex block and two), 1,008 and
# 1,121 (19 x 19, 20 x 20: one group and two), 3,136 with 1,089 vertices (33 x 33)
@pytest.mark.parametrize("n", [3, 5, 6, 19, 20, 33])
def test_pairs_and_hits(n):
    from solidcloth_b200 import api
    from oracle.bridge import PortCloth
    sc, state = scenes.ccd_scene(n)
    sc.params.flags &= ~scenes.CF_SELF
    sc.params.thickness = 0.9 * 30.0 / (n - 1)
    w, p = api.load_scene(sc)
    p.model.set_state(*state)
    p.step(sc.dt)
    PortCloth.set_portable_math(True)
    o2 = PortCloth.from_scene(sc)
    o2.set_state(*state)
    o2.predict_detect(sc.dt / sc.params.substeps, ccd=False)
    tol = sc.params.thickness + 0.5 * sc.params.tolerance
    vt, ee = o2.ccd_broadphase(tol, 0), o2.ccd_broadphase(tol, 1)
    assert len(vt) > 0 and len(ee) > 0
    assert sorted(map(tuple, p.model.ccd_candidates(0)[:, ::-1].tolist())) == sorted(map(tuple, vt.tolist()))
    assert sorted(map(tuple, p.model.ccd_candidates(1).tolist())) == sorted(map(tuple, ee.tolist()))
    o = _oracle(sc, state, p)
    o.step(sc.dt)
    for kind in (3, 4):
        gi, gf = p.model.contacts(kind)
        oi, of = o.contacts(kind)
        assert np.array_equal(gi, oi), (kind, len(gi), len(oi))
        sel = [0, 1, 2, 6]
        assert np.array_equal(gf[:, sel].view(np.uint32), of[:, sel].view(np.uint32)), kind
    assert p.status() & ~16 == 0


def test_batch_instances_do_not_meet():
    """instances that lie in one another: each finds its own pairs only, as many as alone"""
    from solidcloth_b200 import api
    insts = scenes.cfg3_instances(count=5, seed=13, lo=6, hi=40)
    parts = [api.load_scene(s) for s in insts]
    alone = []
    for (w, q), s in zip(parts, insts):
        q.step(s.dt)
        alone.append([q.model.ccd_candidates(k) for k in (0, 1)])
        q.model.set_positions(s.positions)
        q.model.set_state(s.positions, s.positions, np.zeros_like(s.positions))
    b = api.ClothBatch([q for _, q in parts])
    b.step(insts[0].dt)
    first = np.cumsum([0] + [s.num_vertices for s in insts])
    tris = np.cumsum([0] + [q.model.num_tris() for _, q in parts])
    edges = np.cumsum([0] + [q.model.num_edges() for _, q in parts])
    for k, base in ((0, (first, tris)), (1, (edges, edges))):
        got = b.model.ccd_candidates(k)
        want = np.concatenate([a[k] + np.array([base[0][i], base[1][i]], np.int32) for i, a in enumerate(alone)])
        assert sorted(map(tuple, got.tolist())) == sorted(map(tuple, want.tolist())), k
    assert b.status() & ~16 == 0

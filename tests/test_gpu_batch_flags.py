"""A batch whose collision flags are widened by the setter: triangle and edge
collider contacts are solved in the automatic mode as in the per-colour path."""
import numpy as np
import pytest

from solidcloth_b200 import scenes

pytestmark = pytest.mark.gpu


def _run(flags, mode):
    from solidcloth_b200 import api
    insts = scenes.cfg3_instances(count=2, seed=7, lo=16, hi=24)
    for s in insts:
        s.masses = np.ones(s.num_vertices, np.float32)       # these contacts' solves assume them
        s.positions[:, 1] -= np.float32(0.395)               # half a centimetre above the spheres
    b = api.load_batch(insts)
    b.model.set_solver_mode(mode)
    api.lib().scSetCollisionFlags(b.model.h, flags)
    for _ in range(3):
        b.step(insts[0].dt)
    out = [b.model.positions(), b.model.velocities()] + [len(b.model.contacts(k)[0]) for k in (1, 2)] + [b.status()]
    b.free()
    return out


@pytest.mark.parametrize("flags", [scenes.CF_VERTICES | scenes.CF_TRIANGLES, scenes.CF_EDGES, scenes.CF_TRIANGLES | scenes.CF_EDGES])
def test_widened_flags(flags):
    got, want = _run(flags, 0), _run(flags, 3)
    assert want[2] + want[3] > 0                             # there are such contacts
    assert got[2:] == want[2:]
    for a, b in zip(got[:2], want[:2]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))

"""The training pass's GELU on the special-function unit far from and at zero, and its
gradient sums in arrays that the four-float reductions cannot take."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


def _network(seed):
    rng = np.random.default_rng(seed)
    d = M.unpack(M.init_params(seed))
    d["W4"][:] = rng.standard_normal(d["W4"].shape).astype(np.float32) * 0.2
    d["b1"][:] = rng.standard_normal(64).astype(np.float32) * 0.1
    norm = np.concatenate([np.zeros(12), np.ones(12), [1e-3] * 3]).astype(np.float32)
    return M.pack(d), norm


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


@pytest.mark.parametrize("scale", [0.0, 1e-6, 1.0, 30.0])
def test_gradients_over_magnitudes(scale):
    """from the linear range to where the exponential is zero: relative L2 error below 2 %,
    loss within 1 %, the bounds of the BF16 gradients against their oracle"""
    import torch
    from solidcloth_b200.api import lib
    p, norm = _network(5)
    rng = np.random.default_rng(6)
    X = (rng.standard_normal((257, M.IN)) * scale).astype(np.float32)
    X[0] = 0.0
    T = (rng.standard_normal((257, M.OUT)) * 1e-3).astype(np.float32)
    dX, dT, dp, dn = _dev(X), _dev(T), _dev(p), _dev(norm)
    g, loss = torch.zeros(M.NPARAM, device="cuda"), torch.zeros(1, device="cuda")
    assert lib().scMlpGradients(dX.data_ptr(), dT.data_ptr(), 257, dp.data_ptr(), dn.data_ptr(), g.data_ptr(), loss.data_ptr(), None) == 0
    want, want_loss = M.grad(p, norm, X, T)
    got = g.cpu().numpy()
    assert np.isfinite(got).all()
    assert np.linalg.norm(got - want) <= 0.02 * np.linalg.norm(want)
    assert abs(float(loss) - want_loss) <= 0.01 * want_loss


@pytest.mark.parametrize("rows", [1, 300])
def test_gradient_array_at_any_float(rows):
    """the array starts 0 to 3 floats into a 16-byte aligned buffer; nothing around it is
    written. At most 3 blocks add up: 3 x 2^-24 of the largest sum"""
    import torch
    from solidcloth_b200.api import lib
    p, norm = _network(7)
    rng = np.random.default_rng(8)
    dX, dT, dp, dn = _dev(rng.standard_normal((rows, M.IN))), _dev(rng.standard_normal((rows, M.OUT)) * 1e-3), _dev(p), _dev(norm)
    out = []
    for off in range(4):
        buf = torch.full((M.NPARAM + 8,), 7.0, device="cuda")
        loss = torch.zeros(1, device="cuda")
        assert lib().scMlpGradients(dX.data_ptr(), dT.data_ptr(), rows, dp.data_ptr(), dn.data_ptr(),
                                    buf.data_ptr() + 4 * off, loss.data_ptr(), None) == 0
        g = buf.cpu().numpy()
        assert (g[:off] == 7.0).all() and (g[off + M.NPARAM:] == 7.0).all()
        out.append(g[off:off + M.NPARAM])
    assert np.abs(out[0]).max() > 0
    for o in out[1:]:
        assert np.abs(o - out[0]).max() <= 3 * 2.0 ** -24 * np.abs(out[0]).max()

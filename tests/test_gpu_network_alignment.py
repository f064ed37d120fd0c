"""The network's vector loads: arrays that start at any float give the bits that
16-byte aligned ones give, at the row counts where a tile or the grid ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _at(a, off):
    """a copy of `a` that starts `off` floats into a 16-byte aligned buffer"""
    import torch
    buf = torch.zeros(a.size + 4, device="cuda")
    v = buf[off:off + a.size]
    v.copy_(torch.from_numpy(a.reshape(-1)))
    return v


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 148 * 4 * 128 + 5])
def test_unaligned_arrays(rows):
    import torch
    from solidcloth_b200 import learned
    from solidcloth_b200.api import lib
    rng = np.random.default_rng(rows)
    X = rng.standard_normal((rows, learned.IN)).astype(np.float32)
    T = (rng.standard_normal((rows, learned.OUT)) * 1e-3).astype(np.float32)
    prm = (learned.init_params(1) + 0.02 * rng.standard_normal(learned.NPARAM)).astype(np.float32)
    norm = np.concatenate([rng.standard_normal(12) * 0.1, 0.5 + rng.random(12), [1e-3] * 3]).astype(np.float32)
    out = []
    for off in (0, 1, 3):
        dX, dT, dp, dn = (_at(a, off) for a in (X, T, prm, norm))
        Y = torch.zeros(rows * 3 + 4, device="cuda")[off:off + rows * 3]
        assert lib().scMlpForward(dX.data_ptr(), rows, dp.data_ptr(), dn.data_ptr(), Y.data_ptr(), None) == 0
        g, loss = torch.zeros(learned.NPARAM, device="cuda"), torch.zeros(1, device="cuda")
        assert lib().scMlpGradients(dX.data_ptr(), dT.data_ptr(), rows, dp.data_ptr(), dn.data_ptr(), g.data_ptr(),
                                    loss.data_ptr(), None) == 0
        torch.cuda.synchronize()
        out.append((Y.cpu().numpy(), g.cpu().numpy(), float(loss)))
    for o in out[1:]:
        assert np.array_equal(out[0][0].view(np.uint32), o[0].view(np.uint32))
        # the gradients' sums over blocks are in no fixed order: float32 rounding of up to
        # 148 partial sums, 148 x 2^-24 of the largest
        assert np.abs(out[0][1] - o[1]).max() <= 1e-5 * np.abs(out[0][1]).max()
        assert abs(out[0][2] - o[2]) <= 1e-5 * out[0][2]

"""The warm-start network's kernels where a tile, a CTA's run of tiles or the
alignment of the callers' arrays changes: one row, a tile and its neighbours,
more tiles than CTAs (a CTA's accumulators carry over), arrays that start 4
bytes off a 16-byte boundary.  Against the numpy oracle with the bounds of its
own rounding (an activation is rounded to BF16, 2^-9 of its size; a rounding
flipped by FP32 order moves an output by that times a weight): forward 2e-3 of
the largest output, gradients 2e-2 of their norm, loss 1e-4."""
import os
import sys

import numpy as np
import pytest

from cffc_b200 import warmstart

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def on_device(a, off):
    """The array on the device, starting `off` floats past an aligned address."""
    import torch
    t = torch.zeros(a.size + 4, dtype=torch.float32, device="cuda")
    v = t[off:off + a.size].view(a.shape)
    v.copy_(torch.from_numpy(a))
    return v


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 148 * 128 + 1, 2 * 148 * 128 + 300])
def test_sizes(n, off):
    rng = np.random.default_rng(n + off)
    X = rng.standard_normal((n, 16)).astype(np.float32)
    T = (0.5 * np.tanh(X[:, :4] @ rng.standard_normal((4, 4)))).astype(np.float32)
    net = warmstart.Mlp(seed=2)
    p = net.params().astype(np.float64)
    Xd, Td = on_device(X, off), on_device(T, off)
    Y = net.forward(Xd).cpu().numpy()
    ref, _ = mlp_oracle.forward(p, X.astype(np.float64))
    assert np.max(np.abs(Y - ref)) <= 2e-3 * np.max(np.abs(ref))
    loss, g = net.gradient(Xd, Td)
    lref, gref = mlp_oracle.gradient(p, X.astype(np.float64), T.astype(np.float64))
    assert abs(loss - lref) <= 1e-4 * lref
    k = 0
    for name, shape in mlp_oracle.SIZES:
        q = int(np.prod(shape))
        a, b = g[k:k + q].astype(np.float64), gref[k:k + q]
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), name
        k += q
    again, g2 = net.gradient(Xd, Td)
    assert again == loss and np.array_equal(g, g2)  # deterministic
    hist = net.train(Xd, Td, steps=2, lr=1e-3)
    assert abs(hist[0] - loss) <= 1e-6 * loss and np.isfinite(hist[1])
    net.close()

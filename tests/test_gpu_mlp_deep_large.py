"""The deep network's weight gradients over passes whose row groups are several
chunks long, so that the warps issuing their products start at tiles far apart
in the ring of staged tiles: 3 chunks of 64 rows per SM and one row more, where
the fourth warp's first tile lies past the ring, and larger passes.

Against the numpy oracle with the bounds of test_gpu_mlp_deep.py (gradients to
3e-2 per parameter group, the loss to 1e-3); a second call gives the same
bits."""
import os
import sys

import numpy as np
import pytest

from cffc_b200 import warmstart

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_deep_oracle as oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def data(n, seed):
    rng = np.random.default_rng(seed)
    X = np.zeros((n, 16), np.float32)
    X[:, :5] = rng.standard_normal((n, 5)).astype(np.float32)
    # rows whose size grows along the array: a tile taken for another one shows
    X *= np.linspace(0.3, 2.0, n, dtype=np.float32)[:, None]
    T = (0.5 * np.tanh(X[:, :4] @ rng.standard_normal((4, 4)))).astype(np.float32)
    return X, T


def sizes():
    """Multiples of a chunk per SM, for the SM count of the GPU (148 without one)."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148
    return [128 * sms + 1, 192 * sms, 192 * sms + 1, 40000, 65536, 1024 * sms]


@pytest.mark.parametrize("k", range(6))
def test_gradient_matches_oracle(k):
    import torch
    n = sizes()[k]
    net = warmstart.MlpDeep(seed=3)
    p = net.params().astype(np.float64)
    X, T = data(n, n)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    loss, g = net.gradient(Xd, Td)
    loss2, g2 = net.gradient(Xd, Td)
    assert loss == loss2 and np.array_equal(g, g2)
    lref, gref = oracle.gradient(p, X.astype(np.float64), T.astype(np.float64))
    assert abs(loss - lref) <= 1e-3 * lref
    q = 0
    for name, shape in oracle.SIZES:
        m = int(np.prod(shape))
        a, b = g[q:q + m].astype(np.float64), gref[q:q + m]
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b), name
        q += m
    net.close()


def test_training_step_on_a_large_batch():
    """One step on all rows, in the shuffle's order: the loss is that of the rows
    in order, and Adam's first step moves a parameter by lr against its
    gradient's sign.  The other order of the rows changes FP32 sums only, by
    parts in 10^6 of their terms: the sign is sure from a tenth of the group's
    root mean square on."""
    import torch
    n, lr = sizes()[3], 1e-3
    Xd, Td = (torch.from_numpy(a).cuda() for a in data(n, 8))
    out = []
    for _ in range(2):
        net = warmstart.MlpDeep(seed=5)
        p0 = net.params()
        loss, g = net.gradient(Xd, Td)
        hist = net.train(Xd, Td, steps=1, batch=n, lr=lr)
        out.append((hist, net.params()))
        net.close()
    (hist, p1), (hist2, p2) = out
    assert np.array_equal(hist, hist2) and np.array_equal(p1, p2)
    assert abs(hist[0] - loss) <= 1e-5 * loss
    q = 0
    for name, shape in oracle.SIZES:
        m = int(np.prod(shape))
        b, d = g[q:q + m], (p1 - p0)[q:q + m]
        sure = np.abs(b) > 0.1 * np.sqrt(np.mean(b * b))
        assert np.any(sure) and np.all(np.sign(d[sure]) == -np.sign(b[sure])), name
        q += m

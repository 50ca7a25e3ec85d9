"""The deep network's fused kernels at the sizes where their tiling can go
wrong: fewer rows than a 64-row chunk or a 128-row tile, one more and one less,
an odd number of chunks, more rows than one 64-row group per SM (groups of
128), more tiles than CTA pairs, and arrays that are not 16-byte aligned.

Against the numpy oracle with the bounds of test_gpu_mlp_deep.py: outputs to
2e-3 of the largest, gradients to 3e-2 per parameter group (an occasional BF16
rounding of an activation or delta flips), the loss to 1e-3."""
import ctypes as C
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
    T = (0.5 * np.tanh(X[:, :4] @ rng.standard_normal((4, 4)))).astype(np.float32)
    return X, T


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 192, 9473, 20001])
def test_outputs_and_gradient_match_oracle(n):
    import torch
    net = warmstart.MlpDeep(seed=3)
    p = net.params().astype(np.float64)
    X, T = data(n, n)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    ref, _ = oracle.forward(p, X.astype(np.float64))
    Y = net.forward(Xd).cpu().numpy()
    assert np.max(np.abs(Y - ref)) <= 2e-3 * np.max(np.abs(ref))
    loss, g = net.gradient(Xd, Td)
    lref, gref = oracle.gradient(p, X.astype(np.float64), T.astype(np.float64))
    assert abs(loss - lref) <= 1e-3 * lref
    k = 0
    for name, shape in oracle.SIZES:
        m = int(np.prod(shape))
        a, b = g[k:k + m].astype(np.float64), gref[k:k + m]
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b), name
        k += m
    net.close()


@pytest.mark.parametrize("n", [130, 1000])
def test_unaligned_arrays_give_the_same(n):
    """Rows, targets and outputs that start 4 bytes past a 16-byte boundary."""
    import torch
    net = warmstart.MlpDeep(seed=4)
    X, T = (torch.from_numpy(a).cuda() for a in data(n, 5))
    Xu, Tu, Yu = (torch.empty(a.numel() + 1, device="cuda")[1:] for a in (X, T, T))
    Xu.copy_(X.flatten())
    Tu.copy_(T.flatten())
    Y = net.forward(X)
    loss, g = net.gradient(X, T)
    assert Xu.data_ptr() % 16 == 4
    torch.cuda.synchronize()
    assert net.lib.e2d_mlp_deep_forward(net.m, Xu.data_ptr(), n, Yu.data_ptr(), None) == 0
    assert torch.equal(Yu.view(n, 4), Y)
    gu, lu = np.zeros_like(g), C.c_double(0.0)
    assert net.lib.e2d_mlp_deep_gradient(net.m, Xu.data_ptr(), Tu.data_ptr(), n,
                                         gu.ctypes.data_as(C.POINTER(C.c_float)), C.byref(lu), None) == 0
    assert np.array_equal(gu, g) and lu.value == loss
    net.close()


def test_minibatches_cross_epochs():
    """Batches that straddle the shuffles (a ring of row lists, several
    epochs): every step's loss is finite and training is repeatable."""
    import torch
    X, T = (torch.from_numpy(a).cuda() for a in data(300, 6))
    hist = []
    for _ in range(2):
        net = warmstart.MlpDeep(seed=7)
        hist.append(net.train(X, T, steps=23, batch=129, lr=1e-3))
        hist.append(net.params())
        net.close()
    assert np.all(np.isfinite(hist[0])) and np.array_equal(hist[0], hist[2]) and np.array_equal(hist[1], hist[3])

"""The ILU(k) kernels over block shapes and levels of fill: rows of a level
that fill part of a warp, one row a level, more rows than the streamed kernels
take (the kernels on the factors in HBM), levels whose buffers do not fit
(factorization in HBM, streamed solves), a block whose vector does not fit
shared memory.

With the source-terms-only Jacobian the matrix is block diagonal, so ILU(k) of
every shape and level equals block Jacobi's inverse bit for bit (the entries
past the diagonal are zero blocks of the real pattern).  With the HLLE Jacobian
the preconditioner of a block does not depend on the other blocks: a block set
of several equals each block's own, and a second application repeats."""
import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2), (3, 2), (9, 7), (17, 5), (5, 17), (33, 9), (40, 36), (32, 32), (64, 32), (64, 60), (96, 80)]


def apply(bs, level, v, order=capi.JACOBIAN_FIRST_ORDER_HLLE):
    h = capi.Handle(bs)
    h.set_state()
    p = capi.nks_params(1, ilu_level=level, jacobian_order=order)
    z = h.block_precon_apply(p, 5.0, v)
    again = h.block_precon_apply(p, 5.0, v)
    h.close()
    assert np.array_equal(z, again)
    return z


def vector(bs, seed=1):
    return np.random.default_rng(seed).standard_normal((bs.nblk, bs.NCj, bs.NCi, 4))


@pytest.mark.parametrize("level", [0, 1, 2, 4, 5])
@pytest.mark.parametrize("nci, ncj", SHAPES)
def test_block_diagonal_matrix_equals_block_jacobi(nci, ncj, level):
    bs = cases.channel(nbi=2, nbj=1, nci=nci, ncj=ncj, seed=5)
    v = vector(bs)
    g = bs.ng
    z, zj = (apply(bs, k, v, capi.JACOBIAN_SOURCE_TERMS_ONLY) for k in (level, None))
    assert np.array_equal(z[:, g:-g, g:-g], zj[:, g:-g, g:-g])


@pytest.mark.parametrize("level", [0, 2, 4])
@pytest.mark.parametrize("nci, ncj", [(9, 7), (33, 9), (16, 16), (64, 32)])
def test_blocks_are_independent(nci, ncj, level):
    """The same block alone and as each of five: the preconditioner reads the
    state of a block and its ghost cells only."""
    one = cases.channel(nbi=1, nbj=1, nci=nci, ncj=ncj, seed=6)
    v = vector(one)
    z = apply(one, level, v)
    assert np.all(np.isfinite(z)) and np.any(z)
    h = capi.BatchHandle([one] * 5)
    h.set_state()
    p = capi.nks_params(1, ilu_level=level)
    many = h.block_precon_apply(p, 5.0, np.concatenate([v] * 5))
    h.close()
    for b in range(5):
        assert np.array_equal(many[b], z[0])

"""Handles of different block shapes side by side: a kernel's limit of dynamic
shared memory belongs to the process, so a handle of small blocks must not lower
it under one of large blocks made before."""
import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu


def vector(bs, seed=1):
    return np.random.default_rng(seed).standard_normal((bs.nblk, bs.NCj, bs.NCi, 4))


# streamed solves and factorization; factorization in HBM; all in HBM
@pytest.mark.parametrize("nci, ncj, level", [(64, 32, 2), (64, 32, 4), (48, 40, 5)])
def test_ilu(nci, ncj, level):
    p = capi.nks_params(1, ilu_level=level)
    large, small = (cases.channel(nbi=2, nbj=1, nci=a, ncj=b, seed=5) for a, b in ((nci, ncj), (6, 5)))
    h, g = capi.Handle(large), capi.Handle(small)
    for x in (h, g):
        x.set_state()
    v = vector(large)
    z = h.block_precon_apply(p, 5.0, v)
    g.block_precon_apply(p, 5.0, vector(small))
    assert np.array_equal(h.block_precon_apply(p, 5.0, v), z)
    h.close()
    g.close()


def test_residual_smoothing():
    out = []
    for first in (False, True):
        sc = cases.Scheme(cfl=0.4, n_stage=4, local_dt=1, time_integration=cases.TIME_OPTIMAL_SMOOTHING,
                          rs_epsilon=0.5, rs_iterations=2)
        h = capi.Handle(cases.channel(nbi=2, nbj=1, nci=64, ncj=32, seed=5, scheme=sc))
        if first:
            g = capi.Handle(cases.channel(nbi=2, nbj=1, nci=6, ncj=5, seed=5, scheme=sc))
            g.set_state()
            assert g.rk_steps(1)[0] == 0
            g.close()
        h.set_state()
        assert h.rk_steps(3)[0] == 0
        out.append(h.get_state())
        h.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)

"""Explicit runs around the length of a group of captured steps: one call of n
steps against n calls of one step (a graph of one step each), for the marching
and the tiled stage kernel, with frozen limiters and with residual smoothing.
A step's rounding differs between the two (the first time step of a call is
computed by its own kernel): 1e-14 a step and operation, some hundred
operations deep, 1e-11 of the largest value over these lengths."""
import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, {"freeze_limiter": 1, "freeze_level": 0.5}, {"rs_epsilon": 0.5, "rs_iterations": 2}])
@pytest.mark.parametrize("nci", [16, 9])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 66, 71])
def test_lengths(n, nci, kw):
    bs = cases.channel(nbi=2, nbj=2, nci=nci, ncj=7, seed=3,
                       scheme=cases.Scheme(cfl=0.5, n_stage=2, local_dt=0, **kw))
    one, many = capi.Handle(bs), capi.Handle(bs)
    one.set_state()
    many.set_state()
    rc, hist = many.rk_steps(n)
    assert rc == 0
    single = np.concatenate([one.rk_steps(1)[1] for _ in range(n)])
    assert hist.shape == single.shape
    assert np.all(np.abs(hist - single) <= 1e-11 * np.max(np.abs(single), axis=0))
    for a, b in zip(many.get_state(), one.get_state()):
        assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))
    rc, again = many.rk_steps(n)  # the captured groups once more
    assert rc == 0 and np.all(np.isfinite(again)) and again.shape == hist.shape

"""Newton-Krylov on teams of CTAs of which some hold no part of the vector (more
SMs than parts), beside another handle's explicit steps from another host
thread, so that the team's CTAs start at different times: the solve succeeds
and gives the bits of a solve on the idle GPU."""
import threading

import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu


def bump(nbi, nbj, nc, mach=1.4, h=0.03):
    return cases.bump_channel(nbi=nbi, nbj=nbj, nci=nc, ncj=nc, mach=mach, h=h,
                              scheme=cases.Scheme(limiter=cases.LIMITER_ZERO, local_dt=1))


def solve(h, ilu):
    h.set_state()
    rc, hist = h.nks(capi.nks_params(2, gmres_restart=20, max_gmres=40, overall_tol=1e-10, cfl0=10.0, gmres_tol=0.1,
                                     ilu_level=ilu))
    return rc, hist, h.get_state()


# 24 blocks of 32 x 32: 120 parts of the vector, 48 of the cells; 100 of 16 x 16: 100 and 100
@pytest.mark.parametrize("nbi, nbj, nc", [(6, 4, 32), (10, 10, 16)])
@pytest.mark.parametrize("ilu", [None, 1])
def test_beside_another_handle(nbi, nbj, nc, ilu):
    h = capi.Handle(bump(nbi, nbj, nc))
    rc, hist, (W, U) = solve(h, ilu)
    assert rc == 0
    other = capi.Handle(cases.curvilinear_mach2(nbi=8, nbj=8, nc=32, seed=1, scheme=cases.Scheme()))
    other.set_state()
    stop, bad = threading.Event(), []

    def march():
        while not stop.is_set():
            rc, _ = other.rk_steps(16)
            if rc:
                bad.append(rc)
                return
            other.set_state()

    t = threading.Thread(target=march)
    t.start()
    try:
        runs = [solve(h, ilu) for _ in range(6)]
    finally:
        stop.set()
        t.join()
    assert not bad
    for rc2, hist2, (W2, U2) in runs:
        assert rc2 == 0 and hist2 == hist
        assert np.array_equal(W2, W) and np.array_equal(U2, U)
    other.close()
    h.close()

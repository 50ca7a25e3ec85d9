"""The three ways an Arnoldi step runs -- a cluster of CTAs per case, a share
of a cooperative launch per case, separate kernels -- give the same bits: a
case alone (cluster, or the whole GPU's share) against the same case in a
batch of eight or more (shares) and of forty (separate kernels).  Odd block
shapes, chunks that do not divide a block, GMRES restarts and cases that stop
at different steps; block Jacobi and ILU(k)."""
import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu


def bump(nbi, nbj, nci, ncj, mach, h):
    return cases.bump_channel(nbi=nbi, nbj=nbj, nci=nci, ncj=ncj, mach=mach, h=h,
                              scheme=cases.Scheme(limiter=cases.LIMITER_ZERO, local_dt=1))


def solve(bss, ilu, restart):
    p = capi.nks_params(3, gmres_restart=restart, max_gmres=40, overall_tol=1e-10, cfl0=10.0, gmres_tol=0.1,
                        ilu_level=ilu)
    h = capi.BatchHandle(bss) if len(bss) > 1 else capi.Handle(bss[0])
    h.set_state()
    rc, hist = h.nks(p)
    assert rc == 0
    out = h.get_state()
    h.close()
    return ([hist] if len(bss) == 1 else hist), ([out] if len(bss) == 1 else out)


@pytest.mark.parametrize("ilu", [None, 1])
@pytest.mark.parametrize("nci, ncj, restart", [(12, 10, 7), (16, 16, 30), (33, 9, 12), (36, 30, 20)])
def test_routes_give_the_same_bits(ilu, nci, ncj, restart):
    fam = [bump(1 + k % 3, 1 + k % 2, nci, ncj, 1.35 + 0.01 * k, 0.02 + 0.001 * k) for k in range(8)]
    solo = [solve([bs], ilu, restart) for bs in fam]
    for n in (8, 40):
        hists, outs = solve([fam[k % 8] for k in range(n)], ilu, restart)
        for k in range(n):
            (h1,), ((W, U),) = solo[k % 8]
            assert hists[k] == h1, (n, k)
            assert np.array_equal(outs[k][0], W) and np.array_equal(outs[k][1], U), (n, k)


@pytest.mark.parametrize("ilu", [None, 0])
def test_large_case_gives_the_same_bits_in_a_batch(ilu):
    """A case of 24 blocks (a share of the GPU, alone all of it) with seven
    small ones."""
    big = bump(6, 4, 32, 32, 1.4, 0.03)
    small = [bump(2, 1, 32, 32, 1.36 + 0.02 * k, 0.025) for k in range(7)]
    (h1,), ((W, U),) = solve([big], ilu, 30)
    hists, outs = solve(small[:3] + [big] + small[3:], ilu, 30)
    assert hists[3] == h1
    assert np.array_equal(outs[3][0], W) and np.array_equal(outs[3][1], U)

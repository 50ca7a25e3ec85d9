"""The stage kernel of a block set follows from its block width, precision and
flux, whatever the number of blocks: the same case gives the same bits alone, in
batches of other cases, and with any number of rows per chunk.  Widths on both
sides of where the fast precisions change from one kernel to the other."""
import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8), (14, 9), (16, 16), (18, 32), (20, 20), (32, 13), (34, 32), (36, 36), (38, 8), (64, 16)]
SETS = [(1, 1), (2, 2), (6, 5), (12, 8)]


def block_set(nbi, nbj, nci, ncj, precision, flux):
    sc = cases.Scheme(cfl=0.4, precision=precision, flux=flux)
    return cases.channel(nbi=nbi, nbj=nbj, nci=nci, ncj=ncj, seed=nbi, scheme=sc)


def march(h, n):
    h.set_state()
    rc, hist = h.rk_steps(n)
    assert rc == 0
    out = h.get_state()
    config = h.stage_config() if isinstance(h, capi.Handle) else None
    h.close()
    return config, hist, out


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("flux", [cases.FLUX_ROE, cases.FLUX_HLLC])
@pytest.mark.parametrize("nci, ncj", SHAPES)
def test_same_bits_for_any_number_of_blocks(nci, ncj, flux, precision, monkeypatch):
    fam = [block_set(nbi, nbj, nci, ncj, precision, flux) for nbi, nbj in SETS]
    _, hist, states = march(capi.BatchHandle(fam), 5)
    kernels = set()
    for c, bs in enumerate(fam):
        (kernel, rows, _), h1, (W, U) = march(capi.Handle(bs), 5)
        kernels.add(kernel)
        assert np.array_equal(bs.interior(states[c][1]), bs.interior(U)), c
        assert np.array_equal(hist[:, c, 0], h1[:, 0])
        np.testing.assert_allclose(hist[:, c, 1:], h1[:, 1:], rtol=1e-12, atol=0)  # atomically summed norms
    if precision < 2:
        assert len(kernels) == 1
    monkeypatch.setenv("CFFC_E2D_STAGE_KERNEL", "march" if kernel else "tiled")  # the default rows per chunk
    _, _, (W1, U1) = march(capi.Handle(bs), 5)
    assert np.array_equal(W1, W) and np.array_equal(U1, U)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("flux", [cases.FLUX_ROE, cases.FLUX_HLLC])
def test_periodic_and_walled_cases_in_one_batch(flux, precision):
    """A handle with walls takes another instance of the FP32 Roe kernel than a
    periodic one alone."""
    sc = cases.Scheme(cfl=0.4, precision=precision, flux=flux)
    fam = [cases.periodic_box_bumps(nb=3, nc=32, seed=4, scheme=sc), block_set(2, 3, 32, 32, precision, flux)]
    _, hist, states = march(capi.BatchHandle(fam), 8)
    for c, bs in enumerate(fam):
        _, h1, (_, U) = march(capi.Handle(bs), 8)
        assert np.array_equal(bs.interior(states[c][1]), bs.interior(U)), c
        assert np.array_equal(hist[:, c, 0], h1[:, 0])

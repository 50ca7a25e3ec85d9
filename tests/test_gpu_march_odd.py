"""The exact build's marching stage kernel on blocks an odd number of cells
wide (windows by cp.async, no tensor maps) against the tiled kernel: strips of
one column more or less than a full one, chunks with remainders, blocks narrower
than a strip.  Both kernels restate the reference's arithmetic, so state and
residual are equal bit for bit; the history's sums run in each kernel's own
order (1e-12)."""
import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu


def run(bs, kernel, monkeypatch):
    monkeypatch.setenv("CFFC_E2D_STAGE_KERNEL", kernel)
    h = capi.Handle(bs)
    monkeypatch.delenv("CFFC_E2D_STAGE_KERNEL")
    assert h.stage_config()[0] == (kernel != "tiled")
    h.set_state()
    res = bs.interior(h.residual())
    rc, hist = h.rk_steps(3)
    assert rc == 0
    W, U = h.get_state()
    h.close()
    return res, W, U, hist


@pytest.mark.parametrize("nci, ncj", [(3, 2), (5, 9), (31, 7), (33, 16), (37, 29), (65, 8)])
@pytest.mark.parametrize("n_stage, tint, flux", [(2, 0, 2), (4, 8, 4), (4, 7, 6), (1, 0, 2)])
def test_odd_width(nci, ncj, n_stage, tint, flux, monkeypatch):
    sc = cases.Scheme(cfl=0.4, n_stage=n_stage, local_dt=n_stage == 4, time_integration=tint, flux=flux,
                      precision=2)
    bs = cases.channel(nbi=2, nbj=2, nci=nci, ncj=ncj, seed=nci, scheme=sc)
    *got, hist = run(bs, "march_any", monkeypatch)
    *want, hist_t = run(bs, "tiled", monkeypatch)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert np.all(np.abs(hist - hist_t) <= 1e-12 * np.max(np.abs(hist_t), axis=0))

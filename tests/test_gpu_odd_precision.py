"""Handles of odd block width and the exact precision: its geometry is made for
handles that have it, when they first do, and leaves the state alone."""
import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu

FP64, FP32, EXACT = 0, 1, 2


def block_set(precision, nbi=2, nbj=2, nci=37, ncj=29, local=1):
    sc = cases.Scheme(cfl=0.4, n_stage=4, local_dt=local, time_integration=cases.TIME_OPTIMAL_SMOOTHING,
                      precision=precision)
    return cases.channel(nbi=nbi, nbj=nbj, nci=nci, ncj=ncj, seed=3, scheme=sc)


def test_other_precisions_hold_no_exact_geometry():
    """Device memory of a handle of half a million cells: 96 bytes a cell more
    with the exact precision than without."""
    import torch
    capi.Handle(block_set(EXACT)).close()  # what the first handle loads
    used, cells = {}, 30 * 133 * 131
    for precision in (FP64, FP32, EXACT):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        h = capi.Handle(block_set(precision, 6, 5, 129, 127))
        used[precision] = before - torch.cuda.mem_get_info()[0]
        h.close()
    assert used[EXACT] - max(used[FP64], used[FP32]) > 80 * cells


@pytest.mark.parametrize("kernel", [None, "tiled", "march_any"])
@pytest.mark.parametrize("start", [FP64, FP32])
def test_switch_to_exact(start, kernel, monkeypatch):
    """Steps in the first precision, then in the exact one: those of a handle
    created in the exact precision that is given the same state, bit for bit;
    switched back, the first precision's kernel again."""
    if kernel:
        monkeypatch.setenv("CFFC_E2D_STAGE_KERNEL", kernel)
    h = capi.Handle(block_set(start))
    he = capi.Handle(block_set(EXACT))
    h.set_state()
    assert h.rk_steps(3)[0] == 0
    assert h.stage_config()[0] == 0
    before = h.get_state()
    h.set_precision(EXACT)
    after = h.get_state()
    assert all(np.array_equal(a, b) for a, b in zip(before, after))
    assert h.stage_config()[:2] == he.stage_config()[:2]
    for x in (h, he):
        x.set_state(before[0])
    rc, hist = h.rk_steps(4)
    rce, histe = he.rk_steps(4)
    assert rc == 0 and rce == 0
    assert np.array_equal(hist[:, 0], histe[:, 0])
    # (the first entry's norms are of the residual of the steps before, which only h has)
    np.testing.assert_allclose(hist[1:], histe[1:], rtol=1e-12, atol=0)  # atomically summed
    assert all(np.array_equal(a, b) for a, b in zip(h.get_state(), he.get_state()))
    h.set_precision(start)
    assert h.stage_config()[0] == 0
    h.set_precision(EXACT)
    assert h.stage_config()[:2] == he.stage_config()[:2]
    h.close()
    he.close()


def test_switch_of_a_batch():
    """The same for a batch, against its cases alone."""
    fam = [block_set(FP64, 2, 2), block_set(FP64, 3, 1), block_set(FP64, 1, 1)]
    hb = capi.BatchHandle(fam)
    hb.set_precision(EXACT)
    hb.set_state()
    rc, _ = hb.rk_steps(4)
    assert rc == 0
    got = hb.get_state()
    hb.close()
    for c, (nbi, nbj) in enumerate([(2, 2), (3, 1), (1, 1)]):
        bs = block_set(EXACT, nbi, nbj)
        h = capi.Handle(bs)
        h.set_state()
        assert h.rk_steps(4)[0] == 0
        assert np.array_equal(bs.interior(got[c][1]), bs.interior(h.get_state()[1]))
        h.close()

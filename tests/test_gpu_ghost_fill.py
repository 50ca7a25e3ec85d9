"""The ghost fill over what a block's edges may carry: every boundary
condition on whole edges with and without neighbours (the one-round fill and
its corners), conditions on some cells of an edge or on an edge that also
exchanges (the passes one after another), odd and small blocks.  Against the C
restatement bit for bit; 1e-12 where a characteristic condition reaches pow."""
import os
import sys

import numpy as np
import pytest

from cffc_b200 import capi, cases

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import e2d_oracle  # noqa: E402

pytestmark = pytest.mark.gpu

CODES = [cases.BC_NONE, cases.BC_CONSTANT_EXTRAPOLATION, cases.BC_PERIODIC, cases.BC_REFLECTION, cases.BC_FIXED,
         cases.BC_CHARACTERISTIC]


def filled(bs):
    out = []
    for h in (capi.Handle(bs), e2d_oracle.Oracle(bs)):
        h.set_state()
        h.fill_ghosts()
        out.append(h.get_state())
    return out


def check(bs):
    (Wg, Ug), (Wo, Uo) = filled(bs)
    pow_reached = any((a == cases.BC_CHARACTERISTIC).any() for a in (bs.bc_w, bs.bc_e, bs.bc_s, bs.bc_n))
    for a, b in ((Wg, Wo), (Ug, Uo)):
        if pow_reached:
            assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
        else:
            assert np.array_equal(a, b)


@pytest.mark.parametrize("edge", ["W", "E", "S", "N", "all"])
@pytest.mark.parametrize("code", CODES)
@pytest.mark.parametrize("nbi, nbj, nci, ncj", [(1, 1, 8, 6), (2, 2, 7, 5), (3, 1, 2, 3)])
def test_whole_edges(code, edge, nbi, nbj, nci, ncj):
    bc = {k: code if edge in (k, "all") else cases.BC_REFLECTION for k in "WESN"}
    check(cases.channel(nbi=nbi, nbj=nbj, nci=nci, ncj=ncj, bc=bc, seed=4))


@pytest.mark.parametrize("seed", range(8))
def test_mixed_edges(seed):
    """Random codes per edge (none, one code, or a code per cell), on interior
    block edges too."""
    rng = np.random.default_rng(seed)
    bs = cases.channel(nbi=2, nbj=2, nci=9, ncj=6, seed=seed)
    free = np.array([1.0, 0.6, 0.1, 1.0])
    for codes, wo in ((bs.bc_w, bs.wo_w), (bs.bc_e, bs.wo_e), (bs.bc_s, bs.wo_s), (bs.bc_n, bs.wo_n)):
        wo[:] = free[None, :, None]
        for b in range(bs.nblk):
            kind = rng.integers(3)
            codes[b] = (cases.BC_NONE if kind == 0 else rng.choice(CODES[:5]) if kind == 1
                        else rng.choice(CODES[:5], codes.shape[1]))
    check(bs)

"""ILU(k) where the device memory left holds the factors and the inverted
diagonals, but not what the streamed kernels keep beside them: the kernels on
the factors in HBM, the same bits."""
import ctypes as C

import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu


def factor_bytes(bs, level):
    f = capi.load_library().e2d_ilu_pattern
    f.argtypes = [C.c_int32, C.c_int32, C.c_int32, C.POINTER(C.c_int32), C.POINTER(C.c_int32), C.c_int32,
                  C.POINTER(C.c_int32), C.POINTER(C.c_int32)]
    n = bs.nci * bs.ncj
    row_ptr, nnz, levels = np.zeros(n + 1, dtype=np.int32), C.c_int32(0), (C.c_int32 * 2)()
    assert f(bs.nci, bs.ncj, level, row_ptr.ctypes.data_as(C.POINTER(C.c_int32)), None, 0, C.byref(nnz), levels) == 0
    return 128 * (nnz.value + n) * bs.nblk


# streamed solves and factorization; streamed solves, factorization in HBM
@pytest.mark.parametrize("nci, ncj, level", [(32, 32, 2), (64, 32, 4)])
def test_solve_with_little_memory(nci, ncj, level):
    import torch
    bs = cases.channel(nbi=24, nbj=16, nci=nci, ncj=ncj, seed=5)
    p = capi.nks_params(1, ilu_level=level)
    v = np.random.default_rng(1).standard_normal((bs.nblk, bs.NCj, bs.NCi, 4))
    out = []
    for little in (False, True):
        h = capi.Handle(bs)
        h.set_state()
        h.block_precon_apply(capi.nks_params(1), 5.0, v)  # block Jacobi: everything but the factors is allocated
        held = None
        if little:
            torch.cuda.empty_cache()
            left = factor_bytes(bs, level) * 5 // 4 + (64 << 20)  # the streamed kernels' arrays take twice the factors'
            held = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
        out.append(h.block_precon_apply(p, 5.0, v))
        h.close()
        del held
        torch.cuda.empty_cache()
    assert np.array_equal(out[0], out[1])

"""Handles created while another stream keeps the host-to-device copies and the
default stream busy: what creation computes on the handle's own stream (face
normals and kinds of the block edges, geometry) sees the arrays it was given."""
import threading

import numpy as np
import pytest

from cffc_b200 import capi, cases

pytestmark = pytest.mark.gpu


def state(bs):
    h = capi.Handle(bs)
    h.set_state()
    h.fill_ghosts()
    out = h.get_state()
    rc, _ = h.rk_steps(2)
    assert rc == 0
    out += h.get_state()
    h.close()
    return out


@pytest.mark.parametrize("nci, ncj, precision", [(33, 30, 0), (32, 32, 0), (33, 30, 2)])
def test_beside_copies(nci, ncj, precision):
    import torch
    sets = [cases.channel(nbi=5, nbj=4, nci=nci, ncj=ncj, seed=k, skew=0.05 * k,
                          scheme=cases.Scheme(cfl=0.4, precision=precision)) for k in range(1, 5)]
    want = [state(bs) for bs in sets]
    host = torch.empty(1 << 27, dtype=torch.uint8, pin_memory=True)
    dev = torch.empty(1 << 27, dtype=torch.uint8, device="cuda")
    side, stop = torch.cuda.Stream(), threading.Event()

    def copies():
        while not stop.is_set():
            with torch.cuda.stream(side):
                dev.copy_(host, non_blocking=True)
            dev.add_(1)  # the default stream
            side.synchronize()

    t = threading.Thread(target=copies)
    t.start()
    try:
        got = [state(bs) for _ in range(5) for bs in sets]
    finally:
        stop.set()
        t.join()
        torch.cuda.synchronize()
    for k, out in enumerate(got):
        for a, b in zip(out, want[k % len(want)]):
            assert np.array_equal(a, b), k

"""Host-array operators take their streams from a bounded pool: more calls at once than it
keeps, from several threads and with operators that come and go, give the results of calls
one after another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operator(gtb, k):
    n, W, H, P = (24 + 4 * (k % 3), 28, 20), 40, 32, 30
    rng = np.random.default_rng(k)
    proj = rng.uniform(0.0, 2.0, (P, H, W)).astype(np.float32)
    geo = gtb.CBCT_geometry(1000.0, 1500.0, (W * 1.3, H * 1.3), np.linspace(0, 348, P).astype(np.float32),
                            np.zeros((P, 2), np.float32))
    E = gtb.hoCuConebeamProjectionOperator()
    E.setup(gtb.CBCT_acquisition(geo, proj), None, tuple(float(x) for x in n), is_dims=n)
    E.set_use_filtered_backprojection(True)
    return E, proj, (n[2], n[1], n[0])


def test_calls_at_once(gtb, cuda):
    import torch
    want = []
    for k in range(9):
        E, proj, shape = _operator(gtb, k)
        out = torch.zeros(shape, dtype=torch.float32).pin_memory()
        E.mult_MH(torch.from_numpy(proj).pin_memory(), out)
        want.append(out)
    got = [None] * 9
    errors = []

    def work(k):
        try:
            for _ in range(4):                      # a new operator each time: plans come and go
                E, proj, shape = _operator(gtb, k)
                out = torch.zeros(shape, dtype=torch.float32).pin_memory()
                E.mult_MH(torch.from_numpy(proj).pin_memory(), out)
                got[k] = out
        except Exception as e:                      # reported below, by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(9)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    for a, b in zip(got, want):
        assert torch.equal(a, b)

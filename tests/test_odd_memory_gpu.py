"""Row-padded copies are wanted, not needed: plans and served requests of odd sizes do
without them where the device or the budget has no room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_plan_without_room_for_padded_copies(gtb, cuda):
    """A volume of 55 % of the free memory: its transposed copy fits, the row-padded one
    besides does not.  Nothing is launched."""
    import torch
    L = gtb._lib
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    nz = int(0.55 * free / (4 * 1024 * 1023))
    g = L.CbctGeometry(1000.0, 1500.0, 61 * 0.15, 40 * 0.15, 61, 40, 1021, 1023, nz, 102.1, 102.3, 0.1 * nz, 1.5)
    plan = gtb.Plan(g, np.array([10.0, 100.0], np.float32), np.zeros((2, 2), np.float32))
    assert plan.forward_variant().startswith("tma-")      # of volumes that have room
    plan.close()
    assert torch.cuda.mem_get_info()[0] > 0.9 * free


@pytest.mark.parametrize("kind", ["fdk", "osmom"])
def test_served_within_a_budget_without_padded_copies(gtb, cuda, kind):
    import torch
    L = gtb._lib
    n, W, H, P = (45, 42, 33), 71, 50, 40
    g = L.CbctGeometry(1000.0, 1500.0, W * 1.6, H * 1.6, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]), float(n[2]), 1.5)
    ang = gtb.phantom.circular_orbit(P)
    off = np.zeros((P, 2), np.float32)
    proj = torch.from_numpy(np.random.default_rng(4).uniform(0.0, 3.0, (P, H, W)).astype(np.float32))
    vols, recs = [], []
    budget = 4e9
    for _ in range(2):
        vol = torch.full((n[2], n[1], n[0]), -1.0, dtype=torch.float32)
        with gtb.Server(budget, 1) as srv:
            req = srv.fdk_request(g, ang, off, proj, vol) if kind == "fdk" else \
                srv.osmom_request(g, ang, off, proj, vol, 4, iterations=1, nonneg=True)
            rec = srv.wait(srv.submit(req))
        assert rec["status"] == 0 and rec["bytes_peak"] <= rec["bytes_reserved"] <= budget
        vols.append(vol)
        recs.append(rec)
        budget = rec["bytes_reserved"] - 1      # the second run: one byte short of the copies
    assert recs[1]["bytes_reserved"] < recs[0]["bytes_reserved"]
    if kind == "fdk":
        assert torch.equal(vols[0], vols[1])
    else:
        # rays beside the volume are summed in another order
        assert float((vols[0] - vols[1]).norm() / vols[0].norm()) <= 1e-5

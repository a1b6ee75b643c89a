"""Volumes of fewer planes than a run along z, whose detector boxes end at their last
voxels so that thick planes keep the TMA-staged kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# n, plane spacing (mm), pixel (mm): whole runs of the first three would span more than 256
# detector rows
CASES = [((64, 48, 12), 8.0, 0.8), ((64, 48, 3), 10.0, 0.5), ((64, 48, 1), 12.0, 0.8), ((40, 24, 5), 1.0, 1.2),
         ((40, 24, 15), 1.0, 1.2), ((40, 24, 17), 1.0, 1.2)]


@pytest.mark.parametrize("fdk", [False, True])
@pytest.mark.parametrize("n,vz,pitch", CASES)
def test_flat_volumes(gtb, cuda, n, vz, pitch, fdk):
    import torch
    L = gtb._lib
    P = 5
    W, H = int(n[0] * 1.8 / pitch) // 4 * 4, max(8, int(n[2] * vz * 1.8 / pitch))
    g = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                       n[2] * vz, 1.5)
    angles = (5.0 + np.arange(P) * 72.0).astype(np.float32)
    gen = torch.Generator(device=cuda)
    gen.manual_seed(12)
    low = torch.rand((P, 1, H // 8 + 2, W // 8 + 2), generator=gen, device=cuda)
    proj = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=True)[:, 0].contiguous()
    outs = []
    for gather in (1, 0):
        plan = gtb.Plan(g, angles, np.tile(np.array([[1.0, -1.0]], np.float32), (P, 1)))
        plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)
        out = torch.full(plan.vol_shape, 0.5, dtype=torch.float32, device=cuda)
        plan.backproject(proj, out, -1, L.CBCT_BP_FDK_WEIGHT if fdk else 0, True, True)
        assert plan.read_flags() == (0, 0)
        outs.append(out.double())
    # sums of 5 interpolated values; rows within 1e-4 in both kernels (rows up to some 400)
    # against slopes of an eighth
    assert float((outs[1] - outs[0]).norm() / outs[0].norm()) <= 2e-5
    assert plan.autotune()["backproject_tma"] is not None

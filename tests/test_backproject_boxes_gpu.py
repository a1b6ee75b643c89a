"""Detectors much finer than the voxels: runs of 32 voxels along z have detector boxes
twice as high as runs of 16, and the back-projector takes them only where they leave it
the TMA-staged kernel and an SM its CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 640 CTAs of long runs (the line is 592); sums of 3 interpolated values in two kernels,
# rows within 1e-4 (see test_backproject_rows_gpu) and slopes of order 1
CASES = [0.25, 0.3, 0.45, 0.7]


@pytest.mark.parametrize("pitch", CASES)
def test_fine_detectors_keep_the_staged_kernel(gtb, cuda, pitch):
    import torch
    L = gtb._lib
    n, P = (128, 128, 160), 3
    W, H = int(218 / pitch) // 8 * 8, int(256 / pitch) // 8 * 8
    g = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                       float(n[2]), 1.5)
    angles = (7.0 + np.arange(P) * 77.0).astype(np.float32)
    gen = torch.Generator(device=cuda)
    gen.manual_seed(3)
    low = torch.rand((P, 1, H // 8 + 2, W // 8 + 2), generator=gen, device=cuda)
    proj = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=True)[:, 0].contiguous()
    outs = []
    for gather in (1, 0):
        plan = gtb.Plan(g, angles, np.zeros((P, 2), np.float32))
        plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)
        out = torch.empty(plan.vol_shape, dtype=torch.float32, device=cuda)
        plan.backproject(proj, out)
        assert plan.read_flags() == (0, 0)
        outs.append(out.double())
    assert plan.autotune()["backproject_tma"] is not None
    assert float((outs[1] - outs[0]).norm() / outs[0].norm()) <= 1e-4

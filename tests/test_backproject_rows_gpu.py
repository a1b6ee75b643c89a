"""The detector row of a voxel in long runs along z: projections that hold their own row
number, so that a back-projected view is the row coordinate itself.  Its error against
FP64 is that of the coordinates, and must not grow along a run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Detectors of 200 rows: coordinates below 256 and, counted from a box's corner, below 128.
# The kernel's rows differ from FP64 by three roundings of A z (at most 100 rows: 3 x
# 2^-24 x 100), two at detector coordinates (2^-17 each at most), fifteen at box coordinates
# (2^-19 each) and the tap's own three (values below 256, 2^-17 each): below 1e-4.
BOUND = 1e-4


@pytest.mark.parametrize("angle", [20.0, 111.0, 245.0])
@pytest.mark.parametrize("n,W", [((160, 144, 160), 320), ((160, 144, 160), 321), ((64, 64, 48), 160)])
def test_row_coordinates(gtb, cuda, n, W, angle):
    import torch
    L = gtb._lib
    H, pitch = 200, 0.9 * 320 / W
    g = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * 0.9, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                       float(n[2]), 1.5)
    plan = gtb.Plan(g, np.array([angle], np.float32), np.array([[1.0, -1.0]], np.float32))
    proj = torch.arange(H, device=cuda, dtype=torch.float32)[None, :, None].expand(1, H, W).contiguous()
    x, y, z = (torch.arange(m, device=cuda).double() + 0.5 - m / 2 for m in n)
    th = np.deg2rad(angle)
    c, s = np.cos(th), np.sin(th)
    xr, yr = c * x[None, :] + s * y[:, None], -s * x[None, :] + c * y[:, None]
    cu = ((1500.0 * xr / (yr + 1000.0) - 1.0) / float(np.float32(W * pitch)) + 0.5) * W - 0.5
    cv = ((1500.0 * z[:, None, None] / (yr + 1000.0) + 1.0) / float(np.float32(H * 0.9)) + 0.5) * H - 0.5
    ok = (cv > 0.5) & (cv < H - 1.5) & ((cu > 0.5) & (cu < W - 1.5))[None]
    assert float(ok.double().mean()) > 0.2
    for gather in (1, 0):
        plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)   # global loads: runs of 8, a rounding per voxel
        out = torch.empty(plan.vol_shape, dtype=torch.float32, device=cuda)
        plan.backproject(proj, out)
        assert plan.read_flags() == (0, 0)
        d = (out.double() - cv).abs()
        assert float(d[ok].max()) <= BOUND
    k = torch.arange(n[2], device=cuda) % 32 // 8
    rms = [float(d[k == q][ok[k == q]].pow(2).mean().sqrt()) for q in range(4)]
    # The last quarter of a run of 32 is as exact as the first (a rounding per voxel: 1.9
    # times as far off), a quarter more being left for where the quarters lie.
    assert n[2] < 160 or rms[3] <= 1.25 * rms[0], rms

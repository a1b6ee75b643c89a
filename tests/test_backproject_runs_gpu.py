"""TMA-staged back-projection over its z-run lengths and box widths against the
global-load kernel, which takes the same bilinear taps, and the offset weight over
rows that do and do not start on 16-byte boundaries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# sums over at most 40 views of interpolated values of like sign, another arrangement
# of the same multiply-adds; rows accumulate one rounding per voxel of a run of 32 in both
# kernels' coordinates (2^-24 * 128 rows, against slopes of order 1): 1e-5
TOL = 1e-5

# n, W, H, pixel pitch, views: runs of 16 (few CTAs) and 32 (592 CTAs and more), heights that are
# not a multiple of either, footprints for the 40, 48, 56, 72 and 104 wide boxes
CASES = {
    "short_runs": ((40, 24, 37), 64, 48, 1.6, 9),
    "long_runs": ((200, 136, 95), 128, 96, 3.0, 6),
    "long_runs_fine": ((160, 144, 128), 320, 200, 0.9, 6),
    "fine_48": ((64, 40, 32), 160, 120, 0.8, 9),
    "fine_72": ((64, 40, 33), 256, 160, 0.5, 5),
    "fine_104": ((64, 40, 31), 400, 200, 0.32, 5),
    "one_layer": ((48, 40, 1), 80, 24, 1.2, 40),
}


@pytest.mark.parametrize("fdk", [False, True])
@pytest.mark.parametrize("name", list(CASES))
def test_runs_equal_global_loads(gtb, cuda, name, fdk):
    import torch
    L = gtb._lib
    n, W, H, pitch, P = CASES[name]
    cg = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                        float(n[2]), 1.5)
    angles = (3.0 + np.arange(P) * (360.0 / P)).astype(np.float32)
    offsets = np.tile(np.array([[1.0, -1.0]], np.float32), (P, 1))
    gen = torch.Generator(device=cuda)
    gen.manual_seed(8)
    # smooth projections, as real ones are: neighbouring taps differ by a few per cent
    low = torch.rand((P, 1, H // 8 + 2, W // 8 + 2), generator=gen, device=cuda)
    proj = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=True)[:, 0].contiguous()
    outs = []
    for gather in (1, 0):
        plan = gtb.Plan(cg, angles, offsets)
        plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)
        out = torch.full(plan.vol_shape, 0.5, dtype=torch.float32, device=cuda)
        plan.backproject(proj, out, -1, L.CBCT_BP_FDK_WEIGHT if fdk else 0, True, True)
        assert plan.read_flags() == (0, 0)
        outs.append(out.double())
    assert float((outs[0] - 0.5).abs().max()) > 0
    assert float((outs[1] - outs[0]).norm() / outs[0].norm()) <= TOL


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("W,H,P,start", [(64, 48, 3, 0), (64, 48, 3, 1), (63, 65, 2, 0), (129, 130, 2, 0), (4, 1, 1, 0)])
def test_offset_weight_rows(gtb, O, cuda, variant, W, H, P, start):
    """Both column widths of the offset weight, in place and on partial blocks."""
    import torch
    L = gtb._lib
    pitch = 100.0 / W
    cg = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, 8, 8, 8, 8.0, 8.0, 8.0, 1.5)
    og = O.Geometry(8, 8, 8, 8.0, 8.0, 8.0, W, H, W * pitch, H * pitch, 1000.0, 1500.0)
    offsets = np.array([[14.0 - 9.0 * p, 0.0] for p in range(P)], np.float32)
    plan = gtb.Plan(cg, np.linspace(0, 90, P).astype(np.float32), offsets)
    host = np.random.default_rng(2).uniform(0.5, 1.5, (P, H, W)).astype(np.float32)
    flat = torch.zeros(P * H * W + start, dtype=torch.float32, device=cuda)
    proj = flat[start:].view(P, H, W)
    proj.copy_(torch.from_numpy(host))
    plan.offset_correct(proj, -1, variant)
    ref = O.offset_weight(og, host.astype(np.float64), offsets, variant)
    assert O.rel_l2(proj.cpu().numpy(), ref) < 1e-5   # FP32 column position and sine: some 1e-6 of pi/4

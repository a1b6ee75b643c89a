"""The back-projector's rounding does not depend on how it is launched: runs of 32 voxels
along z give bitwise what runs of 16 give, and detectors whose rows TMA cannot read in
place, staged from a padded copy, bitwise what the global-load kernel gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(gtb, n, W, H, pitch, P, ox=1.0, voxel=1.0):
    L = gtb._lib
    m = voxel
    g = L.CbctGeometry(1000.0, 1500.0, W * pitch * m, H * pitch * m, W, H, n[0], n[1], n[2], n[0] * m, n[1] * m,
                       n[2] * m, 1.5)
    return gtb.Plan(g, (5.0 + np.arange(P) * (360.0 / P)).astype(np.float32),
                    np.tile(np.array([[ox, -0.5]], np.float32), (P, 1)))


def _rand(cuda, shape, seed):
    import torch
    gen = torch.Generator(device=cuda)
    gen.manual_seed(seed)
    return torch.rand(shape, generator=gen, device=cuda)


@pytest.mark.parametrize("fdk", [False, True])
@pytest.mark.parametrize("nz", [64, 63, 96, 50])
@pytest.mark.parametrize("pitch,voxel", [(0.6, 1.0), (1.2, 1.0), (1.2, 0.75)])
def test_runs_of_32_are_runs_of_16(gtb, cuda, fdk, nz, pitch, voxel):
    """256 x 256 columns have the CTAs for runs of 32, the 64 x 64 in their middle (the same
    blocks of 16 x 8 columns, exact coordinates) do not."""
    import torch
    L = gtb._lib
    W, H, P = int(300 / pitch) // 4 * 4, int(1.8 * nz / pitch), 5
    proj = _rand(cuda, (P, H, W), 1)
    outs = []
    for m in (256, 64):
        plan = _plan(gtb, (m, m, nz), W, H, pitch, P, voxel=voxel)
        out = torch.full(plan.vol_shape, 0.25, dtype=torch.float32, device=cuda)
        plan.backproject(proj, out, -1, L.CBCT_BP_FDK_WEIGHT if fdk else 0, True, True)
        assert plan.read_flags() == (0, 0)
        outs.append(out)
    assert torch.equal(outs[0][:, 96:160, 96:160], outs[1])


@pytest.mark.parametrize("n,W,H,pitch,P", [((30, 27, 21), 45, 34, 1.2, 7), ((48, 40, 33), 61, 50, 1.2, 128),
                                           ((44, 35, 16), 47, 40, 1.4, 5), ((256, 250, 70), 271, 100, 1.7, 6),
                                           ((256, 256, 64), 401, 220, 0.8, 6), ((64, 48, 5), 90, 30, 1.1, 5)])
@pytest.mark.parametrize("voxel", [1.0, 0.73])
def test_padded_detectors_are_the_global_loads(gtb, cuda, n, W, H, pitch, P, voxel):
    import torch
    L = gtb._lib
    proj = _rand(cuda, (P, H, W), 2)
    start = _rand(cuda, (n[2], n[1], n[0]), 3)
    mask = (_rand(cuda, (n[2], n[1], n[0]), 4) > 0.3).to(torch.uint8)
    for flags in (0, L.CBCT_BP_FDK_WEIGHT):
        for accumulate in (False, True):
            outs = []
            for gather in (1, 0):
                plan = _plan(gtb, n, W, H, pitch, P, 2.5, voxel)
                plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)
                if accumulate:
                    plan.set_mask(mask)
                out = start.clone()
                plan.backproject(proj, out, -1, flags, True, accumulate)
                assert plan.read_flags() == (0, 0)
                outs.append(out)
            assert torch.equal(outs[0], outs[1])


def test_steps_of_odd_sizes(gtb, cuda):
    """Two ordered-subset steps of odd volume and detector: image, momentum image, residual
    and FP64 norm against the gather and global-load kernels."""
    import torch
    L = gtb._lib
    n, W, H, P = (75, 70, 61), 101, 93, 16
    b = 30.0 * _rand(cuda, (P, H, W), 5)
    vol = _rand(cuda, (n[2], n[1], n[0]), 6)
    got = []
    for gather in (1, 0):
        plan = _plan(gtb, n, W, H, 1.3, P, voxel=0.73)
        plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)
        z, xold, pre = vol.clone(), 0.9 * vol, torch.full_like(vol, 1e-4)
        r, n2 = torch.empty_like(b), torch.zeros(1, dtype=torch.float64, device=cuda)
        for _ in range(2):
            plan.osmom_step(0, b, z, xold, pre, r, 4.0, 0.25, True, n2)
        assert plan.read_flags() == (0, 0)
        got.append((z, xold, float(n2)))
    # rays beside the volume are summed in another order (see test_odd_norms_gpu)
    for a, c in zip(got[1][:2], got[0][:2]):
        assert float((a - c).norm() / c.norm()) <= 1e-7
    assert abs(got[1][2] - got[0][2]) <= 1e-9 * got[0][2]

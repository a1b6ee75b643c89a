"""Rays at the volume's silhouette: those that miss the volume box but pass
within half a voxel of it still sample border texels (border 0 interpolation),
so their projections are small and not zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Whole projections against the FP64 oracle: the FP32 path's bound.  A silhouette
# ray alone is ill-conditioned in FP32 whatever kernel samples it (its coordinates
# round at the source distance), so those rays are held to the gather kernel, which
# samples every ray by itself at the same FP32 coordinates: the two sums of up to
# 320 terms differ in order only, N 2^-24 = 2e-5 at most.
TOL = 1e-4
TOL_ORDER = 2e-5


def _misses(W, H, pitch, L, angles, SAD=1000.0, SDD=1500.0):
    """Rays that do not meet the box of size L (FP64): bool (views, H, W)."""
    q = ((np.arange(W) + 0.5) / W - 0.5) * W * pitch
    r = ((np.arange(H) + 0.5) / H - 0.5) * H * pitch
    out = []
    for a in np.deg2rad(angles.astype(np.float64)):
        c, s = np.cos(a), np.sin(a)
        S = np.array([SAD * s, -SAD * c, 0.0])
        d = [np.broadcast_to(c * q - s * (SDD - SAD) - S[0], (H, W)), np.broadcast_to(s * q + c * (SDD - SAD) - S[1], (H, W)),
             np.broadcast_to(r[:, None], (H, W))]
        lo, hi = np.full((H, W), 0.0), np.full((H, W), 1.0)
        for i in range(3):
            t1, t2 = (L[i] / 2 - S[i]) / d[i], (-L[i] / 2 - S[i]) / d[i]
            lo, hi = np.maximum(lo, np.minimum(t1, t2)), np.minimum(hi, np.maximum(t1, t2))
        out.append(hi < lo - 1e-9)
    return np.stack(out)


@pytest.mark.parametrize("kernel", [0, 1, 3, 4, 5])
@pytest.mark.parametrize("n,vox", [((12, 8, 6), 6.0), ((40, 36, 3), 1.5)])
def test_silhouette_rays(gtb, O, cuda, kernel, n, vox):
    import torch
    W, H, pitch = 100, 70, 1.3
    angles = np.array([3.0, 44.0, 90.0, 151.0, 270.0, 333.3], np.float32)
    offsets = np.zeros((angles.size, 2), np.float32)
    L = [k * vox for k in n]
    og = O.Geometry(n[0], n[1], n[2], L[0], L[1], L[2], W, H, W * pitch, H * pitch, 1000.0, 1500.0)
    cg = gtb._lib.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], L[0], L[1], L[2], 8.0)
    vol = np.random.default_rng(5).uniform(0.5, 1.5, (n[2], n[1], n[0])).astype(np.float32)
    ref = O.forward(og, vol.astype(np.float64), angles, offsets, spp=8.0)
    sel = _misses(W, H, pitch, L, angles) & (ref > 0)
    assert sel.sum() > 100
    v = torch.from_numpy(vol).to(cuda)
    outs = []
    for k in (kernel, 2):
        plan = gtb.Plan(cg, angles, offsets)
        plan.set_option(gtb._lib.CBCT_OPT_FORWARD_KERNEL, k)
        plan.set_option(gtb._lib.CBCT_OPT_DEBUG_CHECKS, 1)
        out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
        plan.forward(v, out)
        assert plan.read_flags() == (0, 0)
        outs.append(out.cpu().numpy().astype(np.float64))
    got, gather = outs
    assert np.linalg.norm(got[sel] - gather[sel]) <= TOL_ORDER * np.linalg.norm(gather[sel])
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)

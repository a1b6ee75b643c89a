"""Residuals and their FP64 norms where the gather kernel reads the caller's volume as
it lies: rows of no multiple of 16 bytes, and pixels too wide for a box of 16 x 16
rays.  The TMA kernels that take such launches interpolate in the gather kernel's form, so
rays through the volume are bitwise its rays, and the norm is its norm.  (Rays that pass
beside the volume within half a voxel read border texels and are summed in another order.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# n, W, H, pitch, views.  Sizes of no multiple of four in each axis alone and together;
# launches of a million rays, which take row quads in their warp and wide shapes; pixels of
# several voxels.
CASES = {
    "nx": ((30, 28, 20), 45, 34, 1.2, 7),
    "ny": ((44, 35, 16), 47, 40, 1.2, 7),
    "all": ((41, 43, 37), 61, 51, 1.3, 8),
    "quads_warp": ((75, 70, 101), 301, 151, 0.6, 24),
    "quads_wide": ((61, 67, 93), 383, 207, 0.45, 30),
    "quads_thin": ((75, 70, 201), 201, 203, 1.4, 40),
    "quads_skew": ((75, 70, 221), 201, 203, 1.55, 40),
    "pixels_wide": ((96, 96, 64), 29, 27, 5.0, 3),
}
MEAN = 0.5     # of the volume's values


def _geometry(gtb, name):
    n, W, H, pitch, P = CASES[name]
    g = gtb._lib.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                              float(n[2]), 1.5)
    return g, (4.0 + np.arange(P) * (360.0 / P)).astype(np.float32), np.tile(np.array([[1.0, 0.5]], np.float32), (P, 1))


def _chords(name, angles, offsets, SAD=1000.0, SDD=1500.0):
    """Share of each ray's path inside the volume (FP64), negative where it misses: (views, H, W)."""
    n, W, H, pitch, _ = CASES[name]
    out = []
    for a, (ox, oy) in zip(np.deg2rad(angles.astype(np.float64)), offsets):
        q = ((np.arange(W) + 0.5) / W - 0.5) * W * pitch + ox
        r = ((np.arange(H) + 0.5) / H - 0.5) * H * pitch + oy
        c, s = np.cos(a), np.sin(a)
        S = np.array([SAD * s, -SAD * c, 0.0])
        d = [np.broadcast_to(c * q - s * (SDD - SAD) - S[0], (H, W)), np.broadcast_to(s * q + c * (SDD - SAD) - S[1], (H, W)),
             np.broadcast_to(r[:, None], (H, W))]
        lo, hi = np.full((H, W), 0.0), np.full((H, W), 1.0)
        for i in range(3):
            t1, t2 = (n[i] / 2 - S[i]) / d[i], (-n[i] / 2 - S[i]) / d[i]
            lo, hi = np.maximum(lo, np.minimum(t1, t2)), np.minimum(hi, np.maximum(t1, t2))
        out.append(hi - lo)
    return np.stack(out)


def _close(res, norm, ref, ref_norm, through):
    import torch
    assert torch.equal(res[through], ref[through])
    # Rays beside the volume: sums of up to 400 samples in another order, parts in 1e6 of
    # them at most and 1e-7 mostly, either sign.
    assert float((res - ref).abs().max()) <= 400 * 2.0 ** -24 * float(ref.abs().max())
    assert abs(norm - ref_norm) <= 1e-9 * ref_norm


def _inputs(cuda, name):
    import torch
    n, W, H, _, P = CASES[name]
    gen = torch.Generator(device=cuda)
    gen.manual_seed(19)
    vol = 2.0 * MEAN * torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda)
    b = MEAN * max(n) * torch.rand((P, H, W), generator=gen, device=cuda)
    return vol, b


@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("name", list(CASES))
def test_residual_is_the_gather_kernels(gtb, cuda, name, storage):
    import torch
    L = gtb._lib
    g, angles, offsets = _geometry(gtb, name)
    vol, b = _inputs(cuda, name)
    code = L.CBCT_F32 if storage == "f32" else L.CBCT_BF16
    vol = vol if storage == "f32" else vol.to(torch.bfloat16)
    through = torch.from_numpy(_chords(name, angles, offsets) > 1e-6).to(cuda)
    assert 0.05 < float(through.double().mean())
    res, norms = {}, {}
    for kernel in (2, 0, 1, 3, 4, 5):
        if CASES[name][0][0] % 4 == 0 and CASES[name][0][1] % 4 == 0 and kernel > 2:
            continue       # forced kernels of their own forms over aligned rows
        plan = gtb.Plan(g, angles, offsets)
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        r, n2 = torch.empty_like(b), torch.zeros(1, dtype=torch.float64, device=cuda)
        plan.forward_residual(vol, b, r, -1, 1.0, False, n2, code)
        assert plan.read_flags() == (0, 0)
        res[kernel], norms[kernel] = r, float(n2)
        # FP64 sums of some million equal squares in another order: n 2^-53 at most
        assert abs(float(n2) - float((r.double() ** 2).sum())) <= 1e-9 * float(n2)
    for k, r in res.items():
        _close(r, norms[k], res[2], norms[2], through)


@pytest.mark.parametrize("name", ["nx", "ny", "all"])
def test_step_norm_is_the_gather_kernels(gtb, cuda, name):
    import torch
    L = gtb._lib
    g, angles, offsets = _geometry(gtb, name)
    vol, b = _inputs(cuda, name)
    through = torch.from_numpy(_chords(name, angles, offsets) > 1e-6).to(cuda)
    out = []
    for kernel in (2, 0):
        plan = gtb.Plan(g, angles, offsets)
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        z, xold, pre = vol.clone(), 0.9 * vol, torch.full_like(vol, 1e-3)
        r, n2 = torch.empty_like(b), torch.zeros(1, dtype=torch.float64, device=cuda)
        plan.osmom_step(0, b, z, xold, pre, r, 4.0, 0.25, True, n2)
        assert plan.read_flags() == (0, 0)
        out.append((r, float(n2)))
    _close(out[1][0], out[1][1], out[0][0], out[0][1], through)

"""Per-ray slab forward projector: every box width, long runs of samples in a slab
(dealt over the warp), partial tiles, and the launches that take it in place of the
row-pair and row-quad kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n, W, H, pitch, views, samples per voxel).  Pitches up to 9 mm take every box width
# (8 columns x pitch x 0.7 voxels and the slant of the rays; beyond about 5 mm only under
# a flat volume, whose boxes fit: elsewhere the plan takes the gather kernel); many samples per voxel, flat
# volumes and tall detectors give runs beyond the dealing bound in few and in all lanes.
CASES = {
    "fine": ((40, 48, 24), 67, 45, 0.4, 3, 1.5),
    "one": ((40, 48, 24), 45, 37, 1.5, 3, 1.5),
    "dense": ((24, 24, 16), 41, 35, 1.1, 3, 9.0),
    "flat": ((64, 64, 3), 61, 50, 1.3, 4, 2.0),
    "pitch3": ((64, 48, 40), 33, 30, 3.0, 3, 1.5),
    "pitch5": ((96, 96, 64), 29, 27, 5.0, 3, 1.5),
    "pitch9": ((128, 96, 64), 21, 19, 9.0, 3, 1.5),
    "pitch16": ((192, 160, 96), 19, 18, 16.0, 2, 1.5),
    "flat7": ((96, 96, 3), 23, 19, 7.0, 3, 1.5),
    "flat9": ((128, 96, 3), 21, 19, 9.0, 3, 1.5),
    "one_pixel": ((32, 32, 32), 1, 1, 1.0, 2, 1.5),
}


def _plan(gtb, cuda, name, dtype):
    import torch
    L = gtb._lib
    n, W, H, pitch, P, spp = CASES[name]
    g = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                       float(n[2]), spp)
    angles = (9.0 + np.arange(P) * (360.0 / P)).astype(np.float32)
    offsets = np.tile(np.array([[2.0, -1.0]], np.float32), (P, 1))
    gen = torch.Generator(device=cuda)
    gen.manual_seed(5)
    vol = torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda).to(dtype)
    plan = gtb.Plan(g, angles, offsets)
    plan.set_option(L.CBCT_OPT_DEBUG_CHECKS, 1)
    return plan, vol


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("name", list(CASES))
def test_slab_equals_per_ray_kernels(gtb, cuda, name, storage):
    """Bitwise the fan kernel (where its boxes fit: the same operations, one lane per
    ray); the gather kernel up to the form of its lerps and the order of silhouette
    sums: a lerp rounds three times (1.8e-7 of the values, three levels) and a sum of
    up to 600 nonnegative values in FP32 differs by at most 600 x 2^-24 = 3.6e-5 of
    itself, so 1e-4 of the largest ray."""
    import torch
    L = gtb._lib
    dtype = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[storage]
    code = {"f32": L.CBCT_F32, "f16": L.CBCT_F16, "bf16": L.CBCT_BF16}[storage]
    outs = {}
    for kernel in (0, 1, 2, 3):
        plan, vol = _plan(gtb, cuda, name, dtype)
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
        plan.forward(vol, out, vol_dtype=code)
        assert plan.read_flags() == (0, 0)
        outs["auto" if kernel == 0 else plan.forward_variant()] = out
    if name in ("pitch9", "pitch16"):
        assert "tma-slab" not in outs and torch.equal(outs["auto"], outs["gather"])
        return
    ref = outs["tma-slab"]
    assert float(ref.abs().max()) > 0
    assert torch.equal(ref, outs["auto"])      # few rays: the slab kernel whatever the rows' distance
    if "tma-fan" in outs:
        assert torch.equal(ref, outs["tma-fan"])
    assert float((ref - outs["gather"]).abs().max()) <= 1e-4 * float(ref.abs().max())


@pytest.mark.parametrize("name", ["fine", "one", "dense"])
def test_small_launch_residual_norm(gtb, cuda, name):
    """Residual and FP64 norm of launches that take the slab kernel: its blocks' partial
    sums against the norm of the residual itself, and the residual against the forced
    row-quad kernel's."""
    import torch
    L = gtb._lib
    res = []
    for kernel in (0, 1, 5):
        plan, vol = _plan(gtb, cuda, name, torch.float32)
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        b = torch.linspace(0.0, 3.0, int(np.prod(plan.proj_shape())), device=cuda).reshape(plan.proj_shape())
        r = torch.empty_like(b)
        norm = torch.zeros(1, dtype=torch.float64, device=cuda)
        plan.forward_residual(vol, b, r, -1, 1.0, False, norm)
        assert plan.read_flags() == (0, 0)
        ref = (r.double() ** 2).sum()
        # both are FP64 sums of the same squares
        assert abs(float(norm[0] - ref)) <= 1e-10 * float(ref)
        res.append(r)
    assert torch.equal(res[0], res[1]) and torch.equal(res[0], res[2])

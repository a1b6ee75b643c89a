"""Row-quad forward projector: its tile shapes and row-distance classes against
the per-ray slab kernel, which evaluates the same samples in the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n, W, H, pitch, views): row distances (z texels, 1 mm voxels, rows pitch * t with
# t = 0.62 to 0.72) in every class of the kernel, across the class borders 1/3, 1/2,
# 2/3, 1 and 4/3 inside one volume, beyond them, and with rows far closer than a texel.
# Tall detectors give rays clipped by the top and bottom faces; odd detector sizes leave
# partial tiles; the last entries have launches large enough for the wide and the thin
# tile shape of automatic plans.
CASES = {
    "fine": ((48, 40, 32), 97, 75, 0.1, 5),
    "third": ((48, 40, 32), 97, 75, 0.5, 5),
    "half": ((48, 40, 32), 65, 93, 0.75, 5),
    "two_thirds": ((40, 48, 24), 75, 61, 1.0, 5),
    "one": ((48, 40, 32), 61, 53, 1.5, 5),
    "four_thirds": ((48, 40, 32), 45, 41, 2.0, 5),
    "coarse": ((48, 40, 32), 33, 37, 2.6, 5),
    "short": ((40, 48, 8), 71, 66, 0.8, 5),
    "wide_shape": ((64, 64, 40), 385, 257, 0.3, 26),
    "wide_half": ((64, 64, 40), 385, 257, 0.75, 26),
    "thin_shape": ((64, 64, 40), 129, 97, 1.45, 85),
}


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("name", list(CASES))
def test_quad_equals_slab(gtb, cuda, name, storage):
    import torch
    L = gtb._lib
    n, W, H, pitch, P = CASES[name]
    cg = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                        float(n[2]), 1.5)
    angles = (7.0 + np.arange(P) * (360.0 / P)).astype(np.float32)
    offsets = np.tile(np.array([[3.0, -2.0]], np.float32), (P, 1))
    gen = torch.Generator(device=cuda)
    gen.manual_seed(11)
    td = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[storage]
    code = {"f32": L.CBCT_F32, "f16": L.CBCT_F16, "bf16": L.CBCT_BF16}[storage]
    vol = torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda).to(td)
    outs = []
    for kernel in (1, 5, 0):
        plan = gtb.Plan(cg, angles, offsets)
        plan.set_option(L.CBCT_OPT_DEBUG_CHECKS, 1)
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        if kernel == 1:
            assert plan.forward_variant() == "tma-slab"
        if kernel == 5 or name in ("wide_shape", "wide_half", "thin_shape"):
            assert kernel == 1 or plan.forward_variant() == "tma-quad"
        out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
        plan.forward(vol, out, vol_dtype=code)
        assert plan.read_flags() == (0, 0)
        outs.append(out)
    assert float(outs[0].abs().max()) > 0
    assert torch.equal(outs[0], outs[1])
    assert torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("name", ["half", "one", "short"])
def test_quad_residual_norm(gtb, cuda, name):
    """The fused residual and its FP64 norm: partial sums of every tile shape's
    blocks, own rays and missing rays included."""
    import torch
    L = gtb._lib
    n, W, H, pitch, P = CASES[name]
    cg = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                        float(n[2]), 1.5)
    angles = (np.arange(P) * (360.0 / P)).astype(np.float32)
    offsets = np.zeros((P, 2), np.float32)
    gen = torch.Generator(device=cuda)
    gen.manual_seed(5)
    vol = torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda)
    b = torch.rand((P, H, W), generator=gen, device=cuda)
    plan = gtb.Plan(cg, angles, offsets)
    plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, 5)
    ax = plan.forward(vol, torch.empty_like(b))
    r, n2 = torch.empty_like(b), torch.zeros(1, dtype=torch.float64, device=cuda)
    plan.forward_residual(vol, b, r, -1, 1.0, False, n2)
    assert torch.equal(r, ax - b)
    ref = float(((ax - b).double() ** 2).sum())
    assert abs(float(n2) - ref) <= 4e-12 * ref   # FP64 sums of up to 30225 equal squares in another order: n 2^-53

"""The x/y-transposed and row-padded copies the TMA forward projectors read, at sizes
around their tiles: 32x32 elements of four planes, and 64x64 elements of two planes in
words of two for 16-bit volumes with an even row length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(64, 64, 2), (66, 70, 5), (130, 63, 3), (62, 129, 1), (34, 32, 4), (32, 33, 9), (65, 66, 6)]


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("n", SIZES)
def test_copies(gtb, cuda, n, storage):
    """Views along x and along y against the gather kernel, which reads the caller's
    volume: the same samples of at most 200 values of one sign, another form of the same
    lerps and order of silhouette sums: 200 x 2^-24 + 3 x 1.8e-7 < 2e-5 of the sums."""
    import torch
    L = gtb._lib
    W, H = 2 * max(n), max(16, 2 * n[2])
    g = L.CbctGeometry(1000.0, 1500.0, W * 1.0, H * 1.0, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                       float(n[2]), 1.5)
    angles = np.array([0.0, 90.0, 180.0, 270.0, 33.0, 123.0], np.float32)
    code = {"f32": L.CBCT_F32, "f16": L.CBCT_F16, "bf16": L.CBCT_BF16}[storage]
    dtype = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[storage]
    gen = torch.Generator(device=cuda)
    gen.manual_seed(7)
    vol = torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda).to(dtype)
    outs = []
    for kernel in (2, 1):
        plan = gtb.Plan(g, angles, np.zeros((angles.size, 2), np.float32))
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
        plan.forward(vol, out, vol_dtype=code)
        outs.append(out.double())
        assert plan.forward_variant() == ("gather" if kernel == 2 else "tma-slab")
    assert float(outs[0].abs().max()) > 0
    for v in range(angles.size):
        assert float((outs[1][v] - outs[0][v]).norm()) <= 2e-5 * float(outs[0][v].norm())

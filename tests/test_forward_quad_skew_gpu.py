"""Row quads with rows a texel or more apart: the skewed tile, whose warps hold two
groups of rows beside two others, against the per-ray slab kernel (the same samples in
the same order, so bitwise), at detector sizes that leave partial tiles in both
directions, and the automatic choice of 16-bit and of widely spaced rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# detector columns and rows around the tile's 16 x 16, row distances 0.97 to 1.4 texel
CASES = [(33, 31, 1.45), (16, 16, 1.5), (47, 49, 1.6), (15, 18, 1.8), (64, 40, 1.95)]


@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("case", CASES)
def test_skewed_tiles(gtb, cuda, case, storage):
    import torch
    L = gtb._lib
    W, H, pitch = case
    g = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, 48, 40, 32, 48.0, 40.0, 32.0, 1.5)
    angles = (3.0 + np.arange(6) * 60.0).astype(np.float32)
    offsets = np.tile(np.array([[1.0, -2.0]], np.float32), (6, 1))
    gen = torch.Generator(device=cuda)
    gen.manual_seed(17)
    td, code = (torch.float32, L.CBCT_F32) if storage == "f32" else (torch.bfloat16, L.CBCT_BF16)
    vol = torch.rand((32, 40, 48), generator=gen, device=cuda).to(td)
    outs = []
    for kernel in (1, 5, 0):
        plan = gtb.Plan(g, angles, offsets)
        plan.set_option(L.CBCT_OPT_DEBUG_CHECKS, 1)
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        assert kernel == 0 or plan.forward_variant() == ("tma-slab" if kernel == 1 else "tma-quad")
        out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
        plan.forward(vol, out, vol_dtype=code)
        assert plan.read_flags() == (0, 0)
        outs.append(out)
    assert float(outs[0].abs().max()) > 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])

"""Which projector a launch takes, and row quads in the tile shapes of automatic plans: rows
0.95 texel apart take the thin shape, 1.1 the skewed one, in launches of enough rays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(gtb, n, W, H, pitch, subsets):
    L = gtb._lib
    P = sum(subsets)
    g = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                       float(n[2]), 1.5)
    return gtb.Plan(g, (7.0 + np.arange(P) * (360.0 / P)).astype(np.float32),
                    np.tile(np.array([[1.0, -1.0]], np.float32), (P, 1)), np.array(subsets, np.int32))


# detectors that the volume's height covers, a million rays and more
@pytest.mark.parametrize("n,pitch,storage", [((64, 64, 96), 1.364, "f32"), ((64, 64, 96), 1.364, "bf16"),
                                             ((64, 64, 104), 1.58, "f32"), ((64, 64, 108), 1.58, "f16")])
def test_automatic_thin_and_skewed(gtb, cuda, n, pitch, storage):
    import torch
    L = gtb._lib
    td, code = {"f32": (torch.float32, L.CBCT_F32), "f16": (torch.float16, L.CBCT_F16),
                "bf16": (torch.bfloat16, L.CBCT_BF16)}[storage]
    gen = torch.Generator(device=cuda)
    gen.manual_seed(11)
    vol = torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda).to(td)
    outs = []
    for kernel in (1, 0):
        plan = _plan(gtb, n, 129, 97, pitch, [90])
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        # 16-bit volumes with rows beyond a texel take the slab kernel
        quads = kernel == 0 and not (storage == "f16" and pitch > 1.5)
        assert plan.launch_variant(-1, code) == ("tma-quad" if quads else "tma-slab")
        out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
        plan.forward(vol, out, vol_dtype=code)
        assert plan.read_flags() == (0, 0)
        outs.append(out)
    assert float(outs[0].max()) > 1.0
    assert torch.equal(outs[0], outs[1])


def test_names(gtb, cuda):
    L = gtb._lib
    plan = _plan(gtb, (128, 128, 96), 256, 192, 0.7, [40, 1])
    assert plan.forward_variant() == "tma-quad"
    assert plan.launch_variant(0) == "tma-quad" and plan.launch_variant(1) == "tma-slab"
    assert plan.launch_variant(2) == "" and plan.launch_variant(0, 7) == ""
    # rows 1.3 texels apart: no launch takes quads, and the plan says so
    assert _plan(gtb, (128, 128, 192), 256, 192, 1.8, [60]).forward_variant() == "tma-slab"
    # odd sizes: a forced pair or fan kernel becomes the slab kernel
    plan = _plan(gtb, (127, 125, 96), 256, 192, 0.7, [40])
    assert plan.launch_variant() == "tma-quad"
    for kernel, name in ((4, "tma-slab"), (3, "tma-slab"), (2, "gather"), (5, "tma-quad")):
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        assert plan.launch_variant() == name


def test_autotuned_plans_keep_the_rule_of_small_launches(gtb, cuda):
    """The autotuner times the largest subset; a launch of one view is not that."""
    import torch
    plan = _plan(gtb, (128, 128, 96), 256, 192, 0.7, [60, 1])
    plan.autotune()
    assert plan.launch_variant(0) == "tma-quad"     # three million rays
    assert plan.launch_variant(1) == "tma-slab"
    gen = torch.Generator(device=cuda)
    gen.manual_seed(3)
    vol = torch.rand(plan.vol_shape, generator=gen, device=cuda)
    a = plan.forward(vol, torch.empty(plan.proj_shape(1), device=cuda), 1)
    plan.set_option(gtb._lib.CBCT_OPT_FORWARD_KERNEL, 5)
    assert plan.launch_variant(1) == "tma-quad"     # forced again
    assert torch.equal(a, plan.forward(vol, torch.empty(plan.proj_shape(1), device=cuda), 1))


# rows 0.8 texel apart under covered detectors, 0.5 under detectors taller than the volume:
# scans of some 300,000 rays per subset, which take the slab kernel alone and quads in the
# work lists of a batch (two groups of three)
@pytest.mark.parametrize("W,H,pitch,nz", [(256, 96, 1.15, 80), (160, 144, 0.7, 56)])
def test_batches_promote_quads(gtb, cuda, W, H, pitch, nz):
    import torch
    jobs, alone = [], []
    for i in range(6):
        n = 48 + 8 * (i % 3)
        plan = _plan(gtb, (n, n, nz), W, H, pitch, [12, 12])
        assert plan.forward_variant() == "tma-quad" and plan.launch_variant(0) == "tma-slab"
        gen = torch.Generator(device=cuda)
        gen.manual_seed(23 + i)
        b = 10.0 * torch.rand(plan.proj_shape(), generator=gen, device=cuda)
        z = torch.empty(plan.vol_shape, dtype=torch.float32, device=cuda)
        plan.osmom(b, z, None, 2, nonneg=True)
        alone.append(z)
        jobs.append(dict(plan=plan, b=b, z=torch.empty_like(z), iterations=2, nonneg=True))
    gtb.batch_osmom(jobs, fused=True)
    for z, j in zip(alone, jobs):
        assert float(z.abs().max()) > 0
        assert torch.equal(z, j["z"])

"""Volumes and detectors whose rows are not a multiple of 16 bytes: the TMA
kernels read row-padded copies.  Every call is held to the kernels that load
global memory directly, which take the same samples and differ in rounding only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# sums of at most 320 samples or views of like sign, another order of the same
# multiply-adds: n 2^-24 = 2e-5 at most
TOL = 2e-5

SIZES = [((30, 27, 21), 45, 34, 7), ((33, 40, 18), 38, 51, 6), ((44, 35, 16), 47, 40, 5), ((41, 42, 43), 61, 50, 130)]


def _plan(gtb, n, W, H, P, subsets=None, offcorr=None):
    L = gtb._lib
    pitch = 1.2 * 1.5 * max(n) / W
    cg = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]),
                        float(n[2]), 1.5)
    angles = (5.0 + np.arange(P) * (360.0 / P)).astype(np.float32)
    plan = gtb.Plan(cg, angles, np.tile(np.array([[2.0, 0.5]], np.float32), (P, 1)), subsets, offcorr)
    return plan


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("size", SIZES)
def test_forward_odd(gtb, cuda, size, storage):
    import torch
    L = gtb._lib
    n, W, H, P = size
    gen = torch.Generator(device=cuda)
    gen.manual_seed(3)
    td = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[storage]
    code = {"f32": L.CBCT_F32, "f16": L.CBCT_F16, "bf16": L.CBCT_BF16}[storage]
    flat = torch.rand(n[0] * n[1] * n[2] + 1, generator=gen, device=cuda).to(td)
    plan = _plan(gtb, n, W, H, P)
    for start in (0, 1):      # start 1: an array that does not begin on a 16-byte boundary
        vol = flat[start:start + n[0] * n[1] * n[2]].view(n[2], n[1], n[0])
        outs = []
        for kernel in (2, 1, 4, 5, 0):
            plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
            out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
            plan.forward(vol, out, vol_dtype=code)
            assert plan.read_flags() == (0, 0)
            outs.append(out)
        for o in outs[1:]:
            assert _rel(o, outs[0]) <= TOL
            assert torch.equal(o, outs[1])


@pytest.mark.parametrize("size", SIZES)
def test_backproject_odd(gtb, cuda, size):
    import torch
    L = gtb._lib
    n, W, H, P = size
    gen = torch.Generator(device=cuda)
    gen.manual_seed(4)
    proj = torch.rand((P, H, W), generator=gen, device=cuda)
    start = torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda)
    mask = (torch.rand((n[2], n[1], n[0]), generator=gen, device=cuda) > 0.3).to(torch.uint8)
    for masked in (False, True):
        for accumulate in (False, True):
            for flags in (0, L.CBCT_BP_FDK_WEIGHT):
                outs = []
                for gather in (1, 0):
                    plan = _plan(gtb, n, W, H, P)
                    plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)   # global loads in both projectors
                    if masked:
                        plan.set_mask(mask)
                    out = start.clone()
                    plan.backproject(proj, out, -1, flags, True, accumulate)
                    assert plan.read_flags() == (0, 0)
                    outs.append(out)
                assert _rel(outs[1], outs[0]) <= TOL


def test_solvers_odd(gtb, cuda):
    """The solver epilogues over padded copies, and a solve of more views than a
    padded copy holds (its preconditioner runs in chunks)."""
    import torch
    L = gtb._lib
    n, W, H, P = SIZES[3]
    gen = torch.Generator(device=cuda)
    gen.manual_seed(6)
    b = torch.rand((P, H, W), generator=gen, device=cuda)
    for subsets in ([44, 43, 43], [130]):
        res = []
        for gather in (1, 0):
            plan = _plan(gtb, n, W, H, P, np.array(subsets, np.int32), [1] * len(subsets))
            plan.set_option(L.CBCT_OPT_FORCE_GATHER, gather)
            z = torch.empty(plan.vol_shape, dtype=torch.float32, device=cuda)
            x = torch.empty_like(z)
            pre = plan.osmom_precon(torch.empty_like(z))
            plan.osmom(b, z, None, 1, nonneg=True)
            plan.ossart(b, x, None, 1, nonneg=True)
            res.append((pre, z, x))
        for a, r in zip(res[1], res[0]):
            seen = r.abs() < 1e5      # voxels no view measures keep 1 / 1e-6
            # one iteration: three subset steps, each a few sums of the kind above
            assert _rel(a[seen], r[seen]) <= 10 * TOL

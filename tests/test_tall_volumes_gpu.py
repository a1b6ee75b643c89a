"""Volumes of many planes: the row-quad kernel's element index, counted from the volume's
corner, has to stay below 2^22, the slab kernel's below 2^24.  Plans beyond that take
another kernel; plans just inside it project as the gather kernel does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# planes, whether some shape of quads may run (the smallest box plane of 16-bit volumes, 40 x 5
# elements: 20,900 planes), whether the slab kernel may (fp32, 28 x 10: 59,900 planes)
CASES = [(12800, True, True), (20500, True, True), (31000, False, True), (60400, False, False)]


def _plan(gtb, nz, oy):
    L = gtb._lib
    g = L.CbctGeometry(1000.0, 1500.0, 96 * 0.3, 64 * 0.047, 96, 64, 64, 64, nz, 12.8, 12.8, 0.05 * nz, 1.5)
    angles = np.array([2.0, 95.0, 181.0], np.float32)
    return gtb.Plan(g, angles, np.tile(np.array([[0.5, oy]], np.float32), (3, 1)))


@pytest.mark.parametrize("nz,quads,slabs", CASES)
def test_choice(gtb, cuda, nz, quads, slabs):
    """Plan creation only."""
    L = gtb._lib
    plan = _plan(gtb, nz, 0.0)
    for kernel in (5, 0):
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        assert (plan.forward_variant() == "tma-quad") == quads, (kernel, plan.forward_variant())
    plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, 1)
    assert plan.forward_variant() == ("tma-slab" if slabs else "gather")


@pytest.mark.parametrize("nz,quads,slabs", CASES[:3])
def test_top_planes(gtb, cuda, nz, quads, slabs):
    """A detector shifted to see the volume's topmost planes.  Sums of 96 samples by two
    forms of the lerps: 96 x 2^-24 of the largest ray and three roundings per sample."""
    import torch
    test_choice(gtb, cuda, nz, quads, slabs)    # nothing is launched where the choice is wrong
    L = gtb._lib
    top = 0.5 * 0.05 * nz
    plan = _plan(gtb, nz, 1.5 * (top - 1.0))
    gen = torch.Generator(device=cuda)
    gen.manual_seed(2)
    vol = torch.rand((nz, 64, 64), generator=gen, device=cuda)
    outs = []
    for kernel in (2, 1, 5, 0):
        plan.set_option(L.CBCT_OPT_FORWARD_KERNEL, kernel)
        out = torch.full(plan.proj_shape(), -1.0, dtype=torch.float32, device=cuda)
        plan.forward(vol, out)
        assert plan.read_flags() == (0, 0)
        outs.append(out)
    assert float(outs[0].max()) > 1.0
    assert float((outs[1] - outs[0]).abs().max()) <= 1e-4 * float(outs[0].max())
    if quads:
        assert torch.equal(outs[2], outs[1])
    assert torch.equal(outs[3], outs[1])

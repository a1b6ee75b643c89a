"""Batches of small scans that fill the GPU together: their work lists may run row quads
where each scan alone takes the slab kernel; the volumes are bitwise those of the scans
solved alone either way, with and without residual traces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows about 0.45 and 0.8 texel apart under detectors the volume's height covers, and 0.5
# texel apart under taller ones; 3 scans of 12 views per subset, 300,000 rays or more
@pytest.mark.parametrize("W,H,pitch", [(160, 96, 0.64), (128, 72, 1.15), (160, 120, 0.7)])
@pytest.mark.parametrize("trace", [False, True])
def test_batch_equals_alone(gtb, cuda, W, H, pitch, trace):
    import torch
    L = gtb._lib
    jobs, alone, traces = [], [], []
    for i in range(3):
        n = 48 + 8 * i
        g = L.CbctGeometry(1000.0, 1500.0, W * pitch, H * pitch, W, H, n, n, 56, float(n), float(n), 56.0, 1.5)
        angles = ((np.arange(24) * 15.0 + 2.0 * i) % 360.0).astype(np.float32)
        plan = gtb.Plan(g, angles, np.zeros((24, 2), np.float32), [12, 12], [0, 0])
        gen = torch.Generator(device=cuda)
        gen.manual_seed(23 + i)
        b = 10.0 * torch.rand(plan.proj_shape(), generator=gen, device=cuda)
        z = torch.empty(plan.vol_shape, dtype=torch.float32, device=cuda)
        ra = torch.zeros(4, dtype=torch.float64, device=cuda)
        plan.osmom(b, z, None, 2, nonneg=True, resid=ra if trace else None)
        alone.append(z)
        job = dict(plan=plan, b=b, z=torch.empty_like(z), iterations=2, nonneg=True)
        if trace:
            job["resid"] = torch.zeros(4, dtype=torch.float64, device=cuda)
        traces.append(ra)
        jobs.append(job)
    gtb.batch_osmom(jobs, fused=True)
    for z, ra, j in zip(alone, traces, jobs):
        assert float(z.abs().max()) > 0
        assert torch.equal(z, j["z"])
        assert not trace or torch.equal(ra, j["resid"])

"""Offset weight of more views than a grid has layers (65,535)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [8, 7])
def test_offset_weight_of_70000_views(gtb, O, cuda, W):
    import torch
    L = gtb._lib
    H, P = 2, 70000
    g = L.CbctGeometry(1000.0, 1500.0, 10.0 * W, 10.0 * H, W, H, 8, 8, 8, 8.0, 8.0, 8.0, 1.5)
    og = O.Geometry(8, 8, 8, 8.0, 8.0, 8.0, W, H, 10.0 * W, 10.0 * H, 1000.0, 1500.0)
    offsets = np.zeros((P, 2), np.float32)
    offsets[:, 0] = 5.0 + np.arange(P) % 11
    plan = gtb.Plan(g, (np.arange(P) * (360.0 / P)).astype(np.float32), offsets)
    proj = torch.ones((P, H, W), dtype=torch.float32, device=cuda)
    plan.offset_correct(proj, -1, 0)
    last = O.offset_weight(og, np.ones((11, H, W)), offsets[-11:], 0)
    # FP32 column position and sine: some 1e-6 of pi/4
    assert O.rel_l2(proj[-11:].cpu().numpy(), last) < 1e-5
    assert O.rel_l2(proj[:11].cpu().numpy(), O.offset_weight(og, np.ones((11, H, W)), offsets[:11], 0)) < 1e-5

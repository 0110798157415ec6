"""Saved edge values of soft TRWP cover every entry: what no sweep visits (the first pixel of each chain)
reads zero even in buffers that were not cleared, for every split of the rows over warps."""
import numpy as np
import pytest
import torch

import cases
import gpu_runner as g
from mplayers_b200 import TRWP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,D,H,W", [(1, 4, 3, 5), (3, 4, 1, 1), (8, 8, 5, 4), (9, 16, 4, 6), (16, 4, 18, 3),
                                     (21, 4, 6, 35), (24, 4, 4, 4), (25, 8, 7, 3), (32, 4, 5, 9)])
def test_uncleared_buffers(L, D, H, W):
    rng = np.random.default_rng(L * 100 + D)
    unary = rng.standard_normal((1, 1, H, W, L)).astype(np.float32)
    ctx = cases.make_context("sym2d", L, rng)
    ew = rng.uniform(0.3, 1.4, size=(D, 1, 1, H, W)).astype(np.float32)
    want = g.forward_soft(unary, ctx, ew, D, 2)
    u, c, e = (torch.from_numpy(a).cuda() for a in (unary, ctx, ew))
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    msg = torch.zeros(D, 1, 1, H, W, L, device="cuda")
    el = torch.full((2, D, 1, 1, H, W, L, L), float("nan"), device="cuda")
    ni = torch.full((2, D, 1, 1, H, W), 255, dtype=torch.uint8, device="cuda")
    cost = torch.empty_like(u)
    TRWP.forward_soft(0.5, 2, u, c, e, msg, el, ni, cost, e0, e8)
    assert np.array_equal(el.cpu().numpy(), want["edge_label"])
    assert np.array_equal(ni.cpu().numpy(), want["norm_idx"])
    assert np.array_equal(cost.cpu().numpy(), want["cost"])

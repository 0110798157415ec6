"""Argmin of 17 .. 32 labels among equal minima.  The bulk-copy sweeps find it in two levels (the highest group of three
labels attaining the minimum, then the label inside it), so costs are quantised until minima tie inside one
group and across groups; every value is a small multiple of a power of two, hence exact, and the
indices have to be the oracle's: the highest label among equal ones."""
import numpy as np
import pytest

import gpu_runner as g
from oracle import oracle

pytestmark = pytest.mark.gpu


def tie_case(mode, D, B, H, W, L, weights):
    rng = np.random.default_rng(100 * L + D + W)
    unary = rng.integers(0, 4, size=(B, 1, H, W, L)).astype(np.float32)
    ctx = np.triu(rng.integers(1, 4, size=(L, L)), 1).astype(np.float32) + np.eye(L, dtype=np.float32)
    ew = rng.choice([0.5, 1.0, 2.0], size=(D, B, 1, H, W)).astype(np.float32) if weights else None
    return unary, np.maximum(ctx, ctx.T), ew


def lowest_indices(mode, unary, ctx, ew, D, I):
    """The LOWEST label among equal minima: the oracle on the labels in reverse."""
    L = unary.shape[-1]
    flip = oracle.forward(mode, unary[..., ::-1].copy(), ctx[::-1, ::-1].copy(), ew, D, I)
    return L - 1 - flip["min_idx"][..., ::-1].astype(int)


@pytest.mark.parametrize("L", [17, 18, 19, 24, 25, 28, 31, 32])
@pytest.mark.parametrize("mode,D,B,H,W,I,weights", [
    ("TRWP", 4, 1, 35, 36, 2, True),     # stages of 16 pixels: two full ones and a remainder
    ("TRWP", 4, 2, 16, 20, 1, False),
    ("TRWP", 8, 1, 18, 16, 2, True),
    ("ISGMR", 8, 8, 33, 36, 2, True),    # enough chains for the bulk-copy kernels: three staged arrays
])
def test_highest_label_among_equal_minima(L, mode, D, B, H, W, I, weights):
    unary, ctx, ew = tie_case(mode, D, B, H, W, L, weights)
    want = oracle.forward(mode, unary, ctx, ew, D, I)
    low = lowest_indices(mode, unary, ctx, ew, D, I)[0, :4]
    high = want["min_idx"][0, :4].astype(int)   # (pixels without a predecessor: 0 here, L - 1 there)
    same = (low // 3 == high // 3) & (low < high)
    apart = (low // 3 < high // 3)
    assert same.mean() > 0.01 and apart.mean() > 0.15
    got = g.forward(mode, unary, ctx, ew, D, I)
    assert np.array_equal(got["cost"], want["cost"])
    assert np.array_equal(got["msg"], want["msg"])
    assert np.array_equal(got["min_idx"], want["min_idx"])
    assert np.array_equal(got["norm_idx"], want["norm_idx"])

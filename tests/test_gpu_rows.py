"""Calls on padded label rows and from zero messages (mpl_rows) against the same call on packed rows
and given zeros.  The padding holds NaN, the message buffers of a zero start hold NaN: neither may
reach a result.  Forward results are equal bit for bit (same operations on the same labels); gradients
may sum in another order, so they are held to 1e-5 of the tensor's largest entry, ten times below
the tolerance against the oracle."""
import numpy as np
import pytest
import torch

import cases
import gpu_runner as g
from helpers import rel_err
from mplayers_b200 import ISGMR, TRWP, _lib

pytestmark = pytest.mark.gpu


def _rows(a, row):
    out = torch.full(a.shape[:-1] + (row,), float("nan"), device="cuda")
    out[..., :a.shape[-1]] = torch.from_numpy(a).cuda()
    return out


def _call(mode, unary, ctx, ew, D, I, dcost, window, keep, row):
    """Training-mode forward and backward on rows of `row` elements, cost labels-first."""
    L, rho = unary.shape[-1], 0.5 if mode == "TRWP" else 1.0
    u, c = _rows(unary, row), torch.from_numpy(ctx).cuda()
    b, cv, h, w, _ = u.shape
    e0 = torch.empty(0, device="cuda")
    ewt = torch.from_numpy(ew).cuda() if ew is not None else e0
    nan = lambda *s: torch.full(s, float("nan"), device="cuda")
    msg, mu, cost = nan(D, b, cv, h, w, row), nan(D, b, cv, h, w, row), nan(b, cv, L, h, w)
    mi = torch.full((I, D, b, cv, h, w, row), 255, dtype=torch.uint8, device="cuda")
    ni = torch.zeros(I, D, b, cv, h, w, dtype=torch.uint8, device="cuda")
    lab = torch.zeros(I if keep else 0, b, cv, h, w, dtype=torch.uint8, device="cuda")
    kw = dict(context_window=window, cost_labels_first=True, n_disp=L)
    if mode == "TRWP":
        TRWP.forward(rho, I, 0, u, c, ewt, msg, cost, mi, ni, e0, lab, messages_zero=True, **kw)
    else:
        ISGMR.forward(0, rho, I, 0, u, c, ewt, msg, cost, mi, ni, e0, mu, lab, messages_zero=True, **kw)
    du, dm, dmu = nan(b, cv, h, w, row), nan(D, b, cv, h, w, row), nan(D, b, cv, h, w, row)
    dc, de = torch.zeros_like(c), torch.zeros_like(ewt)
    gr = torch.from_numpy(np.ascontiguousarray(np.moveaxis(dcost, -1, 2))).cuda()
    if mode == "TRWP":
        TRWP.backward(rho, c, ewt, gr, mi, ni, du, dc, de, dm, e0, keep_diag=True, **kw)
    else:
        ISGMR.backward(0, rho, c, ewt, gr, mi, ni, du, dc, de, dm, e0, dmu, keep_diag=True, **kw)
    # inference from zero messages too (other kernels)
    cost2 = nan(b, cv, L, h, w)
    e8 = torch.empty(0, dtype=torch.uint8, device="cuda")
    msg.fill_(float("nan"))
    if mode == "TRWP":
        TRWP.forward(rho, I, 0, u, c, ewt, msg, cost2, e8, e8, e0, e8, messages_zero=True, **kw)
    else:
        mu.fill_(float("nan"))
        ISGMR.forward(0, rho, I, 0, u, c, ewt, msg, cost2, e8, e8, e0, mu, e8, messages_zero=True, **kw)
    return dict(cost=cost, cost2=cost2, msg=msg[..., :L], min_idx=mi[..., :L], norm_idx=ni, lab=lab, dunary=du[..., :L],
                dctx=dc, dew=de)


@pytest.mark.parametrize("mode,D,B,H,W,L,I,kind,ewk", [
    ("TRWP", 4, 1, 7, 9, 21, 3, "sym2d", True),      # odd width: one row per pixel staged in pieces
    ("TRWP", 4, 2, 33, 18, 5, 2, "sym2d", True),     # 16-label kernels, one padded piece
    ("ISGMR", 8, 2, 40, 36, 21, 3, "sym2d", True),   # diagonals; axis directions on padded bulk-copy tiles
    ("ISGMR", 8, 1, 12, 13, 31, 2, "tl1d", False),   # 1-D context, 32-label kernels
    ("TRWP", 8, 1, 9, 10, 13, 2, "sym2d", True),
    ("TRWP", 4, 1, 9, 11, 33, 3, "sym2d", True),     # two labels per lane, an odd count
    ("ISGMR", 8, 1, 10, 9, 63, 2, "sym2d", True),
    ("ISGMR", 4, 2, 8, 11, 46, 1, "sym2d", False),
    ("TRWP", 4, 1, 11, 14, 50, 3, "tl1d", False),    # several labels per lane
    ("TRWP", 8, 1, 9, 12, 67, 2, "tl1d", True),      # zero start beyond direction 3
    ("ISGMR", 8, 1, 13, 10, 101, 3, "tl1d", True),
    ("ISGMR", 8, 1, 375, 380, 34, 1, "tl1d", False), # enough chains that consumers stage for themselves
    ("ISGMR", 4, 1, 9, 8, 255, 2, "tq1d", False),
    ("TRWP", 4, 1, 5, 6, 70, 2, "sym2d", True),      # one CTA per chain
])
def test_padded_rows_and_zero_start(mode, D, B, H, W, L, I, kind, ewk):
    rng = np.random.default_rng(D * 1000 + H * 31 + L)
    unary = rng.standard_normal((B, 1, H, W, L)).astype(np.float32)
    ctx = cases.make_context(kind, L, rng)
    ew = rng.uniform(0.3, 1.4, size=(D, B, 1, H, W)).astype(np.float32) if ewk else None
    dcost = rng.uniform(size=unary.shape).astype(np.float32)
    window = 0 if ctx.ndim == 2 else _lib.analyze_context(torch.from_numpy(ctx).cuda())
    want = g.forward(mode, unary, ctx, ew, D, I, save_labels=True)
    ref = g.backward(mode, ctx, ew, dcost, want["min_idx"], want["norm_idx"], keep_diag=True)
    for row in sorted({L, (L + 3) & ~3}):
        got = {k: v.cpu().numpy() for k, v in _call(mode, unary, ctx, ew, D, I, dcost, max(window, 0), True, row).items()}
        assert np.array_equal(np.moveaxis(got["cost"], 2, -1), want["cost"]), row
        assert np.array_equal(np.moveaxis(got["cost2"], 2, -1), want["cost"]), row
        assert np.array_equal(got["msg"], want["msg"]), row
        assert np.array_equal(got["lab"], want["label_all"]), row
        assert np.array_equal(got["norm_idx"], want["norm_idx"]), row
        seen = got["min_idx"] != 255   # pixels without a predecessor have no index
        assert np.array_equal(got["min_idx"][seen], want["min_idx"][seen]) and not want["min_idx"][~seen].any(), row
        assert rel_err(got["dunary"], ref["dunary"]) < 1e-5, row
        assert rel_err(got["dctx"], ref["dctx"]) < 1e-5, row
        if ewk:
            assert rel_err(got["dew"], ref["dew"]) < 1e-5, row


@pytest.mark.parametrize("L", [33, 34, 35, 37, 63])
@pytest.mark.parametrize("mode,D,I", [("TRWP", 4, 2), ("ISGMR", 4, 2), ("ISGMR", 8, 3)])
def test_blocks_of_two_labels_per_lane(mode, D, I, L):
    """33 .. 64 labels with a table: the backward works in blocks of 16 steps and sums a row of gradients in two halves,
    the upper one of 15 labels at the least.  Chains of more than two blocks, and of one and a bit."""
    test_padded_rows_and_zero_start(mode, D, 1, 18, 35, L, I, "sym2d", True)


def test_rejects_bad_row_strides():
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    for row, n in ((23, 21), (28, 21), (21, 22)):   # no multiple of 4; not the next one; too few elements
        u, m = torch.zeros(1, 1, 4, 4, row, device="cuda"), torch.zeros(4, 1, 1, 4, 4, row, device="cuda")
        c = torch.zeros(n, n, device="cuda")
        with pytest.raises(RuntimeError):
            TRWP.forward(0.5, 1, 0, u, c, e0, m, torch.empty_like(u), e8, e8, e0, e8, n_disp=n)

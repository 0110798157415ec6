"""Sweep kernels that leave out candidates, share a warp between chains or read sums of earlier sweeps, at the sizes and
contexts where they can go wrong.  Forward results and saved indices have to be the oracle's bit for bit
(its arithmetic is followed operation by operation); gradients sum in another order and are held
to the tolerances of helpers.assert_grad_close."""
import types

import numpy as np
import pytest
import torch

import gpu_runner as g
import test_gpu_rows as rows
from helpers import assert_grad_close
from mplayers_b200 import MP_module, TRWP
from oracle import oracle

pytestmark = pytest.mark.gpu


def _table(kind, L, rng):
    if kind == "random":       # few candidates are live once messages have spread
        a = rng.uniform(0.0, 1.0, (L, L))
    elif kind == "potts":      # every column without its diagonal holds one value
        a = np.ones((L, L))
    elif kind == "zero":       # all candidates of a step are equal: all live, the highest label wins
        a = np.zeros((L, L))
    elif kind == "mixed":      # negative entries, a diagonal that is not the smallest
        a = rng.uniform(-1.0, 1.0, (L, L))
    elif kind == "ties":
        a = rng.integers(1, 4, (L, L)).astype(float)
    else:                      # "steep": costs of very different size
        a = 10.0 ** rng.uniform(-6, 6, (L, L))
    a = np.triu(a, 1)
    d = rng.uniform(-0.5, 0.5, L) if kind == "mixed" else np.zeros(L)
    return (a + a.T + np.diag(d)).astype(np.float32)


def _unary(kind, shape, rng):
    if kind in ("ties", "zero", "potts"):
        return rng.integers(0, 4, shape).astype(np.float32)
    return rng.standard_normal(shape).astype(np.float32)


def _same_forward(mode, unary, ctx, ew, D, I, training=True, **kw):
    want = oracle.forward(mode, unary, ctx, ew, D, I, msg_init=kw["msg_init"]) if "msg_init" in kw \
        else oracle.forward(mode, unary, ctx, ew, D, I)
    got = g.forward(mode, unary, ctx, ew, D, I, training=training, **kw)
    for k in ("cost", "msg") + (("min_idx", "norm_idx") if training else ()):
        assert np.array_equal(got[k], want[k]), k
    return want


@pytest.mark.parametrize("kind", ["random", "potts", "zero", "mixed", "ties", "steep"])
@pytest.mark.parametrize("mode,D,I,L,negative", [
    ("ISGMR", 8, 2, 64, False),
    ("ISGMR", 4, 3, 36, True),    # weights of both signs: the bounds change places
    ("TRWP", 4, 2, 60, True),
    ("TRWP", 8, 1, 40, False),
])
def test_live_labels(kind, mode, D, I, L, negative):
    rng = np.random.default_rng(L + D)
    shape = (1, 1, 13, 22, L)
    ew = rng.uniform(-0.5 if negative else 0.2, 1.0, (D,) + shape[:-1]).astype(np.float32)
    if kind in ("ties", "zero", "potts"):
        ew = np.sign(ew) * 2.0 ** np.round(2 * np.abs(ew))
    ctx, unary = _table(kind, L, rng), _unary(kind, shape, rng)
    _same_forward(mode, unary, ctx, ew.astype(np.float32), D, I)
    _same_forward(mode, unary, ctx, None, D, I, training=False)


@pytest.mark.parametrize("kind", ["random", "potts", "zero", "mixed", "ties", "steep"])
@pytest.mark.parametrize("D,L,negative", [(8, 21, False), (8, 32, True), (8, 3, False), (4, 24, True)])
def test_live_labels_up_to_32(kind, D, L, negative):
    """Enough chains in a launch that they fill the schedulers."""
    rng = np.random.default_rng(L + D)
    shape = (10 if D == 4 else 4, 1, 33, 38, L)
    ew = rng.uniform(-0.5 if negative else 0.2, 1.0, (D,) + shape[:-1]).astype(np.float32)
    if kind in ("ties", "zero", "potts"):
        ew = np.sign(ew) * 2.0 ** np.round(2 * np.abs(ew))
    ctx, unary = _table(kind, L, rng), _unary(kind, shape, rng)
    _same_forward("ISGMR", unary, ctx, ew.astype(np.float32), D, 2)
    _same_forward("ISGMR", unary, ctx, None, D, 2, training=False)


@pytest.mark.parametrize("L", [33, 34, 62, 63])
def test_live_labels_odd_counts(L):
    """Label counts that leave a lane with one label or none, on rows padded to a multiple of four."""
    rows.test_padded_rows_and_zero_start("ISGMR", 8, 1, 12, 19, L, 3, "sym2d", True)
    rows.test_padded_rows_and_zero_start("TRWP", 4, 1, 12, 19, L, 2, "sym2d", True)


@pytest.mark.parametrize("L,D,B,H,W", [
    (64, 8, 2, 30, 41),     # diagonal chains of 1 .. 30 pixels share warps
    (36, 8, 1, 35, 64),
    (64, 4, 1, 150, 150),   # chains longer than the table of a warp is kept
    (64, 4, 1, 3, 300),
    (32, 8, 2, 30, 41),     # eight lanes per chain
    (20, 8, 2, 30, 41),
    (4, 4, 2, 150, 151),
    (24, 8, 2, 30, 41),     # a 1-D context, whose table is folded
    # enough chains for the kernel (directions x images x shorter sides >= 2368), and just too few
    (64, 8, 10, 30, 41), (64, 8, 9, 30, 41), (36, 8, 9, 35, 64), (64, 4, 4, 150, 150), (64, 4, 60, 10, 120),
    (32, 8, 10, 30, 41), (20, 8, 10, 30, 41), (4, 4, 4, 150, 151), (24, 8, 10, 30, 41),
])
def test_backward_lanes_share_a_chain(L, D, B, H, W):
    rng = np.random.default_rng(L + W)
    shape = (B, 1, H, W, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _table("random", L, rng)
    if L == 24:
        ctx = _truncated("linear", 3, L)
    ew = rng.uniform(0.2, 1.0, (D,) + shape[:-1]).astype(np.float32)
    want = _same_forward("ISGMR", unary, ctx, ew, D, 2)
    dcost = rng.uniform(-1, 1, shape).astype(np.float32)
    ref = oracle.backward("ISGMR", ctx, ew, dcost, want["min_idx"], want["norm_idx"])
    got = g.backward("ISGMR", ctx, ew, dcost, want["min_idx"], want["norm_idx"])
    again = g.backward("ISGMR", ctx, ew, dcost, want["min_idx"], want["norm_idx"])
    for k in ("dunary", "dctx", "dew"):
        assert_grad_close(got[k], ref[k], k)
        assert np.array_equal(got[k], again[k]), k
    none = g.backward("ISGMR", ctx, None, dcost, want["min_idx"], want["norm_idx"], keep_diag=True)
    assert_grad_close(none["dctx"], oracle.backward("ISGMR", ctx, None, dcost, want["min_idx"], want["norm_idx"],
                                                    keep_diag=True)["dctx"], "dctx")


@pytest.mark.parametrize("L", [5, 21, 31, 33, 38, 63])
def test_backward_lanes_share_a_chain_padded(L):
    for B in (2, 10):
        rows.test_padded_rows_and_zero_start("ISGMR", 8, B, 30, 41, L, 2, "sym2d", True)


def _truncated(kind, R, L):
    """Saturates at offset R; "quantised" costs tie often, "dip" is not smallest at offset 0."""
    k = np.arange(L, dtype=np.float64)
    c = np.minimum(k, R) if kind != "quadratic" else np.minimum(k, R) ** 2
    if kind == "dip":
        c[0] = 0.5
        c[1:R] = 0.25
    return c.astype(np.float32)


@pytest.mark.parametrize("kind", ["linear", "quadratic", "dip"])
@pytest.mark.parametrize("mode,D,B,H,W,L,R", [
    ("TRWP", 4, 1, 19, 36, 16, 2),     # tiled copies
    ("TRWP", 4, 1, 18, 17, 13, 2),     # one row per pixel
    ("TRWP", 8, 1, 12, 20, 21, 4),
    ("ISGMR", 8, 8, 33, 36, 32, 3),
    ("ISGMR", 8, 1, 12, 13, 31, 1),
    ("ISGMR", 4, 8, 32, 36, 2, 1),
    ("TRWP", 4, 1, 20, 24, 24, 6),     # wider than a narrow window
])
def test_narrow_windows(kind, mode, D, B, H, W, L, R):
    rng = np.random.default_rng(L + R)
    shape = (B, 1, H, W, L)
    ctx = _truncated(kind, R, L)
    unary = rng.integers(0, 6, shape).astype(np.float32) / 2
    ew = rng.choice([0.0, 0.5, 1.0, 2.0], (D,) + shape[:-1]).astype(np.float32)
    _same_forward(mode, unary, ctx, ew, D, 2)
    _same_forward(mode, unary, ctx, None, D, 2, training=False)
    ew[:, :, :, H // 2:, W // 3] = -1.0    # stages and steps with a negative weight evaluate every candidate
    _same_forward(mode, unary, ctx, ew, D, 2)
    _same_forward(mode, unary, ctx, ew, D, 2, training=False)


@pytest.mark.parametrize("L", [36, 52, 64])
@pytest.mark.parametrize("R,kind,I", [(1, "linear", 2), (2, "linear", 3), (3, "dip", 2), (4, "quadratic", 2)])
def test_two_chains_per_warp(L, R, kind, I):
    """Chains of one image in eight directions, diagonal ones of different length next to each other."""
    rng = np.random.default_rng(L + R)
    shape = (2, 1, 61, 98, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _truncated(kind, R, L)
    ew = rng.uniform(0.0, 1.4, (8,) + shape[:-1]).astype(np.float32)
    _same_forward("ISGMR", unary, ctx, ew, 8, I, training=False)


@pytest.mark.parametrize("L,R,I", [(68, 3, 2), (128, 8, 1), (132, 2, 2), (256, 6, 1)])
def test_one_chain_per_warp_and_two_pieces(L, R, I):
    rng = np.random.default_rng(L + R)
    shape = (2, 1, 61, 98, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _truncated("linear", R, L)
    ew = rng.uniform(0.0, 1.4, (8,) + shape[:-1]).astype(np.float32)
    _same_forward("ISGMR", unary, ctx, ew, 8, I, training=False)


@pytest.mark.parametrize("L", [35, 50, 99, 137])
def test_many_chains_padded(L):
    rows.test_padded_rows_and_zero_start("ISGMR", 8, 2, 61, 98, L, 2, "tl1d", False)


@pytest.mark.parametrize("L,R,H,W", [(64, 2, 9, 14), (128, 4, 8, 11), (192, 2, 7, 12), (256, 7, 6, 9), (64, 3, 9, 1),
                                     (64, 3, 1, 9)])
@pytest.mark.parametrize("given", [False, True])
def test_sums_of_two_directions(L, R, H, W, given):
    """TRWP with four directions: directions 2 and 3 start from the sums that direction 1 wrote, from given messages too
    (those at the chains' first pixels stay as they are)."""
    rng = np.random.default_rng(L + W)
    shape = (2, 1, H, W, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _truncated("linear", R, L)
    ew = rng.uniform(0.1, 1.4, (4,) + shape[:-1]).astype(np.float32)
    kw = {"msg_init": rng.uniform(0, 1, (4,) + shape).astype(np.float32)} if given else {}
    _same_forward("TRWP", unary, ctx, ew, 4, 3, **kw)
    _same_forward("TRWP", unary, ctx, ew, 4, 2, training=False, **kw)


@pytest.mark.parametrize("L,R,I", [(64, 3, 1), (128, 2, 3), (192, 2, 2), (200, 6, 2)])
@pytest.mark.parametrize("labels_first", [False, True])
def test_costs_from_the_last_sweep(L, R, I, labels_first):
    """The caller does not need the messages: the last sweep stores the costs, in training too."""
    rng = np.random.default_rng(L + I)
    unary, ctx = rng.standard_normal((2, 1, 9, 14, L)).astype(np.float32), _truncated("linear", R, L)
    want = oracle.forward("TRWP", unary, ctx, None, 4, I)
    dev = lambda a: torch.from_numpy(a).cuda()
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    for training in (False, True):
        msg = torch.full((4,) + unary.shape, float("nan"), device="cuda")
        cost = torch.full((2, 1, L, 9, 14) if labels_first else unary.shape, float("nan"), device="cuda")
        mi = torch.zeros((I, 4) + unary.shape, dtype=torch.uint8, device="cuda") if training else e8
        ni = torch.zeros((I, 4) + unary.shape[:-1], dtype=torch.uint8, device="cuda") if training else e8
        TRWP.forward(0.5, I, 0, dev(unary), dev(ctx), e0, msg, cost, mi, ni, e0, e8, context_window=R,
                     cost_labels_first=labels_first, messages_zero=True, messages_needed=False)
        got = cost.cpu().numpy()
        assert np.array_equal(np.moveaxis(got, 2, -1) if labels_first else got, want["cost"])
        if training:
            assert np.array_equal(mi.cpu().numpy(), want["min_idx"]) and np.array_equal(ni.cpu().numpy(), want["norm_idx"])


@pytest.mark.parametrize("L", [1, 2, 21, 32, 33, 255, 256])
@pytest.mark.parametrize("H,W", [(8, 16), (3, 43), (1, 127), (5, 7), (4, 33)])
def test_layout_tiles(L, H, W):
    """Images of one tile, one pixel more, one less, and runs that are no multiple of four; data moves, bit for bit."""
    from mplayers_b200 import glue
    x = torch.from_numpy(np.random.default_rng(L + W).standard_normal((2, 1, L, H, W)).astype(np.float32)).cuda()
    last = glue.labels_last(x)
    assert torch.equal(last, x.permute(0, 1, 3, 4, 2)) and torch.equal(glue.labels_first(last), x)


@pytest.mark.parametrize("R", [2, 12])     # inside a narrow window, all candidates
@pytest.mark.parametrize("L", [4, 8, 12, 16, 20, 24, 28, 32])
def test_row_strides(L, R):
    rng = np.random.default_rng(L)
    unary = rng.standard_normal((2, 1, 9, 20, L)).astype(np.float32)
    ew = rng.uniform(0.2, 1.4, (4,) + unary.shape[:-1]).astype(np.float32)
    _same_forward("TRWP", unary, _truncated("linear", min(R, L - 1), L), ew, 4, 2, training=False)


@pytest.mark.parametrize("L", [1, 7, 10, 15, 18, 23, 27, 30])
def test_row_strides_padded(L):
    rows.test_padded_rows_and_zero_start("TRWP", 4, 2, 9, 20, L, 2, "tl1d", False)


@pytest.mark.parametrize("L,B,H,W", [(20, 8, 1, 40), (20, 6, 40, 1), (32, 8, 7, 23), (32, 8, 23, 7), (64, 3, 19, 20), (64, 2, 41, 30),
                                     (64, 12, 2, 9), (64, 40, 8, 20), (20, 60, 17, 5), (32, 13, 23, 40), (36, 70, 11, 5)])
def test_longest_chains_first(L, B, H, W):
    """Images much wider or higher than the other side, lines, and units of chains that end in mid direction."""
    test_backward_lanes_share_a_chain(L, 8, B, H, W)


@pytest.mark.parametrize("B,H,W", [(12, 7, 23), (12, 23, 7), (9, 1, 50), (8, 20, 21)])
@pytest.mark.parametrize("L", [52, 132])
def test_longest_chains_first_in_a_window(L, B, H, W):
    rng = np.random.default_rng(L + W)
    unary = rng.standard_normal((B, 1, H, W, L)).astype(np.float32)
    _same_forward("ISGMR", unary, _truncated("linear", 2, L), None, 8, 2, training=False)


@pytest.mark.parametrize("mode,D", [("TRWP", 4), ("TRWP", 8), ("ISGMR", 4), ("ISGMR", 8)])
@pytest.mark.parametrize("L,R", [(64, 3), (36, 2), (128, 6), (192, 12), (256, 15)])
@pytest.mark.parametrize("H", [2, 5, 8, 9, 11, 23])
def test_images_of_one_column(mode, D, L, R, H):
    """A column of such an image is contiguous in memory and copied in boxes of rows, of which the last may be a part."""
    rng = np.random.default_rng(L + H)
    unary, ctx = rng.standard_normal((2, 1, H, 1, L)).astype(np.float32), _truncated("linear", R, L)
    _same_forward(mode, unary, ctx, None, D, 2)
    _same_forward(mode, unary, ctx, None, D, 2, training=False)


@pytest.mark.parametrize("H,W", [(1, 9), (9, 1), (1, 2), (2, 1), (2, 2), (1, 1), (37, 6)])
@pytest.mark.parametrize("L,R,I,weights", [(64, 3, 1, False), (64, 2, 2, True), (36, 2, 1, True), (200, 4, 2, False)])
@pytest.mark.parametrize("labels_first", [False, True])
def test_costs_from_the_last_sweep_on_lines(H, W, L, R, I, weights, labels_first):
    """Images of one row or column have chains of one pixel, which no sweep walks; 2 x 2 and a column of several stages
    beside them, lanes with a part of their labels, weights."""
    rng = np.random.default_rng(L + 10 * H + W)
    unary, ctx = rng.standard_normal((2, 1, H, W, L)).astype(np.float32), _truncated("linear", R, L)
    ew = rng.uniform(0.1, 1.4, (4,) + unary.shape[:-1]).astype(np.float32) if weights else None
    want = oracle.forward("TRWP", unary, ctx, ew, 4, I)
    dev = lambda a: torch.from_numpy(a).cuda()
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    for training in (False, True):
        msg = torch.full((4,) + unary.shape, float("nan"), device="cuda")
        cost = torch.full((2, 1, L, H, W) if labels_first else unary.shape, float("nan"), device="cuda")
        mi = torch.zeros((I, 4) + unary.shape, dtype=torch.uint8, device="cuda") if training else e8
        ni = torch.zeros((I, 4) + unary.shape[:-1], dtype=torch.uint8, device="cuda") if training else e8
        TRWP.forward(0.5, I, 0, dev(unary), dev(ctx), dev(ew) if weights else e0, msg, cost, mi, ni, e0, e8,
                     context_window=R, cost_labels_first=labels_first, messages_zero=True, messages_needed=False)
        got = cost.cpu().numpy()
        assert np.array_equal(np.moveaxis(got, 2, -1) if labels_first else got, want["cost"])
        if training:
            assert np.array_equal(mi.cpu().numpy(), want["min_idx"]) and np.array_equal(ni.cpu().numpy(), want["norm_idx"])


@pytest.mark.parametrize("H,W", [(1, 23), (23, 1), (4, 6)])
@pytest.mark.parametrize("train", [False, True])
def test_module_on_lines(H, W, train):
    """The module asks for the costs with the labels first and for no messages."""
    rng = np.random.default_rng(H + W)
    unary, ctx = rng.standard_normal((1, 1, H, W, 64)).astype(np.float32), _truncated("linear", 3, 64)
    want = oracle.forward("TRWP", unary, ctx, None, 4, 3)["cost"]
    args = types.SimpleNamespace(mpnet_mrf_mode="TRWP", mpnet_max_iter=3, mpnet_n_dirs=4, n_classes=64,
                                 mpnet_smoothness_train="on" if train else None, mpnet_term_weight=1.0, mpnet_diag_value=0.0,
                                 enable_symmetric=True, mpnet_smoothness_mode="TL", mpnet_smoothness_trunct_value=-1,
                                 mpnet_smoothness_trunct_loc=-1, enable_cuda=True)
    layer = MP_module.MPModule(args)
    layer.set_label_context(torch.nn.Parameter(torch.from_numpy(ctx).cuda(), requires_grad=train), None, None)
    layer.train(train)
    x = torch.from_numpy(np.ascontiguousarray(np.moveaxis(unary, -1, 2))).cuda().requires_grad_(train)
    got = layer(x)[0].detach().cpu().numpy()
    assert np.array_equal(np.moveaxis(got, 2, -1), want)


@pytest.mark.parametrize("bad", ["nan pixel", "inf pixel", "nan label", "nan table"])
@pytest.mark.parametrize("mode,D,B,H,W,L,R", [    # R = 0: a label-by-label table
    ("TRWP", 4, 2, 9, 20, 21, 0), ("TRWP", 4, 2, 9, 20, 13, 0), ("TRWP", 4, 2, 9, 20, 28, 0), ("TRWP", 4, 2, 9, 20, 30, 0),
    ("TRWP", 4, 2, 9, 20, 31, 0), ("TRWP", 4, 2, 9, 20, 32, 0), ("TRWP", 4, 2, 9, 20, 1, 0),
    ("TRWP", 4, 2, 9, 19, 21, 0), ("TRWP", 4, 2, 9, 19, 15, 0), ("TRWP", 4, 2, 9, 19, 29, 0),
    ("TRWP", 4, 2, 9, 20, 21, 2), ("TRWP", 4, 2, 9, 20, 13, 2), ("TRWP", 4, 2, 9, 20, 32, 1),
    ("ISGMR", 8, 4, 33, 38, 21, 0), ("ISGMR", 8, 4, 33, 38, 19, 2), ("ISGMR", 8, 4, 33, 38, 32, 2),
    ("TRWP", 4, 1, 9, 14, 60, 0), ("ISGMR", 8, 1, 13, 22, 36, 0), ("ISGMR", 8, 3, 30, 41, 64, 0),
    ("TRWP", 4, 1, 9, 14, 37, 0), ("TRWP", 4, 1, 9, 14, 100, 0), ("TRWP", 4, 1, 9, 14, 39, 30),
])
def test_saved_argmin_is_a_label(bad, mode, D, B, H, W, L, R):
    """The backward pass addresses tables with the saved argmin: it is a label also where nothing is a minimum (NaN) or
    every candidate is infinite, in label counts that leave lanes idle too."""
    rng = np.random.default_rng(L + W)
    shape = (B, 1, H, W, L)
    unary = rng.standard_normal(shape).astype(np.float32)
    ctx = _truncated("linear", min(R, L - 1), L) if R else _table("random", L, rng)
    if bad == "nan table":
        if R:
            ctx[0] = np.nan
        else:
            ctx[0, L - 1] = ctx[L - 1, 0] = np.nan
    elif bad == "nan label":
        unary[..., H // 2, W // 2, L // 2] = np.nan
    else:
        unary[..., H // 2, W // 2, :] = np.nan if bad == "nan pixel" else np.inf
    ew = rng.uniform(0.2, 1.0, (D,) + shape[:-1]).astype(np.float32)
    got = g.forward(mode, unary, ctx, ew, D, 2)
    assert got["min_idx"].max() < L


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("mode,D,H,W,L,R", [
    ("TRWP", 4, 9, 14, 36, 2), ("TRWP", 4, 9, 14, 52, 2), ("TRWP", 4, 9, 14, 100, 4), ("TRWP", 4, 9, 14, 132, 7), ("ISGMR", 8, 9, 14, 200, 14),
    ("ISGMR", 4, 9, 14, 64, 16), ("ISGMR", 8, 9, 14, 33, 2),
])
def test_windowed_indices_of_undefined_minima(bad, mode, D, H, W, L, R):
    """A windowed sweep saves any byte where a pixel's costs are all NaN or infinite; the backward pass of the same call
    and calls after it stay sound."""
    rng = np.random.default_rng(L + W)
    shape = (2, 1, H, W, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _truncated("linear", R, L)
    ew = rng.uniform(0.2, 1.0, (D,) + shape[:-1]).astype(np.float32)
    dcost = rng.uniform(-1, 1, shape).astype(np.float32)
    want = _same_forward(mode, unary, ctx, ew, D, 2)
    ref = oracle.backward(mode, ctx, ew, dcost, want["min_idx"], want["norm_idx"])
    spoilt = unary.copy()
    spoilt[0, 0, H // 2, W // 2] = bad
    idx = g.forward(mode, spoilt, ctx, ew, D, 2)
    assert np.array_equal(idx["min_idx"][:, :, 1], want["min_idx"][:, :, 1])   # the other image
    got = g.backward(mode, ctx, ew, dcost, idx["min_idx"], idx["norm_idx"])
    assert_grad_close(got["dunary"][1], ref["dunary"][1], "dunary")
    again = g.backward(mode, ctx, ew, dcost, want["min_idx"], want["norm_idx"])
    for k in ("dunary", "dctx", "dew"):
        assert_grad_close(again[k], ref[k], k)


@pytest.mark.parametrize("L,R,I", [(64, 3, 2), (192, 2, 3), (128, 4, 1), (21, 2, 2)])
@pytest.mark.parametrize("needed", [True, False])
def test_costs_in_place_of_the_unaries(L, R, I, needed):
    """TRWP may write the costs into the buffer that holds the unaries."""
    rng = np.random.default_rng(L + I)
    unary, ctx = rng.standard_normal((2, 1, 9, 14, L)).astype(np.float32), _truncated("linear", R, L)
    want = oracle.forward("TRWP", unary, ctx, None, 4, I)
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    for training in (False, True):
        both = torch.from_numpy(unary).cuda()
        msg = torch.zeros((4,) + unary.shape, device="cuda")
        mi = torch.zeros((I, 4) + unary.shape, dtype=torch.uint8, device="cuda") if training else e8
        ni = torch.zeros((I, 4) + unary.shape[:-1], dtype=torch.uint8, device="cuda") if training else e8
        TRWP.forward(0.5, I, 0, both, torch.from_numpy(ctx).cuda(), e0, msg, both, mi, ni, e0, e8, messages_zero=True,
                     messages_needed=needed)
        assert np.array_equal(both.cpu().numpy(), want["cost"])
        if training:
            assert np.array_equal(mi.cpu().numpy(), want["min_idx"])


@pytest.mark.parametrize("stride", [4096, 4100, 5843, 6001, 12000, 40000])
@pytest.mark.parametrize("L", [3, 32, 40])
def test_layout_of_long_rows(stride, L):
    """The layout entry points take any row stride from the label count on."""
    from mplayers_b200 import _lib
    lib, H, W = _lib.lib(), 5, 53
    x = torch.from_numpy(np.random.default_rng(L).standard_normal((2, L, H, W)).astype(np.float32)).cuda()
    rows_, back = torch.full((2, H, W, stride), float("nan"), device="cuda"), torch.empty_like(x)
    st = torch.cuda.current_stream().cuda_stream
    assert lib.mpl_permute_lhw_to_rows(x.data_ptr(), rows_.data_ptr(), 2, L, H, W, stride, st) == 0
    assert lib.mpl_permute_rows_to_lhw(rows_.data_ptr(), back.data_ptr(), 2, L, H, W, stride, st) == 0
    assert torch.equal(rows_[..., :L], x.permute(0, 2, 3, 1)) and not rows_[..., L:].any() and torch.equal(back, x)


@pytest.mark.parametrize("L,B,H,W", [(64, 10, 30, 41), (20, 10, 30, 41), (36, 10, 30, 41)])
def test_infinite_gradient_stays_in_its_chains(L, B, H, W):
    """A chain whose gradient ends infinite shares its warp with longer ones: the cells of the context gradient that it does
    not touch stay finite."""
    rng = np.random.default_rng(L)
    shape = (B, 1, H, W, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _table("random", L, rng)
    ew = rng.uniform(0.2, 1.0, (8,) + shape[:-1]).astype(np.float32)
    want = _same_forward("ISGMR", unary, ctx, ew, 8, 1)
    dcost = rng.uniform(-1, 1, shape).astype(np.float32)
    dcost[3, 0, 0, 1, L // 2] = np.inf
    ref = oracle.backward("ISGMR", ctx, ew, dcost, want["min_idx"], want["norm_idx"])["dctx"]
    got = g.backward("ISGMR", ctx, ew, dcost, want["min_idx"], want["norm_idx"])["dctx"]
    finite = np.isfinite(ref)   # (the oracle's normalisation sum takes what its chain has scattered too: a few cells more)
    assert finite.any() and not finite.all()
    assert_grad_close(got[finite], ref[finite], "dctx")


@pytest.mark.parametrize("kind", ["random", "potts", "zero", "mixed", "ties", "steep"])
@pytest.mark.parametrize("D,B,H,W,L,I,negative", [
    (8, 16, 13, 22, 64, 2, False),   # steps over the longest chain's: 1664, as far above the line as the test can be
    (8, 4, 50, 52, 64, 1, True),     # 1600, on it
    (8, 4, 49, 62, 36, 2, False),    # just below, elongated: every candidate
    (8, 2, 48, 60, 48, 2, True),     # below, nearly square
    (4, 40, 13, 20, 56, 2, True),
    (4, 12, 30, 24, 40, 1, False),   # more chains than are resident in the other form
    (4, 2, 9, 20, 38, 2, True),      # inference of few labels takes the list, training does not
])
def test_live_labels_of_many_chains(kind, D, B, H, W, L, I, negative):
    """ISGMR on both sides of the line between the two 33 .. 64-label forms."""
    rng = np.random.default_rng(L + D)
    shape = (B, 1, H, W, L)
    ew = rng.uniform(-0.5 if negative else 0.2, 1.0, (D,) + shape[:-1]).astype(np.float32)
    if kind in ("ties", "zero", "potts"):
        ew = np.sign(ew) * 2.0 ** np.round(2 * np.abs(ew))
    ctx, unary = _table(kind, L, rng), _unary(kind, shape, rng)
    _same_forward("ISGMR", unary, ctx, ew.astype(np.float32), D, I)
    _same_forward("ISGMR", unary, ctx, None, D, I, training=False)


@pytest.mark.parametrize("L", [33, 34, 41, 62, 63])
@pytest.mark.parametrize("train", [False, True])
def test_live_labels_of_many_chains_padded(L, train):
    rows.test_padded_rows_and_zero_start("ISGMR", 8, 17, 12, 19, L, 2, "sym2d", train)
    rows.test_padded_rows_and_zero_start("ISGMR", 4, 1, 8, 30, L, 3, "sym2d", train)


@pytest.mark.parametrize("D,L,H,W", [(4, 64, 9, 26), (4, 44, 21, 8), (8, 64, 9, 13), (8, 33, 6, 17), (16, 60, 8, 9)])
def test_every_candidate_from_registers(D, L, H, W):
    """One direction in a launch; with many directions a stage is one or two pixels deep."""
    rng = np.random.default_rng(L + D)
    shape = (2, 1, H, W, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _table("mixed", L, rng)
    ew = rng.uniform(-0.5, 1.0, (D,) + shape[:-1]).astype(np.float32)
    _same_forward("TRWP", unary, ctx, ew, D, 2)
    _same_forward("TRWP", unary, ctx, None, D, 2, training=False)


@pytest.mark.parametrize("kind", ["random", "potts", "zero", "mixed", "ties", "steep"])
@pytest.mark.parametrize("D,B,H,W,L,negative", [
    (8, 10, 33, 38, 21, False), (8, 10, 33, 38, 32, True), (8, 10, 33, 38, 17, False), (8, 8, 33, 38, 3, False),
    (8, 8, 33, 36, 16, True),      # the other way would be one launch per axis direction
    (4, 9, 33, 36, 24, True),      # four directions, training: five rows staged
    (4, 19, 33, 36, 32, False),    # and too many of them
    (8, 3, 33, 95, 29, False),     # 792 steps over the longest chain's, one below the line, and 816
    (8, 3, 34, 95, 29, True),
])
def test_live_labels_up_to_32_by_size(kind, D, B, H, W, L, negative):
    """Both sides of the lines between the forms of several directions in a launch."""
    rng = np.random.default_rng(L + D)
    shape = (B, 1, H, W, L)
    ew = rng.uniform(-0.5 if negative else 0.2, 1.0, (D,) + shape[:-1]).astype(np.float32)
    if kind in ("ties", "zero", "potts"):
        ew = np.sign(ew) * 2.0 ** np.round(2 * np.abs(ew))
    ctx, unary = _table(kind, L, rng), _unary(kind, shape, rng)
    _same_forward("ISGMR", unary, ctx, ew.astype(np.float32), D, 2)
    _same_forward("ISGMR", unary, ctx, None, D, 2, training=False)


@pytest.mark.parametrize("kind", ["linear", "quadratic", "dip"])
@pytest.mark.parametrize("R", [1, 2, 3])     # 3 is no narrow window
@pytest.mark.parametrize("B,H,W,L", [
    (4, 33, 38, 2), (4, 33, 38, 13), (4, 33, 38, 31), (4, 33, 38, 32),   # two kernels, one of which returns at once
    (8, 33, 36, 13), (8, 33, 36, 32),                                     # this kernel for every context
    (10, 33, 70, 28),
])
def test_narrow_windows_of_many_chains(kind, R, B, H, W, L):
    rng = np.random.default_rng(L + R)
    shape = (B, 1, H, W, L)
    ctx = _truncated(kind, min(R, L - 1), L)
    unary = rng.integers(0, 6, shape).astype(np.float32) / 2
    ew = rng.choice([0.0, 0.5, 1.0, 2.0], (8,) + shape[:-1]).astype(np.float32)
    _same_forward("ISGMR", unary, ctx, ew, 8, 2)
    _same_forward("ISGMR", unary, ctx, None, 8, 2, training=False)
    ew[:, :, :, H // 2:, W // 3] = -1.0    # steps with a negative weight evaluate a list of candidates
    _same_forward("ISGMR", unary, ctx, ew, 8, 2)
    _same_forward("ISGMR", unary, ctx, ew, 8, 2, training=False)


@pytest.mark.parametrize("L", [2, 13, 21, 31])
@pytest.mark.parametrize("train", [False, True])
def test_narrow_windows_of_many_chains_padded(L, train):
    rows.test_padded_rows_and_zero_start("ISGMR", 8, 4, 33, 38, L, 2, "tl1d", train)
    rows.test_padded_rows_and_zero_start("ISGMR", 8, 10, 33, 38, L, 2, "tl1d", train)


@pytest.mark.parametrize("L,D,B,H,W", [
    (21, 8, 17, 20, 45), (21, 8, 25, 20, 45),      # elongated: 2720 steps over the longest chain's, and 4000
    (32, 8, 15, 20, 45), (28, 8, 18, 20, 45), (24, 8, 17, 20, 45),
    (48, 8, 17, 20, 39), (40, 8, 17, 20, 45), (40, 8, 18, 20, 45),
    (8, 8, 25, 20, 21), (8, 8, 24, 20, 21), (8, 8, 15, 20, 24),   # few labels; the last one against axis launches
    (64, 8, 296, 1, 9), (64, 8, 296, 9, 1), (20, 8, 500, 1, 9), (20, 8, 500, 9, 1),   # lines
])
def test_backward_lanes_share_a_chain_by_size(L, D, B, H, W):
    """Both sides of the lines between the backward forms, and images of one row or column above them."""
    test_backward_lanes_share_a_chain(L, D, B, H, W)


@pytest.mark.parametrize("L,R,B,H,W", [
    (64, 3, 20, 18, 7), (64, 2, 19, 18, 7),        # images x rows x labels 23040 and 21888
    (72, 2, 30, 13, 5), (72, 4, 28, 13, 5),        # lanes without labels: 28080 and 26208
    (200, 6, 10, 14, 9), (200, 3, 9, 14, 9),       # lanes with a part of theirs: 28000 and 25200
    (60, 2, 40, 20, 5),                            # none
])
def test_sums_of_two_directions_by_size(L, R, B, H, W):
    """Both sides of the line above which TRWP goes through the sums of two directions; the costs with the labels first come
    from the last sweep there."""
    rng = np.random.default_rng(L + B)
    shape = (B, 1, H, W, L)
    unary, ctx = rng.standard_normal(shape).astype(np.float32), _truncated("linear", R, L)
    ew = rng.uniform(0.1, 1.4, (4,) + shape[:-1]).astype(np.float32)
    _same_forward("TRWP", unary, ctx, ew, 4, 2)
    want = _same_forward("TRWP", unary, ctx, None, 4, 2, training=False)
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    msg = torch.full((4,) + shape, float("nan"), device="cuda")
    cost = torch.full((B, 1, L, H, W), float("nan"), device="cuda")
    TRWP.forward(0.5, 2, 0, torch.from_numpy(unary).cuda(), torch.from_numpy(ctx).cuda(), e0, msg, cost, e8, e8, e0, e8,
                 context_window=R, cost_labels_first=True, messages_zero=True, messages_needed=False)
    assert np.array_equal(np.moveaxis(cost.cpu().numpy(), 2, -1), want["cost"])


@pytest.mark.parametrize("L,B", [(64, 4), (64, 12), (61, 4), (60, 4), (56, 4)])
def test_many_chains_of_elongated_images(L, B):
    """Windows of more than four offsets: below 1776 steps over the longest chain's and above, label counts at the line."""
    rng = np.random.default_rng(L + B)
    unary = rng.standard_normal((B, 1, 20, 60, L)).astype(np.float32)
    _same_forward("ISGMR", unary, _truncated("linear", 6, L), None, 8, 2, training=False)
    if L & 3:
        rows.test_padded_rows_and_zero_start("ISGMR", 8, B, 20, 60, L, 2, "tq1d", False)

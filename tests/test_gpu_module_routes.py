"""Routes of the module calls and of wide-window inference against the general paths, bit for bit."""
import types

import numpy as np
import pytest
import torch

import cases
import gpu_runner as g
from mplayers_b200 import ISGMR, TRWP, MP_module, MP_module_hard_soft
from mplayers_b200 import glue
from mplayers_b200.glue import mp_on_scores

pytestmark = pytest.mark.gpu


def _wide_context(L, R, lift):
    """Quadratic up to offset R, then flat; `lift` > 0 makes offset 0 dearer than offset 1."""
    k = np.minimum(np.arange(L), R).astype(np.float64)
    c = 0.02 * k * k
    c[0] = lift
    return c.astype(np.float32)


@pytest.mark.parametrize("mode,D,H,W,L,R,I,lift", [
    ("ISGMR", 4, 9, 8, 36, 9, 2, 0.0),      # two warps of two labels per lane, fewest labels
    ("ISGMR", 4, 11, 13, 128, 15, 3, 0.0),  # the last count of that form
    ("ISGMR", 4, 6, 9, 132, 16, 2, 0.0),    # four warps: few chains, more than 128 labels
    ("ISGMR", 4, 130, 120, 132, 12, 2, 0.0),  # two warps of four labels per lane, partly filled lanes
    ("ISGMR", 8, 20, 18, 256, 15, 2, 0.1),  # aggregate mode; the smallest value not at offset 0
    ("TRWP", 4, 17, 10, 192, 10, 3, 0.0),
    ("TRWP", 8, 9, 12, 68, 15, 2, 0.1),
    ("TRWP", 6, 9, 12, 100, 12, 2, 0.0),    # direction count without an instance of its own
])
def test_wide_window_teams(mode, D, H, W, L, R, I, lift):
    rng = np.random.default_rng(L * 7 + R)
    unary = (3 * rng.standard_normal((1, 1, H, W, L))).astype(np.float32)
    ctx = _wide_context(L, R, lift)
    for ew in (None, rng.uniform(0.0, 1.4, size=(D, 1, 1, H, W)).astype(np.float32)):
        want = g.forward(mode, unary, ctx, ew, D, I, training=False, context_window=-1)   # every candidate
        got = g.forward(mode, unary, ctx, ew, D, I, training=False, context_window=R)
        assert np.array_equal(got["cost"], want["cost"])
        assert np.array_equal(got["msg"], want["msg"])


@pytest.mark.parametrize("shift", [1, 2])
@pytest.mark.parametrize("I", [1, 2])
def test_message_buffer_off_the_alignment(I, shift):
    """ISGMR writes one message buffer while it stages the other: one that takes no 16-byte stores (8 bytes off), or no
    8-byte ones (4 bytes off), goes to kernels that store smaller pieces."""
    D, H, W, L, R = 4, 11, 13, 256, 15   # four labels per lane, several warps per chain
    rng = np.random.default_rng(shift)
    unary = (3 * rng.standard_normal((1, 1, H, W, L))).astype(np.float32)
    ctx = _wide_context(L, R, 0.0)
    u, c = torch.from_numpy(unary).cuda(), torch.from_numpy(ctx).cuda()
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    for training in (False, True):
        want = g.forward("ISGMR", unary, ctx, None, D, I, training=training, context_window=R)
        for zero in (False, True):
            first, other = torch.zeros(D, 1, 1, H, W, L, device="cuda"), torch.zeros(shift + D * H * W * L, device="cuda")
            other = other[shift:].view(first.shape)
            # the buffer written by the first iteration is the second one for an even count
            msg, mu = (other, first) if I % 2 else (first, other)
            cost = torch.empty_like(u)
            mi = torch.zeros(I, D, 1, 1, H, W, L, dtype=torch.uint8, device="cuda") if training else e8
            ni = torch.zeros(I, D, 1, 1, H, W, dtype=torch.uint8, device="cuda") if training else e8
            ISGMR.forward(0, 1.0, I, 0, u, c, e0, msg, cost, mi, ni, e0, mu, e8, context_window=R, messages_zero=zero)
            assert np.array_equal(cost.cpu().numpy(), want["cost"])
            assert np.array_equal(msg.cpu().numpy(), want["msg"])
            if training:
                assert np.array_equal(mi.cpu().numpy(), want["min_idx"])


def _args(mode, D, I, L, train):
    return types.SimpleNamespace(mpnet_mrf_mode=mode, mpnet_max_iter=I, mpnet_n_dirs=D, n_classes=L,
                                 mpnet_smoothness_train="on" if train else None, mpnet_term_weight=1.0,
                                 mpnet_diag_value=0.0, enable_symmetric=True)


@pytest.mark.parametrize("mode,D,H,W,L", [("TRWP", 4, 9, 11, 21), ("TRWP", 4, 8, 12, 21), ("ISGMR", 8, 7, 8, 50),
                                          ("ISGMR", 8, 6, 9, 13)])
def test_labels_last_memory_and_scores(mode, D, H, W, L):
    rng = np.random.default_rng(L + W)
    rows = torch.from_numpy(rng.standard_normal((1, 1, H, W, L)).astype(np.float32)).cuda()
    ctx = torch.from_numpy(cases.make_context("sym2d", L, rng)).cuda()
    ew = torch.from_numpy(rng.uniform(0.3, 1.4, size=(1, D, H, W)).astype(np.float32)).cuda()
    up = torch.from_numpy(rng.uniform(size=(1, 1, L, H, W)).astype(np.float32)).cuda()
    layer = MP_module.MPModule(_args(mode, D, 2, L, True))
    layer.set_label_context(torch.nn.Parameter(ctx), None, None)
    layer.train()

    def run(u):
        u = u.detach().requires_grad_(True)
        out = layer(u, edge_weights=ew)[0]
        return out.detach(), torch.autograd.grad(out, u, up)[0]
    planes = rows.permute(0, 1, 4, 2, 3)                 # labels last in memory
    a, b = run(planes), run(planes.contiguous())
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    # the layer on scores: costs = max - scores, result negated
    scores = rows[:, 0].permute(0, 3, 1, 2).contiguous()
    costs = (scores.amax(1, keepdim=True) - scores).unsqueeze(1)
    want = -layer(costs, edge_weights=ew)[0].squeeze(1)
    assert torch.equal(mp_on_scores(layer, scores, ew)[0], want)


@pytest.mark.parametrize("L", [2, 5, 16, 17, 32, 36, 64, 67, 132, 256])
def test_labels_of_iterations(L):
    """Lowest label among equal minima, across lanes and rounds; costs quantised so that most minima tie."""
    rng = np.random.default_rng(L)
    unary = rng.integers(0, 3, size=(1, 1, 5, 7, L)).astype(np.float32)
    ctx = cases.make_context("potts2d", L, rng)
    got = g.forward("TRWP", unary, ctx, None, 4, 1, training=False, save_labels=True)
    assert np.array_equal(got["label_all"][0], got["cost"].argmin(-1).astype(np.uint8))


@pytest.mark.parametrize("mode", ["TRWP", "ISGMR"])
def test_label_count_argument_given_as_none(mode):
    """The label count is an optional argument of the autograd functions: passing its default changes nothing."""
    L, D, H, W = 7, 4, 5, 8
    rng = np.random.default_rng(3)
    u = torch.from_numpy(rng.standard_normal((1, 1, H, W, L)).astype(np.float32)).cuda().requires_grad_(True)
    c = torch.from_numpy(cases.make_context("sym2d", L, rng)).cuda().requires_grad_(True)
    args = types.SimpleNamespace(rho=0.5, mpnet_max_iter=2, mpnet_n_dirs=D, training=True, enable_min_a_dir=False,
                                 enable_sgm=False, enable_saving_label=False, msg_norm_index=None)
    fn = MP_module.TRWPFunction if mode == "TRWP" else MP_module.ISGMRFunction
    got = []
    for extra in ((), (None,), (L,)):
        cost = fn.apply(u, c, None, args, *extra)[0]
        got.append([cost.detach()] + list(torch.autograd.grad(cost, (u, c), torch.ones_like(cost))))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return None


def test_costs_without_a_gradient():
    """A consumer of the costs that hands back no gradient: zeros, from every autograd function."""
    L, H, W = 5, 6, 8
    u = torch.rand(1, 1, H, W, L, device="cuda", requires_grad=True)
    c = torch.rand(L, L, device="cuda", requires_grad=True)
    ew = torch.rand(4, 1, 1, H, W, device="cuda", requires_grad=True)
    args = types.SimpleNamespace(rho=0.5, mpnet_max_iter=2, mpnet_n_dirs=4, training=True, enable_min_a_dir=False,
                                 enable_sgm=False, enable_saving_label=False, msg_norm_index=None)
    for fn in (MP_module.TRWPFunction, MP_module.ISGMRFunction, MP_module_hard_soft.TRWPSoftFunction):
        out = _NoGradient.apply(fn.apply(u, c, ew, args)[0])
        for grad in torch.autograd.grad(out.sum(), (u, c, ew)):
            assert torch.equal(grad, torch.zeros_like(grad)), fn


def test_labels_last_memory_off_the_alignment():
    """A volume whose labels are last in memory is used as it is only where the 16-byte staging of the sweeps can."""
    buf = torch.rand(1 + 8 * 12 * 21, device="cuda")
    x = buf[1:].view(1, 1, 8, 12, 21).permute(0, 1, 4, 2, 3)
    y = glue.labels_last(x)
    assert y.data_ptr() % 16 == 0 and torch.equal(y, x.permute(0, 1, 3, 4, 2))
    aligned = buf[:-1].view(1, 1, 8, 12, 21).permute(0, 1, 4, 2, 3)
    assert glue.labels_last(aligned).data_ptr() == buf.data_ptr()


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("mode,D,H,W,L,R,I", [
    ("ISGMR", 4, 11, 13, 128, 15, 1),      # the unaries alone, both forms of the first iteration's buffers
    ("ISGMR", 4, 6, 9, 132, 9, 2),
    ("ISGMR", 4, 130, 120, 132, 12, 2),
    ("ISGMR", 8, 20, 18, 256, 16, 3),
    ("ISGMR", 8, 1000, 9, 36, 10, 2),      # enough chains for one warp each
    ("TRWP", 4, 17, 10, 192, 10, 3),       # directions 1 .. 3 of the first iteration: what exists so far
    ("TRWP", 6, 9, 12, 100, 12, 2),        # slices beyond direction 3 hold zeros
    ("TRWP", 8, 9, 12, 68, 16, 2),
])
def test_wide_window_zero_start(mode, D, H, W, L, R, I, training):
    """Messages known to be zero, in buffers of NaN, against the same call on given zeros."""
    rng = np.random.default_rng(L * 3 + R + D)
    unary = (3 * rng.standard_normal((1, 1, H, W, L))).astype(np.float32)
    ctx = _wide_context(L, R, 0.0)
    want = g.forward(mode, unary, ctx, None, D, I, training=training, context_window=R)
    u, c = torch.from_numpy(unary).cuda(), torch.from_numpy(ctx).cuda()
    e0, e8 = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.uint8, device="cuda")
    msg, mu = (torch.full((D, 1, 1, H, W, L), float("nan"), device="cuda") for _ in range(2))
    cost = torch.empty_like(u)
    mi = torch.zeros(I, D, 1, 1, H, W, L, dtype=torch.uint8, device="cuda") if training else e8
    ni = torch.zeros(I, D, 1, 1, H, W, dtype=torch.uint8, device="cuda") if training else e8
    kw = dict(context_window=R, messages_zero=True)
    if mode == "TRWP":
        TRWP.forward(0.5, I, 0, u, c, e0, msg, cost, mi, ni, e0, e8, **kw)
    else:
        ISGMR.forward(0, 1.0, I, 0, u, c, e0, msg, cost, mi, ni, e0, mu, e8, **kw)
    assert np.array_equal(cost.cpu().numpy(), want["cost"])
    assert np.array_equal(msg.cpu().numpy(), want["msg"])
    if training:
        assert np.array_equal(mi.cpu().numpy(), want["min_idx"])
        assert np.array_equal(ni.cpu().numpy(), want["norm_idx"])

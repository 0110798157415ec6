"""What a user of this framework has it compute, as measurable cases.

Every case is one pass through the public entry points: a module call (`MP_module.MPModule`,
`MP_module_hard_soft.MPModule`, `glue.mp_on_scores`) or, for training, that call and its backward
pass; the image-driven stereo case also builds its cost volume from the image pair
(`compute_terms.compute_all_terms`).  Inputs live on the GPU, the way a network or an input builder
hands them over.

Keys of a case:
  task     what the layer is used for: "seg" (class scores of a segmentation network, a learned
           label-by-label table), "stereo" (disparities, truncated linear function), "denoise"
           (grey values, truncated quadratic function), "dense" (arbitrary table, many labels)
  mode     "TRWP", "ISGMR", "SGM" or "SOFT" (TRWP with expected-value messages)
  train    forward and backward with gradients for unaries, pairwise function and edge weights
  batch, height, width, labels, dirs, iters
  trunc    offset at which the truncated function of a stereo / denoise case saturates
  weights  per-direction edge weights [B,D,H,W] are given
  scores   the call goes through glue.mp_on_scores (class scores in, class scores out)
  images   the unaries are built from an image pair inside the pass
  keep_labels  the labelling after every iteration is kept (energy curves)
"""
import math
import types

import torch

from mplayers_b200 import MP_module, MP_module_hard_soft
from mplayers_b200.compute_terms import compute_all_terms
from mplayers_b200.edge_weights import edge_weights_native
from mplayers_b200.glue import mp_on_scores


def _case(task, mode, batch, height, width, labels, dirs, iters, train=False, trunc=0, weights=False,
          scores=False, images=False, keep_labels=False):
    return dict(task=task, mode=mode, train=train, batch=batch, height=height, width=width, labels=labels, dirs=dirs,
                iters=iters, trunc=trunc, weights=weights, scores=scores, images=images, keep_labels=keep_labels)


def listed():
    cases = {
        # The smallest training step: the reference's CPU-runnable configuration; launches and the
        # latency of short chains.
        "seg_train_small": _case("seg", "TRWP", 1, 64, 64, 21, 4, 5, train=True, weights=True),
        # The segmentation training step of the benchmark (21 classes, full 512 x 512 crops).
        "seg_train": _case("seg", "TRWP", 2, 512, 512, 21, 4, 5, train=True, weights=True),
        # Evaluation of one photo of arbitrary size: odd width, no gradients.
        "seg_eval_ragged": _case("seg", "TRWP", 1, 375, 499, 21, 4, 5, weights=True),
        # Training at half resolution with diagonal directions, called on the network's scores.
        "seg_train_8dir": _case("seg", "ISGMR", 2, 256, 256, 21, 8, 5, train=True, weights=True, scores=True),
        # Training with expected-value (soft) messages at half resolution.
        "seg_soft_train": _case("seg", "SOFT", 1, 256, 256, 21, 4, 5, train=True, weights=True),
        # Disparities of a driving-sized image pair, from the two images to the final costs.
        "stereo_eval": _case("stereo", "TRWP", 1, 375, 1242, 192, 4, 3, trunc=2, images=True),
        # Learning the truncated function at that size: forward and backward.
        "stereo_train": _case("stereo", "TRWP", 1, 375, 1242, 192, 4, 3, train=True, trunc=2),
        # One semi-global pass in eight directions with penalties growing over a few disparities.
        "stereo_sgm": _case("stereo", "SGM", 1, 375, 1242, 128, 8, 1, trunc=4),
        # A smaller pair with edge weights from image gradients, a label count and a width that
        # are no multiple of anything, labellings kept after every iteration.
        "stereo_ragged": _case("stereo", "ISGMR", 1, 333, 449, 50, 8, 10, trunc=3, weights=True, keep_labels=True),
        # Energy minimisation with few labels and many iterations.
        "stereo_few_labels": _case("stereo", "TRWP", 1, 288, 384, 16, 4, 50, trunc=2, keep_labels=True),
        # Denoising of a grey image: 256 labels, wide window, many iterations.
        "denoise_eval": _case("denoise", "ISGMR", 1, 256, 256, 256, 4, 50, trunc=15),
        # The largest training step: arbitrary 64 x 64 table, eight directions, one megapixel.
        "dense_train_large": _case("dense", "ISGMR", 1, 1024, 1024, 64, 8, 10, train=True, weights=True),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["seg", "seg", "soft", "stereo", "stereo", "sgm", "denoise", "dense"])
    if kind == "seg":
        mode = rng.choice(["TRWP", "TRWP", "ISGMR"])
        c = _case("seg", mode, rng.randint(1, 2), _log_int(rng, 40, 512), _log_int(rng, 40, 512),
                  rng.choice([21, 21, rng.randint(2, 32)]), rng.choice([4, 8]), rng.randint(1, 5),
                  train=rng.random() < 0.6, weights=rng.random() < 0.7, scores=rng.random() < 0.3)
    elif kind == "soft":
        c = _case("seg", "SOFT", 1, _log_int(rng, 40, 256), _log_int(rng, 40, 256),
                  rng.choice([21, 21, rng.randint(2, 32)]), 4, rng.randint(1, 5), train=rng.random() < 0.7,
                  weights=rng.random() < 0.7)
    elif kind == "stereo":
        train, images = rng.random() < 0.35, False
        if not train:
            images = rng.random() < 0.5
        labels = _log_int(rng, 12, 192)
        c = _case("stereo", rng.choice(["TRWP", "ISGMR"]), 1, _log_int(rng, 96, 375), _log_int(rng, 128, 1242),
                  labels, rng.choice([4, 4, 8]), _log_int(rng, 1, 20) if not train else rng.randint(1, 4), train=train,
                  trunc=rng.randint(2, 4), weights=not images and rng.random() < 0.4, images=images,
                  keep_labels=not train and rng.random() < 0.3)
    elif kind == "sgm":
        c = _case("stereo", "SGM", 1, _log_int(rng, 96, 375), _log_int(rng, 128, 1242), _log_int(rng, 16, 192), 8, 1,
                  trunc=rng.randint(2, 8), weights=rng.random() < 0.3)
    elif kind == "denoise":
        side = _log_int(rng, 64, 256)
        c = _case("denoise", rng.choice(["TRWP", "ISGMR"]), 1, side, rng.randint(side * 3 // 4, side),
                  rng.choice([256, 256, _log_int(rng, 48, 256)]), 4, _log_int(rng, 4, 50), trunc=rng.randint(5, 15))
    else:
        c = _case("dense", "ISGMR", 1, _log_int(rng, 64, 512), _log_int(rng, 64, 512), rng.randint(33, 64),
                  rng.choice([4, 8]), rng.randint(1, 10), train=rng.random() < 0.7, weights=rng.random() < 0.7)
    return c


def _args(case):
    soft = case["mode"] == "SOFT"
    return types.SimpleNamespace(
        mpnet_mrf_mode="TRWP" if soft else case["mode"], mpnet_max_iter=case["iters"], mpnet_n_dirs=case["dirs"],
        n_classes=case["labels"], mpnet_smoothness_train="on" if case["train"] else None, mpnet_term_weight=1.0,
        mpnet_diag_value=0.0, enable_symmetric=True, mpnet_smoothness_mode="TL", mpnet_smoothness_trunct_value=-1,
        mpnet_smoothness_trunct_loc=-1, enable_cuda=True, mpnet_enable_soft=soft)


def _smooth(gen, b, c, h, w, cell):
    """Smooth random field in 0..1: coarse noise, interpolated."""
    coarse = torch.rand(b, c, max(h // cell, 2), max(w // cell, 2), device="cuda", generator=gen)
    return torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=True)


def _disparity(gen, h, w, labels):
    """Piecewise planar disparities: a few planes over random regions."""
    region = (_smooth(gen, 1, 1, h, w, 48)[0, 0] * 12).long()
    ys = torch.linspace(-1, 1, h, device="cuda").view(h, 1)
    xs = torch.linspace(-1, 1, w, device="cuda").view(1, w)
    p = torch.rand(13, 3, device="cuda", generator=gen)
    a, b, c = (p[:, 0] - 0.5) * 0.1 * labels, (p[:, 1] - 0.5) * 0.1 * labels, p[:, 2] * (labels - 1)
    return (a[region] * xs + b[region] * ys + c[region]).clamp(0, labels - 1)


def _image_pair(gen, h, w, labels):
    """A textured uint8 RGB pair whose right image is the left one displaced by the disparities."""
    disp = _disparity(gen, h, w, labels).round().long()
    left = 0.6 * _smooth(gen, 1, 3, h, w, 16)[0] + 0.4 * torch.rand(3, h, w, device="cuda", generator=gen)
    left = (255 * left).to(torch.uint8).permute(1, 2, 0).contiguous()
    src = (torch.arange(w, device="cuda").view(1, w) + disp).clamp(max=w - 1)
    right = torch.gather(left, 1, src.unsqueeze(2).expand(h, w, 3)).contiguous()
    return left, right


def _unary(case, gen):
    """[B,1,L,H,W] (class scores [B,L,H,W] where the call takes scores)."""
    b, h, w, n = case["batch"], case["height"], case["width"], case["labels"]
    if case["task"] == "seg":
        # network scores: noise, and a margin for the class of a blob map
        cls = torch.randint(0, n, (b, 1, max(h // 32, 1), max(w // 32, 1)), device="cuda", generator=gen).float()
        cls = torch.nn.functional.interpolate(cls, size=(h, w), mode="nearest").long()
        score = torch.randn(b, n, h, w, device="cuda", generator=gen)
        score.scatter_add_(1, cls, torch.full_like(score[:, :1], 3.0))
        if case["scores"]:
            return score
        cost = -score
        return (cost - cost.amin(dim=1, keepdim=True)).unsqueeze(1).contiguous()
    if case["task"] == "stereo":
        disp = _disparity(gen, h, w, n)
        lab = torch.arange(n, device="cuda", dtype=torch.float32).view(n, 1, 1)
        u = ((lab - disp).abs() / 8).clamp(max=1.0)
        u += 0.3 * torch.rand(n, h, w, device="cuda", generator=gen)
        outlier = torch.rand(h, w, device="cuda", generator=gen) < 0.1
        u = torch.where(outlier, torch.rand(n, h, w, device="cuda", generator=gen), u)
        return u.view(1, 1, n, h, w)
    if case["task"] == "denoise":
        img = (_smooth(gen, 1, 1, h, w, 32)[0, 0] * 8).floor() / 7 * (n - 1)
        obs = (img + 0.08 * n * torch.randn(h, w, device="cuda", generator=gen)).clamp(0, n - 1)
        lab = torch.arange(n, device="cuda", dtype=torch.float32).view(n, 1, 1)
        return ((lab - obs) ** 2 / n).view(1, 1, n, h, w)
    return torch.rand(b, 1, n, h, w, device="cuda", generator=gen)


def _context(case, gen):
    n = case["labels"]
    k = torch.arange(n, device="cuda", dtype=torch.float32)
    if case["task"] == "stereo":
        # image-driven costs are sums of three colour differences, given ones lie in 0..1.3
        return (20.0 if case["images"] else 1.0) * k.clamp(max=float(case["trunc"]))
    if case["task"] == "denoise":
        return 25.0 * (k * k).clamp(max=case["trunc"] ** 2 - 0.5 * case["trunc"])
    a = torch.triu((2.0 if case["task"] == "seg" else 1.0) * torch.rand(n, n, device="cuda", generator=gen), 1)
    return a + a.t()


def _weights(case, gen):
    """[B,D,H,W], or None."""
    if not case["weights"]:
        return None
    b, h, w, d = case["batch"], case["height"], case["width"], case["dirs"]
    if case["task"] == "dense":
        return 0.2 + 0.8 * torch.rand(b, d, h, w, device="cuda", generator=gen)
    img = 255 * _smooth(gen, b, 3, h, w, 8)
    return edge_weights_native("kernel_cue_real", img, d, sigma=10)[:, :, 0].permute(1, 0, 2, 3).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    args = _args(case)
    if case["mode"] == "SOFT" or (case["task"] == "seg" and case["mode"] == "TRWP" and not case["scores"]):
        layer = MP_module_hard_soft.MPModule(args, enable_saving_label=case["keep_labels"])
    else:
        layer = MP_module.MPModule(args, enable_saving_label=case["keep_labels"])
    context = torch.nn.Parameter(_context(case, gen), requires_grad=case["train"])
    layer.set_label_context(context, None, None)
    layer.train(case["train"])
    state = {"case": case, "layer": layer, "context": context, "weights": _weights(case, gen)}
    if case["images"]:
        state["left"], state["right"] = _image_pair(gen, case["height"], case["width"], case["labels"])
        return state
    state["unary"] = _unary(case, gen)
    if case["train"]:
        state["unary"].requires_grad_(True)
        if state["weights"] is not None:
            state["weights"].requires_grad_(True)
        state["upstream"] = torch.rand(state["unary"].shape, device="cuda", generator=gen)
    return state


def _call(state, unary):
    if state["case"]["scores"]:
        return [mp_on_scores(state["layer"], unary, state["weights"])[0]]
    out = state["layer"](unary, edge_weights=state["weights"])
    return [out[0], out[2]] if state["case"]["keep_labels"] else [out[0]]


def run(state):
    case = state["case"]
    if case["train"]:
        result = _call(state, state["unary"])[0]
        wanted = [state["unary"], state["context"]] + ([state["weights"]] if case["weights"] else [])
        return [result.detach()] + list(torch.autograd.grad(result, wanted, state["upstream"]))
    with torch.no_grad():
        if case["images"]:
            cost = compute_all_terms(state["left"], state["right"], "TL", 8, 2, float(case["trunc"]),
                                     case["labels"])[0]
            return _call(state, cost.permute(2, 0, 1).unsqueeze(0).unsqueeze(0))
        return _call(state, state["unary"])


def work(case):
    n = case["batch"] * case["height"] * case["width"]
    lab, d, it = case["labels"], case["dirs"], case["iters"]
    volume, edges = 4 * n * lab, 4 * n * d if case["weights"] else 0
    table = 4 * lab * (1 if case["trunc"] else lab)
    size = (6 * n if case["images"] else volume) + edges + table + volume
    if case["keep_labels"]:
        size += n * it
    if case["train"]:
        size += 2 * volume + edges + table
    # an addition and a minimum per candidate, the update of the unaries and the normalisation
    candidates = min(lab, 2 * case["trunc"]) if case["trunc"] else lab
    per_label = 2 * candidates + d + 4
    if case["mode"] == "SOFT":
        per_label += 3 * lab   # exponential, weighting and sum
    if case["train"]:
        per_label += 8 + (5 * lab if case["mode"] == "SOFT" else 0)
    return {"bytes": float(size), "flops": float(n * d * it * lab * per_label)}


def tolerance(case):
    """Forward values keep the order of their additions; in the backward pass the order is free.
    Against the same pass with its sums in the order of a direct evaluation the gradients were off by
    at most 1.9e-6 (2-norm) and 8.3e-5 (largest entry), soft costs by 9.6e-8 and 4.6e-7."""
    if case["train"]:
        return {"rel": 8e-6, "max": 4e-4}
    return {"rel": 2e-6, "max": 2e-5, "differ": 1e-4}


def _messages(h, e, ctx, soft):
    """New messages [N,L] of N pixels from their predecessors' terms h [N,L] and edge weights e [N]."""
    v = e.view(-1, 1, 1) * ctx + h.unsqueeze(1)
    m = (torch.softmax(-v, dim=2) * v).sum(2) if soft else v.amin(2)
    return m - m.amin(1, keepdim=True)


def _sweep(direction, uu, rho, e, ctx, soft):
    """Messages [B,H,W,L] of one direction, from uu [B,H,W,L] and edge weights e [B,H,W]."""
    hs, ws = ((0, 1), (0, -1), (1, 0), (-1, 0), (1, 1), (-1, -1), (1, -1), (-1, 1))[direction]
    if hs == 0:   # walk over columns: a vertical sweep of the transposed image
        new = _lines(uu.transpose(1, 2), e.transpose(1, 2), ws, 0, rho, ctx, soft)
        return new.transpose(1, 2)
    return _lines(uu, e, hs, ws, rho, ctx, soft)


def _lines(uu, e, step, shift, rho, ctx, soft):
    b, h, w, n = uu.shape
    new = torch.zeros(uu.shape, device=uu.device, dtype=uu.dtype)
    to, frm = slice(max(shift, 0), w + min(shift, 0)), slice(max(-shift, 0), w + min(-shift, 0))
    order = range(1, h) if step > 0 else range(h - 2, -1, -1)
    for y in order:
        term = rho * new[:, y - step, frm] + uu[:, y - step, frm]
        new[:, y, to] = _messages(term.reshape(-1, n), e[:, y, to].reshape(-1), ctx, soft).view(b, -1, n)
    return new


def exact(case, seed):
    """Final costs in 64 bits.  Gradients have no such value: near-equal candidates resolve to another
    label in another precision, and the gradient follows the label; nor have labellings.  The case
    with images starts from whole-number matching costs of its own and is left out."""
    if case["images"]:
        return None
    state = prepare(case, seed)
    with torch.no_grad():
        u = state["unary"].detach().double()
        if case["scores"]:
            u = u.amax(1, keepdim=True) - u
        else:
            u = u[:, 0]
        u = u.permute(0, 2, 3, 1).contiguous()
        n, dirs = case["labels"], case["dirs"]
        ctx = state["context"].detach().double()
        if ctx.dim() == 1:
            k = torch.arange(n, device="cuda")
            ctx = ctx[(k.view(n, 1) - k).abs()]
        if state["weights"] is None:
            e = torch.ones(u.shape[0], dirs, *u.shape[1:3], device="cuda", dtype=torch.float64)
        else:
            e = state["weights"].detach().double()
        soft, trwp = case["mode"] == "SOFT", case["mode"] in ("SOFT", "TRWP")
        rho = 0.5 if trwp else 1.0
        msg = [torch.zeros_like(u) for _ in range(dirs)]
        for _ in range(case["iters"]):
            read = msg if trwp else list(msg)
            for d in range(dirs):
                rest = u + sum(read[k] for k in range(dirs) if k != d)
                msg[d] = _sweep(d, rho * rest - read[d ^ 1], rho, e[:, d], ctx, soft)
        cost = (dirs if case["mode"] == "SGM" else 1) * u + sum(msg)
        cost = cost.permute(0, 3, 1, 2)
        cost = -cost if case["scores"] else cost.unsqueeze(1)
    return [cost] + [None] * (len(_output_names(case)) - 1)


def _output_names(case):
    """Names of what run returns."""
    names = ["scores" if case["scores"] else "costs"]
    if case["train"]:
        names += ["unary gradient", "context gradient"] + (["weight gradient"] if case["weights"] else [])
    elif case["keep_labels"] and not case["scores"]:
        names += ["labels"]
    return names

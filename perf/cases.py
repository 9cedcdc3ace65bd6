"""Workloads of the BP-Layers hot path, timed and compared through the calls a network makes.

Every case is one pass of a caller: a training step of a BP layer (forward, backward, all
gradients), a disparity or flow inference, a cost-volume layer forward and backward, or the
kernels of one served stereo request.  Sizes are those of this repository's benchmark, tests
and serving mix; `draw` spreads over the same ranges with odd sizes among them.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bp-layers_gb300"))

from bpl_gb300 import ops  # noqa: E402
from bpl_gb300.layers.matching import FlowMpSadFunction, StereoMatchingSadFunction  # noqa: E402
from bpl_gb300.layers.semantic import MessagePassingGlobal, MessagePassingPixel  # noqa: E402
from bpl_gb300.layers.stereo import BP, MessagePassing, pack_affinities  # noqa: E402

DEV = "cuda"
DELTA = 3            # the stereo and flow networks' truncation half-width
L1, L2 = 0.1, 0.5    # the benchmark's pairwise costs
LEFT, RIGHT, UP, DOWN = 0, 1, 2, 3


def _train(name, B, H, W, L, iters, storage="fp32", recompute=False, taps=3):
    return {"name": name, "kind": "train", "B": B, "H": H, "W": W, "L": L, "iters": iters, "storage": storage,
            "recompute": recompute, "taps": taps}


def listed():
    return [
        # the coarsest pyramid level of a small image: one call, launch and latency bound
        {"name": "infer_24x32x32", "kind": "infer", "B": 1, "H": 24, "W": 32, "L": 32, "iters": 1, "mode": "sub-exp"},
        # an ordinary disparity inference at half resolution
        {"name": "infer_188x620x96", "kind": "infer", "B": 1, "H": 188, "W": 620, "L": 96, "iters": 3, "mode": "wta"},
        # optical flow inference: u and v volumes of 65 labels, the reference's order
        {"name": "flow_bp_384x512x65", "kind": "flow_bp", "H": 384, "W": 512, "L": 65, "iters": 1, "mode": "wta"},
        # the full-size training step (scalar learnable L1 / L2, per-edge weights), FP32 and FP16 storage
        _train("train_376x1240x192", 1, 376, 1240, 192, 3),
        _train("train_fp16_376x1240x192", 1, 376, 1240, 192, 3, storage="fp16"),
        # a training batch that recomputes its argmin indices to save memory
        _train("train_recompute_4x256x512x96", 4, 256, 512, 96, 3, recompute=True),
        # learned per-pixel affinities (8 taps), an odd crop with an odd label count
        _train("train_affinities_187x311x70", 1, 187, 311, 70, 2, taps=5),
        # semantic segmentation layers, 19 classes, forward and backward
        {"name": "semantic_global_512x1024x19", "kind": "global", "B": 2, "H": 512, "W": 1024, "L": 19, "iters": 2},
        {"name": "semantic_pixel_512x1024x19", "kind": "pixel", "B": 1, "H": 512, "W": 1024, "L": 19, "iters": 1},
        # the cost-volume layers, forward and backward
        {"name": "sad_376x1240_C64_D192", "kind": "sad", "B": 1, "C": 64, "H": 376, "W": 1240, "L": 192},
        {"name": "flow_sad_384x512_C32_w65", "kind": "flow_sad", "B": 1, "C": 32, "H": 384, "W": 512, "L": 65},
        # a served request of the mix's most frequent size: features in, disparity map out
        {"name": "serve_376x1240x128", "kind": "serve", "B": 1, "C": 64, "H": 376, "W": 1240, "L": 128, "iters": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["infer", "flow_bp", "train", "train", "train", "global", "pixel", "sad", "flow_sad", "serve"])
    iters = rng.randint(1, 3)
    B, H, W = rng.choice([1, 1, 2, 4]), _log_int(rng, 24, 512), _log_int(rng, 32, 1240)
    if kind in ("global", "pixel"):
        L = rng.randint(5, 32)
        most = 2 * 512 * 1024 * 19 * (2 if kind == "global" else 0.5) // iters
    elif kind == "flow_sad":
        L = 2 * rng.randint(8, 54) + 1
        most = 384 * 512 * 65 * 65 // L
    else:
        L = _log_int(rng, 16, 256)
        most = 376 * 1240 * 192 * (2 if kind in ("infer", "serve", "train") else 1) // iters
    recompute = kind == "train" and rng.random() < 0.25
    if recompute:
        most //= 3
    while B * H * W * max(L, 64 if kind in ("infer", "flow_bp", "train", "serve") else 1) > most:
        B, H, W = max(1, B // 2), max(24, int(H * 0.8)), max(32, int(W * 0.8))
    case = {"kind": kind, "B": B, "H": H, "W": W, "L": L, "iters": iters}
    if kind == "train":
        taps = rng.choice([3, 3, 5])
        storage = "fp16" if not recompute and rng.random() < 0.3 else "fp32"
        case.update(storage=storage, recompute=recompute, taps=taps)
    elif kind in ("infer", "flow_bp"):
        case.update(mode=rng.choice(["wta", "sub-exp"]))
        if kind == "flow_bp":
            del case["B"]
            case["iters"] = 1
    elif kind in ("sad", "flow_sad", "serve"):
        case["C"] = rng.choice([16, 32, 48, 64]) if kind != "flow_sad" else rng.choice([16, 24, 32])
    if kind in ("sad", "flow_sad"):
        del case["iters"]
    return case


# ---------------------------------------------------------------------------
# inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(shape, device=DEV, generator=g)


def _planes(g, B, H, W, D, n=6):
    """Piecewise-planar disparities in [0, D-1]."""
    u = torch.rand((B, n, 5), device=DEV, generator=g)
    ys = torch.arange(H, device=DEV, dtype=torch.float32).view(1, 1, H, 1)
    xs = torch.arange(W, device=DEV, dtype=torch.float32).view(1, 1, 1, W)
    k = [u[:, :, i].view(B, n, 1, 1) for i in range(5)]
    cy, cx = k[0] * H, k[1] * W
    disp = (0.1 + 0.8 * k[2]) * D + (k[3] - 0.5) * 0.3 * D / W * (xs - cx) + (k[4] - 0.5) * 0.3 * D / H * (ys - cy)
    near = ((ys - cy) ** 2 + (xs - cx) ** 2).argmin(1, keepdim=True)
    return disp.gather(1, near)[:, 0].clamp(0, D - 1)


def _features(g, B, C, H, W, D):
    """Left features N(0,1), right ones the left warped by a planar scene plus N(0,0.1)."""
    f0 = _randn(g, B, C, H, W)
    src = (torch.arange(W, device=DEV).view(1, 1, W) + _planes(g, B, H, W, D).round().long()).clamp(0, W - 1)
    f1 = torch.gather(f0, 3, src.view(B, 1, H, W).expand(B, C, H, W)) + 0.1 * _randn(g, B, C, H, W)
    return f0, f1.contiguous()


def _prob_volume(g, B, H, W, L):
    """A matching network's probabilities: a peak at the scene's disparity over noise."""
    labels = torch.arange(L, device=DEV, dtype=torch.float32)
    score = 2.0 * _randn(g, B, H, W, L)
    score -= 2.0 * (labels - _planes(g, B, H, W, L).unsqueeze(-1)).abs().clamp(max=4.0)
    return torch.softmax(score, dim=-1).contiguous()


def _affinities(g, B, H, W):
    """Monotone positive affinities [L2-, L2+, L1-, L1+, L3] per direction, as the affinity network hands them over."""
    a = 0.05 + 1.45 * torch.rand((B, 4, 5, H, W), device=DEV, generator=g)
    a[:, :, 0] = torch.maximum(a[:, :, 0], a[:, :, 2])
    a[:, :, 1] = torch.maximum(a[:, :, 1], a[:, :, 3])
    a[:, :, 4] = torch.maximum(a[:, :, 4], torch.maximum(a[:, :, 0], a[:, :, 1]))
    return a


def _set_l1l2(mp):
    with torch.no_grad():
        mp._L1.fill_(L1)
        mp._L2.fill_(L2)
    return mp


def prepare(case, seed):
    g = _gen(seed)
    kind, H, W, L = case["kind"], case["H"], case["W"], case["L"]
    B = case.get("B", 1)
    s = dict(case)
    if kind == "train":
        s["prob"] = _prob_volume(g, B, H, W, L).requires_grad_(True)
        s["edge"] = torch.exp(0.3 * _randn(g, B, 4, H, W)).requires_grad_(True)
        s["aff"] = _affinities(g, B, H, W).requires_grad_(True) if case["taps"] == 5 else None
        # the gradient of an expected truncated disparity error, plus noise
        labels = torch.arange(L, device=DEV, dtype=torch.float32)
        s["up"] = (labels - _planes(g, B, H, W, L).unsqueeze(-1)).abs().clamp(max=8.0) / 8.0 + 0.1 * _randn(g, B, H, W, L)
        s["mp"] = _set_l1l2(MessagePassing(DEV, case["iters"], L, DELTA, storage=case["storage"],
                                           recompute_argmin=case["recompute"]))
    elif kind in ("infer", "flow_bp"):
        if kind == "infer":
            s["prob"] = _prob_volume(g, B, H, W, L)
        else:
            s["prob"] = torch.stack((_prob_volume(g, 1, H, W, L), _prob_volume(g, 1, H, W, L)), dim=1).contiguous()
        s["edge"] = torch.exp(0.3 * _randn(g, B, 4, H, W))
        s["bp"] = BP(DEV, None, case["iters"], L, DELTA, mode_inference=case["mode"])
        _set_l1l2(s["bp"].message_passing)
    elif kind in ("global", "pixel"):
        logits = 2.0 * _randn(g, B, H, W, L)
        bias = 2.0 * _randn(g, B, (H + 31) // 32, (W + 31) // 32, L)
        logits += bias.repeat_interleave(32, 1)[:, :H].repeat_interleave(32, 2)[:, :, :W]
        s["prob"] = torch.log_softmax(logits, dim=-1).requires_grad_(True)
        base = 0.2 + 1.3 * torch.rand((2, L, L), device=DEV, generator=g)
        base = 0.5 * (base + base.transpose(1, 2)) * (1.0 - torch.eye(L, device=DEV))
        if kind == "global":
            s["edge"] = torch.exp(0.3 * _randn(g, B, 4, H, W)).requires_grad_(True)
            s["jump"] = base.unsqueeze(0).contiguous().requires_grad_(True)
            s["mp"] = MessagePassingGlobal(DEV, case["iters"], L, L)
        else:
            s["jump"] = (base.view(2, 1, 1, L, L) * torch.exp(0.3 * _randn(g, 2, H, W, 1, 1))).requires_grad_(True)
            s["mp"] = MessagePassingPixel(DEV, case["iters"], L, L)
        s["up"] = _randn(g, B, H, W, L)
    elif kind == "sad":
        f0, f1 = _features(g, B, case["C"], H, W, L)
        s["f0"], s["f1"] = f0.requires_grad_(True), f1.requires_grad_(True)
        s["up"] = _randn(g, B, H, W, L)
    elif kind == "flow_sad":
        f0 = _randn(g, B, case["C"], H, W)
        # the second image: the first one moved by a few pixels, plus noise
        f1 = torch.roll(f0, (2, -3), (2, 3)) + 0.1 * _randn(g, B, case["C"], H, W)
        s["f0"], s["f1"] = f0.requires_grad_(True), f1.requires_grad_(True)
        s["up"] = [_randn(g, B, H, W, L) for _ in range(2)]
    else:
        # a serving slot: features, resident taps, cost, messages and result
        s["f0"], s["f1"] = _features(g, B, case["C"], H, W, L)
        aff = torch.full((1, 4, 3, H, W), L1, device=DEV)
        aff[:, :, 2] = L2
        s["taps"] = pack_affinities(aff, torch.zeros((1, 4, H, W), device=DEV))
        s["edge"] = torch.ones((1, 4, H, W), device=DEV)
        lp = ops.padded_labels(L)
        s["sad"] = torch.zeros((B, H, W, L), device=DEV)
        s["cost"] = torch.zeros((B, H, W, lp), dtype=torch.float16, device=DEV)
        s["msgs"] = torch.zeros((B, 4, H, W, lp), dtype=torch.float16, device=DEV)
        s["disp"] = torch.zeros((B, H, W), dtype=torch.int64, device=DEV)
    return s


# ---------------------------------------------------------------------------
# one pass

def _clear(*tensors):
    for t in tensors:
        if t is not None:
            t.grad = None


def run(s):
    kind, H, W, L = s["kind"], s["H"], s["W"], s["L"]
    B = s.get("B", 1)
    if kind == "train":
        mp, prob, edge, aff = s["mp"], s["prob"], s["edge"], s["aff"]
        _clear(prob, edge, aff, *mp.parameters())
        m0 = torch.zeros((B, 4, H, W, L), device=DEV, requires_grad=True) if s["storage"] == "fp32" else None
        beliefs, messages = mp(prob, edge, aff, None, m0)
        beliefs.backward(s["up"])
        out = {"beliefs": beliefs.detach(), "messages": messages.detach(), "g_prob": prob.grad, "g_edge": edge.grad,
               "g_T": mp.softmin.T.grad}
        if m0 is not None:
            out["g_messages"] = m0.grad
        if aff is not None:
            out["g_aff"] = aff.grad
        else:
            out["g_L1"], out["g_L2"] = mp._L1.grad, mp._L2.grad
        return out
    if kind in ("infer", "flow_bp"):
        with torch.no_grad():
            disp, beliefs, messages = s["bp"](s["prob"], s["edge"])
        return {"disp": disp, "beliefs": beliefs, "messages": messages}
    if kind in ("global", "pixel"):
        prob, jump, edge = s["prob"], s["jump"], s.get("edge")
        _clear(prob, jump, edge)
        m0 = torch.zeros((B, 4, H, W, L), device=DEV, requires_grad=True)
        beliefs = s["mp"](prob, edge, m0, jump)
        beliefs.backward(s["up"])
        out = {"beliefs": beliefs.detach(), "messages": m0.detach(), "g_prob": prob.grad, "g_jump": jump.grad,
               "g_messages": m0.grad}
        if edge is not None:
            out["g_edge"] = edge.grad
        return out
    if kind == "sad":
        _clear(s["f0"], s["f1"])
        sad = StereoMatchingSadFunction.apply(s["f0"], s["f1"], 0, L - 1)
        sad.backward(s["up"])
        return {"sad": sad.detach(), "g_f0": s["f0"].grad, "g_f1": s["f1"].grad}
    if kind == "flow_sad":
        _clear(s["f0"], s["f1"])
        cu, cv, us, vs = FlowMpSadFunction.apply(s["f0"], s["f1"], L - 1)
        torch.autograd.backward([cu, cv], s["up"])
        return {"cv_u": cu.detach(), "cv_v": cv.detach(), "u_star": us, "v_star": vs, "g_f0": s["f0"].grad,
                "g_f1": s["f1"].grad}
    ops.sad_forward(s["f0"], s["f1"], 0, L - 1, out=s["sad"])
    ops.cost_from_sad(s["sad"], 1.0, half=True, out=s["cost"])
    s["msgs"].zero_()
    for _ in range(s["iters"]):
        ops.lbp_forward_f16(ops.LBP_STEREO, s["cost"], s["taps"], s["edge"], s["msgs"], DELTA, L, argmin_dtype=None)
    ops.messages_argmin(s["msgs"], s["cost"], L, out=s["disp"])
    return {"disp": s["disp"], "messages": s["msgs"], "cost": s["cost"], "sad": s["sad"]}


def work(case):
    """Bytes: the inputs and outputs of a pass, each once.  Flops: the additions and comparisons of its updates
    (a min-sum message-label update about 12, its adjoint about 8; an absolute difference and its sum 2)."""
    kind, H, W, L = case["kind"], case["H"], case["W"], case["L"]
    B, it = case.get("B", 1), case.get("iters", 1)
    vol, px = B * H * W * L, B * H * W
    upd = 2 * L * B * (H * (W - 1) + W * (H - 1)) * it
    if kind == "train":
        m = 4 if case["storage"] == "fp32" else 2
        fp32 = case["storage"] == "fp32"
        return {"bytes": vol * (4 * 4 + 4 * m + (16 if fp32 else 0)) + px * 4 * 4 * (2 + (2 * 5 if case["taps"] == 5 else 0)),
                "flops": upd * 20}
    if kind == "infer":
        return {"bytes": vol * (4 + 4 + 16) + px * (16 + 8), "flops": upd * 12}
    if kind == "flow_bp":
        return {"bytes": 2 * vol * (4 + 4 + 16) + px * (16 + 16), "flops": 2 * upd * 12}
    if kind in ("global", "pixel"):
        jump = 2 * 2 * L * L * 4 * (1 if kind == "global" else H * W)
        return {"bytes": vol * (4 * 4 + 16 + 16) + jump + (px * 32 if kind == "global" else 0),
                "flops": upd * (2 * L + 8)}
    if kind == "sad":
        return {"bytes": 2 * vol * 4 + 4 * px * case["C"] * 4, "flops": 6 * vol * case["C"]}
    if kind == "flow_sad":
        return {"bytes": 6 * vol * 4 + 4 * px * case["C"] * 4, "flops": 2 * vol * L * case["C"] + 8 * vol * case["C"]}
    lp = (L + 7) // 8 * 8
    return {"bytes": 2 * px * case["C"] * 4 + vol * 4 + px * lp * 10 + px * 8, "flops": 2 * vol * case["C"] + upd * 8}


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch

def _pack64(aff):
    """(B,4,K,H,W) affinities -> (B,4,K+3,H,W) taps [offset, L3, L2-, L1-, 0, L1+, L2+, L3]."""
    B, _, K, H, W = aff.shape
    fwd = torch.zeros((B, 2, K + 3, H, W), dtype=torch.float64, device=DEV)
    rev = fwd.clone()
    even, odd = aff[:, 0::2], aff[:, 1::2]
    for t, a in ((fwd, even), (rev, odd)):
        t[:, :, 1] = t[:, :, K + 2] = a[:, :, K - 1]
    for i in range((K - 1) // 2):
        lo, hi = 2 + i, K + 1 - i
        fwd[:, :, lo], fwd[:, :, hi] = even[:, :, 2 * i], even[:, :, 2 * i + 1]
        rev[:, :, lo], rev[:, :, hi] = odd[:, :, 2 * i + 1], odd[:, :, 2 * i]
    return torch.stack((fwd[:, 0], rev[:, 0], fwd[:, 1], rev[:, 1]), dim=1)


class _Min64:
    """Min-sum passes and their adjoint over (B,H,W,L) in 64 bits, one line of pixels at a time."""

    def __init__(self, cost, edge, taps=None, jump=None, delta=DELTA, log_normalise=True):
        self.cost, self.edge, self.taps, self.jump, self.delta = cost, edge, taps, jump, delta
        self.B, self.H, self.W, self.L = cost.shape
        self.log_normalise = log_normalise
        self.msgs = torch.zeros((self.B, 4) + tuple(cost.shape[1:]), dtype=torch.float64, device=DEV)
        self.args = []
        labels = torch.arange(self.L, device=DEV)
        self.labels = labels
        if taps is not None:
            self.Lv = taps.shape[2]
            self.tap_of = (self.Lv // 2 + labels.view(1, -1) - torch.arange(self.L, device=DEV).view(-1, 1)).clamp(1, self.Lv - 1)

    def line(self, t, d, i):
        """Pixels of line i of a (B,H,W,...) tensor: a column for the horizontal directions."""
        return t[:, :, i] if d in (LEFT, RIGHT) else t[:, i]

    def steps(self, d):
        n = self.W if d in (LEFT, RIGHT) else self.H
        return [(i, i + 1) for i in range(n - 1)] if d in (RIGHT, DOWN) else [(i, i - 1) for i in range(n - 1, 0, -1)]

    def pairwise(self, d, i):
        """(..., s, t) costs of the senders of line i."""
        if self.jump.dim() == 4:   # (1,2,L,L): one matrix per axis
            j = self.jump[0, d >> 1]
            return (j.t() if d & 1 else j).view(1, 1, self.L, self.L)
        j = self.jump[d >> 1]      # (H,W,L,L): the reverse directions read the neighbour's matrix, transposed
        if not d & 1:
            return self.line(j.unsqueeze(0), d, i)
        if i == 0:
            return torch.zeros_like(self.line(j.unsqueeze(0), d, 0))
        return self.line(j.unsqueeze(0), d, i - 1).transpose(-1, -2)

    def send(self, d, i, h):
        """(values, argmin) of the messages that line i sends."""
        w = self.line(self.edge[:, d], d, i).unsqueeze(-1)
        if self.jump is not None:
            v = self.pairwise(d, i) * w.unsqueeze(-1) + h.unsqueeze(-1)
            return v.min(dim=-2)
        taps = self.line(self.taps[:, d].movedim(1, -1), d, i)
        best, low = h.min(dim=-1, keepdim=True)
        m = (taps[..., -1:] * w + best).expand_as(h).clone()
        arg = low.expand_as(h).clone()
        for k in range(-self.delta, self.delta + 1):
            if abs(k) >= self.L:
                continue
            lo, hi = max(0, -k), min(self.L, self.L - k)
            f = taps[..., max(1, min(self.Lv - 1, self.Lv // 2 - k))].unsqueeze(-1)
            v = f * w + h[..., lo + k:hi + k]
            take = v < m[..., lo:hi]
            m[..., lo:hi] = torch.where(take, v, m[..., lo:hi])
            arg[..., lo:hi] = torch.where(take, self.labels[lo + k:hi + k].expand_as(v), arg[..., lo:hi])
        return m, arg

    def forward(self, keep=True):
        args = torch.zeros(self.msgs.shape, dtype=torch.int64, device=DEV) if keep else None
        for d in (RIGHT, LEFT, DOWN, UP):
            e = d ^ 1
            for i, q in self.steps(d):
                h = self.line(self.cost, d, i).clone()
                for k in range(4):
                    if k != d:
                        h += self.line(self.msgs[:, k], d, i)
                m, a = self.send(d, i, h)
                low = torch.logsumexp(m, dim=-1, keepdim=True) if self.log_normalise else h.min(dim=-1, keepdim=True)[0]
                self.line(self.msgs[:, e], d, q).copy_(m - low)
                if keep:
                    self.line(args[:, e], d, q).copy_(a)
        if keep:
            self.args.append(args)

    def adjoint(self, g, args):
        """Cost, pairwise and edge gradients of one pass, the messages' gradient g the same in every slot."""
        gc = torch.zeros_like(self.cost)
        ge = torch.zeros_like(self.edge)
        gp = torch.zeros_like(self.taps if self.taps is not None else self.jump)
        saved = {}
        for e in (DOWN, UP, LEFT, RIGHT):
            d = e ^ 1
            acc = torch.zeros_like(self.line(self.cost, d, 0))
            rows = torch.zeros_like(self.cost)
            for i, q in reversed(self.steps(d)):
                a = self.line(g, d, q) + acc
                if e in (LEFT, RIGHT):
                    a = a + self.line(saved[UP], d, q) + self.line(saved[DOWN], d, q)
                m = self.line(self.msgs[:, e], d, q)
                add = a - torch.softmax(m, dim=-1) * a.sum(-1, keepdim=True)
                s = self.line(args[:, e], d, q)
                acc = torch.zeros_like(add).scatter_add_(-1, s, add)
                self.line(gc, d, i).add_(acc)
                self.line(rows, d, i).copy_(acc)
                w = self.line(self.edge[:, d], d, i)
                if self.taps is not None:
                    idx = (self.Lv // 2 + self.labels - s).clamp(1, self.Lv - 1)
                    t = self.line(self.taps[:, d].movedim(1, -1), d, i)
                    bins = torch.zeros_like(t).scatter_add_(-1, idx, add)
                    self.line(gp[:, d].movedim(1, -1), d, i).add_(bins * w.unsqueeze(-1))
                    self.line(ge[:, d], d, i).add_((bins * t).sum(-1))
                    continue
                full = torch.zeros(add.shape[:-1] + (self.L, self.L), dtype=torch.float64, device=DEV)
                full.scatter_(-2, s.unsqueeze(-2), add.unsqueeze(-2))
                self.line(ge[:, d], d, i).add_((full * self.pairwise(d, i)).sum((-1, -2)))
                full *= w.unsqueeze(-1).unsqueeze(-1)
                if self.jump.dim() == 4:
                    full = full.sum((0, 1))
                    gp[0, d >> 1] += full.t() if d & 1 else full
                elif not d & 1:
                    self.line(gp[d >> 1].unsqueeze(0), d, i).add_(full.sum(0, keepdim=True))
                elif i > 0:
                    self.line(gp[d >> 1].unsqueeze(0), d, i - 1).add_(full.sum(0, keepdim=True).transpose(-1, -2))
            saved[e] = rows
        return gc, gp, ge


def _beliefs64(z):
    return torch.softmax(-z, dim=-1)


def _sub_exp64(b, support=3):
    win = (torch.arange(-support, support + 1, device=DEV) + b.argmax(-1, keepdim=True)).clamp(0, b.shape[-1] - 1)
    bw = torch.gather(b, -1, win)
    return ((bw / bw.sum(-1, keepdim=True)) * win).sum(-1, keepdim=True)


def _scalar_taps64(B, H, W):
    row = torch.tensor([0.0, L2, L1, 0.0, L1, L2], dtype=torch.float32, device=DEV).double()
    return row.view(1, 1, 6, 1, 1).expand(B, 4, 6, H, W).contiguous()


def _sad64(f0, f1, D):
    B, C, H, W = f0.shape
    sad = torch.full((B, H, W, D), 40.0, dtype=torch.float64, device=DEV)
    for d in range(min(D, W)):
        sad[:, :, d:, d] = (f0[..., d:] - f1[..., :W - d]).abs().sum(1)
    return sad


def _exact_layer(case, s):
    """The BP layers' training passes: beliefs, messages and the gradients of the reference's adjoint."""
    B, H, W, L, it = case["B"], case["H"], case["W"], case["L"], case["iters"]
    prob = s["prob"].detach().double()
    edge = s["edge"].detach().double() if s.get("edge") is not None else torch.ones((B, 4, H, W), device=DEV).double()
    half = case.get("storage") == "fp16"
    aff = None
    if case["kind"] == "train":
        if s["aff"] is not None:
            aff = s["aff"].detach().double().requires_grad_(True)
            packed = _pack64(aff)
        else:
            packed = _scalar_taps64(B, H, W)
        m = _Min64(-prob, edge, taps=packed.detach(), log_normalise=not half)
    else:
        m = _Min64(-prob, edge, jump=s["jump"].detach().double(), delta=L)
    for _ in range(it):
        m.forward(keep=not half)
    z = m.msgs.sum(1) - prob
    b = _beliefs64(z)
    msgs = m.msgs
    if half:
        # the half rows carry padding; their gradients follow the half rounding of every message
        msgs = torch.nn.functional.pad(msgs, (0, (L + 7) // 8 * 8 - L))
        out = {"beliefs": b, "messages": msgs, "g_prob": None, "g_edge": None, "g_T": None}
        out.update({"g_aff": None} if aff is not None else {"g_L1": None, "g_L2": None})
        return out
    up = s["up"].double()
    gz = -b * (up - (up * b).sum(-1, keepdim=True))
    gp, ge, gpair = -gz, torch.zeros_like(edge), 0.0
    for args in m.args:
        c, p, e = m.adjoint(gz, args)
        gp, ge, gpair = gp - c, ge + e, gpair + p
    out = {"beliefs": b, "messages": msgs, "g_prob": gp, "g_messages": gz.unsqueeze(1).expand(B, 4, H, W, L)}
    if case["kind"] != "train":
        out["g_jump"] = gpair
        if s.get("edge") is not None:
            out["g_edge"] = ge
        return out
    out["g_edge"] = ge
    out["g_T"] = -(gz * z).sum()
    if aff is not None:
        out["g_aff"] = torch.autograd.grad(packed, aff, gpair)[0]
    else:
        out["g_L1"], out["g_L2"] = gpair[:, :, [2, 4]].sum(), gpair[:, :, [1, 5]].sum()
    return out


def _exact_infer(case, s):
    H, W, L = case["H"], case["W"], case["L"]
    B = case.get("B", 1)
    m = None
    beliefs, disps = [], []
    volumes = [s["prob"]] if case["kind"] == "infer" else [s["prob"][:, 0], s["prob"][:, 1]]
    for v in volumes:  # the flow path starts v from u's final messages
        v = v.double()
        n = _Min64(-v, s["edge"].double(), taps=_scalar_taps64(B, H, W))
        if m is not None:
            n.msgs.copy_(m.msgs)
        m = n
        for _ in range(case["iters"]):
            m.forward(keep=False)
        beliefs.append(_beliefs64(m.msgs.sum(1) - v))
        disps.append(_sub_exp64(beliefs[-1]) if case["mode"] == "sub-exp" else None)
    if case["kind"] == "infer":
        disp = None if disps[0] is None else disps[0].permute(0, 3, 1, 2)
        return {"disp": disp, "beliefs": beliefs[0], "messages": m.msgs}
    disp = None if disps[0] is None else torch.cat(disps, -1).permute(0, 3, 1, 2)
    msgs = torch.cat((m.msgs.unsqueeze(1), m.msgs.unsqueeze(1)), dim=1)
    return {"disp": disp, "beliefs": torch.stack(beliefs, dim=1), "messages": msgs}


def _exact_sad(s):
    f0, f1, up = s["f0"].detach().double(), s["f1"].detach().double(), s["up"].double()
    B, C, H, W = f0.shape
    D = up.shape[-1]
    g0, g1 = torch.zeros_like(f0), torch.zeros_like(f1)
    for d in range(min(D, W)):
        sg = torch.sign(f0[..., d:] - f1[..., :W - d]) * up[:, :, d:, d].unsqueeze(1)
        g0[..., d:] += sg
        g1[..., :W - d] -= sg
    return {"sad": _sad64(f0, f1, D), "g_f0": g0, "g_f1": g1}


def _exact_flow_sad(s):
    f0, f1 = s["f0"].detach().double(), s["f1"].detach().double()
    B, C, H, W = f0.shape
    K = s["L"]
    hs = (K - 1) // 2
    best = [torch.full((B, H, W, K), 9999999.0, dtype=torch.float64, device=DEV) for _ in range(2)]
    star = [torch.zeros((B, H, W, K), dtype=torch.int64, device=DEV) for _ in range(2)]
    for v in range(-hs, hs + 1):
        for u in range(-hs, hs + 1):
            sad = torch.full((B, H, W), 40.0, dtype=torch.float64, device=DEV)
            y0, y1, x0, x1 = max(0, -v), min(H, H - v), max(0, -u), min(W, W - u)
            if y0 < y1 and x0 < x1:
                sad[:, y0:y1, x0:x1] = (f0[:, :, y0:y1, x0:x1] - f1[:, :, y0 + v:y1 + v, x0 + u:x1 + u]).abs().sum(1)
            for k, (i, j) in enumerate(((u + hs, v + hs), (v + hs, u + hs))):
                less = sad < best[k][..., i]
                best[k][..., i] = torch.where(less, sad, best[k][..., i])
                star[k][..., i] = torch.where(less, j, star[k][..., i])
    g0, g1 = torch.zeros_like(f0), torch.zeros_like(f1).view(B, C, H * W)
    ys = torch.arange(H, device=DEV).view(1, H, 1)
    xs = torch.arange(W, device=DEV).view(1, 1, W)
    for k in range(2):
        up = s["up"][k].double()
        for i in range(K):
            u, v = (i - hs, star[0][..., i] - hs) if k == 0 else (star[1][..., i] - hs, i - hs)
            y, x = ys + v, xs + u
            inside = (y >= 0) & (y < H) & (x >= 0) & (x < W)
            at = (y.clamp(0, H - 1) * W + x.clamp(0, W - 1)).view(B, 1, H * W).expand(B, C, H * W)
            sg = torch.sign(f0 - torch.gather(f1.view(B, C, H * W), 2, at).view(B, C, H, W))
            sg = sg * (up[..., i] * inside).unsqueeze(1)
            g0 += sg
            g1.scatter_add_(2, at, -sg.reshape(B, C, H * W))
    return {"cv_u": best[0], "cv_v": best[1], "u_star": None, "v_star": None, "g_f0": g0, "g_f1": g1.view(B, C, H, W)}


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind in ("train", "global", "pixel"):
        return _exact_layer(case, s)
    if kind in ("infer", "flow_bp"):
        return _exact_infer(case, s)
    if kind == "sad":
        return _exact_sad(s)
    if kind == "flow_sad":
        return _exact_flow_sad(s)
    sad = _sad64(s["f0"].double(), s["f1"].double(), case["L"])
    cost = torch.nn.functional.pad(-torch.softmax(-sad, dim=-1), (0, (-case["L"]) % 8))
    m = _Min64(cost[..., :case["L"]], s["edge"].double(), taps=s["taps"].double(), log_normalise=False)
    if m.edge.shape[0] != m.B:
        m.edge, m.taps = m.edge.expand(m.B, -1, -1, -1), m.taps.expand(m.B, -1, -1, -1, -1)
    for _ in range(case["iters"]):
        m.forward(keep=False)
    return {"disp": None, "messages": torch.nn.functional.pad(m.msgs, (0, (-case["L"]) % 8)), "cost": cost, "sad": sad}

"""The calls whose speed is followed: Polynomial-Mixer layers, the aggregation operator and the residual stack, each
through the entry point a program calls (``PoM.forward``, ``PoMRoPE.forward``, ``polynomial_aggregation_``,
``PoMStack.frame_forward``), with a plain float64 restatement of the same arithmetic beside it.

A case is a dict of plain values:

* ``kind``   "layer" | "op" | "frame"
* ``family`` what the case stands for; :func:`draw` varies the sizes inside a family
* ``dtype``  "bf16" | "fp32"; ``train``: with the gradients of the tokens and of every parameter
* ``B, N, D, K, E, heads``  samples, query tokens, channels, degree, expansion, gate heads (1: one gate per channel)
* ``ctx``    context tokens of a cross-mixing layer (0: self-mixing)
* ``mask``   "none" | "keypad" (valid lengths) | "causal" | "packed" (documents side by side, a (B, N, N) mask)
* ``rope``   "none" | "1d" | "2d" (``gh`` x ``gw`` grid in raster order, N = gh * gw)
* ``layers`` mixers of a stack ("frame")
"""
import math

import torch
import torch.nn.functional as F

from pom_b200 import PoM, PoMRoPE
from pom_b200.functional import polynomial_aggregation_
from pom_b200.stack import PoMStack

_BASE = dict(kind="layer", dtype="bf16", train=True, heads=1, ctx=0, mask="none", rope="none", gh=0, gw=0, layers=0)


def _case(**kw):
    c = dict(_BASE)
    c.update(kw)
    return c


def listed():
    return [
        # A float32 layer as nn.Module makes it (nobody called .bfloat16()), at the size of a first experiment: the
        # smallest call, all latency and launches.
        _case(name="fp32_small_forward", family="fp32_forward", dtype="fp32", train=False, B=2, N=256, D=256, K=2, E=2),
        # One training step of a float32 image-generation layer (a 30 x 34 patch grid: an ordinary, odd length).
        _case(name="fp32_train", family="fp32_train", dtype="fp32", B=4, N=1020, D=1152, K=2, E=2),
        # One training step of the bf16 image-generation layer: 32 x 32 patches, 32 images.
        _case(name="dit_train", family="dit_train", B=32, N=1024, D=1152, K=2, E=2),
        # The same layer while sampling with guidance: two images, forward only.
        _case(name="dit_sample", family="dit_sample", train=False, B=2, N=1024, D=1152, K=2, E=2),
        # The same training step with one gate value per head (16 heads).
        _case(name="heads16_train", family="heads_train", B=32, N=1024, D=1152, K=2, E=2, heads=16),
        # Variable-length batches, padded to the longest sample; degree 3.
        _case(name="masked_train", family="masked_train", B=32, N=1987, D=1024, K=3, E=2, mask="keypad"),
        # Image layer with axial rotary positions on a 24 x 24 grid (384-pixel images).
        _case(name="rope2d_train", family="rope2d_train", B=32, N=576, D=1152, K=2, E=2, rope="2d", gh=24, gw=24),
        # One long sequence, a 256 x 256 grid with axial rotary positions and the token-causal prefix mean: the
        # largest call.
        _case(name="long_causal_train", family="causal_train", B=1, N=65536, D=1152, K=2, E=2, mask="causal",
              rope="2d", gh=256, gw=256),
        # One 256-token frame of 8 videos through a 12-layer stack that carries its state from frame to frame.
        _case(name="video_frame", family="frame", kind="frame", train=False, B=8, N=256, D=1024, K=2, E=4, layers=12),
        # Image tokens read from text: 1024 queries against up to 120 context tokens, padded.
        _case(name="cross_train", family="cross_train", B=16, N=1024, ctx=120, D=1152, K=2, E=2, mask="keypad"),
        # Documents packed side by side in one sequence: a (B, N, N) mask.
        _case(name="packed_train", family="packed_train", B=4, N=1536, D=1024, K=2, E=2, mask="packed"),
        # The aggregation operator alone on features that the caller projected: causal, forward and backward.
        _case(name="op_causal_train", family="op_train", kind="op", B=8, N=2047, D=2304, K=3, E=1, mask="causal"),
    ]


# ---------------------------------------------------------------------------- drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fit(rng, tokens, n):
    """A batch size between 1 and what keeps batch * n at or below ``tokens``."""
    return _log_int(rng, 1, max(1, tokens // n))


def draw(rng):
    family = rng.choice(sorted({c["family"] for c in listed()}))
    D = 8 * rng.randint(16, 144)  # 128 .. 1152 channels, multiples of 8 (what bf16 rows need)
    K, E = rng.randint(1, 4), rng.choice([1, 2, 2, 4])
    N = _log_int(rng, 128, 2048)
    small = dict(family=family, D=D, K=K, E=min(E, 2))
    if family == "fp32_forward":
        return _case(**{**small, "D": rng.randint(96, 1152)}, dtype="fp32", train=False, N=N, B=_fit(rng, 4096, N),
                     mask=rng.choice(["none", "causal"]))
    if family == "fp32_train":
        return _case(**small, dtype="fp32", N=N, B=_fit(rng, 4096, N), mask=rng.choice(["none", "keypad", "causal"]))
    if family == "dit_train":
        return _case(**small, N=N, B=_fit(rng, 32768, N))
    if family == "dit_sample":
        return _case(**small, train=False, N=N, B=_fit(rng, 8192, N))
    if family == "heads_train":
        return _case(**{**small, "D": 64 * rng.randint(2, 18)}, N=N, B=_fit(rng, 32768, N), heads=rng.choice([8, 16]),
                     mask=rng.choice(["none", "keypad"]))
    if family == "masked_train":
        return _case(**small, N=N, B=_fit(rng, 65536, N), mask="keypad")
    if family == "rope2d_train":
        gh, gw = rng.randint(8, 48), rng.randint(8, 48)
        return _case(**small, N=gh * gw, B=_fit(rng, 32768, gh * gw), rope="2d", gh=gh, gw=gw)
    if family == "causal_train":
        N = _log_int(rng, 512, 32768)
        return _case(**small, N=N, B=_fit(rng, 32768, N), mask="causal", rope=rng.choice(["none", "1d"]))
    if family == "frame":
        L = _log_int(rng, 32, 512)
        return _case(family=family, kind="frame", train=False, N=L, B=_fit(rng, 2048, L), D=8 * rng.randint(16, 128),
                     K=rng.randint(1, 4), E=E, layers=rng.randint(1, 12))
    if family == "cross_train":
        return _case(**small, N=N, B=_fit(rng, 16384, N), ctx=_log_int(rng, 16, 512), mask="keypad")
    if family == "packed_train":
        N = _log_int(rng, 128, 1536)
        return _case(**small, N=N, B=_fit(rng, 6144, N), mask="packed")
    return _case(**{**small, "E": 1, "D": 8 * rng.randint(16, 288)}, kind="op", N=N, B=_fit(rng, 16384, N),
                 mask=rng.choice(["none", "causal", "keypad"]), dtype=rng.choice(["bf16", "bf16", "fp32"]))


# ---------------------------------------------------------------------------- inputs
def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float32


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def _linear(gen, rows, cols, dt):
    """nn.Linear's own start: uniform within 1 / sqrt(inputs)."""
    return ((torch.rand(rows, cols, generator=gen, device="cuda") * 2 - 1) / math.sqrt(cols)).to(dt)


def _mixer_weights(gen, case, dt):
    D, K, P = case["D"], case["K"], case["D"] * case["E"]
    S = case["heads"] if case["heads"] > 1 else P
    scale = 0.2 / (torch.arange(K, device="cuda") + 1.0)  # polynomial coefficients as training leaves them
    return dict(qc=_linear(gen, P + S, D, dt), bias=(0.1 * torch.randn(S, generator=gen, device="cuda")).to(dt),
                coeff=(torch.randn(P, K, generator=gen, device="cuda") * scale).to(dt), ag=_linear(gen, D, P, dt))


def _positions(case):
    """Row and column of every token of a raster-ordered grid, or 0..N-1."""
    n = torch.arange(case["N"], device="cuda")
    return torch.stack([n // case["gw"], n % case["gw"]], dim=1) if case["rope"] == "2d" else n


def _mask(gen, case):
    B, N = case["B"], case["ctx"] or case["N"]
    if case["mask"] == "keypad":  # valid lengths between an eighth of the longest sample and all of it
        lens = torch.randint(max(1, N // 8), N + 1, (B,), generator=gen, device="cuda")
        lens[0] = N
        return torch.arange(N, device="cuda")[None, :] < lens[:, None]
    if case["mask"] == "packed":  # four documents per row on average, each token reading its own document
        starts = torch.rand(B, N, generator=gen, device="cuda") < 3.0 / N
        doc = starts.cumsum(1)
        return doc[:, :, None] == doc[:, None, :]
    return None if case["mask"] == "none" else "causal"


def _inputs(case, seed):
    """Every tensor of the call, from the seed alone."""
    gen, dt = _generator(seed), _dtype(case)
    B, N, D = case["B"], case["N"], case["D"]
    P = D * case["E"]
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dt)
    t = dict(x=randn(B, N, D), mask=_mask(gen, case))
    if case["kind"] == "op":
        scale = 0.2 / (torch.arange(case["K"], device="cuda") + 1.0)
        t["coeff"] = (torch.randn(D, case["K"], generator=gen, device="cuda") * scale).to(dt)
        t["dy"] = randn(B, N if case["mask"] == "causal" else 1, D)
        return t
    if case["kind"] == "frame":
        t["layers"] = [dict(_mixer_weights(gen, case, dt), w1=_linear(gen, 4 * D, D, dt), w2=_linear(gen, D, 4 * D, dt),
                            h=0.06 * torch.randn(B, 1, P, generator=gen, device="cuda")) for _ in range(case["layers"])]
        return t
    t.update(_mixer_weights(gen, case, dt))
    if case["ctx"]:
        t["xc"] = randn(B, case["ctx"], D)
    if case["rope"] != "none":
        t["pos"] = _positions(case)
    if case["train"]:
        t["dy"] = randn(B, N, D)
    return t


def _load(mixer, w):
    with torch.no_grad():
        mixer.qc_proj.weight.copy_(w["qc"])
        mixer.se_bias.copy_(w["bias"])
        mixer.po_coeff.copy_(w["coeff"])
        mixer.ag_proj.weight.copy_(w["ag"])


def prepare(case, seed):
    t, dt = _inputs(case, seed), _dtype(case)
    D, K, E = case["D"], case["K"], case["E"]
    s = dict(case=case, x=t["x"], mask=t["mask"])
    if case["kind"] == "op":
        s.update(coeff=t["coeff"].requires_grad_(), dy=t["dy"])
        s["x"].requires_grad_()
        return s
    with torch.device("cuda"):
        if case["kind"] == "frame":
            model = PoMStack(D, K, E, case["layers"]).to(dt)
        elif case["rope"] == "2d":
            model = PoMRoPE(D, K, E, n_sel_heads=case["heads"], rope_2d=True, max_h=case["gh"], max_w=case["gw"]).to(dt)
        elif case["rope"] == "1d":
            model = PoMRoPE(D, K, E, n_sel_heads=case["heads"], max_seq_len=case["N"]).to(dt)
        else:
            model = PoM(D, K, E, n_sel_heads=case["heads"]).to(dt)
    for name in ("row_cos", "row_sin", "col_cos", "col_sin", "freqs_cos", "freqs_sin"):
        if hasattr(model, name):  # the rotary tables stay in float32 whatever the weights are cast to
            setattr(model, name, _tables(case)[name])
    s["model"] = model
    if case["kind"] == "frame":
        for i, w in enumerate(t["layers"]):
            _load(model.mixers[i], w)
            with torch.no_grad():
                model.ffn_in[i].weight.copy_(w["w1"])
                model.ffn_out[i].weight.copy_(w["w2"])
        s["states"] = [dict(h=w["h"], n=3) for w in t["layers"]]
        return s
    _load(model, t)
    s["kw"] = {}
    if case["rope"] != "none":
        s["kw"] = {"positions_hw" if case["rope"] == "2d" else "positions": t["pos"]}
    s["xc"] = t.get("xc")
    if case["train"]:
        s["dy"] = t["dy"]
        s["params"] = [model.qc_proj.weight, model.se_bias, model.po_coeff, model.ag_proj.weight]
        s["wrt"] = [v.requires_grad_() for v in (s["x"], s["xc"]) if v is not None] + s["params"]
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "op":
        y = polynomial_aggregation_(state["x"], state["coeff"], case["K"], state["mask"])
        return [y.detach(), *torch.autograd.grad(y, [state["x"], state["coeff"]], state["dy"])]
    if case["kind"] == "frame":
        y, states = state["model"].frame_forward(state["x"], state["states"])
        return [y] + [s["h"] for s in states]
    if not case["train"]:
        with torch.no_grad():
            return [state["model"](state["x"], state["xc"], state["mask"], **state["kw"])]
    y = state["model"](state["x"], state["xc"], state["mask"], **state["kw"])
    return [y.detach(), *torch.autograd.grad(y, state["wrt"], state["dy"])]


# ---------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    B, N, D, K = case["B"], case["N"], case["D"], case["K"]
    e = 2 if case["dtype"] == "bf16" else 4
    P, C = D * case["E"], case["ctx"] or case["N"]
    S = case["heads"] if case["heads"] > 1 else P
    if case["kind"] == "op":
        out = N if case["mask"] == "causal" else 1
        mask = B * N if case["mask"] == "keypad" else 0
        return dict(bytes=e * B * D * (2 * N + 2 * out) + 2 * e * D * K + mask, flops=B * N * D * (6 * K + 4))
    weights = (P + S) * D + S + P * K + D * P
    if case["kind"] == "frame":
        L = case["layers"]
        flops = L * (2 * B * N * D * 3 * P + 2 * B * N * D * 8 * D)
        return dict(bytes=e * (L * (weights + 8 * D * D) + 2 * B * N * D) + L * 2 * 4 * B * P, flops=flops)
    gate, out = 2 * B * N * D * S, 2 * B * N * P * D
    if case["heads"] > 1 and case["mask"] in ("none", "keypad"):  # the output side collapses to one small matrix
        out = 2 * B * N * S * D + 2 * B * P * D
    flops = 2 * B * C * D * P + gate + out
    mask = 0
    if case["mask"] == "packed":
        flops += 2 * B * N * C * P
        mask = B * N * C
    elif case["mask"] == "keypad":
        mask = B * C
    tokens = B * (N + (case["ctx"] or 0)) * D
    nbytes = e * (tokens + weights + B * N * D) + mask
    if case["train"]:
        flops = 3 * flops - (2 * B * N * C * P if case["mask"] == "packed" else 0)  # the mask gets no gradient
        nbytes += e * (B * N * D + tokens + weights)
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    # About four times the distance measured between the layers and exact(): 1e-6 in float32; in bf16 1.7e-3 for the
    # operator, 2.5e-3 for a layer, 4.2e-3 where the gate itself (heads) or the per-token aggregate (packed) is
    # rounded too, 8e-3 after the 48 roundings of a 12-layer residual stream.
    if case["dtype"] == "fp32":
        return dict(rel=6e-6)
    if case["kind"] == "frame":
        return dict(rel=3.3e-2)
    if case["kind"] == "op":
        return dict(rel=7e-3)
    return dict(rel=1.7e-2 if case["heads"] > 1 or case["mask"] == "packed" else 1.2e-2)


# ---------------------------------------------------------------------------- the same in float64
def _tables(case):
    """cos and sin of position x base^(-j / pairs), float32 as the layer keeps them."""
    P = case["D"] * case["E"]
    pairs = P // 4 if case["rope"] == "2d" else P // 2
    inv = 1.0 / (10000.0 ** (torch.arange(pairs, device="cuda", dtype=torch.float32) / pairs))
    ang = lambda n: torch.outer(torch.arange(n, device="cuda", dtype=torch.float32), inv)
    if case["rope"] == "2d":
        r, c = ang(case["gh"]), ang(case["gw"])
        return dict(row_cos=r.cos(), row_sin=r.sin(), col_cos=c.cos(), col_sin=c.sin())
    a = ang(case["N"])
    return dict(freqs_cos=a.cos(), freqs_sin=a.sin())


def _turn(v, cos, sin):
    lo, hi = v.chunk(2, dim=-1)
    return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], dim=-1)


def _rotate(case, v, pos):
    t = {k: a.double() for k, a in _tables(case).items()}
    if case["rope"] == "1d":
        return _turn(v, t["freqs_cos"][pos], t["freqs_sin"][pos])
    top, bot = v.chunk(2, dim=-1)
    r, c = pos[:, 0], pos[:, 1]
    return torch.cat([_turn(top, t["row_cos"][r], t["row_sin"][r]), _turn(bot, t["col_cos"][c], t["col_sin"][c])], -1)


def _features(hp, coeff):
    a = F.leaky_relu(hp, 0.01).clamp(-0.1, 6.0)
    total = torch.zeros_like(a)
    for i in reversed(range(coeff.shape[1])):
        total = (total + coeff[:, i]) * a
    return total


def _aggregate(f, mask):
    if mask is None:
        return f.mean(dim=1, keepdim=True)
    if isinstance(mask, str):
        return f.cumsum(dim=1) / torch.arange(1, f.shape[1] + 1, device=f.device, dtype=f.dtype)[:, None]
    w = mask.double()
    if w.dim() == 2:
        return (f * w[..., None]).sum(1, keepdim=True) / w.sum(1)[:, None, None]
    return (w @ f) / w.sum(-1, keepdim=True)


def _mix(case, x, xc, qc, bias, coeff, ag, mask=None, pos=None, past=None):
    P = coeff.shape[0]
    f = _features(xc @ qc[:P].t(), coeff)
    s = F.relu6(x @ qc[P:].t() + bias + 3.0) / 6.0
    if pos is not None:
        f, s = _rotate(case, f, pos), _rotate(case, s, pos)
    h = _aggregate(f, mask)
    if past is not None:
        h = (3.0 * past + h) / 4.0
    if case["heads"] > 1:
        s = s.repeat_interleave(P // case["heads"], dim=-1)
    return (s * h) @ ag.t(), h


def exact(case, seed):
    t = _inputs(case, seed)
    wide = lambda v: v.double().requires_grad_(case["train"])
    if case["kind"] == "op":
        x, coeff = wide(t["x"]), wide(t["coeff"])
        y = _aggregate(_features(x, coeff), t["mask"])
        return [y.detach(), *torch.autograd.grad(y, [x, coeff], t["dy"].double())]
    if case["kind"] == "frame":
        x, hs = t["x"].double(), []
        for w in t["layers"]:
            w = {k: v.double() for k, v in w.items()}
            y, h = _mix(case, x, x, w["qc"], w["bias"], w["coeff"], w["ag"], past=w["h"])
            x = x + y
            x = x + F.gelu(x @ w["w1"].t()) @ w["w2"].t()
            hs.append(h)
        return [x] + hs
    x, params = wide(t["x"]), [wide(t[k]) for k in ("qc", "bias", "coeff", "ag")]
    xc = wide(t["xc"]) if case["ctx"] else None
    y, _ = _mix(case, x, x if xc is None else xc, *params, mask=t["mask"], pos=t.get("pos"))
    if not case["train"]:
        return [y]
    wrt = [x] + ([] if xc is None else [xc]) + params
    return [y.detach(), *torch.autograd.grad(y, wrt, t["dy"].double())]

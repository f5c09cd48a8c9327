"""Performance cases: the layers that Triune and universal (dense) models are made of, and whole requests to a served model.

Kinds, each through the entry point that a program uses for it:

* ``train``: forward and backward of one ``TransformerBlock`` (norm, gated-linear-attention or Gated-DeltaNet mixer, norm, dense
  feed-forward) on activations of a training batch; gradients of the input and of every weight.
* ``moe``: forward and backward of ``MoE_FFN`` (router, grouped experts, shared expert) on a training batch.
* ``prefill``: a ``TransformerBlock`` in evaluation over a prompt with a recurrent cache; ``carry`` tokens were consumed before
  (a chat's next turn, or the next portion of a long prompt).
* ``generate``: ``GraphedGreedyDecoder.generate`` on a ``UniversalDenseTransformer``: the prompt, then greedy tokens.

Widths are those of the model presets (``triune_b200/config.py``): 6 to 16 heads of 64 (triune-base to triune-1.5b, the 90M
benchmark model), 8 to 16 heads of 128 (triune-default, bench-dense-1.5b, the published 4 x 2048 x 8 x 128 mixer shape).
All weights and activations are bfloat16, the only type these models are trained and served in on a GPU.
"""

import math

import torch
import torch.nn.functional as F

from triune_b200.config import ModelConfig
from triune_b200.inference import GraphedGreedyDecoder
from triune_b200.models import MoE_FFN, TransformerBlock
from triune_b200.models.factory import build_model
from triune_b200.utils import place_model

WIDTHS = {384: (6, 64), 512: (8, 64), 768: (12, 64), 1024: (8, 128), 1536: (12, 128), 2048: (16, 128)}  # width: heads, head size
VOCAB = 32000
MOST_WORK = 32768 * 384.0  # tokens x width of the largest training batch and of the largest expert batch
EPS, ROPE_BASE = 1e-6, 10000.0


def _mixer_case(kind, name, mixer, batch, seq, dim, **more):
    heads, head = WIDTHS[dim]
    return {"name": name, "kind": kind, "mixer": mixer, "batch": batch, "seq": seq, "dim": dim, "heads": heads, "head_dim": head, **more}


def listed():
    return [
        # a step of the 90M benchmark model (16 x 2048 tokens): one layer, forward and backward
        _mixer_case("train", "train gla 16x2048 6x64", "gla", 16, 2048, 384),
        # the default model (12 heads of 128), an ordinary batch
        _mixer_case("train", "train gla 8x1024 12x128", "gla", 8, 1024, 1536),
        # fine-tuning on documents of a length that is no multiple of anything
        _mixer_case("train", "train gla 3x777 16x128", "gla", 3, 777, 2048),
        # Gated DeltaNet at the published mixer shape
        _mixer_case("train", "train gdn 4x2048 8x128", "gdn", 4, 2048, 1024),
        # a small fine-tuning batch, short ragged rows
        _mixer_case("train", "train gdn 2x300 6x64", "gdn", 2, 300, 384),
        # the experts of the 90M benchmark model over a whole batch
        {"name": "moe 16x2048 d384 top2", "kind": "moe", "batch": 16, "seq": 2048, "dim": 384, "experts": 8, "top_k": 2, "hidden": 1536},
        # the long prompts of the serving benchmark
        _mixer_case("prefill", "prefill gla 4x16384 6x64", "gla", 4, 16384, 384, carry=0),
        # one long prompt to a model with wide heads, both mixers
        _mixer_case("prefill", "prefill gla 1x8192 16x128", "gla", 1, 8192, 2048, carry=0),
        _mixer_case("prefill", "prefill gdn 1x8192 16x128", "gdn", 1, 8192, 2048, carry=0),
        # the next turn of a chat: few tokens after many
        _mixer_case("prefill", "turn gla 1x37 12x128", "gla", 1, 37, 1536, carry=333),
        # a served request: latency of single tokens
        _mixer_case("generate", "generate gla 1x200+32 16x128", "gla", 1, 200, 2048, layers=6, new=32),
        # requests served together
        _mixer_case("generate", "generate gdn 4x512+32 16x128", "gdn", 4, 512, 2048, layers=6, new=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "moe", "prefill", "prefill", "prefill", "generate", "generate"])
    dim = rng.choice(sorted(WIDTHS))
    mixer = rng.choice(["gla", "gdn"])
    heads, head = WIDTHS[dim]
    case = {"kind": kind, "mixer": mixer, "batch": 1, "seq": 1, "dim": dim, "heads": heads, "head_dim": head}
    if kind in ("train", "moe"):
        case["batch"] = _log(rng, 1, 16)
        case["seq"] = min(_log(rng, 48, 2048), int(MOST_WORK / dim / case["batch"]))
        if rng.random() < 0.4:  # packed rows come in round lengths
            case["seq"] = max(64, case["seq"] // 64 * 64)
        if kind == "moe":
            for k in ("mixer", "heads", "head_dim"):
                del case[k]
            case.update(dim=min(dim, 1024), experts=8, top_k=rng.choice([1, 2]))
            case["hidden"] = 4 * case["dim"]
    elif kind == "prefill":
        case["batch"] = _log(rng, 1, 4)
        most = {384: 16384, 512: 16384, 768: 8192, 1024: 8192, 1536: 8192, 2048: 8192}[dim] // (1 if dim < 768 else case["batch"])
        case["seq"] = _log(rng, 16, most)
        if rng.random() < 0.3:
            case["seq"] = max(64, case["seq"] // 64 * 64)
        case["carry"] = rng.choice([0, _log(rng, 64, 1024)])
    else:
        case.update(batch=_log(rng, 1, 8), seq=_log(rng, 16, 512), layers=rng.choice([4, 6]), new=_log(rng, 8, 32))
    return case


# ------------------------------------------------------------------------------------------------ inputs and weights
def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _normal(gen, shape, std, mean=0.0):
    return torch.empty(shape, device="cuda", dtype=torch.float32).normal_(mean, std, generator=gen).to(torch.bfloat16)


def _mixer_weights(gen, case, prefix, beta=True):
    d, hd = case["dim"], case["heads"] * case["head_dim"]
    w = {f"{prefix}{n}_proj.weight": _normal(gen, (hd, d), 0.02) for n in "qkvg"}
    w[prefix + "out_proj.weight"] = _normal(gen, (d, hd), 0.02)
    if case["mixer"] == "gdn":
        w[prefix + "beta_proj.weight"] = _normal(gen, (case["heads"], d), 0.02)
    return w


def _block_weights(case, seed):
    """Weights of a TransformerBlock under the names of its state dict."""
    gen, d = _generator(seed, 1), case["dim"]
    w = _mixer_weights(gen, case, "attn.gla.")
    w.update({"ffn.0.weight": _normal(gen, (4 * d, d), 0.02), "ffn.0.bias": _normal(gen, (4 * d,), 0.02),
              "ffn.2.weight": _normal(gen, (d, 4 * d), 0.02), "ffn.2.bias": _normal(gen, (d,), 0.02),
              "norm1.weight": _normal(gen, (d,), 0.1, 1.0), "norm2.weight": _normal(gen, (d,), 0.1, 1.0)})
    return w


def _moe_weights(case, seed):
    gen, d, h, w = _generator(seed, 2), case["dim"], case["hidden"], {}
    for p in [f"experts.{e}." for e in range(case["experts"])] + ["shared."]:
        w.update({p + "0.weight": _normal(gen, (h, d), 0.02), p + "0.bias": _normal(gen, (h,), 0.02),
                  p + "2.weight": _normal(gen, (d, h), 0.02), p + "2.bias": _normal(gen, (d,), 0.02)})
    w.update({"router.weight": _normal(gen, (case["experts"], d), 0.02), "router.bias": _normal(gen, (case["experts"],), 0.02)})
    return w


def _model_weights(case, seed):
    """Weights of a dense model that, like a trained one, is sure of its next token: the head's row of the token after ``t``
    (a fixed random order of the vocabulary) is the embedding of ``t``."""
    gen, d = _generator(seed, 3), case["dim"]
    hidden = _swiglu_hidden(d)
    emb = _normal(gen, (VOCAB, d), 1.0)
    order = torch.randperm(VOCAB, device="cuda", generator=gen)
    head = torch.empty_like(emb)
    head[order] = emb * 0.0625
    w = {"embed_tokens.weight": emb, "lm_head.weight": head, "norm.weight": _normal(gen, (d,), 0.1, 1.0)}
    for i in range(case["layers"]):
        p = f"layers.{i}."
        w.update(_mixer_weights(gen, case, p + "attn."))
        w.update({p + "mlp.gate_proj.weight": _normal(gen, (hidden, d), 0.02), p + "mlp.up_proj.weight": _normal(gen, (hidden, d), 0.02),
                  p + "mlp.down_proj.weight": _normal(gen, (d, hidden), 0.02),
                  p + "input_norm.weight": _normal(gen, (d,), 0.1, 1.0), p + "post_attn_norm.weight": _normal(gen, (d,), 0.1, 1.0)})
    return w, order


def _swiglu_hidden(d):
    return d * 11 // 4 // 32 * 32


def _rows(case, seed, salt, seq=None):
    """Activations of the residual stream: [batch, seq, dim]."""
    return _normal(_generator(seed, salt), (case["batch"], seq or case["seq"], case["dim"]), 1.0)


def _load(module, weights):
    buffers = dict(module.named_buffers())
    module.load_state_dict({**{k: v for k, v in module.state_dict().items() if k in buffers}, **weights}, strict=True)
    return module


# ------------------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind, dev = case["kind"], torch.device("cuda")
    if kind == "generate":
        cfg = ModelConfig(family="universal", vocab_size=VOCAB, hidden_dim=case["dim"], num_layers=case["layers"], num_heads=case["heads"],
                          head_dim=case["head_dim"], mixer={"gla": "gla", "gdn": "gated_deltanet"}[case["mixer"]], ffn="swiglu",
                          dense_hidden=_swiglu_hidden(case["dim"]), tie_embeddings=False).validate()
        with torch.device(dev):
            model = build_model(cfg)
        weights, _ = _model_weights(case, seed)
        _load(place_model(model, dev, torch.bfloat16), weights).eval()
        decoder = GraphedGreedyDecoder(model, batch_size=case["batch"])
        prompt = torch.randint(0, VOCAB, (case["batch"], case["seq"]), device=dev, generator=_generator(seed, 4))
        decoder.generate(prompt.flip(1), case["new"])  # a server's first request captures the decoder's graph
        return {"case": case, "decoder": decoder, "prompt": prompt}
    with torch.device(dev):
        if kind == "moe":
            layer = MoE_FFN(case["dim"], num_experts=case["experts"], top_k=case["top_k"], expert_hidden=case["hidden"])
        else:
            gdn = case["mixer"] == "gdn"
            layer = TransformerBlock(case["dim"], case["heads"], 0, VOCAB, [], use_moe=False, head_dim=case["head_dim"],
                                     use_delta_rule=gdn, learn_beta=gdn)
    layer = _load(place_model(layer, dev, torch.bfloat16), (_moe_weights if kind == "moe" else _block_weights)(case, seed))
    state = {"case": case, "layer": layer.train(kind != "prefill"), "x": _rows(case, seed, 5)}
    if kind == "prefill":
        state["cache"] = (None, 0)
        if case["carry"]:
            with torch.no_grad():
                state["cache"] = layer(_rows(case, seed, 6, case["carry"]), cache=(None, 0))[2]
    else:
        state["x"].requires_grad_(True)
        state["dy"] = _rows(case, seed, 7)
        state["names"], state["weights"] = zip(*layer.named_parameters())
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "generate":
        decoder = state["decoder"]
        with torch.no_grad():
            tokens = decoder.generate(state["prompt"], state["case"]["new"])
        return {"tokens": tokens, "states": list(decoder.states)}
    if kind == "prefill":
        with torch.no_grad():
            y, _, cache = state["layer"](state["x"], cache=state["cache"])
        return {"y": y, "state": cache[0]}
    x, layer = state["x"], state["layer"]
    y = layer(x) if kind == "moe" else layer(x)[0]
    grads = torch.autograd.grad(y, (x, *state["weights"]), state["dy"])
    return {"y": y.detach(), "dx": grads[0], **{"d " + n: g for n, g in zip(state["names"], grads[1:])}}


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Bytes: inputs, weights and outputs once each. Operations: two for each multiply-add of the projections, the feed-forward and
    the recurrence (three state-sized products a token for GLA: decay, write, read; four for the delta rule), three times
    that where gradients are formed. A generated token reads every weight once."""
    d, n = case["dim"], case["batch"] * case["seq"]
    if case["kind"] == "moe":
        h, e, k = case["hidden"], case["experts"], case["top_k"]
        params = (e + 1) * 2 * d * h + e * d
        return {"bytes": 2.0 * (4 * n * d + 2 * params), "flops": 3 * 2.0 * n * (k + 1) * 2 * d * h}
    hd, state = case["heads"] * case["head_dim"], case["heads"] * case["head_dim"] ** 2
    per_token = 2.0 * state * (3 if case["mixer"] == "gla" else 4)
    if case["kind"] == "generate":
        layer = 5 * d * hd + 3 * d * _swiglu_hidden(d)
        params = case["layers"] * layer + VOCAB * d
        tokens, new = case["batch"] * (case["seq"] + case["new"]), case["new"]
        flops = tokens * case["layers"] * (2.0 * layer + per_token) + case["batch"] * (new + 1) * 2.0 * VOCAB * d
        return {"bytes": 2.0 * params * (new + 1) + 8.0 * case["batch"] * state * case["layers"] * (new + 1), "flops": flops}
    params = 5 * d * hd + 8 * d * d
    flops = n * (2.0 * params + per_token)
    if case["kind"] == "prefill":
        return {"bytes": 2.0 * (2 * n * d + params) + 4.0 * case["batch"] * state * (2 if case["carry"] else 1), "flops": flops}
    return {"bytes": 2.0 * (4 * n * d + 2 * params), "flops": 3 * flops}


def tolerance(case):
    return {"rel": 0.02, "max": 0.5}


# ------------------------------------------------------------------------------------------------ 64-bit statement
def _norm(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _turned(x, start):
    """Half-split rotary embedding of [B, T, H, D] from position ``start``; angles are the 32-bit ones of the models."""
    half = x.shape[-1] // 2
    freq = 1.0 / (ROPE_BASE ** (torch.arange(0, half, dtype=torch.float32, device=x.device) / half))
    angle = torch.outer(torch.arange(start, start + x.shape[1], dtype=torch.float32, device=x.device), freq).double()
    c, s = angle.cos()[None, :, None, :], angle.sin()[None, :, None, :]
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _recurrence(q, k, v, g, beta, state):
    """Gated linear attention (``beta`` None) or the gated delta rule over [B, T, H, D] in chunks of 64 tokens:
    S_t = exp(g_t) S_{t-1} + k_t u_t^T with u_t = v_t, or beta_t (v_t - S_{t-1}^T k_t); o_t = S_t^T q_t."""
    q, k, v, g = (t.transpose(1, 2) for t in (q, k, v, g))
    outs = []
    for c in range(0, q.shape[2], 64):
        qc, kc, vc, gc = (t[:, :, c:c + 64] for t in (q, k, v, g))
        b = gc.cumsum(2)
        grown = kc * torch.exp(-b)  # at most 64 tokens of decay: far inside the range of 64-bit numbers
        u = vc
        if beta is not None:
            bc = beta[:, c:c + 64].transpose(1, 2).unsqueeze(-1)
            seen = kc * torch.exp(b - gc)
            low = torch.tril(bc * (seen @ grown.transpose(-1, -2)), -1)
            u = torch.linalg.solve_triangular(low, bc * (vc - seen @ state), upper=False, unitriangular=True)
        read = qc * torch.exp(b)
        outs.append(torch.tril(read @ grown.transpose(-1, -2)) @ u + read @ state)
        last = b[:, :, -1:]
        state = torch.exp(last).transpose(-1, -2) * state + (kc * torch.exp(last - b)).transpose(-1, -2) @ u
    return torch.cat(outs, 2).transpose(1, 2), state


def _mixer(case, w, prefix, x, state, start):
    B, T, _ = x.shape
    H, D = case["heads"], case["head_dim"]
    q, k, v, g = ((x @ w[f"{prefix}{n}_proj.weight"].t()).view(B, T, H, D) for n in "qkvg")
    q, k = (_turned(F.normalize(F.elu(t) + 1.0, dim=-1, eps=1e-6), start) for t in (q, k))
    beta = torch.sigmoid(x @ w[prefix + "beta_proj.weight"].t()) if case["mixer"] == "gdn" else None
    if state is None:
        state = x.new_zeros(B, H, D, D)
    o, state = _recurrence(q, k, v, F.logsigmoid(g), beta, state)
    return o.reshape(B, T, H * D) @ w[prefix + "out_proj.weight"].t(), state


def _gelu_mlp(x, w, p):
    return F.gelu(x @ w[p + "0.weight"].t() + w[p + "0.bias"], approximate="tanh") @ w[p + "2.weight"].t() + w[p + "2.bias"]


def _block(case, w, x, state, start):
    a, state = _mixer(case, w, "attn.gla.", _norm(x, w["norm1.weight"]), state, start)
    x = x + a
    return x + _gelu_mlp(_norm(x, w["norm2.weight"]), w, "ffn."), state


def _moe(case, w, x):
    """Training mode with every expert below its capacity, which random routing of these batches stays (else None)."""
    x2 = x.reshape(-1, case["dim"])
    n, e, k = x2.shape[0], case["experts"], case["top_k"]
    # routing logits are bfloat16, so are the decisions that follow from them
    logits = x2 @ w["router.weight"].t() + w["router.bias"]
    logits = logits + (logits.detach().bfloat16().double() - logits.detach())
    probs = torch.softmax(logits, -1)
    order = torch.sort(logits.detach(), dim=-1, descending=True, stable=True)[1][:, :k]
    if any(int(c) > math.ceil(n / e * 1.5) for j in range(k) for c in torch.bincount(order[:, j], minlength=e)):
        return None
    mix = probs.gather(1, order)
    mix = mix / mix.sum(-1, keepdim=True) if k > 1 else mix
    out = 0.5 * _gelu_mlp(x2, w, "shared.")
    for i in range(e):
        rows, slot = (order == i).nonzero(as_tuple=True)
        out = out.index_add(0, rows, mix[rows, slot].unsqueeze(1) * _gelu_mlp(x2[rows], w, f"experts.{i}."))
    return out.view_as(x)


def exact(case, seed):
    kind = case["kind"]
    if kind == "generate":
        return _exact_generate(case, seed)
    w = {n: t.double() for n, t in (_moe_weights if kind == "moe" else _block_weights)(case, seed).items()}
    x = _rows(case, seed, 5).double()
    if kind == "prefill":
        state, start = None, case["carry"]
        with torch.no_grad():
            if start:
                _, state = _block(case, w, _rows(case, seed, 6, start).double(), None, 0)
            y, state = _block(case, w, x, state, start)
        return {"y": y, "state": state}
    names = list(w)
    for t in (x, *w.values()):
        t.requires_grad_(True)
    y = _moe(case, w, x) if kind == "moe" else _block(case, w, x, None, 0)[0]
    if y is None:
        return None
    grads = torch.autograd.grad(y, (x, *w.values()), _rows(case, seed, 7).double())
    g = dict(zip(names, grads[1:]))
    out = {"y": y.detach(), "dx": grads[0]}
    if kind == "moe":
        for i, n in ((1, "0.weight"), (1, "0.bias"), (2, "2.weight"), (2, "2.bias")):
            out[f"d {n[2]}{i}"] = torch.stack([g.pop(f"experts.{e}.{n}") for e in range(case["experts"])])
    else:
        out["d attn.gla.qkvg_weight"] = torch.cat([g.pop(f"attn.gla.{n}_proj.weight") for n in "qkvg"])
    out.update({"d " + n: t for n, t in g.items()})
    return out


@torch.no_grad()
def _exact_generate(case, seed):
    w16, order = _model_weights(case, seed)
    prompt = torch.randint(0, VOCAB, (case["batch"], case["seq"]), device="cuda", generator=_generator(seed, 4))
    tokens = prompt
    for _ in range(case["new"]):
        tokens = torch.cat((tokens, order[tokens[:, -1:]]), 1)
    w = {n: t.double() for n, t in w16.items() if not n.startswith(("embed", "lm_head"))}
    x, states = w16["embed_tokens.weight"][tokens].double(), []
    for i in range(case["layers"]):
        p = f"layers.{i}."
        a, s = _mixer(case, w, p + "attn.", _norm(x, w[p + "input_norm.weight"]), None, 0)
        x = x + a
        n = _norm(x, w[p + "post_attn_norm.weight"])
        x = x + (F.silu(n @ w[p + "mlp.gate_proj.weight"].t()) * (n @ w[p + "mlp.up_proj.weight"].t())) @ w[p + "mlp.down_proj.weight"].t()
        states.append(s)
    h = _norm(x[:, case["seq"] - 1:], w["norm.weight"])
    best = torch.cat([(h[:, i:i + 4] @ w16["lm_head.weight"].double().t()).argmax(-1) for i in range(0, h.shape[1], 4)], 1)
    if not torch.equal(best[:, :-1], tokens[:, case["seq"]:]):
        return None  # the order of the vocabulary is not what this model says: no other statement of its tokens at hand
    return {"tokens": tokens, "states": states}

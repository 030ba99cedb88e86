"""Performance cases: what users of this framework have it do, through ``Engine``.

A case is one of two calls on one of the registered models, at the sizes the repository's benchmark and tests use (depth cut
where three copies of a request's state have to fit one GPU):

``reply``
    ``Engine.generate``: a prompt comes in, ``new`` tokens go out.  The prompt takes whichever path the engine picks for its
    length, decoding runs as captured rounds.  With the speculative target a round is draft, verification and sampler.
``extend``
    ``StackEngine.extend``: ``feed`` given tokens behind a sequence of ``context`` tokens, logits of the last ``want`` of them
    back.  One token is a decode step driven by the caller, more are the chunk path: a prompt (``context`` 0) or a later turn.

Weights are the repository's random initialisation from a fixed seed, with a larger embedding.  Where a model would otherwise
have no preferred next token, its head is tied to its embedding through a permutation, and the draft proposes the same successor
for 70 % of the tokens: peaked distributions, as trained models have, so that neither a generated sequence nor the choice of
experts hangs on the last bit of a product.  Prompts come from the case's seed.
"""
import math

import torch
import torch.nn.functional as F

from naivert_b200.models.device_init import init_draft_rank_weights_device, init_rank_weights_device, init_stack_weights_device
from naivert_b200.models.registry import resolve_model
from naivert_b200.models.spec import SamplingParams
from naivert_b200.runtime.engine import Engine

CHUNK = 2048                     # rows of a prompt chunk, the benchmark's and the layer stacks' default
# model of a case -> (registered name, layers kept, longest sequence)
MODELS = {
    "target": ("naive-n0.5", 6, 17408),            # both attention kinds, dense and routed feed-forward
    "experts": ("tumatar-bench", 4, 25600),
    "dense": ("tumatar-bench-dense", 4, 25600),
    "states": ("zuzupel-bench", 6, 25600),
    "experts-small": ("tumatar-small", 0, 4096),
    "states-small": ("zuzupel-small", 0, 4096),
}
WEIGHT_SEED = 20


def listed():
    return [
        # chat with the speculative target: a short message below the chunk path's threshold, then a short answer
        {"name": "target-turn", "model": "target", "call": "reply", "prompt": 53, "new": 40},
        # the same with an ordinary prompt and a longer answer: rounds dominate
        {"name": "target-reply", "model": "target", "call": "reply", "prompt": 1021, "new": 192},
        # a long document is read and summarised: sparse attention past 2048 keys, prompt chunks dominate
        {"name": "target-document", "model": "target", "call": "reply", "prompt": 16001, "new": 24},
        # an answer of a model with routed experts: captured one-token rounds
        {"name": "experts-reply", "model": "experts", "call": "reply", "prompt": 300, "new": 96},
        # a prompt of the benchmark's length, the continuation's logits read back (scoring)
        {"name": "experts-prompt", "model": "experts", "call": "extend", "form": "bf16", "context": 0, "feed": 8192, "want": 64},
        # a follow-up message behind a long conversation
        {"name": "dense-turn", "model": "dense", "call": "extend", "form": "bf16", "context": 11003, "feed": 187, "want": 1},
        # a step of a caller that samples for itself, far into a sequence (latent attention over 24,000 tokens)
        {"name": "dense-step", "model": "dense", "call": "extend", "form": "bf16", "context": 24001, "feed": 1, "want": 1},
        # a model of matrix states and chunked attention: answer, prompt of odd length, step
        {"name": "states-reply", "model": "states", "call": "reply", "prompt": 777, "new": 96},
        {"name": "states-prompt", "model": "states", "call": "extend", "form": "bf16", "context": 0, "feed": 6131, "want": 64},
        {"name": "states-step", "model": "states", "call": "extend", "form": "bf16", "context": 12289, "feed": 1, "want": 1},
        # small models: launches and host work are what counts; the 32-bit form is what a port is checked against
        {"name": "small-step", "model": "states-small", "call": "extend", "form": "bf16", "context": 150, "feed": 1, "want": 1},
        {"name": "small-prompt-fp32", "model": "experts-small", "call": "extend", "form": "fp32", "context": 0, "feed": 301, "want": 301},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["target", "target", "target", "experts", "dense", "states", "states", "experts-small", "states-small"])
    if model == "target":
        prompt = _log(rng, 20, 16001)
        return {"model": model, "call": "reply", "prompt": prompt, "new": _log(rng, 8, 192 if prompt < 3000 else 24)}
    small = model.endswith("small")
    longest = 3000 if small else 12000
    kind = rng.choice(["reply", "prompt", "turn", "step"])
    if kind == "reply":
        return {"model": model, "call": "reply", "prompt": _log(rng, 8, 1200), "new": _log(rng, 16, 96)}
    form = rng.choice(["bf16", "fp32"]) if small else "bf16"
    if kind == "prompt":
        feed = _log(rng, 33, 1200 if small else 8192)
        return {"model": model, "call": "extend", "form": form, "context": 0, "feed": feed, "want": min(feed, 64)}
    if kind == "turn":
        return {"model": model, "call": "extend", "form": form, "context": _log(rng, 100, longest), "feed": _log(rng, 2, 800), "want": 1}
    return {"model": model, "call": "extend", "form": form, "context": _log(rng, 16, longest if small else 24001), "feed": 1, "want": 1}


# --------------------------------------------------------------------------- models and engines
_KEPT = {}                       # weights, successors and engine of the model in use: a program serves one


def _spec(case):
    name, layers, _ = MODELS[case["model"]]
    spec = resolve_model(name)
    return spec.with_layers(layers) if layers else spec


def _weights(case):
    """(weights, draft weights or None, successors the model prefers, successors the draft proposes)."""
    if _KEPT.get("model") != case["model"]:
        _KEPT.clear()
        torch.cuda.empty_cache()
        spec, dev = _spec(case), torch.device("cuda", torch.cuda.current_device())
        g = torch.Generator(device=dev).manual_seed(WEIGHT_SEED)
        draft = None
        after = proposed = torch.arange(spec.vocab, device=dev)          # a tied head prefers the token itself
        if case["model"] == "target":
            w = init_rank_weights_device(spec, 0, 1, seed=WEIGHT_SEED, device=dev)
            draft = init_draft_rank_weights_device(spec, 0, 1, seed=WEIGHT_SEED, device=dev)
            after = torch.randperm(spec.vocab, generator=g, device=dev)
            differs = torch.nonzero(torch.rand(spec.vocab, generator=g, device=dev) >= 0.7)[:, 0]
            proposed = after.clone()
            proposed[differs] = after[differs.roll(1)]
            w["embed"] = w["embed"] * 600                                # the stream keeps its token through the layers
            w["lm_head"] = torch.empty_like(w["lm_head"]).index_copy_(0, after, w["embed"] * (0.02 / 12))
            draft["markov_w1"] = draft["markov_w1"] * 8
            draft["markov_w2"] = torch.empty_like(draft["markov_w2"]).index_copy_(0, proposed, draft["markov_w1"])
        else:
            w = init_stack_weights_device(spec, WEIGHT_SEED, dev)
            w["embed"] = w["embed"] * 4
            if not spec.tied_head:
                after = proposed = torch.randperm(spec.vocab, generator=g, device=dev)
                w["head"] = torch.empty_like(w["head"]).index_copy_(0, after, w["embed"] * (33.0 / spec.hidden))
        _KEPT.update(model=case["model"], weights=(w, draft, after.cpu(), proposed.cpu()))
    return _KEPT["weights"]


class _Owned:
    """An engine that gives its pinned and peer memory back when the last state that uses it is dropped."""

    def __init__(self, case):
        spec = _spec(case)
        w, draft, _, _ = _weights(case)
        more = {"draft_weights": draft} if draft is not None else {"dtype": case.get("form", "bf16")}
        self.engine = Engine.build(spec, capacity=MODELS[case["model"]][2], weights=w, prefill_chunk=CHUNK, **more)

    def __del__(self):
        if hasattr(self, "engine"):
            self.engine.close()


def _engine(case):
    """The engine of a program that serves one request after the other."""
    _weights(case)
    form = case.get("form", "bf16")
    if _KEPT.get("form") != form:
        _KEPT["engine"], _KEPT["form"] = _Owned(case), form
    return _KEPT["engine"]


def _tokens(case, seed):
    """Prompt, or context and the tokens behind it, on the host."""
    spec = _spec(case)
    n = case["prompt"] if case["call"] == "reply" else case["context"] + case["feed"]
    g = torch.Generator().manual_seed(int(seed) * 7919 + 3)
    return torch.randint(0, spec.vocab - 1024 if spec.vocab > 4096 else spec.vocab - 8, (n,), generator=g, dtype=torch.int32)


SAMPLING = {"temperature": 0.4, "top_p": 0.95}       # the benchmark's


def prepare(case, seed):
    tokens = _tokens(case, seed)
    if case["call"] == "reply":
        return {"case": case, "own": _engine(case), "prompt": tokens.pin_memory(), "sampling": SamplingParams(seed=int(seed), **SAMPLING)}
    n = case["context"]
    if n == 0:
        return {"case": case, "own": _engine(case), "tokens": tokens.tolist(), "want": range(case["feed"] - case["want"], case["feed"])}
    own = _Owned(case)                                # the sequence lives in the engine's caches
    own.engine.extend(tokens[:n].tolist())
    return {"case": case, "own": own, "tokens": tokens[n:].tolist(), "want": range(case["feed"] - case["want"], case["feed"])}


def run(state):
    case, eng = state["case"], state["own"].engine
    if case["call"] == "reply":
        result = eng.generate(state["prompt"], case["new"], state["sampling"])
        rows = 1 if eng.round.draft is None else eng.spec.draft.rows
        return {"tokens": torch.tensor(result.tokens), "logits": eng.target.logits[:rows].clone()}
    eng.position = case["context"]                    # the same turn again: steps and chunks may be repeated at a position
    return {"logits": eng.extend(state["tokens"], state["want"])}


# --------------------------------------------------------------------------- work
def _stack_matrices(spec):
    """Per layer run: (elements of its dense matrices, elements of one expert, experts, top k, attention width, state elements)."""
    out = []
    for r in spec.runs():
        layer = spec.layers[r.layer]
        m, f, W = layer.mixer, layer.mlp, spec.hidden
        attn = state = 0
        if m.kind == "latent_attention":
            n = (W + m.heads * m.dim) * m.q_rank + (W + m.heads * (m.dim + m.vdim)) * m.kv_rank + 2 * W * m.heads * m.vdim
            attn = (m.heads * (m.dim + m.vdim), m.kv_rank, 0)
        elif m.kind == "rglru":
            n = 3 * W * m.width + 2 * m.width * m.block
        elif m.kind == "channel_delta":
            n = W * (2 * m.kv_heads * m.dim + 2 * m.heads * m.vdim + m.heads + m.decay_rank + m.gate_rank) \
                + m.heads * (m.dim * m.decay_rank + m.vdim * m.gate_rank)
            state = m.heads * m.dim * m.vdim
        elif m.kind == "wkv":
            n = m.heads * m.dim * (5 * W + m.decay_rank) + W * m.decay_rank
            state = m.heads * m.dim * m.dim
        else:
            a, b = m.left, m.right
            n = W * (a.heads * (a.dim + a.vdim) + a.kv_heads * (a.dim + a.vdim) + b.heads * (2 * b.dim + 3 * b.vdim + 2))
            attn = (a.heads * (a.dim + a.vdim), a.kv_heads * (a.dim + a.vdim), a.window)
            state = b.heads * b.dim * b.vdim
        expert = experts = top = 0
        if f is not None and f.kind == "moe":
            n += W * f.routing.expert_count
            expert, experts, top = 3 * W * f.ff, f.routing.expert_count, f.routing.top_k
        elif f is not None:
            n += (2 if f.kind == "relu2" else 3) * W * f.ff
        out.append((n, expert, experts, top, attn, state))
    return out


def _hit(experts, top, rows):
    """Experts that ``rows`` tokens are expected to reach."""
    return experts * (1 - (1 - top / experts) ** rows) if experts else 0


def _stack_work(spec, pos, rows, want, es):
    """Bytes and operations of ``rows`` tokens behind ``pos``, ``want`` rows of logits."""
    nbytes, flops = 2.0 * rows * spec.hidden, 0.0
    for n, expert, experts, top, attn, state in _stack_matrices(spec):
        nbytes += 2.0 * (n + _hit(experts, top, rows) * expert)
        flops += 2.0 * rows * (n + top * expert)
        if attn:
            per_key, cached, window = attn
            seen = pos + rows if not window else min(pos + rows, window)
            nbytes += es * cached * float(seen + rows)
            flops += 2.0 * per_key * rows * (seen - min(rows, seen) / 2)
        nbytes += 8.0 * state
        flops += 6.0 * rows * state
    nbytes += 2.0 * spec.vocab * spec.hidden + 4.0 * want * spec.vocab
    return nbytes, flops + 2.0 * want * spec.vocab * spec.hidden


def _target_rows(spec, pos, rows):
    """Bytes (e4m3 experts and output projections, bf16 q/k/v) and operations of ``rows`` target rows behind ``pos``."""
    H, rt, ix = spec.hidden, spec.routing, spec.indexer
    nbytes = flops = 0.0
    for layer, kind in enumerate(spec.layer_kinds):
        a = spec.attention[kind]
        qkv = H * (a.head_count * a.head_dim + a.kv_head_count * (a.head_dim + a.v_head_dim))
        o = H * a.head_count * a.v_head_dim
        row = a.kv_head_count * (a.head_dim + a.v_head_dim) * 2.0
        if a.sliding_window is None:
            qkv += H * (ix.head_count * (ix.head_dim + 1) + ix.head_dim)
            mean = max(1.0, pos + rows / 2)
            keys, touched = min(ix.top_k, mean), min(pos + rows, ix.top_k * rows)
            if pos + rows > ix.top_k:
                flops += 2.0 * rows * mean * ix.head_count * ix.head_dim
                nbytes += (pos + rows) * (ix.head_dim + 4.0)
        else:
            keys, touched = a.sliding_window, min(pos + rows, a.sliding_window + rows)
        flops += 2.0 * rows * (qkv + o + keys * a.head_count * (a.head_dim + a.v_head_dim))
        nbytes += 2.0 * qkv + o + row * (touched + rows)
        if spec.is_dense(layer):
            flops += 6.0 * rows * H * spec.dense_intermediate
            nbytes += 3.0 * H * spec.dense_intermediate
        else:
            flops += 2.0 * rows * (H * rt.expert_count + 3 * rt.top_k * H * rt.intermediate)
            nbytes += 4.0 * H * rt.expert_count + 3.0 * H * rt.intermediate * _hit(rt.expert_count, rt.top_k, rows)
    return nbytes, flops


def work(case):
    spec = _spec(case)
    es = 4 if case.get("form") == "fp32" else 2
    if case["call"] == "extend":
        nbytes, flops = _stack_work(spec, case["context"], case["feed"], case["want"], es)
    elif case["model"] != "target":
        n, new = case["prompt"], case["new"]
        nbytes, flops = _stack_work(spec, 0, n - 1, 0, es) if n > 1 else (0.0, 0.0)
        step = _stack_work(spec, n + new // 2, 1, 1, es)
        nbytes, flops = nbytes + new * step[0], flops + new * step[1]
    else:
        n, d = case["prompt"], spec.draft
        rounds = max(1.0, case["new"] / 3.14)           # tokens of a round at an acceptance of 0.7
        nbytes, flops = _target_rows(spec, 0, n - 1)
        rows = _target_rows(spec, n + case["new"] // 2, d.rows)
        head = spec.vocab * spec.hidden
        layer = spec.hidden * (2 * d.head_count + 2 * d.kv_head_count) * d.head_dim + 3 * spec.hidden * d.intermediate
        fixed = len(d.target_layer_ids) * spec.hidden * d.hidden + d.layer_count * layer
        nbytes += rounds * (rows[0] + 2.0 * fixed + 2 * 2.0 * head + 2.0 * spec.vocab * d.markov_rank + 15 * 4.0 * spec.vocab)
        flops += rounds * (rows[1] + 2.0 * d.rows * (fixed + 2 * head) + 2.0 * d.block_size * spec.vocab * d.markov_rank)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what other correct orders of the same sums differ by.  32-bit form: 1e-6 from 64 bits.  bf16 stacks: other
    chunk sizes differ by 0.006 (0.16 at one logit, where a token's last expert changes).  Target: its paths without fused steps and
    wide tiles differ by 0.015 (0.11), mostly e4m3 codes that round the other way."""
    if case.get("form") == "fp32":
        return {"rel": 1e-5}
    return {"rel": 0.03, "max": 0.45} if case["model"] == "target" else {"rel": 0.025, "max": 0.6}


# --------------------------------------------------------------------------- the same in 64 bits
D = torch.float64


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, eps):
    return F.layer_norm(x, x.shape[-1:], eps=eps) * w


def _lin(x, w):
    """x W^T with the matrix taken to 64 bits a few rows at a time."""
    out = torch.empty(x.shape[0], w.shape[0], dtype=D, device=x.device)
    for lo in range(0, w.shape[0], 16384):
        out[:, lo:lo + 16384] = x @ w[lo:lo + 16384].to(D).T
    return out


def _attend(q, k, v, scale, lowest, sink=None, chosen=None):
    """Causal softmax attention, a block of queries at a time; q [T, H, D], k and v [T, G, .]; query i sees keys lowest(i) .. i,
    of those the ones in ``chosen`` (rows lo .. hi -> mask)."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=D, device=q.device)
    at = torch.arange(T, device=q.device)
    for lo in range(0, T, 256):
        hi = min(T, lo + 256)
        first = int(lowest(at[lo:hi]).min())
        keys = at[first:hi]
        dead = (keys[None] > at[lo:hi, None]) | (keys[None] < lowest(at[lo:hi])[:, None])
        if chosen is not None:
            mask = chosen(lo, hi)
            dead = dead if mask is None else dead | ~mask[:, first:hi]
        for g in range(G):
            hs = slice(g * H // G, (g + 1) * H // G)
            s = torch.einsum("ihd,jd->hij", q[lo:hi, hs], k[first:hi, g]) * scale
            s.masked_fill_(dead, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[hs].view(-1, 1, 1).expand(-1, hi - lo, 1)], -1)
            p = torch.softmax(s, -1)
            out[lo:hi, hs] = torch.einsum("hij,jv->ihv", p[..., : hi - first], v[first:hi, g])
    return out


def _routed(h, scores, choice, top, normalise, expert):
    """Sum over a token's chosen experts; ``expert(e)`` -> (gate, up, down) in 64 bits."""
    ids = torch.sort(-choice, dim=-1, stable=True).indices[:, :top]
    p = scores.gather(1, ids)
    p = p / (p.sum(-1, keepdim=True) + 1e-20) if normalise else p
    out = torch.zeros_like(h)
    for e in range(scores.shape[1]):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            gate, up, down = expert(e)
            out.index_add_(0, t, p[t, j, None] * ((F.silu(h[t] @ gate.T) * (h[t] @ up.T)) @ down.T))
    return out


# ---- latent attention, gated linear recurrence
def _latent_attention(h, w, m, eps):
    T = h.shape[0]
    q = _lin(_rms(_lin(h, w["dq"]), w["dq.norm"].to(D), eps), w["uq"]).view(T, m.heads, m.dim)
    c = _rms(_lin(h, w["dkv"]), w["dkv.norm"].to(D), eps)
    k, v = _lin(c, w["uk"]).view(T, m.heads, m.dim), _lin(c, w["uv"]).view(T, m.heads, m.vdim)
    o = _attend(q, k, v, m.scale, lambda i: i * 0).reshape(T, -1)
    return _lin(o * torch.sigmoid(_lin(h, w["g"])), w["o"])


def _conv(x, taps):
    out = torch.zeros_like(x)
    n = taps.shape[1]
    for back in range(min(n, x.shape[0])):
        out[back:] += taps[:, n - 1 - back].to(D) * x[: x.shape[0] - back]
    return out


def _recurrence(h, w, m, eps):
    T = h.shape[0]
    y = F.gelu(_lin(h, w["y"]) + w["y.b"].to(D), approximate="tanh")
    u = _conv(_lin(h, w["x"]) + w["x.b"].to(D), w["conv"]) + w["conv.b"].to(D)
    ub = u.view(T, m.blocks, m.block)
    r, i = (torch.sigmoid(torch.einsum("tbi,bji->tbj", ub, w[n].to(D)) + w[n + ".b"].to(D)).reshape(T, -1) for n in ("ra", "ri"))
    log_a = -m.decay * r * F.softplus(w["lam"].to(D), threshold=100.0)
    a, s = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
    for t in range(1, T):
        s[t].addcmul_(a[t], s[t - 1])
    return _lin(s * y, w["o"])


# ---- matrix states
def _unit(x):
    return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _heads(x, H):
    """Key heads repeated for the value heads they serve."""
    return x.repeat_interleave(H // x.shape[1], 1)


def _delta(h, w, m, eps):
    T, H = h.shape[0], m.heads
    q, k, v = (F.silu(_conv(_lin(h, w[n]), w[n + ".conv"])) for n in "qkv")
    q = _heads(_unit(q.view(T, m.kv_heads, m.dim)) * m.dim ** -0.5, H)
    k, v = _heads(_unit(k.view(T, m.kv_heads, m.dim)), H), v.view(T, H, m.vdim)
    beta = torch.sigmoid(_lin(h, w["b"]))[..., None]
    rate = F.softplus(_lin(_lin(h, w["a1"]), w["a2"]) + w["dt_bias"].to(D), threshold=100.0).view(T, H, m.dim)
    g = torch.exp(-torch.exp(w["A_log"].to(D))[:, None] * rate)
    S, out = torch.zeros(H, m.dim, m.vdim, dtype=D, device=h.device), torch.empty_like(v)
    for t in range(T):
        S *= g[t, :, :, None]
        S.baddbmm_(k[t, :, :, None], (beta[t] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0]))[:, None])
        out[t] = torch.bmm(q[t, :, None], S)[:, 0]
    gate = torch.sigmoid(_lin(_lin(h, w["g1"]), w["g2"]))
    return _lin(_rms(out, w["norm"].to(D), eps).reshape(T, -1) * gate, w["o"])


def _wkv(h, w, m, eps):
    T, H = h.shape[0], m.heads
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])

    def mix(s):
        return h + (before - h) * w["mu." + s].to(D)

    r, k, v = (_lin(mix(s), w[s]).view(T, H, m.dim) for s in "rkv")
    decay = torch.exp(-torch.exp(_lin(torch.tanh(_lin(mix("w"), w["w1"])), w["w2"]) + w["w0"].to(D))).view(T, H, m.dim)
    now = (r * w["u"].to(D) * k).sum(-1, keepdim=True) * v                  # the current token's own part of the read-out
    S, out = torch.zeros(H, m.dim, m.dim, dtype=D, device=h.device), torch.empty_like(v)
    for t in range(T):
        out[t] = torch.bmm(r[t, :, None], S)[:, 0]
        S *= decay[t, :, :, None]
        S.baddbmm_(k[t, :, :, None], v[t, :, None])
    o = _rms(out + now, 1.0, eps).reshape(T, -1) * w["norm"].to(D) * F.silu(_lin(mix("g"), w["g"]))
    return _lin(o, w["o"])


def _rotate(x, rot):
    half = rot.dims // 2
    f = torch.tensor([rot.base ** (-2.0 * i / rot.dims) / rot.factor for i in range(half)], dtype=D, device=x.device)
    a = torch.arange(x.shape[0], dtype=D, device=x.device)[:, None, None] * f
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., 2 * half:]], -1)


def _grouped(h, w, m, eps):
    T = h.shape[0]
    q, k, v = (_lin(h, w["left." + n]) + w["left." + n + ".b"].to(D) for n in "qkv")
    q, k = q.view(T, m.heads, m.dim), k.view(T, m.kv_heads, m.dim)
    q, k = _rotate(_rms(q, w["left.q.norm"].to(D), eps), m.rotary), _rotate(_rms(k, w["left.k.norm"].to(D), eps), m.rotary)
    o = _attend(q, k, v.view(T, m.kv_heads, m.vdim), m.scale, lambda i: i // m.window * m.window)
    return _lin(o.reshape(T, -1), w["left.o"])


def _memory(h, w, m, eps):
    T, H = h.shape[0], m.heads
    q, k = _lin(h, w["right.q"]).view(T, H, m.dim) * m.dim ** -0.5, _lin(h, w["right.k"]).view(T, H, m.dim)
    v = _lin(h, w["right.v"]).view(T, H, m.vdim)
    i = m.cap * torch.tanh((_lin(h, w["right.i"]) + w["right.i.b"].to(D)) / m.cap)
    f = F.logsigmoid(m.cap * torch.tanh((_lin(h, w["right.f"]) + w["right.f.b"].to(D)) / m.cap))
    # running maximum of the stabilised state: max over s <= t of i_s + sum of f behind s, and of the start's 0
    F_ = f.cumsum(0)
    top = torch.maximum(F_, F_ + torch.cummax(i - F_, 0).values)
    a = torch.exp(f + torch.cat([torch.zeros_like(top[:1]), top[:-1]]) - top)[..., None]
    b = torch.exp(i - top)[..., None]
    S = torch.zeros(H, m.dim, m.vdim + 1, dtype=D, device=h.device)         # the last column is the normaliser
    v1, out = torch.cat([v, torch.ones_like(v[..., :1])], -1), torch.empty(T, H, m.vdim + 1, dtype=D, device=h.device)
    for t in range(T):
        S *= a[t, :, :, None]
        S.baddbmm_((b[t] * k[t])[:, :, None], v1[t, :, None])
        out[t] = torch.bmm(q[t, :, None], S)[:, 0]
    o = out[..., :-1] / (torch.maximum(out[..., -1:].abs(), torch.exp(-top)[..., None]) + 1e-6)
    return _lin(_rms(o, 1.0, eps).reshape(T, -1) * w["right.norm"].to(D) * torch.sigmoid(_lin(h, w["right.g"])), w["right.o"])


def _parallel(h, w, m, eps):
    return (_rms(_grouped(h, w, m.left, eps), w["left.out"].to(D), eps) + _rms(_memory(h, w, m.right, eps), w["right.out"].to(D), eps)) / 2


MIXERS = {"latent_attention": _latent_attention, "rglru": _recurrence, "channel_delta": _delta, "wkv": _wkv, "parallel": _parallel}


def _stack_ffn(h, w, f):
    if f.kind == "relu2":
        return _lin(F.relu(_lin(h, w["up"])) ** 2, w["down"])
    if f.kind == "dense":
        g, u = _lin(h, w["gate"]).clamp(max=f.limit), _lin(h, w["up"]).clamp(-f.limit, f.limit)
        return _lin(g * torch.sigmoid(1.702 * g) * (u + 1), w["down"])
    rt = f.routing
    s = torch.sigmoid(_lin(h, w["router"]))
    choice = s + w["correction"].to(D)
    groups = choice.view(len(h), rt.group_count, -1)
    best = torch.sort(-groups.topk(2, -1).values.sum(-1), dim=-1, stable=True).indices[:, :rt.limited_group_count]
    out_of = torch.ones_like(groups[..., 0], dtype=torch.bool).scatter_(1, best, False)
    choice = groups.masked_fill(out_of[..., None], -math.inf).view_as(choice)
    return _routed(h, s, choice, rt.top_k, rt.normalize_top_k, lambda e: tuple(w[n][e].to(D) for n in ("gate", "up", "down")))


def _stack_logits(spec, w, tokens, want):
    eps = spec.norm_eps
    norm = _layer_norm if spec.norm == "layer" else _rms
    x = w["embed"][tokens].to(D) * spec.embed_scale
    for r in spec.runs():
        layer, lw = spec.layers[r.layer], w["layers"][spec.owner(r.layer)]
        if r.pass_start is not None:
            x = x + w["loop"][r.pass_start].to(D)
        h = _rms(x, lw["norm1"].to(D), eps) if spec.pre_norm else x
        x = x + norm(MIXERS[layer.mixer.kind](h, lw["mix"], layer.mixer, eps), lw["norm1b"].to(D), eps)
        if layer.mlp is not None:
            h = _rms(x, lw["norm2"].to(D), eps) if spec.pre_norm else x
            x = x + norm(_stack_ffn(h, lw["mlp"], layer.mlp), lw["norm2b"].to(D), eps)
    return _lin(norm(x[want], w["norm"].to(D), eps), w["embed"] if spec.tied_head else w["head"]) * spec.logit_scale


# ---- the speculative target
def _whole(q, e=None):
    """A block-scaled matrix in 64 bits."""
    w, s = (q["w"], q["s"]) if e is None else (q["w"][e], q["s"][e])
    n, k = w.shape
    return (w.to(D).view(n // 128, 128, k // 128, 128) * s.to(D)[:, None, :, None]).view(n, k)


def _pairs(x, dims, theta):
    """Rotation of adjacent pairs of the first ``dims`` columns; x [T, heads, dim]."""
    f = theta ** (-2.0 * torch.arange(dims // 2, dtype=D, device=x.device) / dims)
    a = torch.arange(x.shape[0], dtype=D, device=x.device)[:, None, None] * f
    p = x[..., :dims].reshape(*x.shape[:-1], dims // 2, 2)
    turned = torch.stack([p[..., 0] * a.cos() - p[..., 1] * a.sin(), p[..., 0] * a.sin() + p[..., 1] * a.cos()], -1)
    return torch.cat([turned.reshape(*x.shape[:-1], dims), x[..., dims:]], -1)


def _target_logits(spec, w, tokens, want):
    eps, ix, rt, T = spec.norm_eps, spec.indexer, spec.routing, len(tokens)
    x = w["embed"][tokens].to(D)
    for layer, kind in enumerate(spec.layer_kinds):
        a, lw = spec.attention[kind], w["layers"][layer]
        h = _rms(x, lw["g_in"].to(D), eps)
        q = _pairs(_lin(h, lw["wq"]).view(T, -1, a.head_dim), a.rope_dim, a.rope_theta)
        k = _pairs(_lin(h, lw["wk"]).view(T, -1, a.head_dim), a.rope_dim, a.rope_theta)
        v = _lin(h, lw["wv"]).view(T, -1, a.v_head_dim) * a.value_scale
        if a.sliding_window is not None:
            o = _attend(q, k, v, a.softmax_scale, lambda i: (i - a.sliding_window + 1).clamp(min=0), sink=lw["sink"].to(D))
        else:
            iq = _pairs(_lin(h, lw["iwq"]).view(T, -1, ix.head_dim), ix.rope_dim, a.rope_theta)
            ik = _layer_norm(_lin(h, lw["iwk"]), lw["ik_w"].to(D), eps) + lw["ik_b"].to(D)
            ik, weight = _pairs(ik[:, None], ix.rope_dim, a.rope_theta)[:, 0], _lin(h, lw["iww"]) * ix.weight_scale

            def chosen(lo, hi):
                if hi <= ix.top_k:
                    return None
                s = torch.zeros(hi - lo, hi, dtype=D, device=x.device)
                for j in range(ix.head_count):
                    s += torch.relu(iq[lo:hi, j] @ ik[:hi].T) * weight[lo:hi, j, None]
                s.masked_fill_(torch.arange(hi, device=x.device)[None] > torch.arange(lo, hi, device=x.device)[:, None], -math.inf)
                return torch.zeros_like(s, dtype=torch.bool).scatter_(1, s.topk(ix.top_k, -1).indices, True)

            o = _attend(q, k, v, a.softmax_scale, lambda i: i * 0, chosen=chosen)
        x = x + o.reshape(T, -1) @ _whole(lw["wo"]).T
        h = _rms(x, lw["g_post"].to(D), eps)
        if "dense" in lw:
            gate, up, down = (_whole(lw["dense"][n]) for n in ("gate", "up", "down"))
            x = x + (F.silu(h @ gate.T) * (h @ up.T)) @ down.T
        else:
            s = torch.sigmoid(_lin(h, lw["router_w"]))
            x = x + rt.route_scale * _routed(h, s, s + lw["router_b"].to(D), rt.top_k, rt.normalize_top_k,
                                             lambda e: tuple(_whole(lw[n], e) for n in ("gate", "up", "down")))
    return _lin(_rms(x[want], w["norm"].to(D), eps), w["lm_head"])


def exact(case, seed):
    spec, tokens = _spec(case), _tokens(case, seed).tolist()
    w, _, after, proposed = _weights(case)
    dev = w["embed"].device
    if case["call"] == "extend":
        want = list(range(len(tokens) - case["want"], len(tokens)))
        return {"logits": _stack_logits(spec, w, torch.tensor(tokens, device=dev), want)}
    for _ in range(case["new"]):                        # the preferred successors, one after the other
        tokens.append(int(after[tokens[-1]]))
        if tokens[-1] in spec.stop_token_ids:
            break
    if case["model"] != "target":
        return {"tokens": None, "logits": _stack_logits(spec, w, torch.tensor(tokens, device=dev), [len(tokens) - 1])}
    for _ in range(spec.draft.block_size):              # the rows of the last verification: the last token and the draft's proposals
        tokens.append(int(proposed[tokens[-1]]))
    want = list(range(len(tokens) - spec.draft.rows, len(tokens)))
    return {"tokens": None, "logits": _target_logits(spec, w, torch.tensor(tokens, device=dev), want)}

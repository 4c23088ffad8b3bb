"""The work this engine is used for, as cases that can be timed: what a serving program asks of it, step by step.

A case is one model shape and one job. The shapes are the presets of :func:`mlxcel_b200.config.preset` at their full widths, heads,
vocabularies and experts, with a few layers of each, so that weights are drawn in a moment and the same numbers can be had in 64 bits.
The jobs are what one pass through a serving engine consists of:

* ``chat``    sequences are opened, their prompts read, tokens generated one by one, sequences closed
* ``decode``  running sequences with their context in the cache get their next tokens, one step after the other
* ``verify``  a speculative round: every running sequence gets its pending token and the drafts behind it in one step
* ``prefill`` prompts are read in portions, with the logits behind each; the last ones are what the first generated token is drawn from
* ``admit``   one step of continuous batching: a new prompt is read beside the rows that are decoding

Every token is given (nothing is sampled), so that results can be compared; all goes through ``LLM`` and the engine's
``open_sequence`` / ``feed`` / ``close_sequence``. Jobs on running sequences end by taking the fed tokens back, as a speculative
round takes rejected drafts back, so that a pass can be repeated.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

PORTION = 2048          # prompt tokens of one sequence in a step: the engine's default chunk
BUDGET = 8192           # tokens of one step: the engine's default
SMALL = 0.005           # spread of the projections that write into the residual stream

# preset and layers kept of it; "pack": stored weights; "kv": bits of a cached value
MODELS = {
    "tiny": dict(preset="tiny-llama", layers=2),
    "dense": dict(preset="llama-3.1-8b", layers=8),
    "dense 4-bit": dict(preset="llama-3.1-8b", layers=8, pack="affine", kv=8),
    "wide": dict(preset="qwen3-32b", layers=3),
    "experts": dict(preset="gpt-oss-120b", layers=2, pack="mxfp4"),
    "state space": dict(preset="mamba2-2.7b", layers=8),
}


def listed():
    def c(name, model, job, rows, length, new, spread=0.0):
        return dict(name=name, model=model, job=job, rows=rows, length=length, new=new, spread=spread)
    return [
        # The smallest call: one short chat with the tiny model of the first benchmark configuration (16 tokens in, 32 logits
        # out). Launches, graph replays and the host's part of a step are all there is.
        c("tiny chat", "tiny", "chat", 1, 16, 31),
        # The headline benchmark's steady state: 64 requests around 1024 tokens, one token each per step.
        c("decode 64 rows", "dense", "decode", 64, 1279, 4, 0.2),
        # A few users with long documents in the cache: few rows, so the weights and the long contexts are read for little work.
        c("decode long contexts", "dense", "decode", 3, 12001, 4, 0.3),
        # The headline benchmark's admission: 8 prompts of 1024 tokens in one step.
        c("prefill 8 x 1024", "dense", "prefill", 8, 1024, 0),
        # One long document, read in the engine's portions: attention over a context that grows to 12 thousand tokens.
        c("prefill one long prompt", "dense", "prefill", 1, 12001, 0),
        # A speculative round of the 16-request configuration: pending token + 3 drafts on contexts up to 4096.
        c("verify 16 x 4", "wide", "verify", 16, 4090, 4, 0.25),
        # One chat with a 4-bit checkpoint and an 8-bit cache: the interactive single user.
        c("4-bit decode 1 row", "dense 4-bit", "decode", 1, 777, 8),
        # The same model serving 32 requests.
        c("4-bit decode 32 rows", "dense 4-bit", "decode", 32, 1100, 4, 0.4),
        # The same model in a step that reads a 512-token prompt while 31 rows decode (the engine's chunk when rows are waiting).
        c("4-bit admit", "dense 4-bit", "admit", 31, 900, 512, 0.4),
        # Mixture of experts with 4-bit experts, windowed and full attention: 128 requests decode.
        c("experts decode 128 rows", "experts", "decode", 128, 1025, 4, 0.5),
        # The same model reading prompts: 4 x 2048 tokens in one step.
        c("experts prefill 4 x 2048", "experts", "prefill", 4, 2048, 0),
        # A state-space model: ragged prompts are read, then tokens generated from the state.
        c("state space chat", "state space", "chat", 4, 1500, 6, 0.5),
    ]


def draw(rng):
    def log(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))

    def case(model, job, rows, length, new):
        return dict(model=model, job=job, rows=rows, length=max(2, length), new=new, spread=round(rng.uniform(0.0, 0.6), 2))
    kind = rng.randrange(10)
    if kind == 0:
        return case("tiny", "chat", rng.randint(1, 4), log(4, 200), rng.randint(8, 31))
    if kind == 1:
        rows = log(1, 64)
        return case("dense", "decode", rows, log(64, min(12001, 65536 // rows)), rng.randint(1, 4))
    if kind == 2:
        rows = log(1, 8)
        return case("dense", "prefill", rows, log(24, 8192 // rows), 0)
    if kind == 3:
        return case("dense", "prefill", 1, log(1500, 12001), 0)
    if kind == 4:
        return case("wide", "verify", log(1, 16), log(64, 4090), rng.randint(2, 4))
    if kind == 5:
        rows = log(1, 32)
        return case("dense 4-bit", "decode", rows, log(64, 1100), rng.randint(2, 4))
    if kind == 6:
        return case("dense 4-bit", "admit", log(1, 31), log(64, 900), log(17, 512))
    if kind == 7:
        return case("experts", "decode", log(1, 128), log(64, 1025), rng.randint(1, 4))
    if kind == 8:
        rows = log(1, 4)
        return case("experts", "prefill", rows, log(64, 8192 // rows // 2), 0)
    return case("state space", "chat", log(1, 4), log(32, 1500), rng.randint(1, 6))


# ----------------------------------------------------------------------------- what is asked, token by token
def _plan(case):
    """(tokens each sequence has in the cache beforehand, steps, all tokens of each sequence). A step lists (sequence, first token, tokens,
    places whose logits are wanted)."""
    rows, new, job = case["rows"], case["new"], case["job"]
    lens = [max(2, case["length"] - int(case["spread"] * case["length"] * i / rows)) for i in range(rows)]
    if case["model"] == "experts" and job == "decode":
        # The windowed layers give blocks of 16 tokens back once nothing can reach them; a context that ends right behind a block edge can
        # be extended by a few tokens and taken back without crossing the next edge.
        lens = [max(1, (n - 1) // 16) * 16 + 1 for n in lens]
    single = [[(i, n + t, 1, [0]) for i, n in enumerate(lens)] for t in range(new)]
    if job == "decode":
        return lens, single, [n + new for n in lens]
    if job == "verify":
        return lens, [[(i, n, new, list(range(new))) for i, n in enumerate(lens)]], [n + new for n in lens]
    if job == "admit":
        return lens + [0], [[(i, n, 1, [0]) for i, n in enumerate(lens)] + [(rows, 0, new, [new - 1])]], [n + 1 for n in lens] + [new]
    steps = _portions([0] * rows, lens)
    if job == "chat":
        steps, lens = steps + single, [n + new for n in lens]
    return [0] * rows, steps, lens


def _portions(start, stop, seqs=8):
    """Steps that bring every sequence from ``start`` to ``stop`` tokens: at most 8 sequences and BUDGET tokens each. The logits behind
    every portion are wanted: the host then waits for a portion before it builds the next one."""
    at, steps = list(start), []
    while any(a < b for a, b in zip(at, stop)):
        step, left = [], BUDGET
        for i, b in enumerate(stop):
            n = min(PORTION, b - at[i], left)
            if n > 0 and len(step) < seqs:
                step.append((i, at[i], n, [n - 1]))
                at[i] += n
                left -= n
        steps.append(step)
    return steps


def _config(case):
    from mlxcel_b200.config import preset
    m = MODELS[case["model"]]
    cfg = preset(m["preset"])
    cfg.num_hidden_layers = m["layers"]
    cfg.rope_scaling = None                   # a table of other frequencies: the same work
    if cfg.layer_types:
        cfg.layer_types = cfg.layer_types[:m["layers"]]
    return cfg, m


# ----------------------------------------------------------------------------- weights and tokens, from the seed alone
class _Draw:
    def __init__(self, seed, device):
        self.g = torch.Generator(device=device).manual_seed(1_000_003 * int(seed) + 17)
        self.device = device

    def normal(self, *shape, std=0.02, mean=0.0, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=self.device).normal_(mean, std, generator=self.g)

    def uniform(self, n, lo, hi):
        return torch.empty(n, dtype=torch.float32, device=self.device).uniform_(lo, hi, generator=self.g)

    def affine(self, n, k, std=0.02):
        """4-bit codes, 8 to a word, with a scale and an offset for each 64: values spread like N(0, std) weights."""
        words = torch.randint(-2 ** 31, 2 ** 31, (n, k // 8), dtype=torch.int32, device=self.device, generator=self.g)
        scale = self.uniform(n * k // 64, 0.18 * std, 0.25 * std).view(n, k // 64)
        offset = -7.5 * scale + self.uniform(n * k // 64, -0.15 * std, 0.15 * std).view(n, k // 64)
        return words, scale.to(torch.bfloat16), offset.to(torch.bfloat16)

    def mxfp4(self, e, n, k, std=0.02):
        """e2m1 codes with one of two powers of two for each 32, around the spread of N(0, std)."""
        words = torch.randint(-2 ** 31, 2 ** 31, (e, n, k // 8), dtype=torch.int32, device=self.device, generator=self.g)
        low = 127 + math.floor(math.log2(std / 2.93))
        return words, torch.randint(low, low + 2, (e, n, k // 32), dtype=torch.uint8, device=self.device, generator=self.g), None


def _weights(cfg, m, seed, device="cuda"):
    """The model's tensors by name, as plain tensors (packed matrices: words, scales, offsets). As in a trained model, a layer's two results
    are small beside the residual stream they are added to."""
    d = _Draw(seed, device)
    H, D, Hq, Hkv, V = cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.vocab_size
    mat = d.affine if m.get("pack") == "affine" else d.normal
    gain = lambda n: d.normal(n, std=0.1, mean=1.0)                                                       # noqa: E731
    w = dict(embed=d.normal(V, H, std=1.0), final_norm=gain(H), layers=[])
    for _ in range(cfg.num_hidden_layers):
        if "mamba" in cfg.extra:
            s = cfg.extra["mamba"]
            inner, heads, conv = s["d_inner"], s["d_inner"] // s["head_dim"], s["d_inner"] + 2 * s["n_groups"] * s["d_state"]
            w["layers"].append(dict(
                norm=gain(H), in_proj=d.normal(inner + conv + heads, H), conv_w=d.normal(conv, s["d_conv"], std=0.2), conv_b=d.normal(conv, std=0.1),
                dt_bias=d.uniform(heads, -3.0, -1.0), A_log=torch.log(d.uniform(heads, 1.0, 16.0)), D=torch.ones(heads, device=device),
                gnorm=gain(inner), out_proj=d.normal(H, inner, std=SMALL)))
            continue
        lw = dict(ln1=gain(H), ln2=gain(H), wqkv=mat((Hq + 2 * Hkv) * D, H), wo=mat(H, Hq * D, std=SMALL))
        if cfg.qk_norm:
            lw.update(q_norm=gain(D), k_norm=gain(D))
        if cfg.attention_sinks:
            lw.update(bqkv=d.normal((Hq + 2 * Hkv) * D), bo=d.normal(H), sinks=d.normal(Hq, std=1.0, dtype=torch.float32))
        if cfg.num_experts:
            E, I = cfg.num_experts, cfg.moe_intermediate_size
            # a trained router is sure of its choice: logits of a few units, not of noise
            lw.update(router_w=d.normal(E, H, std=0.05), router_b=d.normal(E), experts_gate_up=d.mxfp4(E, 2 * I, H), experts_down=d.mxfp4(E, H, I, std=SMALL),
                      experts_gate_up_b=d.normal(E, 2 * I), experts_down_b=d.normal(E, H))
        else:
            lw.update(w_gate_up=mat(2 * cfg.intermediate_size, H), w_down=mat(H, cfg.intermediate_size, std=SMALL))
        w["layers"].append(lw)
    w["lm_head"] = w["embed"] if cfg.tie_word_embeddings else mat(V, H)
    return w


def _tokens(case, cfg, seed):
    lens = _plan(case)[2]
    g = torch.Generator().manual_seed(1_000_003 * int(seed) + 71)
    return [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in lens]


# ----------------------------------------------------------------------------- the framework's side
def prepare(case, seed):
    from mlxcel_b200.engine import EngineConfig
    from mlxcel_b200.llm import LLM
    from mlxcel_b200.models.mamba2 import Mamba2LayerWeights, Mamba2Weights
    from mlxcel_b200.models.weights import LayerWeights, ModelWeights, QuantizedTensor
    cfg, m = _config(case)
    cached, steps, lens = _plan(case)

    def stored(v):
        if not isinstance(v, tuple):
            return v
        return QuantizedTensor(*v, 4, *((32, "mxfp4") if v[2] is None else (64, "affine")))
    w = _weights(cfg, m, seed)
    parts = [{k: stored(v) for k, v in lw.items()} for lw in w["layers"]]
    if "mamba" in cfg.extra:
        weights = Mamba2Weights(w["embed"], [Mamba2LayerWeights(**p) for p in parts], w["final_norm"], w["lm_head"])
    else:
        weights = ModelWeights(w["embed"], [LayerWeights(**p) for p in parts], w["final_norm"], stored(w["lm_head"]))
    del w, parts
    ecfg = EngineConfig(max_batch=max(2, case["rows"]), max_num_batched_tokens=BUDGET, max_prefill_seqs=max(8, case["rows"] if case["job"] == "verify" else 0),
                        num_blocks=sum(n // 16 + 2 for n in lens) + 8, max_model_len=(max(lens) // 16 + 2) * 16, kv_bits=m.get("kv", 16))
    llm = LLM(cfg, weights, ecfg, fold_norms="mamba" not in cfg.extra)
    state = dict(llm=llm, cached=cached, steps=steps, tokens=_tokens(case, cfg, seed), ids={})
    for i, n in enumerate(cached):
        if n:
            state["ids"][i] = llm.engine.open_sequence()
    for step in _portions([0] * len(cached), cached):
        _feed(state, step)
    if any(cached) and all(n == 1 for _, _, n, _ in steps[0]):
        # a serving engine has met its decode batch before: the graph of this one exists
        _feed(state, steps[0])
        _take_back(state)
    return state


def _feed(state, step):
    ids, tokens = state["ids"], state["tokens"]
    return state["llm"].engine.feed([(ids[i], tokens[i][a:a + n], want) for i, a, n, want in step])


def _take_back(state):
    """Sequences with a cached context lose what was fed behind it."""
    eng = state["llm"].engine
    for i, n in enumerate(state["cached"]):
        if n:
            sid = state["ids"][i]
            eng.bm.truncate(sid, n)
            if eng.bm_win is not None:
                eng.bm_win.truncate(sid, n)
            seq = eng.seqs[sid]
            del seq.prompt[n:]
            seq.num_computed = n


def run(state):
    eng, ids, cached = state["llm"].engine, state["ids"], state["cached"]
    for i, n in enumerate(cached):
        if not n:
            ids[i] = eng.open_sequence()
    out = [_feed(state, step) for step in state["steps"]]
    _take_back(state)
    for i, n in enumerate(cached):
        if not n:
            eng.close_sequence(ids.pop(i))
    return [x for x in out if x is not None]


# ----------------------------------------------------------------------------- what a pass cannot do without
def _sizes(cfg, m):
    """Parameters every token meets in a layer, bytes they are stored in, parameters of the head, bytes of a parameter there."""
    H, D, Hq, Hkv, V = cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.vocab_size
    if "mamba" in cfg.extra:
        s = cfg.extra["mamba"]
        inner, heads = s["d_inner"], s["d_inner"] // s["head_dim"]
        n = H * (2 * inner + 2 * s["n_groups"] * s["d_state"] + heads) + H * inner
        return n, 2.0 * n, V * H, 2.0
    per = 0.5 + 4 / 64 if m.get("pack") == "affine" else 2.0
    n = H * (Hq + 2 * Hkv) * D + H * Hq * D
    if not cfg.num_experts:
        n += 3 * H * cfg.intermediate_size
    return n, per * n, V * H, per


def work(case):
    cfg, m = _config(case)
    cached, steps, _ = _plan(case)
    n, nbytes, head, per = _sizes(cfg, m)
    L, D, Hq, Hkv = cfg.num_hidden_layers, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads
    recurrent = "mamba" in cfg.extra
    kv = 2 * Hkv * D * (1.0625 if m.get("kv") == 8 else 2.0)             # bytes of a cached token in a layer (8 bits: a scale and offset per 64)
    total = flops = 0.0
    for step in steps:
        tokens, wanted = sum(s[2] for s in step), sum(len(s[3]) for s in step)
        total += L * nbytes + (per * head if wanted else 0) + tokens * cfg.hidden_size * 2 + wanted * cfg.vocab_size * 2
        flops += 2.0 * L * n * tokens + 2.0 * head * wanted
        if cfg.num_experts:
            E, k, one = cfg.num_experts, cfg.num_experts_per_tok, 3 * cfg.hidden_size * cfg.moe_intermediate_size
            used = E * (1 - (1 - k / E) ** tokens)                       # experts that some token is expected to choose
            total += L * used * one * (0.5 + 1 / 32)
            flops += 2.0 * L * k * one * tokens
        for layer in range(L):
            if recurrent:
                s = cfg.extra["mamba"]
                state = s["d_inner"] * s["d_state"]
                total += len(step) * state * 4 * 2
                flops += 6.0 * state * tokens
                continue
            window = cfg.layer_window(layer)
            for _, a, c, _ in step:
                seen = min(a + c, window + c) if window else a + c
                total += kv * (seen + c)
                keys = sum(min(a + t + 1, window) if window else a + t + 1 for t in range(c)) if window else c * a + c * (c + 1) / 2
                flops += 4.0 * Hq * D * keys
    return dict(bytes=total, flops=flops)


def tolerance(case):
    # Two correct bf16 implementations differ by the rounding of the activations between kernels, layer after layer: against 64 bits the
    # outputs are 0.004 (2 layers) to 0.012 (8 layers) off. Where a router's choice is a tie up to rounding, one row may differ by more.
    return {"rel": 0.02, "max": 0.5 if case["model"] == "experts" else 0.15}


# ----------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """Logits of every step from a plain statement of the model: whole sequences at once, weights as stored, all sums in fp64."""
    cfg, m = _config(case)
    _, steps, lens = _plan(case)
    w = _weights(cfg, m, seed)
    tokens = _tokens(case, cfg, seed)
    first = [0]
    for n in lens:
        first.append(first[-1] + n)
    h = w["embed"][torch.tensor(sum(tokens, []), device="cuda")].double()
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    for li, lw in enumerate(w["layers"]):
        if "mamba" in cfg.extra:
            h = h + _mixer(cfg, lw, h, lens, first)
            continue
        x = _rms(h, lw["ln1"], cfg.rms_norm_eps)
        h = h + _attention(cfg, li, lw, x, pos, lens, first)
        x = _rms(h, lw["ln2"], cfg.rms_norm_eps)
        if cfg.num_experts:
            h = h + _experts(cfg, lw, x)
        else:
            I = cfg.intermediate_size
            h = h + _lin(x, lw["w_gate_up"], lambda z: _lin(F.silu(z[:, :I]) * z[:, I:], lw["w_down"]))
    out = []
    for step in steps:
        rows = [first[i] + a + p for i, a, _, want in step for p in want]
        if rows:
            out.append(_lin(_rms(h[rows], w["final_norm"], cfg.rms_norm_eps), w["lm_head"]))
    return out


def _dense(w):
    if not isinstance(w, tuple):
        return w.double()
    words, scale, offset = w
    codes = ((words.unsqueeze(-1) >> torch.arange(0, 32, 4, dtype=torch.int32, device=words.device)) & 15).flatten(-2)
    if offset is not None:
        return (codes.view(*codes.shape[:-1], -1, 64).double() * scale.double().unsqueeze(-1) + offset.double().unsqueeze(-1)).view(codes.shape)
    table = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0], dtype=torch.float64, device=words.device)
    v = table[codes.long()].view(*codes.shape[:-1], -1, 32)
    return (v * torch.exp2(scale.double() - 127.0).unsqueeze(-1)).view(codes.shape)


def _lin(x, w, then=None):
    """x w^T, and ``then`` of it, for a few thousand rows at a time."""
    d = _dense(w).t()
    parts = [p @ d if then is None else then(p @ d) for p in x.split(8192)]
    return torch.cat(parts)


def _rms(x, g, eps):
    return torch.cat([p * torch.rsqrt(p.square().mean(-1, keepdim=True) + eps) * g.double() for p in x.split(16384)])


def _attention(cfg, li, lw, x, pos, lens, first):
    D, Hq, Hkv, window = cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.layer_window(li)
    z = _lin(x, lw["wqkv"])
    if "bqkv" in lw:
        z += lw["bqkv"].double()
    z = z.view(-1, Hq + 2 * Hkv, D)
    q, k, v = z[:, :Hq], z[:, Hq:Hq + Hkv], z[:, Hq + Hkv:]
    if "q_norm" in lw:
        q, k = _rms(q, lw["q_norm"], cfg.rms_norm_eps), _rms(k, lw["k_norm"], cfg.rms_norm_eps)
    ang = pos.double()[:, None] / cfg.rope_theta ** (torch.arange(0, D, 2, dtype=torch.float64, device=x.device) / D)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def turn(t):
        a, b = t[..., :D // 2], t[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    q, k = turn(q), turn(k)
    o = torch.empty_like(q)
    for s, n in zip(first, lens):
        ks, vs = (t[s:s + n].transpose(0, 1).repeat_interleave(Hq // Hkv, 0) for t in (k, v))
        for a in range(0, n, 1024):
            b, lo = min(n, a + 1024), max(0, a - window) if window else 0
            sc = q[s + a:s + b].transpose(0, 1) @ ks[:, lo:b].transpose(1, 2) * D ** -0.5
            i, j = torch.arange(a, b, device=x.device)[:, None], torch.arange(lo, b, device=x.device)[None]
            sc.masked_fill_((j > i) | ((j <= i - window) if window else False), -math.inf)
            if "sinks" in lw:
                sc = torch.cat([sc, lw["sinks"].double()[:, None, None].expand(Hq, b - a, 1)], -1)
            o[s + a:s + b] = (torch.softmax(sc, -1)[..., :b - lo] @ vs[:, lo:b]).transpose(0, 1)
    o = _lin(o.reshape(-1, Hq * D), lw["wo"])
    return o + lw["bo"].double() if "bo" in lw else o


def _experts(cfg, lw, x):
    I, k = cfg.moe_intermediate_size, cfg.num_experts_per_tok
    top, ids = (_lin(x, lw["router_w"]) + lw["router_b"].double()).topk(k, -1)
    share = torch.softmax(top, -1)
    out = torch.zeros_like(x)
    for e in range(cfg.num_experts):
        row, slot = torch.nonzero(ids == e, as_tuple=True)
        if not row.numel():
            continue
        z = x[row] @ _dense(tuple(None if t is None else t[e] for t in lw["experts_gate_up"])).t() + lw["experts_gate_up_b"][e].double()
        gate, up = z[:, :I].clamp(max=cfg.swiglu_limit), z[:, I:].clamp(-cfg.swiglu_limit, cfg.swiglu_limit)
        a = gate * torch.sigmoid(cfg.swiglu_alpha * gate) * (up + 1.0)
        y = a @ _dense(tuple(None if t is None else t[e] for t in lw["experts_down"])).t() + lw["experts_down_b"][e].double()
        out.index_add_(0, row, y * share[row, slot][:, None])
    return out


def _mixer(cfg, lw, h, lens, first):
    s = cfg.extra["mamba"]
    inner, P, G, N, K = s["d_inner"], s["head_dim"], s["n_groups"], s["d_state"], s["d_conv"]
    heads = inner // P
    z = _lin(_rms(h, lw["norm"], cfg.rms_norm_eps), lw["in_proj"])
    B, T = len(lens), max(lens)
    pad = torch.zeros(B, T + K - 1, z.shape[1], dtype=torch.float64, device=h.device)
    for i, (a, n) in enumerate(zip(first, lens)):
        pad[i, K - 1:K - 1 + n] = z[a:a + n]
    conv = inner + 2 * G * N
    c = sum(pad[:, j:j + T, inner:inner + conv] * lw["conv_w"][:, j].double() for j in range(K)) + lw["conv_b"].double()
    c = F.silu(c)
    dt = F.softplus(pad[:, K - 1:, inner + conv:] + lw["dt_bias"].double())
    keep = torch.exp(-dt * torch.exp(lw["A_log"].double()))
    xs = c[..., :inner].view(B, T, heads, P)
    bs, cs = (c[..., inner + j * G * N:inner + (j + 1) * G * N].reshape(B, T, G, N).repeat_interleave(heads // G, 2) for j in (0, 1))
    state = torch.zeros(B, heads, P, N, dtype=torch.float64, device=h.device)
    ys = torch.empty(B, T, heads, P, dtype=torch.float64, device=h.device)
    for t in range(T):
        state.mul_(keep[:, t, :, None, None]).add_((dt[:, t, :, None] * xs[:, t])[..., None] * bs[:, t, :, None, :])
        ys[:, t] = (state @ cs[:, t, :, :, None])[..., 0]
    ys = (ys + lw["D"].double()[:, None] * xs).view(B, T, inner) * F.silu(pad[:, K - 1:, :inner])
    ys = _rms(torch.cat([ys[i, :n] for i, n in enumerate(lens)]), lw["gnorm"], cfg.rms_norm_eps)
    return _lin(ys, lw["out_proj"])

"""Performance cases: steps of GGUF-quantised decoders through `LLMEngine`, the way a program that generates or scores text
takes them.

A decode case is one step of one new token for each of `batch` sequences that hold about `ctx` tokens of context; after the
step the sequences are set back by the one token, so that every pass is the step at the same place.  A prefill case is one step
of about `rows` new tokens for each of `batch` sequences, from nothing or behind `ctx` tokens of context.  Both return the
logits of the last token of every sequence.

Models have the package's shapes, some with fewer layers so that a case is set up quickly: every layer of a shape does the same
work.  Their checkpoints are blocks of random codes with scales that give matrices of standard deviation 0.02 and mean 0,
in the block formats that the recipe names for each tensor.  As in models that are trained, the embedding is as large as what a
layer reads, and what all layers together add to the residual stream is no larger, so that rounding errors do not grow from
layer to layer.
"""
import math

import torch

from llaminar_b200.engine.engine import LLMEngine
from llaminar_b200.engine.kv_cache import Q8
from llaminar_b200.gguf import GGMLType
from llaminar_b200.models.config import RECIPES, SHAPES
from llaminar_b200.models.weights import ModelWeights, QTensor

DEVICE = "cuda"


def _case(name, model, layers, recipe, kind, batch, rows, ctx, kv="bf16"):
    return {"name": name, "model": model, "layers": layers, "recipe": recipe, "kind": kind, "batch": batch, "rows": rows, "ctx": ctx, "kv": kv}


def listed():
    return [
        # one user's chat, a few hundred tokens in: the smallest step there is, and the one that a single user waits for
        _case("decode_8b_1", "qwen3-8b", 36, "Q4_K_M", "decode", 1, 1, 700),
        # a few long documents at once, 8-bit weights and cache
        _case("decode_8b_q8_3_long", "qwen3-8b", 18, "Q8_0", "decode", 3, 1, 6001, "q8_0"),
        # a server with 32 lanes taken, the usual 4-bit mix
        _case("decode_8b_32", "qwen3-8b", 18, "Q4_K_M", "decode", 32, 1, 1024),
        # the same at the larger dense shape
        _case("decode_32b_32", "qwen3-32b", 16, "Q4_K_S", "decode", 32, 1, 512),
        # a half-full server, an odd number of lanes, 5-bit weights and the 8-bit cache
        _case("decode_8b_q5_13", "qwen3-8b", 12, "Q5_K", "decode", 13, 1, 333, "q8_0"),
        # a busy server with short contexts, the family with biases and without query and key norms
        _case("decode_7b_100", "qwen2.5-7b", 14, "Q4_K_M", "decode", 100, 1, 200),
        # a few lanes of the model with routed experts
        _case("decode_30b_a3b_8", "qwen3-30b-a3b", 12, "Q4_K_M", "decode", 8, 1, 256),
        # a short question: the prompt's own latency
        _case("prefill_8b_37", "qwen3-8b", 36, "Q4_K_M", "prefill", 1, 37, 0),
        # one ordinary prompt: time to the first token
        _case("prefill_8b_2048", "qwen3-8b", 36, "Q4_K_M", "prefill", 1, 2048, 0),
        # the next turn of a long chat, or a chunk of a long document, behind what is cached
        _case("prefill_8b_q8_500_behind", "qwen3-8b", 18, "Q8_0", "prefill", 1, 500, 7000),
        # prompts of several users in one step, the largest an engine takes by default
        _case("prefill_32b_8x1020", "qwen3-32b", 16, "Q4_K_S", "prefill", 8, 1020, 0),
        # prompts of a few users for the model with routed experts
        _case("prefill_30b_a3b_3x700", "qwen3-30b-a3b", 12, "Q4_K_M", "prefill", 3, 700, 0),
    ]


_MODELS = (("qwen3-8b", 12, 36), ("qwen3-8b", 12, 36), ("qwen3-32b", 8, 16), ("qwen2.5-7b", 14, 28), ("qwen3-30b-a3b", 6, 12))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    top = [work(c) for c in listed()]
    most = {k: max(w[k] for w in top) for k in ("bytes", "flops")}
    while True:
        model, lo, hi = rng.choice(_MODELS)
        recipe = rng.choice(("Q4_K_M", "Q4_K_M", "Q4_K_S", "Q5_K", "Q6_K", "Q8_0")) if model != "qwen3-30b-a3b" else rng.choice(("Q4_K_M", "Q8_0"))
        c = {"model": model, "layers": rng.randint(lo, hi), "recipe": recipe, "kind": rng.choice(("decode", "prefill"))}
        if c["kind"] == "decode":
            c.update(batch=_log(rng, 1, 128), rows=1, ctx=_log(rng, 30, 8000))
        else:
            c.update(batch=rng.choice((1, 1, 1, 2, 3, 5, 8)), rows=_log(rng, 5, 4096), ctx=rng.choice((0, 0, _log(rng, 64, 7000))))
        c["kv"] = rng.choice(("bf16", "bf16", "q8_0"))
        w = work(c)
        if c["batch"] * (c["ctx"] + 1) <= 33000 and c["batch"] * c["rows"] <= 8192 and all(w[k] <= most[k] for k in most):
            return c


# -- checkpoints ---------------------------------------------------------------------------------------------------------

_BLOCK = {"Q4_K": (256, 144), "Q5_K": (256, 176), "Q6_K": (256, 210), "Q8_0": (32, 34)}


def _half(x):
    """The bytes of 16-bit floats, [n] -> [n, 2]."""
    return x.to(torch.float16).view(-1, 1).view(torch.uint8)


def _blocks(fmt, n, gen, shift=0):
    """`n` blocks of random codes, flat bytes, of standard deviation 0.02 * 2^-shift.  The two k-quant formats with minima get the
    minimum that centres their codes."""
    size = _BLOCK[fmt][1]
    b = torch.randint(0, 256, (n, size), dtype=torch.uint8, device=DEVICE, generator=gen)

    def numbers(lo, hi, cols=1):
        return torch.randint(lo, hi, (n, cols), device=DEVICE, generator=gen, dtype=torch.int32)

    if fmt in ("Q4_K", "Q5_K"):
        r = numbers(5, 8)[:, 0].float()
        unit, centre = (2.0 ** (-16 - shift), 7.5) if fmt == "Q4_K" else (2.0 ** (-17 - shift), 15.5)
        b[:, 0:2], b[:, 2:4] = _half(r * unit), _half(r * unit * centre)
        s = numbers(32, 64, 8)                                    # scale and minimum of a sub-block are the same number
        lo, hi = s[:, :4], s[:, 4:]
        b[:, 4:8] = (lo | (hi >> 4) << 6).to(torch.uint8)
        b[:, 8:12] = b[:, 4:8]
        b[:, 12:16] = ((hi & 15) | (hi & 15) << 4).to(torch.uint8)
    elif fmt == "Q6_K":
        s = numbers(64, 128, 16) * (1 - 2 * numbers(0, 2, 16))
        b[:, 192:208] = s.to(torch.int8).view(torch.uint8)
        b[:, 208:210] = _half(numbers(160, 220)[:, 0].float() * 2.0 ** (-24 - shift))
    else:
        b[:, 0:2] = _half(numbers(240, 330)[:, 0].float() * 2.0 ** (-20 - shift))
    return b.reshape(-1)


def _values(fmt, raw, shape):
    """Block bytes -> 64-bit values, written from the published layouts of the formats."""
    if fmt == "F32":
        return raw.view(torch.float32).view(shape).double()
    b = raw.view(-1, _BLOCK[fmt][1])
    n = b.shape[0]

    def half(at):
        return b[:, at:at + 2].contiguous().view(torch.float16).double()

    if fmt == "Q8_0":
        return (half(0) * b[:, 2:].view(torch.int8).double()).view(shape)
    if fmt == "Q6_K":
        ql, qh = b[:, :128].reshape(n, 2, 64), b[:, 128:192].reshape(n, 2, 32)
        sc = b[:, 192:208].contiguous().view(torch.int8).double().view(n, 2, 8, 1)
        low = torch.cat([ql & 15, ql >> 4], 2)                    # 128 columns of a half block in order
        high = torch.cat([(qh >> 2 * i) & 3 for i in range(4)], 2)
        q = (low | high << 4).double() - 32.0
        return (half(208).view(n, 1, 1, 1) * sc * q.view(n, 2, 8, 16)).view(shape)
    sb = b[:, 4:16].int()
    sc = torch.cat([sb[:, :4] & 63, (sb[:, 8:] & 15) | (sb[:, :4] >> 6) << 4], 1).double()
    mn = torch.cat([sb[:, 4:8] & 63, sb[:, 8:] >> 4 | (sb[:, 4:8] >> 6) << 4], 1).double()
    qs = b[:, -128:].reshape(n, 4, 32)
    q = torch.stack([qs & 15, qs >> 4], 2).reshape(n, 8, 32)
    if fmt == "Q5_K":
        q = q | torch.stack([(b[:, 16:48] >> i) & 1 for i in range(8)], 1) << 4
    return ((half(0) * sc).unsqueeze(2) * q.double() - (half(2) * mn).unsqueeze(2)).view(shape)


def _config(case):
    return SHAPES[case["model"]].with_(n_layers=case["layers"])


def _tensors(case, seed):
    """name -> (format, shape, bytes) of the whole checkpoint."""
    cfg, recipe = _config(case), RECIPES[case["recipe"]]
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    out = {}

    def mat(name, *shape, layer=None):
        fmt = recipe.for_tensor(name, layer, cfg.n_layers).name
        shift = -6 if "embd" in name else round(math.log2(0.02 * math.sqrt(2 * cfg.n_layers * shape[-1]))) if "_output" in name or "_down" in name else 0
        out[name] = (fmt, shape, _blocks(fmt, math.prod(shape) // _BLOCK[fmt][0], gen, shift))

    def plain(name, *shape, mean=0.0, std=0.02):
        x = torch.randn(*shape, device=DEVICE, generator=gen) * std + mean
        out[name] = ("F32", shape, x.reshape(-1).view(torch.uint8))

    d, hd = cfg.d_model, cfg.head_dim
    qd, kvd = cfg.n_heads * hd, cfg.n_kv_heads * hd
    mat("token_embd.weight", cfg.vocab_size, d)
    plain("output_norm.weight", d, mean=1.0, std=0.1)
    mat("output.weight", cfg.vocab_size, d)
    for i in range(cfg.n_layers):
        p = f"blk.{i}."
        plain(p + "attn_norm.weight", d, mean=1.0, std=0.1)
        for name, rows, cols in (("attn_q", qd, d), ("attn_k", kvd, d), ("attn_v", kvd, d), ("attn_output", d, qd)):
            mat(f"{p}{name}.weight", rows, cols, layer=i)
            if cfg.qkv_bias and name != "attn_output":
                plain(f"{p}{name}.bias", rows, std=0.1)
        if cfg.qk_norm:
            plain(p + "attn_q_norm.weight", hd, mean=1.0, std=0.1)
            plain(p + "attn_k_norm.weight", hd, mean=1.0, std=0.1)
        plain(p + cfg.ffn_norm_name, d, mean=1.0, std=0.1)
        if cfg.is_moe:
            # a trained router is sure of its first choices: logits of a standard deviation of about 3
            plain(p + "ffn_gate_inp.weight", cfg.n_experts, d, std=3.0 / d ** 0.5)
            mat(p + "ffn_gate_exps.weight", cfg.n_experts, cfg.expert_ff, d, layer=i)
            mat(p + "ffn_up_exps.weight", cfg.n_experts, cfg.expert_ff, d, layer=i)
            mat(p + "ffn_down_exps.weight", cfg.n_experts, d, cfg.expert_ff, layer=i)
        else:
            mat(p + "ffn_gate.weight", cfg.d_ff, d, layer=i)
            mat(p + "ffn_up.weight", cfg.d_ff, d, layer=i)
            mat(p + "ffn_down.weight", d, cfg.d_ff, layer=i)
    return out


def _lengths(n, batch):
    """Lengths of the sequences of a batch: about `n`, ragged."""
    return [max(1, n - (i * 37) % (n // 4 + 1)) if n else 0 for i in range(batch)]


def _texts(case, seed):
    """Per sequence: the tokens of its context, and the tokens of the step."""
    gen = torch.Generator().manual_seed(seed + 1)
    ctx, new = _lengths(case["ctx"], case["batch"]), _lengths(case["rows"], case["batch"])
    vocab = SHAPES[case["model"]].vocab_size
    return [(torch.randint(0, vocab, (c,), generator=gen).tolist(), torch.randint(0, vocab, (n,), generator=gen).tolist()) for c, n in zip(ctx, new)]


# -- the calls -------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    weights = ModelWeights(_config(case), {k: QTensor(GGMLType[f], shape, raw) for k, (f, shape, raw) in _tensors(case, seed).items()})
    texts = _texts(case, seed)
    engine = LLMEngine(weights, device=DEVICE, max_batch=case["batch"], max_context=case["ctx"] + case["rows"] + 64,
                       kv_dtype=Q8 if case["kv"] == "q8_0" else None)
    state = {"engine": engine, "new": [new for _, new in texts], "held": None}
    if case["ctx"]:
        state["held"] = seqs = [engine.open_sequence() for _ in texts]
        at = 0
        while at < case["ctx"]:                                   # contexts in portions that an engine takes in one step
            n = min(case["ctx"] - at, engine.max_prefill_tokens // len(seqs))
            entries = [(r, c[at:at + n], []) for r, (c, _) in zip(seqs, texts) if c[at:at + n]]
            engine.feed(entries)
            at += n
    return state


def run(state):
    engine, held = state["engine"], state["held"]
    seqs = held or [engine.open_sequence() for _ in state["new"]]
    logits = engine.feed([(r, new, [len(new) - 1]) for r, new in zip(seqs, state["new"])])
    for r, new in zip(seqs, state["new"]):
        if held:
            r.kv.length -= len(new)
            del r.output[-len(new):]
        else:
            engine.close_sequence(r)
    return logits


# -- what is asked of them ---------------------------------------------------------------------------------------------------

def _matrices(case):
    """(bytes, multiplications per token, whether it is a routed expert's) of every matrix."""
    cfg, recipe = _config(case), RECIPES[case["recipe"]]
    d, qd, kvd = cfg.d_model, cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
    for i in range(cfg.n_layers):
        ff = cfg.expert_ff if cfg.is_moe else cfg.d_ff
        x = "_exps" if cfg.is_moe else ""
        for name, n, k in (("attn_q", qd, d), ("attn_k", kvd, d), ("attn_v", kvd, d), ("attn_output", d, qd),
                           ("ffn_gate" + x, ff, d), ("ffn_up" + x, ff, d), ("ffn_down" + x, d, ff)):
            cols, size = _BLOCK[recipe.for_tensor(f"blk.{i}.{name}.weight", i, cfg.n_layers).name]
            yield n * k // cols * size, n * k, name.endswith("_exps")


def work(case):
    cfg = _config(case)
    ctx, new = _lengths(case["ctx"], case["batch"]), _lengths(case["rows"], case["batch"])
    T, B = sum(new), case["batch"]
    cols, size = _BLOCK[RECIPES[case["recipe"]].for_tensor("output.weight").name]
    head = cfg.vocab_size * cfg.d_model
    moved, macs = head // cols * size + B * cfg.vocab_size * 4, head * B
    for nbytes, mults, routed in _matrices(case):
        if routed:                                                # experts that T tokens choose, on average
            E, k = cfg.n_experts, cfg.n_experts_used
            moved, macs = moved + nbytes * E * (1 - (1 - k / E) ** T), macs + mults * k * T
        else:
            moved, macs = moved + nbytes, macs + mults * T
    row = 2 * cfg.n_kv_heads * cfg.head_dim * (2 if case["kv"] == "bf16" else 17 / 16) * cfg.n_layers
    moved += row * sum(c + n for c, n in zip(ctx, new))           # the context is read, the new rows are written
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in zip(ctx, new))
    macs += 2 * pairs * cfg.n_heads * cfg.head_dim * cfg.n_layers
    return {"bytes": float(moved), "flops": 2.0 * macs}


def tolerance(case):
    # measured: up to 0.011 against 64 bits (bf16 operands, 8-bit activation blocks in the steps of a few rows), and up to 0.007
    # between two passes on the same inputs where partial sums meet in another order
    return {"rel": 0.03}


def exact(case, seed):
    cfg = _config(case)
    texts = _texts(case, seed)
    tokens = sum(len(c) + len(n) for c, n in texts)
    macs = sum(m * (cfg.n_experts_used if routed else 1) for _, m, routed in _matrices(case))
    if 2.0 * macs * tokens > 4e14:                                # about 20 seconds of 64-bit products
        return None
    w = {k: v for k, v in _tensors(case, seed).items()}

    def get(name):
        return _values(w[name][0], w[name][2], w[name][1])

    def norm(x, gain):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + cfg.rms_eps) * gain

    ids = torch.tensor([t for c, n in texts for t in c + n], device=DEVICE)
    cuts, pos = [0], []
    for c, n in texts:
        cuts.append(cuts[-1] + len(c) + len(n))
        pos += range(len(c) + len(n))
    fmt, shape, raw = w["token_embd.weight"]
    h = _values(fmt, raw.view(shape[0], -1)[ids].reshape(-1), (tokens, shape[1]))
    H, Hk, D = cfg.n_heads, cfg.n_kv_heads, cfg.head_dim
    turn = torch.tensor(pos, device=DEVICE).double()[:, None] * cfg.rope_theta ** (-torch.arange(0, D, 2, device=DEVICE).double() / D)
    cos, sin = turn.cos()[:, None], turn.sin()[:, None]

    def rotate(x):
        a, b = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for i in range(cfg.n_layers):
        p = f"blk.{i}."
        x = norm(h, get(p + "attn_norm.weight"))
        q, k, v = (x @ get(f"{p}attn_{n}.weight").T + (get(f"{p}attn_{n}.bias") if cfg.qkv_bias else 0.0) for n in "qkv")
        q, k, v = q.view(-1, H, D), k.view(-1, Hk, D), v.view(-1, Hk, D)
        if cfg.qk_norm:
            q, k = norm(q, get(p + "attn_q_norm.weight")), norm(k, get(p + "attn_k_norm.weight"))
        q, k = rotate(q), rotate(k)
        o = torch.empty_like(q)
        for a, b in zip(cuts, cuts[1:]):
            future = torch.ones(b - a, b - a, dtype=torch.bool, device=DEVICE).triu(1)
            for g in range(Hk):
                mine = slice(g * (H // Hk), (g + 1) * (H // Hk))
                s = q[a:b, mine].transpose(0, 1) @ k[a:b, g].T / D ** 0.5
                o[a:b, mine] = (torch.softmax(s.masked_fill_(future, -math.inf), -1) @ v[a:b, g]).transpose(0, 1)
        h = h + o.reshape(tokens, H * D) @ get(p + "attn_output.weight").T
        x = norm(h, get(p + cfg.ffn_norm_name))
        if not cfg.is_moe:
            h = h + (torch.nn.functional.silu(x @ get(p + "ffn_gate.weight").T) * (x @ get(p + "ffn_up.weight").T)) @ get(p + "ffn_down.weight").T
            continue
        share, chosen = torch.softmax(x @ get(p + "ffn_gate_inp.weight").T, -1).topk(cfg.n_experts_used, -1)
        if cfg.norm_topk_prob:
            share = share / share.sum(-1, keepdim=True)

        def expert(name, e):
            f, (_, r, c), data = w[f"{p}ffn_{name}_exps.weight"]
            return _values(f, data.view(cfg.n_experts, -1)[e], (r, c))

        for e in range(cfg.n_experts):
            rows, slot = (chosen == e).nonzero(as_tuple=True)
            if rows.numel():
                y = torch.nn.functional.silu(x[rows] @ expert("gate", e).T) * (x[rows] @ expert("up", e).T)
                h[rows] += share[rows, slot, None] * (y @ expert("down", e).T)
    last = torch.tensor(cuts[1:], device=DEVICE) - 1
    return norm(h[last], get("output_norm.weight")) @ get("output.weight").T

"""The work this framework is used for, as cases whose time can be taken: the delta projections of a decoder
layer from one token to a prompt batch, the attention and recurrent steps of the three decoders, a whole decode
pass of a small model, and the compression of a delta.

A case is a dict of plain values with a "kind"; every kind prepares seeded inputs on the GPU, runs one pass through
the package's public entry points, says which bytes and operations the pass cannot do without, and gives the same
results in 64 bits with plain torch."""
from __future__ import annotations

import math
import random
from types import SimpleNamespace

import torch

from deltazip_b200 import compress, ops
from deltazip_b200.cache import AttnMeta, PagedKVCache
from deltazip_b200.config import DeltaConfig
from deltazip_b200.layers import DeltaMapping
from deltazip_b200.llama import LlamaConfig, LlamaForCausalLM
from deltazip_b200.models import DeltaModelManager

DEV = "cuda"
TYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
#: What an output of this type is off by when only its last rounding differs, about four times.
ROUNDING = {"fp16": 1.5e-3, "bf16": 9e-3}
HEAD = 128                              # head size of every decoder here
BLOCK = 16                              # tokens of a cache block
I32, I64, F64 = torch.int32, torch.int64, torch.float64


def _gen(seed: int, *tags: int) -> torch.Generator:
    for t in tags:
        seed = (seed * 1000003 + 7919 * t + 12345) % (1 << 62)
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(gen, *shape, dtype=torch.float32, std: float = 1.0) -> torch.Tensor:
    return torch.empty(shape, dtype=dtype, device=DEV).normal_(0, std, generator=gen)


def _rng(c: dict, tag: int) -> random.Random:
    """Lengths and block tables belong to the case, so that its outputs have one shape whatever the seed."""
    return random.Random(repr(sorted((k, v) for k, v in c.items() if k != "name")) + str(tag))


def _ints(values, dtype=I32) -> torch.Tensor:
    return torch.tensor(values, dtype=dtype).to(DEV)


def _lengths(rng: random.Random, count: int, longest: int, shortest: int) -> list:
    """`count` lengths up to `longest`, one of them `longest` itself."""
    lens = [rng.randint(shortest, longest) for _ in range(count)]
    lens[rng.randrange(count)] = longest
    return lens


def _block_tables(rng: random.Random, blocks: list) -> list:
    """Cache blocks of every sequence, scattered over the pool; rows filled up with block 0."""
    pool = list(range(sum(blocks)))
    rng.shuffle(pool)
    wide, tables = max(blocks), []
    for n in blocks:
        tables.append(pool[:n] + [0] * (wide - n))
        pool = pool[n:]
    return tables


# ---------------------------------------------------------------------------
# deltas: 2:4-pruned, symmetric codes per output channel, as a compressor leaves them
# ---------------------------------------------------------------------------

def _delta(gen, n: int, k: int, bits: int):
    """(codes uint8 [k, n] with pruned entries at the zero point, scale fp16 [n]) of a normal delta."""
    g = _normal(gen, k // 4, 4, n, std=5e-3)
    size, zero = g.abs(), 1 << (bits - 1)
    parts = size.unbind(1)
    keep = torch.empty(g.shape, dtype=torch.bool, device=DEV)
    for i, a in enumerate(parts):       # kept: fewer than two of the other three are larger (the lower index wins ties)
        larger = sum((b >= a).to(torch.uint8) if j < i else (b > a).to(torch.uint8) for j, b in enumerate(parts) if j != i)
        keep[:, i] = larger < 2
    scale = (size.amax((0, 1)) * 2 / ((1 << bits) - 1)).half()
    codes = (g / scale.float()).round_().add_(zero).clamp_(0, 2 * zero - 1)
    return torch.where(keep, codes, zero).to(torch.uint8).view(k, n), scale


def _gptq(codes: torch.Tensor, scale: torch.Tensor, bits: int):
    """The tensors a checkpoint holds: qweight int32 [k * bits / 32, n], qzeros, scales."""
    per, (k, n) = 32 // bits, codes.shape
    c, word = codes.view(k // per, per, n), torch.zeros((k // per, n), dtype=I32, device=DEV)
    for j in range(per):
        word |= c[:, j].to(I32) << (bits * j)
    zeros = torch.full((1, n * bits // 32), 0x77777777 if bits == 4 else 0x55555555, dtype=I32, device=DEV)
    return word, zeros, scale.view(1, n)


def _dense(codes: torch.Tensor, scale: torch.Tensor, bits: int) -> torch.Tensor:
    """The delta [k, n] in 64 bits."""
    return (codes.to(F64) - (1 << (bits - 1))) * scale.to(F64)


# ---------------------------------------------------------------------------
# kind "linear" (one matrix) and "layer" (the four of a decoder layer): y = x W^T + x delta_slot^T
# ---------------------------------------------------------------------------

def _shapes(c: dict) -> list:
    if c["kind"] == "linear":
        return [(c["n"], c["k"])]
    h, i, kv = c["hidden"], c["inter"], c["kv"]
    return [(h + 2 * kv, h), (h, h), (2 * i, h), (h, i)]


def _popularity(c: dict) -> list:
    """Share of the tokens that the base model (first) and each delta get."""
    w = [1.0 / (i + 1) if c["spread"] == "zipf" else 1.0 for i in range(c["deltas"])]
    return [c["base"]] + [(1 - c["base"]) * v / sum(w) for v in w]


def _runs(c: dict, seed: int) -> list:
    """[(slot, tokens)]: a token each for a decode batch, a prompt each otherwise; sorted by slot (-1 first) unless
    the batch comes in any order."""
    rng, p = random.Random(seed * 31 + 5), _popularity(c)
    count = c["prompts"] or c["tokens"]
    slots = rng.choices(range(-1, c["deltas"]), p, k=count)
    if c["sorted"]:
        slots.sort()
    if not c["prompts"]:
        return [(s, 1) for s in slots]
    cuts = sorted(rng.sample(range(1, c["tokens"]), count - 1))
    return [(s, b - a) for s, a, b in zip(slots, [0] + cuts, cuts + [c["tokens"]])]


def _linear_inputs(c: dict, seed: int):
    """Per matrix its weight and activations; the rows of one matrix' input are the same for qkv and gate/up."""
    dt, xs, out = TYPES[c["dtype"]], {}, []
    for j, (n, k) in enumerate(_shapes(c)):
        tag = {2: 0}.get(j, j)
        if tag not in xs:
            xs[tag] = _normal(_gen(seed, 1, tag), c["tokens"], k, dtype=dt)
        out.append((_normal(_gen(seed, 2, j), n, k, dtype=dt, std=0.02), xs[tag]))
    return out


def _linear_prepare(c: dict, seed: int):
    s = SimpleNamespace(layers=[], by_row=not c["sorted"])
    for j, ((n, k), (w, x)) in enumerate(zip(_shapes(c), _linear_inputs(c, seed))):
        q, m, sc = ops.alloc_slots(c["deltas"], n, k, c["bits"], DEV)
        for d in range(c["deltas"]):
            ops.convert_from_gptq(*_gptq(*_delta(_gen(seed, 3, j, d), n, k, c["bits"]), c["bits"]), c["bits"],
                                  out=(q[d], m[d], sc[d]), check_status=False)
        s.layers.append((x, q, sc, m, w))
    runs = _runs(c, seed)
    s.indices = _ints([slot for slot, t in runs for _ in range(t)], I64)
    s.segments = ops.Segments(c["tokens"], c["deltas"], DEV)
    s.host_runs, at = [], 0
    for slot, t in runs:                # neighbouring rows of one slot are one run
        if s.host_runs and s.host_runs[-1][0] == slot:
            s.host_runs[-1] = (slot, s.host_runs[-1][1], at + t)
        else:
            s.host_runs.append((slot, at, at + t))
        at += t
    if c["tokens"] <= ops.FUSED_MAX_TOKENS:
        s.host_runs = None
    return s


def _linear_run(s):
    if s.by_row:                        # slot ids in any order: the call that takes them as they are
        return [ops.apply_delta(x, q, sc, m, s.indices, w) for x, q, sc, m, w in s.layers]
    seg = s.segments.build(s.indices, sorted_hint=True)
    seg.host_runs = s.host_runs
    return [ops.sbmm(x, q, sc, m, seg, w, stable=True) for x, q, sc, m, w in s.layers]


def _linear_work(c: dict) -> dict:
    p, draws = _popularity(c), c["prompts"] or c["tokens"]
    present = sum(1 - (1 - v) ** draws for v in p[1:])
    m, nbytes, flops = c["tokens"], 0.0, 0.0
    for n, k in _shapes(c):
        nbytes += 2.0 * n * k + present * ((c["bits"] / 16 + 1 / 8) * n * k + 2 * n) + 2.0 * m * (n + k)
        flops += 2.0 * m * n * k + (1 - c["base"]) * m * n * k      # half of a delta's entries are zero
    return {"bytes": nbytes, "flops": flops}


def _linear_exact(c: dict, seed: int):
    out, rows = [], {}
    at = 0
    for slot, t in _runs(c, seed):
        rows.setdefault(slot, []).extend(range(at, at + t))
        at += t
    for j, ((n, k), (w, x)) in enumerate(zip(_shapes(c), _linear_inputs(c, seed))):
        y = x.to(F64) @ w.to(F64).t()
        for d, r in rows.items():
            if d >= 0:
                r = _ints(r, I64)
                y[r] += x[r].to(F64) @ _dense(*_delta(_gen(seed, 3, j, d), n, k, c["bits"]), c["bits"])
        out.append(y)
    return out


# ---------------------------------------------------------------------------
# kind "step": a whole decode pass of a Llama with deltas, cache, output matrix
# ---------------------------------------------------------------------------

def _step_weights(c: dict, seed: int) -> dict:
    h, i, kv, dt = c["hidden"], c["inter"], c["kv_heads"] * HEAD, TYPES[c["dtype"]]
    shapes = {"model.embed_tokens.weight": (c["vocab"], h), "lm_head.weight": (c["vocab"], h), "model.norm.weight": (h,)}
    for n in range(c["layers"]):
        pre = f"model.layers.{n}."
        shapes.update({pre + "input_layernorm.weight": (h,), pre + "post_attention_layernorm.weight": (h,),
                       pre + "self_attn.q_proj.weight": (h, h), pre + "self_attn.k_proj.weight": (kv, h),
                       pre + "self_attn.v_proj.weight": (kv, h), pre + "self_attn.o_proj.weight": (h, h),
                       pre + "mlp.gate_proj.weight": (i, h), pre + "mlp.up_proj.weight": (i, h),
                       pre + "mlp.down_proj.weight": (h, i)})
    out = {}
    for t, (name, shape) in enumerate(shapes.items()):
        std = 0.1 if len(shape) == 1 else 1.0 if "embed" in name else 0.02
        out[name] = _normal(_gen(seed, 11, t), *shape, dtype=dt, std=std)
        if len(shape) == 1:
            out[name] += 1
    return out


def _step_batch(c: dict):
    """(length before this token, delta (0: base model), block table, token) of every sequence, sorted by delta."""
    rng = _rng(c, 1)
    lens = _lengths(rng, c["seqs"], c["context"], c["context"] // 2)
    ids = sorted(rng.randrange(c["deltas"] + 1) for _ in lens)
    tables = _block_tables(rng, [n // BLOCK + 1 for n in lens])
    return lens, ids, tables, [rng.randrange(c["vocab"]) for _ in lens]


def _step_cache(c: dict, seed: int, tables: list, layer: int):
    rows = (1 + max(max(t) for t in tables)) * BLOCK
    return [_normal(_gen(seed, 12, layer, side), rows, c["kv_heads"], HEAD, dtype=TYPES[c["dtype"]]) for side in range(2)]


def _step_prepare(c: dict, seed: int):
    cfg = LlamaConfig(c["hidden"], c["inter"], c["layers"], c["hidden"] // HEAD, c["kv_heads"], c["vocab"])
    s = SimpleNamespace(model=LlamaForCausalLM(cfg, device=DEV, seed=0, dtype=TYPES[c["dtype"]]))
    s.model.load_weights(_step_weights(c, seed))
    s.manager = DeltaModelManager(s.model, c["seqs"], c["seqs"], c["vocab"],
                                  DeltaConfig(max_deltas=c["deltas"], max_bitwidth=c["bits"]), device=DEV)
    for j, module in enumerate(s.manager.modules.values()):
        n, k = module.weight.shape
        for d in range(c["deltas"]):
            module.set_delta(d, c["bits"], *_gptq(*_delta(_gen(seed, 13, j, d), n, k, c["bits"]), c["bits"]))
    for d in range(c["deltas"]):
        s.manager.adopt_resident(d + 1, d)
    lens, ids, tables, tokens = _step_batch(c)
    s.manager.set_delta_mapping(DeltaMapping(ids, ids))
    s.cache = s.model.make_cache(1 + max(max(t) for t in tables), BLOCK, c["seqs"])
    for layer in range(c["layers"]):
        for pool, data in zip((s.cache.k[layer], s.cache.v[layer]), _step_cache(c, seed, tables, layer)):
            pool.copy_(data)
    s.tokens, s.positions = _ints(tokens, I64), _ints(lens, I64)
    splits = max(1, min(8, 296 // (c["seqs"] * c["kv_heads"])))
    s.meta = AttnMeta(slot_mapping=_ints([t[n // BLOCK] * BLOCK + n % BLOCK for n, t in zip(lens, tables)], I64),
                      block_tables=_ints(tables), seq_lens=_ints([n + 1 for n in lens]), splits=splits)
    return s


def _step_run(s):
    with torch.inference_mode():
        hidden = s.model(s.tokens, s.positions, s.cache, s.meta)
        return {"hidden": hidden, "logits": ops.base_gemm(hidden, s.model.lm_head)}


def _step_work(c: dict) -> dict:
    h, i, kv, m = c["hidden"], c["inter"], c["kv_heads"] * HEAD, c["seqs"]
    per = h * (h + 2 * kv) + h * h + 3 * h * i
    present = c["deltas"] * (1 - (1 - 1 / (c["deltas"] + 1)) ** m)
    keys = m * c["context"] * 0.75
    return {"bytes": c["layers"] * (per * (2 + present * (c["bits"] / 16 + 1 / 8)) + 4 * keys * kv) + 2 * c["vocab"] * (h + m),
            "flops": m * (c["layers"] * 3 * per + 2 * c["vocab"] * h) + 4 * keys * h * c["layers"]}


def _rms(x, w, eps):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt() * w


def _turned(x: torch.Tensor, positions: torch.Tensor, theta: float) -> torch.Tensor:
    """Rotary embedding of [rows, heads, 128], first half against second half."""
    half = HEAD // 2
    angle = positions.to(F64)[:, None, None] * theta ** (-torch.arange(half, dtype=F64, device=DEV) / half)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1)


def _attend(q, k, v, scale, bias=None, hidden=None):
    """q [rows, heads, d], k and v [keys, kv_heads, d]; bias and hidden [heads or 1, rows, keys]."""
    r, heads, d = q.shape
    kvh = k.shape[1]
    s = torch.einsum("rghd,kgd->ghrk", q.reshape(r, kvh, heads // kvh, d), k).reshape(heads, r, -1) * scale
    if bias is not None:
        s = s + bias
    if hidden is not None:
        s = s.masked_fill(hidden, -math.inf)
    p = s.softmax(-1).reshape(kvh, heads // kvh, r, -1)
    return torch.einsum("ghrk,kgd->rghd", p, v).reshape(r, -1)


def _step_exact(c: dict, seed: int):
    w = {name: t.to(F64) for name, t in _step_weights(c, seed).items()}
    lens, ids, tables, tokens = _step_batch(c)
    heads, kvh, eps, positions = c["hidden"] // HEAD, c["kv_heads"], 1e-5, _ints(lens, I64)

    def linear(j, x, *names):
        weight = torch.cat([w[n + "_proj.weight"] for n in names])
        y = x @ weight.t()
        for d in sorted(set(ids) - {0}):
            r = _ints([a for a, i in enumerate(ids) if i == d], I64)
            y[r] += x[r] @ _dense(*_delta(_gen(seed, 13, j, d - 1), *weight.shape, c["bits"]), c["bits"])
        return y

    x = w["model.embed_tokens.weight"][_ints(tokens, I64)]
    for n in range(c["layers"]):
        pre = f"model.layers.{n}."
        h = _rms(x, w[pre + "input_layernorm.weight"], eps)
        qkv = linear(4 * n, h, *[pre + "self_attn." + t for t in "qkv"]).view(len(lens), -1, HEAD)
        q, k = (_turned(t, positions, 1e4) for t in (qkv[:, :heads], qkv[:, heads:heads + kvh]))
        pools, att = _step_cache(c, seed, tables, n), []
        for a, t in enumerate(lens):
            at = _ints([tables[a][p // BLOCK] * BLOCK + p % BLOCK for p in range(t)], I64)
            keys, vals = (torch.cat([pool[at].to(F64), new[a:a + 1]]) for pool, new in zip(pools, (k, qkv[:, heads + kvh:])))
            att.append(_attend(q[a:a + 1], keys, vals, HEAD ** -0.5))
        x = x + linear(4 * n + 1, torch.cat(att), pre + "self_attn.o")
        h = _rms(x, w[pre + "post_attention_layernorm.weight"], eps)
        gate, up = linear(4 * n + 2, h, pre + "mlp.gate", pre + "mlp.up").chunk(2, -1)
        x = x + linear(4 * n + 3, torch.nn.functional.silu(gate) * up, pre + "mlp.down")
    h = _rms(x, w["model.norm.weight"], eps)
    return {"hidden": h, "logits": h @ w["lm_head.weight"].t()}


# ---------------------------------------------------------------------------
# kind "paged": a decode batch's rotary embedding, cache append and attention over the paged cache
# ---------------------------------------------------------------------------

def _paged_batch(c: dict):
    rng = _rng(c, 2)
    lens = _lengths(rng, c["seqs"], c["context"], max(1, c["context"] // 4))      # this token included
    return lens, _block_tables(rng, [-(-n // BLOCK) for n in lens])


def _paged_inputs(c: dict, seed: int, tables: list):
    dt, kvh = TYPES[c["dtype"]], c["kv_heads"]
    rows = (1 + max(max(t) for t in tables)) * BLOCK
    return (_normal(_gen(seed, 21), c["seqs"], (c["heads"] + 2 * kvh) * HEAD, dtype=dt),
            _normal(_gen(seed, 22), rows, kvh, HEAD, dtype=dt), _normal(_gen(seed, 23), rows, kvh, HEAD, dtype=dt))


def _slot(table: list, position: int) -> int:
    return table[position // BLOCK] * BLOCK + position % BLOCK


def _paged_prepare(c: dict, seed: int):
    lens, tables = _paged_batch(c)
    s = SimpleNamespace(heads=c["heads"], kvh=c["kv_heads"])
    s.qkv, s.k, s.v = _paged_inputs(c, seed, tables)
    s.positions, s.lens, s.tables = _ints([n - 1 for n in lens], I64), _ints(lens), _ints(tables)
    s.slots = _ints([_slot(t, n - 1) for n, t in zip(lens, tables)], I64)
    s.splits = max(1, min(8, 296 // (c["seqs"] * c["kv_heads"])))        # as the decode engine chooses them
    return s


def _paged_run(s):
    ops.rotary_and_cache(s.qkv, s.positions, s.heads, s.kvh, 1e4, s.k, s.v, s.slots)
    out = ops.paged_attention_decode(s.qkv, s.k, s.v, s.tables, s.lens, s.heads, s.kvh, BLOCK, HEAD ** -0.5, s.splits)
    return {"out": out, "qkv": s.qkv, "k": s.k, "v": s.v}


def _paged_work(c: dict) -> dict:
    keys = c["seqs"] * (c["context"] + max(1, c["context"] // 4)) / 2
    return {"bytes": 4 * HEAD * (keys * c["kv_heads"] + c["seqs"] * (c["heads"] + c["kv_heads"])) + 2 * HEAD * c["seqs"] * c["heads"],
            "flops": 4 * HEAD * keys * c["heads"]}


def _paged_exact(c: dict, seed: int):
    lens, tables = _paged_batch(c)
    qkv, k, v = (t.to(F64) for t in _paged_inputs(c, seed, tables))
    heads, kvh = c["heads"], c["kv_heads"]
    qkv = qkv.view(len(lens), -1, HEAD)
    qkv[:, :heads + kvh] = _turned(qkv[:, :heads + kvh], _ints([n - 1 for n in lens], I64), 1e4)
    slots = _ints([_slot(t, n - 1) for n, t in zip(lens, tables)], I64)
    k[slots], v[slots] = qkv[:, heads:heads + kvh], qkv[:, heads + kvh:]
    out = []
    for a, n in enumerate(lens):
        at = _ints([_slot(tables[a], p) for p in range(n)], I64)
        out.append(_attend(qkv[a:a + 1, :heads], k[at], v[at], HEAD ** -0.5))
    return {"out": torch.cat(out), "qkv": qkv.reshape(len(lens), -1), "k": k, "v": v}


# ---------------------------------------------------------------------------
# kind "window": query/key norm, sliding-window attention with a distance bias, cache append -- prompt portions, or one
# token per sequence
# ---------------------------------------------------------------------------

def _window_batch(c: dict):
    rng = _rng(c, 3)
    if c["decode"]:
        lens = [1] * c["seqs"]
        ctx = _lengths(rng, c["seqs"], c["context"], c["context"] // 2)
    else:
        lens = _lengths(rng, c["seqs"], c["prompt"], max(1, c["prompt"] // 2))
        ctx = [rng.randint(0, c["context"]) for _ in lens]
    ring = -(-c["window"] // BLOCK)
    return lens, ctx, _block_tables(rng, [ring] * c["seqs"])


def _ring_slot(table: list, position: int) -> int:
    return table[position // BLOCK % len(table)] * BLOCK + position % BLOCK


def _window_inputs(c: dict, seed: int, rows: int):
    dt, h, kvh = TYPES[c["dtype"]], c["heads"], c["kv_heads"]
    pool = c["seqs"] * -(-c["window"] // BLOCK) * BLOCK
    return SimpleNamespace(qkv=_normal(_gen(seed, 31), rows, (h + 2 * kvh) * HEAD, dtype=dt),
                           k=_normal(_gen(seed, 32), pool, kvh, HEAD, dtype=dt), v=_normal(_gen(seed, 33), pool, kvh, HEAD, dtype=dt),
                           wq=1 + _normal(_gen(seed, 34), h * HEAD, std=0.1), wk=1 + _normal(_gen(seed, 35), kvh * HEAD, std=0.1),
                           bias=_normal(_gen(seed, 36), h, min(c["window"], 513)))


def _kept(lens, ctx, tables):
    """Slots of the rows the rings keep, -1 for those that leave them again at once."""
    return [_ring_slot(t, p) if p >= c + n - len(t) * BLOCK else -1 for n, c, t in zip(lens, ctx, tables) for p in range(c, c + n)]


def _window_prepare(c: dict, seed: int):
    lens, ctx, tables = _window_batch(c)
    s = _window_inputs(c, seed, sum(lens))
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    s.starts, s.ctx, s.tables, s.slots = _ints(starts), _ints(ctx), _ints(tables), _ints(_kept(lens, ctx, tables), I64)
    s.most, s.c = max(lens), c
    return s


def _window_run(s):
    c = s.c
    kw = dict(k_cache=s.k, v_cache=s.v, slot_mapping=s.slots) if c["decode"] else {}
    ops.qk_norm(s.qkv, s.wq, s.wk, c["kv_heads"] * HEAD, 1e-6, **kw)
    out = ops.window_attention(s.qkv, s.k, s.v, s.tables, s.starts, s.ctx, s.most, c["decode"], c["heads"], BLOCK,
                               HEAD ** -0.5, c["window"], s.bias)
    if not c["decode"]:
        ops.kv_append(s.qkv, c["heads"] * HEAD, s.k, s.v, s.slots)
    return {"out": out, "qkv": s.qkv, "k": s.k, "v": s.v}


def _window_work(c: dict) -> dict:
    """With sequences of the mean length."""
    n = 1 if c["decode"] else 0.75 * c["prompt"]
    ctx = c["context"] * (0.75 if c["decode"] else 0.5)
    old, w = min(ctx, c["window"]), c["window"]
    full = min(n, max(0.0, w - ctx))                    # rows that see everything before them
    pairs = full * (ctx + (full + 1) / 2) + (n - full) * w
    rows, kvh = c["seqs"] * n, c["kv_heads"]
    return {"bytes": 2 * HEAD * (rows * (2 * (c["heads"] + kvh) + kvh + c["heads"]) + 2 * kvh * c["seqs"] * (old + min(n, w))),
            "flops": 4 * HEAD * c["heads"] * c["seqs"] * pairs}


def _window_exact(c: dict, seed: int):
    lens, ctx, tables = _window_batch(c)
    s = _window_inputs(c, seed, sum(lens))
    h, kvh, w = c["heads"], c["kv_heads"], c["window"]
    qkv, old = s.qkv.to(F64), [s.k.to(F64), s.v.to(F64)]
    q, k, v = qkv.split([h * HEAD, kvh * HEAD, kvh * HEAD], 1)
    q, k = _rms(q, s.wq.to(F64), 1e-6), _rms(k, s.wk.to(F64), 1e-6)
    out, at = [], 0
    for a, n in enumerate(lens):
        first = max(0, ctx[a] + 1 - w)                  # what the ring still holds for the first row
        held = _ints([_ring_slot(tables[a], p) for p in range(first, ctx[a])], I64)
        keys, vals = (torch.cat([o[held], t[at:at + n].view(n, kvh, HEAD)]) for o, t in zip(old, (k, v)))
        rows = torch.arange(ctx[a], ctx[a] + n, device=DEV)
        far = rows[:, None] - torch.arange(first, ctx[a] + n, device=DEV)[None]
        hidden, near = (far < 0) | (far >= w), far.clamp(0, s.bias.shape[1] - 1)
        part = []
        for g in range(kvh):                            # a head group at a time: scores take rows x keys x 8 bytes
            hs = slice(g * (h // kvh), (g + 1) * (h // kvh))
            part.append(_attend(q[at:at + n].view(n, h, HEAD)[:, hs], keys[:, g:g + 1], vals[:, g:g + 1], HEAD ** -0.5,
                                s.bias[hs].to(F64)[:, near], hidden))
        out.append(torch.cat(part, 1))
        at += n
    slots = _ints(_kept(lens, ctx, tables), I64)
    keep = slots >= 0
    for o, t in zip(old, (k, v)):
        o[slots[keep]] = t.reshape(-1, kvh, HEAD)[keep]
    return {"out": torch.cat(out), "qkv": torch.cat([q, k, v], 1), "k": old[0], "v": old[1]}


# ---------------------------------------------------------------------------
# kinds "mlstm" and "lightning": the recurrent layers, over prompts or one token per sequence
# ---------------------------------------------------------------------------

def _rec_batch(c: dict):
    rng = _rng(c, 4)
    lens = [1] * c["seqs"] if c["decode"] else _lengths(rng, c["seqs"], c["prompt"], max(5, c["prompt"] // 2))
    ctx = [rng.randint(1, 2048) if c["decode"] or c["continued"] else 0 for _ in lens]
    return lens, ctx, rng.sample(range(c["seqs"] + 3), c["seqs"])


def _rec_inputs(c: dict, seed: int, rows: int):
    dt, h, pool = TYPES[c["dtype"]], c["heads"], c["seqs"] + 3
    s = SimpleNamespace(x=_normal(_gen(seed, 41), rows, 4 * h * HEAD, dtype=dt), norm=1 + _normal(_gen(seed, 42), h * HEAD, std=0.1),
                        S=_normal(_gen(seed, 43), pool, h, HEAD, HEAD))
    if c["kind"] == "mlstm":
        width = h * HEAD
        s.h = _normal(_gen(seed, 44), rows, width, dtype=dt)
        s.w_if = _normal(_gen(seed, 45), 2 * h, width, dtype=dt, std=width ** -0.5)
        s.b_if = torch.cat([_normal(_gen(seed, 46), h), 4 + _normal(_gen(seed, 47), h)])       # forget gates start open
        s.n, s.m = _normal(_gen(seed, 48), pool, h, HEAD), _normal(_gen(seed, 49), pool, h)
    else:
        decay = torch.tensor([1 - 2.0 ** (-1 - 7 * i / h) for i in range(h)], dtype=F64)
        s.decay = decay.to(DEV)
        s.powers = (decay[:, None] ** torch.arange(ops.LIGHTNING_POWERS, dtype=F64)).float().to(DEV)
    return s


def _rec_prepare(c: dict, seed: int):
    lens, ctx, slots = _rec_batch(c)
    s = _rec_inputs(c, seed, sum(lens))
    s.starts, s.ctx, s.slots, s.c = _ints([sum(lens[:i]) for i in range(len(lens) + 1)]), _ints(ctx), _ints(slots), c
    return s


def _mlstm_run(s):
    out = ops.mlstm(s.x, s.h, s.w_if, s.b_if, s.norm, s.S, s.n, s.m, s.slots, s.starts, s.ctx, 15.0, HEAD ** -0.5, 1e-6,
                    not s.c["decode"])
    return {"out": out, "S": s.S, "n": s.n, "m": s.m}


def _lightning_run(s):
    out = ops.lightning(s.x, s.powers, s.norm, s.S, s.slots, s.starts, s.ctx, 1e-6, not s.c["decode"])
    return {"out": out, "S": s.S}


def _rec_work(c: dict) -> dict:
    rows, h = c["seqs"] * (1 if c["decode"] else 0.75 * c["prompt"]), c["heads"]
    read = 2 if c["decode"] or c["continued"] else 1
    nbytes = 2 * rows * 5 * h * HEAD + 4 * read * c["seqs"] * h * HEAD * (HEAD + 1)
    if c["kind"] == "mlstm":
        nbytes += 2 * rows * h * HEAD + 4 * h * h * HEAD
    per = 6 * HEAD * HEAD if c["decode"] else 2 * 33 * 2 * HEAD + 4 * HEAD * HEAD     # prompts: 64 tokens at a time
    return {"bytes": nbytes, "flops": rows * h * per}


def _mlstm_exact(c: dict, seed: int):
    lens, ctx, slots = _rec_batch(c)
    s = _rec_inputs(c, seed, sum(lens))
    heads, out, at = c["heads"], [], 0
    S, n, m = s.S.to(F64), s.n.to(F64), s.m.to(F64)
    for a, t in enumerate(lens):
        rows = slice(at, at + t)
        q, k, v, g = s.x[rows].to(F64).view(t, 4, heads, HEAD).permute(1, 2, 0, 3)       # [heads, t, 128]
        q = q * HEAD ** -0.5
        pre = 15 * torch.tanh((s.h[rows].to(F64) @ s.w_if.to(F64).t() + s.b_if.to(F64)) / 15)
        i, f = pre[:, :heads].t(), torch.nn.functional.logsigmoid(pre[:, heads:]).t()    # [heads, t]
        j = slots[a]
        if ctx[a] == 0:
            S[j], n[j], m[j] = 0, 0, 0
        F = f.cumsum(1)
        top = torch.maximum(m[j][:, None], (i - F).cummax(1).values)                      # running maximum less F
        old = (m[j][:, None] - top).exp()
        later = torch.ones((t, t), dtype=torch.bool, device=DEV).triu(1)
        o = torch.empty((heads, t, HEAD), dtype=F64, device=DEV)
        for b in range(heads):
            w = ((i - F)[b][None] - top[b][:, None]).masked_fill(later, -math.inf).exp() * (q[b] @ k[b].t())
            num = w @ v[b] + old[b][:, None] * (q[b] @ S[j][b])
            den = w.sum(1) + old[b] * (q[b] @ n[j][b])
            o[b] = num / (torch.maximum(den.abs(), (-F[b] - top[b]).exp())[:, None] + 1e-6)
        last = (i - F - top[:, -1:]).exp()
        S[j] = torch.einsum("ht,htd,htv->hdv", last, k, v) + old[:, -1, None, None] * S[j]
        n[j] = torch.einsum("ht,htd->hd", last, k) + old[:, -1, None] * n[j]
        m[j] = F[:, -1] + top[:, -1]
        o = o / (o.square().mean(-1, keepdim=True) + 1e-6).sqrt()
        out.append((o * torch.sigmoid(g)).transpose(0, 1).reshape(t, -1) * s.norm.to(F64))
        at += t
    return {"out": torch.cat(out), "S": S, "n": n, "m": m}


def _lightning_exact(c: dict, seed: int):
    lens, ctx, slots = _rec_batch(c)
    s = _rec_inputs(c, seed, sum(lens))
    heads, out, at, S = c["heads"], [], 0, s.S.to(F64)
    for a, t in enumerate(lens):
        x = s.x[at:at + t].to(F64).view(t, 4, heads, HEAD).permute(1, 2, 0, 3)
        (q, k, v), g = torch.nn.functional.silu(x[:3]), x[3]
        j = slots[a]
        if ctx[a] == 0:
            S[j] = 0
        pos = torch.arange(t, device=DEV)
        far = (pos[:, None] - pos[None]).to(F64)
        o = torch.empty((heads, t, HEAD), dtype=F64, device=DEV)
        for b in range(heads):
            w = torch.where(far >= 0, s.decay[b] ** far.clamp(min=0), 0.0) * (q[b] @ k[b].t())
            o[b] = w @ v[b] + s.decay[b] ** (pos + 1)[:, None] * (q[b] @ S[j][b])
            S[j, b] = (k[b] * s.decay[b] ** (t - 1 - pos)[:, None]).t() @ v[b] + s.decay[b] ** t * S[j, b]
        o = o.transpose(0, 1).reshape(t, -1)
        out.append(_rms(o, s.norm.to(F64), 1e-6) * torch.sigmoid(g.transpose(0, 1).reshape(t, -1)))
        at += t
    return {"out": torch.cat(out), "S": S}


# ---------------------------------------------------------------------------
# kind "latent": decode attention over cached latents with a sink per head
# ---------------------------------------------------------------------------

def _latent_inputs(c: dict, seed: int):
    rng = _rng(c, 5)
    ctx = _lengths(rng, c["seqs"], c["context"], c["context"] // 2)
    tables = _block_tables(rng, [n // BLOCK + 1 for n in ctx])
    dt, row = TYPES[c["dtype"]], c["rank"] + c["rot"]
    return ctx, tables, SimpleNamespace(
        q=_normal(_gen(seed, 51), c["seqs"], c["heads"], row, dtype=dt),
        cache=_normal(_gen(seed, 52), (1 + max(max(t) for t in tables)) * BLOCK, 1, row, dtype=dt), sink=_normal(_gen(seed, 53), c["heads"]))


def _latent_prepare(c: dict, seed: int):
    ctx, tables, s = _latent_inputs(c, seed)
    s.ctx, s.tables, s.starts, s.c = _ints(ctx), _ints(tables), _ints(list(range(len(ctx) + 1))), c
    return s


def _latent_run(s):
    return ops.latent_attention(s.q, s.cache, s.tables, s.starts, s.ctx, s.c["rank"], BLOCK, (HEAD + s.c["rot"]) ** -0.5, s.sink)


def _latent_work(c: dict) -> dict:
    keys, row = c["seqs"] * 0.75 * c["context"], c["rank"] + c["rot"]
    return {"bytes": 2 * keys * row + 2 * c["seqs"] * c["heads"] * (row + c["rank"]), "flops": 2 * keys * c["heads"] * (row + c["rank"])}


def _latent_exact(c: dict, seed: int):
    ctx, tables, s = _latent_inputs(c, seed)
    out, sink = [], s.sink.to(F64)
    for a, n in enumerate(ctx):
        rows = s.cache[_ints([_slot(tables[a], p) for p in range(n + 1)], I64), 0].to(F64)
        e = s.q[a].to(F64) @ rows.t() * (HEAD + c["rot"]) ** -0.5
        p = torch.cat([e, sink[:, None]], 1).softmax(1)[:, :-1]
        out.append(p @ rows[:, :c["rank"]])
    return torch.stack(out)


# ---------------------------------------------------------------------------
# kind "compress": a dense delta and its layer's calibration Hessian to the tensors of a checkpoint
# ---------------------------------------------------------------------------

def _compress_inputs(c: dict, seed: int):
    k = c["k"]
    mix = _normal(_gen(seed, 61), k, k, std=0.3 * k ** -0.5)
    x = _normal(_gen(seed, 62), 2 * k, k)
    x = x + x @ mix                     # correlated inputs
    return SimpleNamespace(delta=_normal(_gen(seed, 63), c["n"], k, std=5e-3), H=x.t() @ x * (2 / x.shape[0]), bits=c["bits"])


def _compress_run(s):
    return dict(zip(("qweight", "qzeros", "scales", "loss"), compress.compress_delta(s.delta, s.bits, s.H)))


def _compress_work(c: dict) -> dict:
    n, k = c["n"], c["k"]               # two factorisations and an inverse of H, and the error's way through the columns
    return {"bytes": 4.0 * n * k + 4.0 * k * k + n * k * c["bits"] / 8, "flops": 4 / 3 * k ** 3 + 1.0 * n * k * k}


def _compress_exact(c: dict, seed: int):
    """The loss; codes are whole numbers whose ties another order of sums may turn."""
    s = _compress_inputs(c, seed)
    n, k, bits = c["n"], c["k"], c["bits"]
    W, H, zero = s.delta.to(F64), s.H.to(F64), 1 << (bits - 1)
    scale = W.abs().amax(1, keepdim=True) * 2 / ((1 << bits) - 1)
    H.diagonal().add_(0.01 * H.diagonal().mean())
    U = torch.linalg.cholesky(torch.cholesky_inverse(torch.linalg.cholesky(H)), upper=True)
    loss = torch.zeros(n, dtype=F64, device=DEV)
    for a in range(0, k, 128):
        b = min(a + 128, k)
        E = torch.empty((n, b - a), dtype=F64, device=DEV)
        for i in range(a, b):
            if i % 4 == 0:
                drop = (W[:, i:i + 4].square() / U.diagonal()[i:i + 4].square()).topk(2, 1, largest=False).indices
                gone = torch.zeros((n, 4), dtype=torch.bool, device=DEV).scatter_(1, drop, True)
            w = W[:, i].clone()
            q = ((w.masked_fill(gone[:, i % 4], 0)[:, None] / scale).round() + zero).clamp(0, 2 * zero - 1)
            q = (scale * (q - zero))[:, 0]
            E[:, i - a] = (w - q) / U[i, i]
            loss += E[:, i - a].square() / 2
            W[:, i:b] -= E[:, i - a, None] * U[i, i:b]
        W[:, b:] -= E @ U[a:b, b:]
    return {"qweight": None, "qzeros": None, "scales": scale.view(1, n), "loss": loss}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

KINDS = {
    "linear": (_linear_prepare, _linear_run, _linear_work, _linear_exact),
    "layer": (_linear_prepare, _linear_run, _linear_work, _linear_exact),
    "step": (_step_prepare, _step_run, _step_work, _step_exact),
    "paged": (_paged_prepare, _paged_run, _paged_work, _paged_exact),
    "window": (_window_prepare, _window_run, _window_work, _window_exact),
    "mlstm": (_rec_prepare, _mlstm_run, _rec_work, _mlstm_exact),
    "lightning": (_rec_prepare, _lightning_run, _rec_work, _lightning_exact),
    "latent": (_latent_prepare, _latent_run, _latent_work, _latent_exact),
    "compress": (_compress_inputs, _compress_run, _compress_work, _compress_exact),
}


def _layer(**kw) -> dict:
    return {"kind": "layer", "hidden": 4096, "inter": 11008, "kv": 4096, "dtype": "fp16", "bits": 4, "spread": "even",
            "base": 0.0, "prompts": 0, "sorted": True, **kw}


def listed() -> list:
    return [
        # one request alone in the server: a single matrix, slot ids as the caller has them
        {"name": "one_token", "kind": "linear", "n": 4096, "k": 4096, "tokens": 1, "deltas": 8, "dtype": "fp16", "bits": 4,
         "spread": "even", "base": 0.0, "prompts": 0, "sorted": False},
        # a decode batch over a handful of fine-tuned 7B models, one decoder layer
        _layer(name="layer_7b_decode", tokens=64, deltas=8),
        # many users of many models: nearly every delta has only a few tokens of the batch
        _layer(name="layer_7b_many_2bit", tokens=128, deltas=31, bits=2, base=0.03),
        # a full server of a 13B model, a few deltas popular and a long tail
        _layer(name="layer_13b_zipf", hidden=5120, inter=13824, kv=5120, tokens=250, deltas=64, dtype="bf16", spread="zipf", base=0.05),
        # new requests of several models enter together: their prompts in one pass
        _layer(name="layer_7b_prompts", tokens=1999, deltas=8, prompts=7, base=0.1),
        # a small model under light load, where launches count: the whole decode pass
        {"name": "step_small", "kind": "step", "hidden": 2048, "inter": 5632, "layers": 4, "kv_heads": 16, "vocab": 32000,
         "seqs": 5, "context": 301, "deltas": 3, "bits": 4, "dtype": "fp16"},
        # decode attention of a 70B model: eight query heads share a key
        {"name": "paged_gqa", "kind": "paged", "seqs": 64, "heads": 64, "kv_heads": 8, "context": 1501, "dtype": "fp16"},
        # prompts through windowed attention
        {"name": "window_prompts", "kind": "window", "decode": False, "seqs": 4, "prompt": 2048, "context": 0, "window": 1024,
         "heads": 32, "kv_heads": 32, "dtype": "bf16"},
        # prompts through the matrix memory
        {"name": "mlstm_prompts", "kind": "mlstm", "decode": False, "continued": False, "seqs": 4, "prompt": 2048, "heads": 32,
         "dtype": "bf16"},
        # later portions of prompts through linear attention
        {"name": "lightning_prompts", "kind": "lightning", "decode": False, "continued": True, "seqs": 5, "prompt": 1500, "heads": 16,
         "dtype": "bf16"},
        # decode attention over latents, all heads on one row per token
        {"name": "latent_decode", "kind": "latent", "seqs": 64, "heads": 32, "rank": 512, "rot": 64, "context": 2047, "dtype": "bf16"},
        # offline: one projection of a fine-tuned 7B model
        {"name": "compress_7b", "kind": "compress", "n": 4096, "k": 4096, "bits": 4},
    ]


def _between(rng: random.Random, low: float, high: float) -> int:
    return round(math.exp(rng.uniform(math.log(low), math.log(high))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["linear", "layer", "layer", "layer", "step", "paged", "window", "mlstm", "lightning", "latent", "compress"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind in ("linear", "layer"):
        prompt = kind == "layer" and rng.random() < 0.3
        c = {"kind": kind, "tokens": _between(rng, 513, 3000) if prompt else _between(rng, 1, 320), "dtype": dtype,
             "deltas": _between(rng, 1, 16 if prompt else 64), "bits": rng.choice([2, 4]), "spread": rng.choice(["even", "zipf"]),
             "base": rng.choice([0.0, 0.1, 0.3]), "prompts": _between(rng, 1, 24) if prompt else 0,
             "sorted": prompt or rng.random() < 0.7}
        if kind == "linear":
            return {**c, "n": 128 * _between(rng, 8, 172), "k": 64 * _between(rng, 16, 216)}
        hidden = 256 * _between(rng, 4, 20)
        return {**c, "hidden": hidden, "inter": 64 * round(hidden * rng.uniform(2.5, 3.5) / 64), "kv": rng.choice([hidden, hidden // 4])}
    if kind == "step":
        heads = 4 * rng.randint(2, 6)
        return {"kind": kind, "hidden": heads * HEAD, "inter": 64 * round(heads * HEAD * rng.uniform(2.5, 3.5) / 64),
                "layers": rng.randint(1, 4), "kv_heads": heads // rng.choice([1, 4]), "vocab": 128 * rng.randint(60, 260),
                "seqs": _between(rng, 1, 48), "context": _between(rng, 16, 1000), "deltas": rng.randint(1, 8),
                "bits": rng.choice([2, 4]), "dtype": dtype}
    if kind == "paged":
        kvh, ratio = rng.choice([1, 2, 4, 8, 16]), rng.choice([1, 2, 4, 8])
        return {"kind": kind, "seqs": _between(rng, 1, 160), "heads": kvh * ratio, "kv_heads": kvh, "context": _between(rng, 20, 4000),
                "dtype": dtype}
    if kind == "window":
        kvh, ratio, decode = rng.choice([4, 8, 16]), rng.choice([1, 1, 2, 4]), rng.random() < 0.4
        return {"kind": kind, "decode": decode, "seqs": _between(rng, 1, 96) if decode else rng.randint(1, 5),
                "prompt": 1 if decode else _between(rng, 65, 2048), "context": _between(rng, 40, 6000) if decode else rng.choice([0, 1500]),
                "window": rng.choice([512, 1000, 1024, 4096]), "heads": kvh * ratio, "kv_heads": kvh, "dtype": dtype}
    if kind in ("mlstm", "lightning"):
        decode = rng.random() < 0.4
        return {"kind": kind, "decode": decode, "continued": rng.random() < 0.5, "seqs": _between(rng, 1, 96) if decode else rng.randint(1, 6),
                "prompt": 1 if decode else _between(rng, 65, 2048), "heads": rng.choice([8, 16, 32]), "dtype": dtype}
    if kind == "latent":
        return {"kind": kind, "seqs": _between(rng, 1, 96), "heads": rng.choice([16, 32]), "rank": rng.choice([256, 512]), "rot": 64,
                "context": _between(rng, 40, 4000), "dtype": dtype}
    return {"kind": kind, "n": 128 * _between(rng, 4, 32), "k": 128 * _between(rng, 8, 32), "bits": rng.choice([2, 4])}


def prepare(case: dict, seed: int):
    state = KINDS[case["kind"]][0](case, seed)
    state.kind = case["kind"]
    return state


def run(state):
    return KINDS[state.kind][1](state)


def work(case: dict) -> dict:
    return KINDS[case["kind"]][2](case)


def tolerance(case: dict):
    if case["kind"] == "compress":
        return {"rel": 2e-3, "differ": 1e-2}
    # several layers round the hidden state one after the other
    return {"rel": min(3e-2, ROUNDING[case["dtype"]] * (4 if case["kind"] == "step" else 1))}


def exact(case: dict, seed: int):
    return KINDS[case["kind"]][3](case, seed)

"""Decode attention with several query heads per key/value head (warp MMAs) against softmax attention in 64 bits:
lengths around its 16-key tiles, four warps and splits, group sizes that fill the eight MMA rows or not, windows,
distance bias and sinks.

Tolerance: scores, sums and weights (three 16-bit parts) are 32-bit, so what is left is the output's
rounding, at most half a unit in the last place: 2^-11 (fp16) or 2^-8 (bf16) of every element; twice that for the
relative 2-norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BLOCK = 16
TOL = {torch.float16: 2 * 2.0 ** -11, torch.bfloat16: 2 * 2.0 ** -8}
LENS = [1, 15, 16, 17, 63, 64, 65, 130, 257, 700]


def batch(kvh, heads, dtype, seed, blocks_per_seq, lens):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(dtype)
    n = len(lens)
    tables = torch.randperm(n * blocks_per_seq, generator=g, device="cuda").to(torch.int32).view(n, blocks_per_seq)
    rows = n * blocks_per_seq * BLOCK
    return rnd(n, (heads + 2 * kvh) * 128), 2 * rnd(rows, kvh, 128), rnd(rows, kvh, 128), tables.contiguous()


def reference(q, k, v, scale, bias=None, sink=None):
    """q [heads, 128], k and v [keys, kv_heads, 128], bias [heads, keys], sink [heads]; 64 bits."""
    rep = q.shape[0] // k.shape[1]
    k, v = (t.double().repeat_interleave(rep, 1) for t in (k, v))
    s = torch.einsum("hd,khd->hk", q.double(), k) * scale
    if bias is not None:
        s = s + bias.double()
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None]], 1)
    p = s.softmax(1)[:, :k.shape[0]]
    return torch.einsum("hk,khd->hd", p, v).reshape(-1)


def check(out, want, dtype):
    assert torch.isfinite(out).all()
    err = (out.double() - want).norm() / want.norm()
    assert err <= TOL[dtype], float(err)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("heads,kvh", [(4, 1), (8, 1), (12, 3), (32, 4)])
@pytest.mark.parametrize("splits", [1, 3, 33])
def test_paged(heads, kvh, splits, dtype):
    from deltazip_b200 import ops
    qkv, k, v, tables = batch(kvh, heads, dtype, heads + splits, -(-max(LENS) // BLOCK), LENS)
    lens = torch.tensor(LENS, dtype=torch.int32, device="cuda")
    for rep in range(2):                           # twice: the tickets are back at zero
        out = ops.paged_attention_decode(qkv, k, v, tables, lens, heads, kvh, BLOCK, 128 ** -0.5, splits)
        for i, n in enumerate(LENS):
            at = (tables[i].long()[:, None] * BLOCK + torch.arange(BLOCK, device="cuda")).flatten()[:n]
            check(out[i], reference(qkv[i, :heads * 128].view(heads, 128), k[at], v[at], 128 ** -0.5), dtype)


def test_paged_without_keys():
    from deltazip_b200 import ops
    qkv, k, v, tables = batch(1, 8, torch.float16, 1, 2, [0, 5])
    out = ops.paged_attention_decode(qkv, k, v, tables, torch.tensor([0, 5], dtype=torch.int32, device="cuda"), 8, 1, BLOCK, 0.1)
    assert not out[0].any() and out[1].any()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("heads,kvh", [(3, 1), (10, 2), (8, 1), (20, 2)])
@pytest.mark.parametrize("window,splits,extra", [(300, 0, True), (300, 5, False), (33, 2, True), (5000, 0, True), (0, 3, False)])
def test_window(heads, kvh, window, splits, extra, dtype):
    from deltazip_b200 import ops
    most = max(LENS) if window == 0 else min(window, max(LENS))
    ring = -(-most // BLOCK)
    qkv, k, v, tables = batch(kvh, heads, dtype, heads + window, ring, LENS)
    g = torch.Generator(device="cuda").manual_seed(7)
    bias = torch.randn((heads, 40), generator=g, device="cuda") * 2 if extra else None
    sink = torch.randn(heads, generator=g, device="cuda") if extra else None
    starts = torch.arange(len(LENS) + 1, dtype=torch.int32, device="cuda")
    ctx = torch.tensor([n - 1 for n in LENS], dtype=torch.int32, device="cuda")
    for rep in range(2):
        out = ops.window_attention(qkv, k, v, tables, starts, ctx, 1, True, heads, BLOCK, 0.11, window, bias, splits, sink)
        for i, n in enumerate(LENS):
            pos = torch.arange(max(0, n - window) if window else 0, n, device="cuda")
            at = tables[i].long()[pos // BLOCK % ring] * BLOCK + pos % BLOCK
            b = bias[:, (n - 1 - pos).clamp(max=39)] if extra else None
            check(out[i], reference(qkv[i, :heads * 128].view(heads, 128), k[at], v[at], 0.11, b, sink), dtype)


@pytest.mark.parametrize("mask", [float("-inf"), torch.finfo(torch.float32).min, -1e9, -1e6, -1e4])
@pytest.mark.parametrize("splits", [1, 4])
def test_bias_that_masks_far_keys(mask, splits):
    """The last bias of the table, which all farther keys share, hides them: near keys keep their scores."""
    from deltazip_b200 import ops
    heads, kvh, dtype, length = 8, 1, torch.float16, 40
    qkv, k, v, tables = batch(kvh, heads, dtype, 3, -(-max(LENS) // BLOCK), LENS)
    bias = torch.randn((heads, length), generator=torch.Generator("cuda").manual_seed(4), device="cuda")
    bias[:, 21:] = mask                            # hidden beyond distance 20, the shared entry among them
    starts = torch.arange(len(LENS) + 1, dtype=torch.int32, device="cuda")
    ctx = torch.tensor([n - 1 for n in LENS], dtype=torch.int32, device="cuda")
    out = ops.window_attention(qkv, k, v, tables, starts, ctx, 1, True, heads, BLOCK, 0.3, 0, bias, splits, None)
    for i, n in enumerate(LENS):
        pos = torch.arange(n, device="cuda")
        at = tables[i].long()[pos // BLOCK] * BLOCK + pos % BLOCK
        b = bias[:, (n - 1 - pos).clamp(max=length - 1)]
        check(out[i], reference(qkv[i, :heads * 128].view(heads, 128), k[at], v[at], 0.3, b), dtype)


@pytest.mark.parametrize("splits", [1, 3])
def test_every_key_masked_by_the_lowest_value(splits):
    """Finite masks over all keys leave equal weights: the mean of the values."""
    from deltazip_b200 import ops
    heads, kvh, dtype = 8, 1, torch.float16
    qkv, k, v, tables = batch(kvh, heads, dtype, 3, -(-max(LENS) // BLOCK), LENS)
    bias = torch.full((heads, 40), torch.finfo(torch.float32).min, device="cuda")
    starts = torch.arange(len(LENS) + 1, dtype=torch.int32, device="cuda")
    ctx = torch.tensor([n - 1 for n in LENS], dtype=torch.int32, device="cuda")
    out = ops.window_attention(qkv, k, v, tables, starts, ctx, 1, True, heads, BLOCK, 0.3, 0, bias, splits, None)
    for i, n in enumerate(LENS):
        pos = torch.arange(n, device="cuda")
        at = tables[i].long()[pos // BLOCK] * BLOCK + pos % BLOCK
        check(out[i].view(heads, 128), v[at, 0].double().mean(0).expand(heads, 128), dtype)


def test_weights_keep_32_bits():
    """bf16, four keys a sequence whose products with the weights cancel down to 2^-16 of themselves, so that the output's
    own rounding is out of the way.  Error allowed against the sum of absolute products: 2^-19.5, from two units of the
    exponential and three 32-bit sums (2^-21); a weight of two 16-bit parts is off by up to 2^-18."""
    from deltazip_b200 import ops
    n, heads, dtype = 64, 8, torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(6)
    q = torch.randn((n, 1, 128), generator=g, device="cuda").to(dtype)
    k = torch.randn((n * BLOCK, 1, 128), generator=g, device="cuda").to(dtype)
    v = (1 + torch.rand((n, BLOCK, 128), generator=g, device="cuda")).to(dtype)
    w = torch.einsum("nd,nkd->nk", q[:, 0].double(), k.view(n, BLOCK, 128)[:, :4].double()).mul(128 ** -0.5).softmax(1)
    for key in (2, 3):                             # each takes away what the keys before it leave
        v[:, key] = (-(w[:, :key, None] * v[:, :key].double()).sum(1) / w[:, key, None]).to(dtype)
    qkv = torch.cat([q.expand(n, heads, 128).reshape(n, -1), torch.zeros((n, 256), device="cuda", dtype=dtype)], 1).contiguous()
    tables, lens = (t.int().cuda() for t in (torch.arange(n)[:, None], torch.full((n,), 4)))
    out = ops.paged_attention_decode(qkv, k, v.reshape(-1, 1, 128), tables.contiguous(), lens, heads, 1, BLOCK, 128 ** -0.5)
    parts = w[:, :, None] * v[:, :4].double()
    err = (out.view(n, heads, 128).double() - parts.sum(1)[:, None]).abs() / parts.abs().sum(1)[:, None]
    assert float(err.max()) <= 2.0 ** -19.5, float(err.max())


def test_small_weights_add_up():
    """fp16: 6000 keys at 2^-26 of the largest weight each, alone in having values."""
    from deltazip_b200 import ops
    heads, n, dtype = 4, 6000, torch.float16
    blocks = -(-n // BLOCK)
    v = torch.ones((blocks * BLOCK, 1, 128), device="cuda", dtype=dtype)
    v[n - 1] = 0
    bias = torch.tensor([[0.0, -26 * 0.6931471805599453]] * heads, device="cuda")
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    out = ops.window_attention(torch.zeros((1, (heads + 2) * 128), device="cuda", dtype=dtype), torch.zeros_like(v), v,
                               torch.arange(blocks, dtype=torch.int32, device="cuda")[None], i32([0, 1]), i32([n - 1]), 1, True,
                               heads, BLOCK, 1.0, 0, bias, 1, None)
    tail = (n - 1) * 2.0 ** -26
    check(out[0], torch.full_like(out[0], tail / (1 + tail), dtype=torch.float64), dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("length,key", [(16, 3), (21, 20), (70, 69), (70, 5)])
def test_infinities_among_the_values(length, key, dtype):
    """An infinite component of a value gives that infinity, and leaves the other components alone; values that repeat
    behind a sequence's end do not count."""
    from deltazip_b200 import ops
    heads = 8
    qkv, k, v, tables = batch(1, heads, dtype, length, 5, [length])
    v[int(tables[0, key // BLOCK]) * BLOCK + key % BLOCK, 0, 7] = float("inf")
    v[int(tables[0, key // BLOCK]) * BLOCK + key % BLOCK, 0, 12] = float("-inf")
    out = ops.paged_attention_decode(qkv, k, v, tables, torch.tensor([length], dtype=torch.int32, device="cuda"), heads, 1, BLOCK, 0.02)
    at = (tables[0].long()[:, None] * BLOCK + torch.arange(BLOCK, device="cuda")).flatten()[:length]
    want = reference(qkv[0, :heads * 128].view(heads, 128), k[at], v[at], 0.02)
    bad = torch.isinf(want)
    assert torch.equal(torch.where(bad, out[0].double(), 0), torch.where(bad, want, 0)) and int(bad.sum()) == 2 * heads
    check(out[0][~bad], want[~bad], dtype)


@pytest.mark.parametrize("heads", [2, 8])
@pytest.mark.parametrize("splits", [0, -1, 65])
def test_split_counts_out_of_range_are_refused(heads, splits):
    from deltazip_b200 import ops
    from deltazip_b200._lib import DeltaZipError
    qkv, k, v, tables = batch(1, heads, torch.float16, 1, 40, [600])
    with pytest.raises(DeltaZipError):
        ops.paged_attention_decode(qkv, k, v, tables, torch.tensor([600], dtype=torch.int32, device="cuda"), heads, 1, BLOCK, 0.1, splits)


@pytest.mark.parametrize("heads,kvh", [(8, 1), (32, 8)])
def test_short_sequences_in_wide_tables(heads, kvh):
    """The number of splits follows from the tables' width; splits that a sequence has no keys for take no part, in the
    merge and in the tickets."""
    from deltazip_b200 import ops
    dtype, lens = torch.float16, [1, 64, 65, 300, 1000, 0]
    qkv, k, v, tables = batch(kvh, heads, dtype, 9, 256, lens)
    for rep in range(3):
        order = list(range(len(lens)))[::-1] if rep == 1 else list(range(len(lens)))     # the tickets are back at zero
        n = torch.tensor([lens[i] for i in order], dtype=torch.int32, device="cuda")
        out = ops.paged_attention_decode(qkv, k, v, tables, n, heads, kvh, BLOCK, 128 ** -0.5)
        for row, i in enumerate(order):
            at = (tables[row].long()[:, None] * BLOCK + torch.arange(BLOCK, device="cuda")).flatten()[:lens[i]]
            if lens[i] == 0:
                assert not out[row].any()
            else:
                check(out[row], reference(qkv[row, :heads * 128].view(heads, 128), k[at], v[at], 128 ** -0.5), dtype)

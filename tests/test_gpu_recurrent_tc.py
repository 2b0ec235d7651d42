"""Chunkwise recurrences with heads of 128 x 128 (the tcgen05 kernel): chunk borders, continued sequences, decays and
gates at their ends, unequal batches -- against the 64-bit recurrences of the oracle."""
import pytest
import torch

from tests.test_gpu_buzalorn import BF16, EXACT, F16, MlstmRun, i32, rel
from tests.test_gpu_movarax import LightningRun

pytestmark = pytest.mark.gpu

# whole chunks, one token more and less, single tokens between portions; then prompts continued from decoding
CUTS = [[600], [127, 1, 128, 129, 215], [256, 256, 88], [5, 300], [1, 130]]
CHUNKS = lambda n: n > 4


@pytest.mark.parametrize("dtype", [BF16, F16])
@pytest.mark.parametrize("run", [MlstmRun, LightningRun])
def test_chunk_borders(run, dtype):
    r = run(2, 128, 128, 600, dtype)
    for cuts in CUTS:
        always = len(cuts) != 2
        assert rel(r.run(cuts, chunk=lambda n: always or n > 4), r.want) < EXACT[dtype], cuts
    assert torch.isnan(r.S[0]).all() and torch.isnan(r.S[2]).all()


@pytest.mark.parametrize("kw", [dict(f_mean=-30.0, cap=12.0), dict(f_mean=30.0, cap=14.0), dict(i_std=40.0, cap=13.0)])
def test_gates_at_their_ends(kw):
    r = MlstmRun(2, 128, 128, 300, BF16, seed=5, **kw)
    for cuts in ([300], [130, 40]):
        assert rel(r.run(cuts, chunk=CHUNKS), r.want) < EXACT[BF16] * 1.5, cuts


def test_decays_at_their_ends():
    r = LightningRun(3, 128, 128, 400, BF16, decay=[0.0, 1.0, 0.999])
    for cuts in ([400], [129, 131]):
        assert rel(r.run(cuts, chunk=CHUNKS), r.want) < EXACT[BF16], cuts


def test_absent_tokens_bring_nothing_from_their_neighbours():
    """Rows behind a sequence's end hold infinities: they belong to the next one."""
    from deltazip_b200 import ops
    a = LightningRun(2, 128, 128, 131, BF16, seed=3)
    x = torch.cat([a.x, torch.full_like(a.x[:100], float("inf"))])
    S = torch.zeros(3, 2, 128, 128, device="cuda")
    got = ops.lightning(x, a.powers, a.norm, S, i32([1, 2]), i32([0, 131, 231]), i32([0, 0]), a.eps, True)
    assert rel(got[:131].double().cpu().numpy(), a.want) < EXACT[BF16] and torch.isfinite(S[1]).all()
    b = MlstmRun(2, 128, 128, 131, BF16, seed=3)
    x = torch.cat([b.x, torch.full_like(b.x[:100], float("inf"))])
    h = torch.cat([b.h, b.h[:100]])
    S, n, m = torch.zeros(3, 2, 128, 128, device="cuda"), torch.zeros(3, 2, 128, device="cuda"), torch.zeros(3, 2, device="cuda")
    got = ops.mlstm(x, h, b.w, b.b, b.norm, S, n, m, i32([1, 2]), i32([0, 131, 231]), i32([0, 0]), b.cap, b.scale, b.eps, True)
    assert rel(got[:131].double().cpu().numpy(), b.want) < EXACT[BF16] and torch.isfinite(S[1]).all()


def test_unequal_sequences_in_one_batch():
    from deltazip_b200 import ops
    runs = [MlstmRun(2, 128, 128, t, BF16, seed=t) for t in (290, 3, 128)]
    w, b, norm = runs[0].w, runs[0].b, runs[0].norm
    S, n, m = torch.zeros(5, 2, 128, 128, device="cuda"), torch.zeros(5, 2, 128, device="cuda"), torch.zeros(5, 2, device="cuda")
    x, h = torch.cat([r.x for r in runs]), torch.cat([r.h for r in runs])
    args = (runs[0].cap, runs[0].scale, runs[0].eps)
    got = ops.mlstm(x, h, w, b, norm, S, n, m, i32([3, 0, 4, 2]), i32([0, 290, 293, 293, 421]), i32([0, 0, 0, 0]), *args, True)
    at = 0
    for r, slot in zip(runs, (3, 0, 2)):
        s1, n1, m1 = torch.zeros_like(S), torch.zeros_like(n), torch.zeros_like(m)
        alone = ops.mlstm(r.x, r.h, w, b, norm, s1, n1, m1, i32([1]), i32([0, r.t]), i32([0]), *args, True)
        assert torch.equal(alone, got[at:at + r.t]) and torch.equal(s1[1], S[slot]) and torch.equal(n1[1], n[slot])
        assert torch.equal(m1[1], m[slot])
        at += r.t
    assert not S[4].any() and not m[4].any()              # no tokens: the slot is left alone
    assert ops.read_status(x.device) == 0


@pytest.mark.parametrize("kind", ["mlstm", "lightning"])
def test_results_do_not_depend_on_when_tiles_arrive(kind):
    """Whole chunks come by one bulk copy per tile, which complete in any order when the memory is busy: the results next
    to large copies on another stream equal those on an idle GPU bit for bit."""
    from deltazip_b200 import ops
    heads, t = 8, 1024
    r = (MlstmRun if kind == "mlstm" else LightningRun)(heads, 128, 128, t, BF16, seed=11)
    slots, starts, ctx = i32([2, 0]), i32([0, 512, t]), i32([0, 7])
    g = torch.Generator(device="cuda").manual_seed(2)
    start = [torch.randn(s, generator=g, device="cuda") for s in ((3, heads, 128, 128), (3, heads, 128), (3, heads))]

    def run():
        S, n, m = (x.clone() for x in start)
        if kind == "mlstm":
            out = ops.mlstm(r.x, r.h, r.w, r.b, r.norm, S, n, m, slots, starts, ctx, r.cap, r.scale, r.eps, True)
        else:
            out = ops.lightning(r.x, r.powers, r.norm, S, slots, starts, ctx, r.eps, True)
        return out, S, n, m

    quiet = run()
    big = torch.empty((2, 1 << 28), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(200):
            big[1].copy_(big[0])
    busy = [run() for _ in range(20)]
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for other in busy for a, b in zip(quiet, other))
    assert ops.read_status() == 0


def test_status_word_of_a_workspace():
    """A word that a kernel left is read from the first word of the workspace, also after a larger one took its place; a
    call without room for it takes the kernel that waits for nothing, or is refused where a workspace is asked for."""
    import ctypes
    from deltazip_b200 import _lib, ops
    L = _lib.lib()
    assert L.dz_lightning_workspace_bytes(200, 1, 2, 128, 1) >= 4
    assert L.dz_mlstm_workspace_bytes(3, 2) >= 4 + 3 * 2 * 4
    assert ops.read_status() == 0
    a = MlstmRun(2, 128, 128, 140, BF16, seed=3)
    a.run([140])
    ops._zeroed_scratch("mlstm", a.x.device, 4)[:4].view(torch.int32).fill_(_lib.DZ_ERR_TIMEOUT)
    many = 4096                                    # more (sequence, head) pairs than the workspace has room for
    starts = torch.zeros(many + 1, dtype=torch.int32, device="cuda")
    ops.mlstm(a.x, a.h, a.w, a.b, a.norm, a.S, a.n, a.m, i32([0] * many), starts, i32([0] * many), a.cap, a.scale, a.eps, True)
    assert ops.read_status() == _lib.DZ_ERR_TIMEOUT and ops.read_status() == 0

    b = LightningRun(2, 128, 128, 200, BF16, seed=3)
    ops._zeroed_scratch("lightning_chunk", b.x.device, 4)[:4].view(torch.int32).fill_(_lib.DZ_ERR_TIMEOUT)
    assert ops.read_status() == _lib.DZ_ERR_TIMEOUT and ops.read_status() == 0
    out, S = torch.empty((200, 256), dtype=BF16, device="cuda"), torch.zeros((1, 2, 128, 128), device="cuda")
    slots, starts, ctx = i32([0]), i32([0, 200]), i32([0])
    args = _lib.LightningArgs(
        x=b.x.data_ptr(), row_stride=b.x.stride(0), k_off=256, v_off=512, g_off=768, powers=b.powers.data_ptr(),
        norm_weight=b.norm.data_ptr(), eps=b.eps, out=out.data_ptr(), S=S.data_ptr(), slots=slots.data_ptr(),
        q_starts=starts.data_ptr(), ctx_lens=ctx.data_ptr(), num_seqs=1, rows=200, heads=2, dim=128, vdim=128, chunkwise=1,
        dtype=_lib.DZ_DTYPE_BF16)
    assert L.dz_lightning(ctypes.byref(args), ops._stream()) == 0
    assert rel(out.double().cpu().numpy(), b.want) < EXACT[BF16]
    small = torch.zeros(64, dtype=torch.uint8, device="cuda")
    x = a.x
    margs = _lib.MlstmArgs(
        x=x.data_ptr(), row_stride=x.stride(0), k_off=256, v_off=512, g_off=768, b_if=a.b.data_ptr(), pre_if=S.data_ptr(), width=48,
        cap=a.cap, scale=a.scale, norm_weight=a.norm.data_ptr(), eps=a.eps, out=out.data_ptr(), S=a.S.data_ptr(), n=a.n.data_ptr(),
        m=a.m.data_ptr(), slots=slots.data_ptr(), q_starts=starts.data_ptr(), ctx_lens=ctx.data_ptr(), num_seqs=1, rows=140,
        heads=2, dim=128, vdim=128, chunkwise=1, workspace=small.data_ptr(), workspace_bytes=64, dtype=_lib.DZ_DTYPE_BF16)
    assert L.dz_mlstm(ctypes.byref(margs), ops._stream()) == _lib.DZ_ERR_WORKSPACE


@pytest.mark.parametrize("dim", [64, 128])
def test_silu_far_below_zero_and_next_to_a_nan(dim):
    """SiLU of -50 is -1e-20, which bf16 holds; a NaN stays in its own column of the state."""
    from deltazip_b200 import ops
    r = LightningRun(1, dim, dim, 70, BF16, seed=8, decay=[0.9])
    x = r.x[:, :4 * dim].clone()
    x[:, 2 * dim + 3] = -50
    S = torch.zeros((1, 1, dim, dim), device="cuda")
    ops.lightning(x, r.powers, r.norm, S, i32([0]), i32([0, 70]), i32([0]), r.eps, True)
    silu = lambda t: torch.nn.functional.silu(t.double()).to(BF16).double()
    decay = 0.9 ** torch.arange(69, -1, -1, device="cuda", dtype=torch.float64)
    want = (silu(x[:, dim:2 * dim]) * decay[:, None]).t() @ silu(x[:, 2 * dim:3 * dim])
    err = (S[0, 0].double() - want).norm(dim=0) / want.norm(dim=0)          # a column of the state per component of v
    assert float(err.max()) < 1e-2 and float(S[0, 0, :, 3].abs().max()) > 0
    x[9, 2 * dim + 5] = float("nan")
    S.zero_()
    ops.lightning(x, r.powers, r.norm, S, i32([0]), i32([0, 70]), i32([0]), r.eps, True)
    assert torch.isnan(S[0, 0]).any(0).nonzero().flatten().tolist() == [5]


def test_gate_sums_of_a_chunk_keep_their_precision():
    """Forget gates near 0.1: the logarithms of a chunk add up to -300, whose last place is 3e-5.  What a weight's logarithm
    may be off by is the roundings of a gate of size 3 (cap, tanh, logarithm: 2^-22 each) for the few tokens that count;
    the gates' inputs are exact in 32 bits.  The bound is 2^-19."""
    from deltazip_b200 import ops
    t, heads = 600, 2
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn((t, heads * 512), generator=g, device="cuda").to(BF16)
    h = torch.randint(-3, 4, (t, 16), generator=g, device="cuda").to(BF16)
    w = (torch.randint(-1, 2, (2 * heads, 16), generator=g, device="cuda") / 8).to(BF16)
    b = torch.tensor([0.5, -1.0, -2.25, -2.5], device="cuda")
    S, n, m = (torch.zeros(s, device="cuda") for s in ((1, heads, 128, 128), (1, heads, 128), (1, heads)))
    ops.mlstm(x, h, w, b, torch.ones(heads * 128, device="cuda"), S, n, m, i32([0]), i32([0, t]), i32([0]), 64.0, 0.1, 1e-6, True)
    pre = 64 * torch.tanh((h.double() @ w.double().t() + b.double()) / 64)
    i, F = pre[:, :heads].t(), torch.nn.functional.logsigmoid(pre[:, heads:]).t().cumsum(1)
    top = torch.maximum((i - F).cummax(1).values, torch.zeros((), device="cuda", dtype=torch.float64))[:, -1:]
    last = (i - F - top).exp()
    k = x[:, heads * 128:heads * 256].double().view(t, heads, 128)
    want = torch.einsum("ht,thd->hd", last, k)
    assert float(F.min()) < -1000
    assert float((n[0].double() - want).norm() / want.norm()) <= 2.0 ** -19
    assert float((m[0].double() - (F[:, -1:] + top)[:, 0]).abs().max()) <= 2.0 ** -19

"""Delta products of prompt batches (more than 512 tokens, added in place) against 64-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(n, k, runs, bits, dtype, seed=5):
    """runs: [(slot, tokens)] in slot order.  Scales are powers of two, so that the unpacked delta is exact."""
    from deltazip_b200 import ops, synth
    dev = torch.device("cuda")
    slots = max(s for s, _ in runs) + 2                    # the last one has no tokens
    qw, meta, sc = synth.random_delta_slots(slots, n, k, bits, seed=seed, device=dev, std=1e-2)
    sc.copy_((2.0 ** torch.randint(-9, -5, sc.shape, generator=torch.Generator(dev).manual_seed(seed), device=dev)).half())
    g = torch.Generator(device=dev).manual_seed(seed + 1)
    m = sum(t for _, t in runs)
    x = torch.randn((m, k), generator=g, device=dev).to(dtype)
    y = torch.randn((m, n), generator=g, device=dev).to(dtype)
    idx = torch.tensor([s for s, t in runs for _ in range(t)], device=dev)
    want = y.double()
    for s in {s for s, _ in runs if s >= 0}:
        rows = idx == s
        want[rows] += x[rows].double() @ ops.unpack(qw[s], meta[s], sc[s], n, k, bits).double().t()
    return x, y, idx, qw, meta, sc, want


def _close(got, want, dtype):
    """One rounding of the sum to the type, and the 32-bit accumulation's far smaller error (2^-24 a step over at
    most 1536 kept products of comparable size)."""
    unit = 2.0 ** (-11 if dtype == torch.float16 else -8)
    err = (got.double() - want).abs()
    assert bool((err <= unit * want.abs() + 2.0 ** -11 * want.square().mean().sqrt()).all()), err.max()


# run lengths around the token block (176), the TMA box (88) and the MMA's column step (16); base-only rows between
RUNS = [(-1, 30), (0, 1), (2, 16), (3, 17), (4, 88), (5, 89), (6, 176), (7, 177), (9, 353)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits", [2, 4])
@pytest.mark.parametrize("n,k", [(128, 64), (384, 192), (12288, 256), (256, 3072)])
def test_prompt_batch_adds_the_delta_products(n, k, bits, dtype):
    from deltazip_b200 import ops
    x, y, idx, qw, meta, sc, want = _case(n, k, RUNS, bits, dtype)
    seg = ops.Segments(len(idx), qw.shape[0], x.device).build(idx, sorted_hint=True)
    got = ops.sbmm(x, qw, sc, meta, seg, None, out=y, accumulate=True)
    _close(got, want, dtype)
    assert ops.read_status(x.device) == 0


@pytest.mark.parametrize("bits", [2, 4])
def test_prompt_batch_in_any_order_and_into_a_slice(bits):
    from deltazip_b200 import ops
    n, k = 256, 320
    x, y, idx, qw, meta, sc, want = _case(n, k, RUNS, bits, torch.float16)
    order = torch.randperm(len(idx), generator=torch.Generator("cuda").manual_seed(1), device=x.device)
    wide = torch.zeros((len(idx), n + 64), dtype=torch.float16, device=x.device)
    wide[:, 8:8 + n] = y[order]
    seg = ops.Segments(len(idx), qw.shape[0], x.device).build(idx[order])
    ops.sbmm(x[order].contiguous(), qw, sc, meta, seg, None, out=wide[:, 8:8 + n], accumulate=True)
    _close(wide[:, 8:8 + n], want[order], torch.float16)
    assert not wide[:, :8].any() and not wide[:, 8 + n:].any()


@pytest.mark.parametrize("tokens", [512, 513])
def test_edge_of_the_prompt_path(tokens):
    from deltazip_b200 import ops
    x, y, idx, qw, meta, sc, want = _case(256, 256, [(0, tokens - 1), (1, 1)], 4, torch.float16)
    seg = ops.Segments(tokens, qw.shape[0], x.device).build(idx, sorted_hint=True)
    _close(ops.sbmm(x, qw, sc, meta, seg, None, out=y, accumulate=True), want, torch.float16)


def test_a_wrong_promise_of_order_leaves_y_alone():
    from deltazip_b200 import ops
    x, y, idx, qw, meta, sc, _ = _case(256, 256, [(0, 300), (1, 300)], 4, torch.float16)
    before = y.clone()
    seg = ops.Segments(600, qw.shape[0], x.device).build(idx.flip(0), sorted_hint=True)
    ops.sbmm(x, qw, sc, meta, seg, None, out=y, accumulate=True)
    assert ops.read_status(x.device) == 1 and torch.equal(y, before)

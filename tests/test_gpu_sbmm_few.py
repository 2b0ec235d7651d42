"""The SBMM form of at most 16 tokens at its edges: both numbers of token blocks, one and several stages of deltas, slices of
16 and of 32 features, blocks of k that leave warps without work, both types and code widths, added products, and columns
that must not see each other."""
import numpy as np
import pytest
import torch

from oracle import deltazip_oracle as O
from tests.gpu_util import DeviceLayer, dev
from tests.test_gpu_sbmm import check, run_sbmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("n,k,m,nd", [(128, 64, 1, 1), (128, 448, 8, 8), (256, 1088, 9, 4), (1024, 512, 16, 16), (384, 576, 16, 11),
                                      (4864, 128, 3, 2), (4864, 192, 16, 6), (9600, 64, 5, 5)])
def test_shapes(n, k, m, nd, bits):
    layer = DeviceLayer(n, k, nd, bits, seed=n + m)
    x, idx = O.make_tokens(m, k, nd, seed=k + m, sort=False, base_frac=0.2)
    if m >= nd:
        idx[:nd] = np.arange(nd)[::-1]               # every delta present
    y, _ = run_sbmm(layer, x, idx)
    check(layer, x, idx, y)


@pytest.mark.parametrize("n,m", [(256, 5), (256, 13), (4864, 2), (9600, 16)])
def test_bf16_and_base_alone(n, m):
    from deltazip_b200 import ops
    k, nd = 320, 3
    layer = DeviceLayer(n, k, nd, 4, seed=m)
    x, idx = O.make_tokens(m, k, nd, seed=m, sort=False, base_frac=0.1)
    seg = ops.Segments(m, nd, "cuda").build(torch.from_numpy(idx).cuda())
    xb, wb = dev(x).bfloat16(), layer.w.bfloat16()
    y = ops.sbmm(xb, layer.qweight, layer.scales, layer.meta, seg, wb)
    want = xb.double() @ wb.double().t()
    alone = ops.base_gemm(xb, wb)
    # one rounding to 8 bits of the result, and sums of k products in 32 bits of mixed sign
    room = lambda w, v: (w - v.double()).abs() <= 2.0 ** -8 * w.abs() + 2.0 ** -22 * k ** 0.5 * w.abs().max()
    assert room(want, alone).all()
    for i, d in enumerate(idx):
        if d >= 0:
            dense = ops.unpack(layer.qweight[d], layer.meta[d], layer.scales[d], n, k, 4).double()
            want[i] += xb[i].double() @ dense.t()
    # unpack rounds code * scale to 16 bits: 2^-11 of a delta's share, which is smaller than the sum's largest entry
    assert ((want - y.double()).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -10 * want.abs().max()).all()


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("k,m", [(64, 2), (192, 7), (320, 16), (384, 9)])
def test_second_slices(k, m, bits):
    """More slices of 32 features than four CTAs on each of 148 SMs: a CTA goes on to a second one, its rings as they are."""
    n = 19328                                        # 604 slices
    layer = DeviceLayer(n, k, 2, bits, seed=m)
    x, idx = O.make_tokens(m, k, 2, seed=k, sort=False, base_frac=0.2)
    y, _ = run_sbmm(layer, x, idx)
    check(layer, x, idx, y)
    from deltazip_b200 import ops
    alone = ops.base_gemm(dev(x), layer.w)
    base, _ = run_sbmm(layer, x, np.full(m, -1))
    np.testing.assert_array_equal(alone.cpu().numpy().view(np.uint16), base.view(np.uint16))


def test_columns_do_not_see_each_other():
    layer = DeviceLayer(256, 256, 4, 4, seed=1)
    x, _ = O.make_tokens(12, 256, 4, seed=1)
    idx = np.array([3, 0, -1, 0, 2, 1, 3, -1, 2, 0, 1, 1])
    y, _ = run_sbmm(layer, x, idx)
    bad = x.copy()
    bad[[1, 7, 8]] = np.array([[np.nan], [np.inf], [65504.0]], dtype=np.float16)
    z, _ = run_sbmm(layer, bad, idx)
    rest = [i for i in range(12) if i not in (1, 7, 8)]
    np.testing.assert_array_equal(z[rest].view(np.uint16), y[rest].view(np.uint16))
    # a batch of one has the same sums as its row in a larger one
    one, _ = run_sbmm(layer, x[4:5], idx[4:5])
    np.testing.assert_array_equal(one.view(np.uint16), y[4:5].view(np.uint16))


@pytest.mark.parametrize("m", [1, 7, 16])
def test_a_reset_slot_adds_nothing(m):
    from deltazip_b200 import ops
    from deltazip_b200._lib import check as ok, lib
    layer = DeviceLayer(384, 192, 2, 4, seed=m)
    for t in (layer.qweight, layer.meta, layer.scales):
        ok(lib().dz_slot_reset(t[1].data_ptr(), t[1].numel() * t.element_size(), torch.cuda.current_stream().cuda_stream), "reset")
    x, _ = O.make_tokens(m, 192, 2, seed=m)
    idx = np.full(m, 1)
    y, _ = run_sbmm(layer, x, idx)
    base, _ = run_sbmm(layer, x, np.full(m, -1))
    np.testing.assert_array_equal(y.view(np.uint16), base.view(np.uint16))


def test_wrong_promise_is_reported_and_y_left():
    from deltazip_b200 import _lib, ops
    layer = DeviceLayer(128, 128, 3, 4, seed=0)
    x, _ = O.make_tokens(6, 128, 3, seed=0)
    seg = ops.Segments(6, 3, "cuda").build(torch.tensor([2, 1, 0, 0, -1, 1], device="cuda"), sorted_hint=True)
    y = torch.full((6, 128), 5.0, dtype=torch.float16, device="cuda")
    ops.read_status()
    ops.sbmm(dev(x), layer.qweight, layer.scales, layer.meta, seg, layer.w, out=y)
    assert ops.read_status() == _lib.DZ_ERR_INVALID_ARG
    assert (y == 5).all()


@pytest.mark.parametrize("m,slots", [(6, 3), (32, 3)])
def test_rejected_among_early_starting_calls(m, slots):
    """Calls that start under their predecessor's tail, each reading what the one before wrote, with a rejected table in
    between: its grid ends no sooner than the call before it, and the chain goes on.  (32 tokens: the form for larger batches.)"""
    from deltazip_b200 import _lib, ops
    layer = DeviceLayer(256, 256, slots, 4, seed=m)
    x_np, idx = O.make_tokens(m, 256, slots, seed=m, sort=False, base_frac=0.2)
    idx[:2] = [2, 0]
    index = torch.from_numpy(idx).cuda()
    seg = ops.Segments(m, slots, "cuda").build(index)
    wrong = ops.Segments(m, slots, "cuda").build(index, sorted_hint=True)

    def chain(reject):
        x, ys = dev(x_np), [torch.full((m, 256), 5.0, dtype=torch.float16, device="cuda") for _ in range(12)]
        torch.cuda.synchronize()                     # table, slots and weight are written before the chain begins
        for y, kept in zip(ys[::2], ys[1::2]):
            ops.sbmm(x, layer.qweight, layer.scales, layer.meta, seg, layer.w, out=y, stable=True)
            if reject:
                ops.sbmm(y, layer.qweight, layer.scales, layer.meta, wrong, layer.w, out=kept, stable=True)
            x = y
        return ys
    ops.read_status()
    want, got = chain(False), chain(True)
    assert want[0].any() and torch.isfinite(want[10]).all()
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    assert ops.read_status() == _lib.DZ_ERR_INVALID_ARG and ops.read_status() == 0

"""Batches of at most 16 tokens in any order: the kernels take them as they come, without a gather of x in front, and larger
ones through the gather as before.  Small k go to the form for few tokens, k above 6144 (or 8192 over the number of deltas)
to that of 16 columns with tcgen05.mma."""
import numpy as np
import pytest
import torch

from oracle import deltazip_oracle as O
from tests.gpu_util import DeviceLayer, dev
from tests.test_gpu_sbmm import check, run_sbmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("m", [1, 2, 7, 15, 16, 17])
def test_any_order(m, bits):
    layer = DeviceLayer(256, 448, 6, bits, seed=m, num_slots=8)
    x, idx = O.make_tokens(m, 448, 6, seed=m + 1, sort=False, base_frac=0.2)
    if m > 2:
        idx = np.concatenate([[5, 0], idx[2:]])      # descending at the start, whatever was drawn
    y, seg = run_sbmm(layer, x, idx)
    assert m <= 2 or seg.header()[3] == 0
    check(layer, x, idx, y)
    # the same rows in the table's order: the same sums
    order = np.argsort(idx, kind="stable")
    z, _ = run_sbmm(layer, x[order], idx[order])
    np.testing.assert_array_equal(z.view(np.uint16), y[order].view(np.uint16))


@pytest.mark.parametrize("m", [3, 16])
def test_added_into_a_slice(m):
    from deltazip_b200 import ops
    layer = DeviceLayer(256, 192, 4, 4, seed=m)
    x, _ = O.make_tokens(m, 192, 4, seed=m)
    idx = np.array([(3 * i + 2) % 5 - 1 for i in range(m)])
    y = torch.zeros((m, 512), dtype=torch.float16, device="cuda")
    ops.add_delta_slice(y, dev(x), layer.qweight, None, layer.scales, None, torch.from_numpy(idx).cuda(), 1.0, 128, 256,
                        meta=layer.meta)
    full, _ = run_sbmm(layer, x, idx)
    base, _ = run_sbmm(layer, x, np.full(m, -1, dtype=np.int64))
    got = y.cpu().numpy().astype(np.float32)
    assert not got[:, :128].any() and not got[:, 384:].any()
    want = full.astype(np.float32) - base.astype(np.float32)
    # each of the three results is rounded to 16 bits once
    limit = 2.0 ** -11 * (np.abs(full).astype(np.float32) + np.abs(base) + np.abs(got[:, 128:384])) + 1e-6
    assert (np.abs(got[:, 128:384] - want) <= limit).all()


def long_k(n, k, nd, bits, m):
    """A layer above the few-token form's limit on k, and unsorted tokens that are never all of one delta or in order."""
    layer = DeviceLayer(n, k, nd, bits, seed=m + k)
    x, idx = O.make_tokens(m, k, nd, seed=k + m, sort=False, base_frac=0.2)
    if m > 2:
        idx[:3] = [nd - 1, 0, -1]
    return layer, x, idx


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("n,k,m,nd", [(256, 6208, 1, 1), (128, 6272, 2, 2), (256, 6208, 8, 8), (256, 6272, 9, 3), (384, 6208, 16, 1),
                                      (128, 6208, 16, 16), (256, 2112, 15, 8), (128, 1088, 16, 16), (2432, 4160, 8, 4)])
def test_sixteen_columns_any_order(n, k, m, nd, bits):
    """Whole units of k and ones of 64 (6208, 2112, 1088, 4160); the last three lie above the limit by their deltas."""
    layer, x, idx = long_k(n, k, nd, bits, m)
    if m >= nd:
        idx[:nd] = np.arange(nd)[::-1]                 # every delta present
    y, seg = run_sbmm(layer, x, idx)
    assert m <= 2 or nd == 1 or seg.header()[3] == 0
    check(layer, x, idx, y)
    order = np.argsort(idx, kind="stable")
    z, _ = run_sbmm(layer, x[order], idx[order])
    np.testing.assert_array_equal(z.view(np.uint16), y[order].view(np.uint16))


@pytest.mark.parametrize("k,m", [(6208, 5), (6272, 13)])
def test_sixteen_columns_bf16(k, m):
    from deltazip_b200 import ops
    n, nd = 256, 3
    layer, x, idx = long_k(n, k, nd, 4, m)
    seg = ops.Segments(m, nd, "cuda").build(torch.from_numpy(idx).cuda())
    xb, wb = dev(x).bfloat16(), layer.w.bfloat16()
    y = ops.sbmm(xb, layer.qweight, layer.scales, layer.meta, seg, wb)
    want = xb.double() @ wb.double().t()
    for i, d in enumerate(idx):
        if d >= 0:
            want[i] += xb[i].double() @ ops.unpack(layer.qweight[d], layer.meta[d], layer.scales[d], n, k, 4).double().t()
    # one rounding to 8 bits of the result; unpack rounds code * scale to 16 bits, 2^-11 of a delta's share
    assert ((want - y.double()).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -10 * want.abs().max()).all()


@pytest.mark.parametrize("k,m", [(6208, 3), (6272, 16)])
def test_sixteen_columns_added_into_a_slice(k, m):
    from deltazip_b200 import ops
    layer, x, idx = long_k(256, k, 4, 2, m)
    before = torch.randn((m, 512), generator=torch.Generator().manual_seed(k)).half().cuda()
    y = before.clone()
    ops.add_delta_slice(y, dev(x), layer.qweight, None, layer.scales, None, torch.from_numpy(idx).cuda(), 1.0, 128, 256,
                        meta=layer.meta)
    assert torch.equal(y[:, :128], before[:, :128]) and torch.equal(y[:, 384:], before[:, 384:])
    want = before[:, 128:384].double()
    for i, d in enumerate(idx):
        if d >= 0:
            dense = ops.unpack(layer.qweight[d], layer.meta[d], layer.scales[d], 256, k, 2).double()
            want[i] += dev(x)[i].double() @ dense.t()
    # one rounding of the sum to 16 bits; unpack's rounding of code * scale, 2^-11 of a delta's share
    assert ((want - y[:, 128:384].double()).abs() <= 2.0 ** -10 * (want.abs() + want.abs().max())).all()


def test_sixteen_columns_do_not_see_each_other():
    layer, x, _ = long_k(256, 6272, 4, 4, 12)
    idx = np.array([3, 0, -1, 0, 2, 1, 3, -1, 2, 0, 1, 1])
    y, _ = run_sbmm(layer, x, idx)
    bad = x.copy()
    bad[[1, 7, 8]] = np.array([[np.nan], [np.inf], [65504.0]], dtype=np.float16)
    z, _ = run_sbmm(layer, bad, idx)
    rest = [i for i in range(12) if i not in (1, 7, 8)]
    np.testing.assert_array_equal(z[rest].view(np.uint16), y[rest].view(np.uint16))

"""Batches that are no larger than the narrow form's 16 columns, in any order: the kernel takes them as they come, without
a gather of x in front, and larger ones through the gather as before."""
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

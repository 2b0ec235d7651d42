"""The compressor's kernels at their edges: one block of columns against the arithmetic step by step in numpy (bit for bit,
in place and not, rows that do not fill a thread block, divisions outside the quick form's range)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F = np.float32


def one_block(W, h, scale, zero, maxq):
    """One block of error feedback in 32 bits, every operation rounded by itself."""
    W = W.copy()
    n, count = W.shape
    Q, E = np.zeros_like(W), np.zeros_like(W)
    with np.errstate(all="ignore"):
        for i in range(count):
            if i % 4 == 0:
                d = np.diagonal(h)[i:i + 4]
                rank = (W[:, i:i + 4] * W[:, i:i + 4]) / (d * d)[None]
                order = np.argsort(rank, axis=1, kind="stable")[:, :2]
                pruned = np.zeros((n, 4), dtype=bool)
                np.put_along_axis(pruned, order, True, 1)
            w = W[:, i]
            v = np.where(pruned[:, i % 4], F(0), w)
            q = np.clip(np.rint(v / scale) + zero, F(0), F(maxq))
            Q[:, i] = scale * (q - zero)
            E[:, i] = (w - Q[:, i]) / h[i, i]
            W[:, i + 1:] -= E[:, i:i + 1] * h[i:i + 1, i + 1:]
    return Q, E


def call(W, h, scale, zero, bits, in_place, lead=0):
    from deltazip_b200._lib import check, lib
    n, count = W.shape
    wide = torch.zeros((n, lead + count + 8), device="cuda")
    wide[:, lead:lead + count] = torch.from_numpy(W)
    H = torch.from_numpy(h).cuda()
    s, z, loss = torch.from_numpy(scale).cuda(), torch.from_numpy(zero).cuda(), torch.zeros(n, device="cuda")
    E = torch.full((n, count + 4), 7.0, device="cuda")
    Q = wide if in_place else torch.empty((n, count), device="cuda")
    at = wide.data_ptr() + 4 * lead
    check(lib().dz_sparsegpt_block_strided(at, wide.stride(0), H.data_ptr(), count, s.data_ptr(), z.data_ptr(), bits, n, count,
                                           at if in_place else Q.data_ptr(), Q.stride(0), E.data_ptr(), E.stride(0),
                                           loss.data_ptr(), torch.cuda.current_stream().cuda_stream), "block")
    assert (E[:, count:] == 7).all()
    if in_place:
        assert not wide[:, :lead].any() and not wide[:, lead + count:].any()
        Q = wide[:, lead:lead + count]
    return Q.cpu().numpy(), E[:, :count].cpu().numpy(), loss.cpu().numpy()


@pytest.mark.parametrize("size", [1.0, 1e-12, 1e-25, 1e12])
@pytest.mark.parametrize("n,count,lead", [(1, 4, 0), (5, 128, 1), (31, 60, 4), (33, 128, 0), (70, 36, 3)])
def test_one_block(n, count, lead, size):
    rng = np.random.default_rng(n * count)
    W = (rng.standard_normal((n, count)) * size).astype(F)
    W[:, 1] = 0
    h = (np.triu(rng.standard_normal((count, count)) * 0.2, 1) + np.diag(0.5 + rng.random(count))).astype(F)
    scale, zero = (np.abs(W).max(1) * F(2 / 15)).astype(F), np.full(n, 8, F)
    if n > 4:
        W[3] = 0
        scale[3] = F(0.1)
    want_q, want_e = one_block(W, h, scale, zero, 15)
    for in_place in (True, False):
        q, e, loss = call(W, h, scale, zero, 4, in_place, lead)
        assert np.array_equal(q.view(np.uint32), want_q.view(np.uint32))
        assert np.array_equal(e, want_e)
        # `count` terms in 32 bits, each of them three roundings of its own
        true = (want_e.astype(np.float64) ** 2).sum(1) / 2
        assert (np.abs(loss - true) <= (count + 4) * 2.0 ** -23 * true + 1e-37).all()

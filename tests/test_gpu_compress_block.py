"""The compressor's kernels at their edges: one block of columns against the arithmetic step by step in numpy (bit for bit,
in place and not, rows that do not fill a thread block, divisions outside the quick form's range), the inverses of
diagonal blocks and the operands of the update against 64 bits."""
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


@pytest.mark.parametrize("n,count", [(5, 128), (33, 36)])
def test_one_block_into_matrices_of_its_own(n, count):
    """dz_sparsegpt_block: rows of the results `count` apart, the block left as it was."""
    from deltazip_b200._lib import check, lib
    rng = np.random.default_rng(n)
    W = rng.standard_normal((n, count)).astype(F)
    h = (np.triu(rng.standard_normal((count, count)) * 0.2, 1) + np.diag(0.5 + rng.random(count))).astype(F)
    scale, zero = (np.abs(W).max(1) * F(2 / 15)).astype(F), np.full(n, 8, F)
    w, H, s, z = (torch.from_numpy(a).cuda() for a in (W, h, scale, zero))
    Q, E = torch.empty((n, count), device="cuda"), torch.empty((n, count), device="cuda")
    check(lib().dz_sparsegpt_block(w.data_ptr(), count, H.data_ptr(), count, s.data_ptr(), z.data_ptr(), 4, n, count,
                                   Q.data_ptr(), E.data_ptr(), None, torch.cuda.current_stream().cuda_stream), "block")
    want_q, want_e = one_block(W, h, scale, zero, 15)
    assert np.array_equal(Q.cpu().numpy(), want_q) and np.array_equal(E.cpu().numpy(), want_e)
    assert np.array_equal(w.cpu().numpy(), W)


@pytest.mark.parametrize("k", [1, 7, 128, 129, 300, 512])
def test_inverses_of_diagonal_blocks(k):
    from deltazip_b200._lib import check, lib
    g = torch.Generator().manual_seed(k)
    R = torch.randn((k, k + 2), generator=g, dtype=torch.float64).cuda() * 0.1      # what lies below the diagonal is not read
    R.diagonal().copy_(1 + torch.rand(k, generator=g, dtype=torch.float64))
    X = torch.full((k, k), 9.0, dtype=torch.float64, device="cuda")
    check(lib().dz_triangular_inverse_blocks(R.data_ptr(), k + 2, k, X.data_ptr(), k,
                                             torch.cuda.current_stream().cuda_stream), "inverse")
    for b in range(0, k, 128):
        e = min(b + 128, k)
        block, got = R[b:e, b:e].triu(), X[b:e, b:e]
        assert not got.tril(-1).any()
        # back substitution: a column's residual is below n * 2^-53 times |R| |X| (Higham, Accuracy and Stability, 8.5)
        residual = (block @ got - torch.eye(e - b, dtype=torch.float64, device="cuda")).abs()
        assert (residual <= (e - b + 2) * 2.0 ** -52 * (block.abs() @ got.abs())).all()
        X[b:e, b:e] = 9
    assert (X == 9).all()


@pytest.mark.parametrize("n,count,c", [(1, 4, 4), (5, 128, 12), (33, 60, 100), (64, 128, 516)])
def test_operands_of_the_update(n, count, c):
    from deltazip_b200._lib import check, lib
    g = torch.Generator().manual_seed(n + c)
    E = (torch.randn((n, count + 4), generator=g) * 1e-4).cuda()
    U = torch.randn((count, c + 8), generator=g).cuda()
    A = torch.empty((n, 6, count), dtype=torch.bfloat16, device="cuda")
    B = torch.empty((6, count, c), dtype=torch.bfloat16, device="cuda")
    check(lib().dz_split_update(E.data_ptr(), count + 4, n, count, U.data_ptr(), c + 8, c, A.data_ptr(), B.data_ptr(),
                                torch.cuda.current_stream().cuda_stream), "split")
    e, u = E[:, :count].double(), U[:, :c].double()
    a, b = A.double(), B.double()
    # h, m, l in their places; three roundings to 8 bits each leave 2^-27 at most
    for parts, order, x in ((a.transpose(0, 1), "lmhmhh", e), (b, "hmlhmh", u)):
        by = {ch: parts[order.index(ch)] for ch in "hml"}
        assert all(torch.equal(parts[i], by[ch]) for i, ch in enumerate(order))
        assert ((by["h"] + by["m"] + by["l"] - x).abs() <= 2.0 ** -26 * x.abs()).all()
    product = a.reshape(n, -1) @ b.reshape(-1, c)
    # what is left out: m l, l m and l l, and the splits' own rest
    assert ((product - e @ u).abs() <= 2.0 ** -23 * (e.abs() @ u.abs())).all()


def test_inputs_that_carry_gradients():
    from deltazip_b200 import compress
    g = torch.Generator(device="cuda").manual_seed(0)
    delta = torch.randn((32, 256), generator=g, device="cuda")
    x = torch.randn((512, 256), generator=g, device="cuda")
    H = x.t() @ x / 256
    plain = compress.sparsegpt_2_4(delta, 4, H)
    # the factor's other form differs by its roundings, and a code that lies between two values by one step
    carried = compress.sparsegpt_2_4(delta.clone().requires_grad_(), 4, H.clone().requires_grad_())
    assert (plain[0] != carried[0]).float().mean() <= 1e-3
    torch.testing.assert_close(plain[3], carried[3].detach(), rtol=1e-2, atol=0)


@pytest.mark.parametrize("of", ["delta", "H", "both"])
def test_a_quantised_delta_has_no_slope(of):
    """The result lies on a grid: its gradient is zero in the delta and in the Hessian, and its tangent is."""
    from deltazip_b200 import compress
    g = torch.Generator(device="cuda").manual_seed(1)
    delta = torch.randn((32, 256), generator=g, device="cuda").requires_grad_(of != "H")
    x = torch.randn((512, 256), generator=g, device="cuda")
    H = (x.t() @ x / 256).requires_grad_(of != "delta")
    Wq = compress.sparsegpt_2_4(delta, 4, H)[0]
    (Wq * torch.randn(Wq.shape, generator=g, device="cuda")).sum().backward()
    for t in (delta, H):
        assert t.grad is None if not t.requires_grad else not t.grad.any()
    with torch.no_grad():
        assert not compress.sparsegpt_2_4(delta, 4, H)[0].requires_grad
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(delta.detach(), torch.ones_like(delta))
        tangent = torch.autograd.forward_ad.unpack_dual(compress.sparsegpt_2_4(dual, 4, H.detach())[0]).tangent
        assert tangent is None or not tangent.any()


def fed_back(W, E, U):
    from deltazip_b200 import compress
    (n, count), c = E.shape, U.shape[1]
    wide = torch.zeros((n, c + 8), device="cuda")
    later = wide[:, 4:4 + c].copy_(W)
    room = [torch.full((6 * s * count,), 3.0, dtype=torch.bfloat16, device="cuda") for s in (n, c)]
    compress._feed_back(later, E.cuda(), U.cuda(), *room)
    assert not wide[:, :4].any() and not wide[:, 4 + c:].any()
    return later.double().cpu()


@pytest.mark.parametrize("n,count,c", [(1, 4, 4), (33, 60, 100), (512, 128, 1028)])
def test_update_of_the_columns_behind(n, count, c):
    g = torch.Generator().manual_seed(n + c)
    W, E, U = (torch.randn(s, generator=g) * f for s, f in (((n, c), 1e-3), ((n, count), 1e-4), ((count, c), 1.0)))
    want, size = W.double() - E.double() @ U.double(), E.double().abs() @ U.double().abs()
    error = (fed_back(W, E, U) - want).abs()
    # what the split leaves out, and sums of 6 count terms in 32 bits that may be cut
    assert (error <= (2.0 ** -23 + 6 * count * 2.0 ** -23) * size + 2.0 ** -23 * W.abs()).all()
    if n == 512:                                   # in all no further off than a product in 32 bits
        plain = torch.addmm(W.cuda(), E.cuda(), U.cuda(), alpha=-1).double().cpu()
        assert error.norm() <= (plain - want).norm()


@pytest.mark.parametrize("size", [2.0 ** -60, 2.0 ** -70, 2.0 ** -112, 2.0 ** -120, 2.0 ** 25, 2.0 ** 34, 2.0 ** 100])
def test_update_by_errors_of_any_size(size):
    """A third bf16 part has no bits left below 2^-109; the update is one of 32 bits at all sizes."""
    n, count, c = 9, 128, 132
    g = torch.Generator().manual_seed(0)
    W, E, U = (torch.randn(s, generator=g) * f for s, f in (((n, c), size), ((n, count), size), ((count, c), 1.0)))
    E[3:5] = torch.randn((2, count), generator=g)      # (rows of another size, and one of zeros)
    E[7] = 0
    got, want = fed_back(W, E, U), W.double() - E.double() @ U.double()
    # sums of `count` rounded terms, or of 6 count terms that may be cut where the sizes are those of the tensor cores
    terms = torch.full((n, 1), count * 0.5 if abs(np.log2(size)) > 64 or size > 2 ** 32 else 6.0 * count, dtype=torch.float64)
    terms[3:5] = 6.0 * count
    room = (E.double().abs() @ U.double().abs()) * 2.0 ** -23 * (terms + 1) + 2.0 ** -23 * W.abs() + 2.0 ** -148
    assert ((got - want).abs() <= room).all()
    assert torch.equal(got[7], W[7].double())


def test_update_by_errors_that_are_not_finite():
    n, count, c = 6, 8, 12
    W, E, U = torch.zeros((n, c)), torch.ones((n, count)), torch.ones((count, c)) * (1 + 2.0 ** -20)
    U[1] = 2.0 ** -40
    E[1, 2], E[2, 1], E[3, 0], E[4, 5] = float("inf"), float("-inf"), float("nan"), 3.4e38
    got = fed_back(W, E, U)
    assert (got[1] == float("-inf")).all() and (got[2] == float("inf")).all() and got[3].isnan().all()
    assert torch.allclose(got[4], torch.full((c,), -3.4e38, dtype=torch.float64) * (1 + 2.0 ** -20), rtol=2.0 ** -22)
    assert torch.allclose(got[[0, 5]], -(E.double() @ U.double())[[0, 5]], rtol=2.0 ** -20)


@pytest.mark.parametrize("shape", [(128, 128), (256, 128), (512, 512), (256,)])
def test_a_factor_of_another_size_is_refused(shape):
    from deltazip_b200 import compress
    with pytest.raises(ValueError, match="256, 256"):
        compress.sparsegpt_2_4(torch.zeros((8, 256), device="cuda"), 4, hinv=torch.ones(shape, device="cuda"))

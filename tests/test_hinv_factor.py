"""The factor of H^-1 that error feedback goes by, on the CPU and on the GPU, against 64 bits: sizes around the halves
and levels of the triangular inverse, a Hessian whose other triangle is not kept up, reduced-precision products."""
import pytest
import torch
import torch.fx.experimental.proxy_tensor

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


def hessian(k, device):
    g = torch.Generator().manual_seed(k)
    x = torch.randn((k + 50, k), generator=g, dtype=torch.float64) * (0.5 + torch.rand(k, generator=g, dtype=torch.float64))
    H = x.t() @ x / k
    H[3], H[:, 3] = 0, 0                           # a column the calibration never touched
    return H.float().to(device)


def want(H, percdamp):
    H = H.double()
    dead = H.diag() == 0
    H[dead, dead] = 1
    H += percdamp * H.diag().mean() * torch.eye(H.shape[0], dtype=torch.float64, device=H.device)
    return torch.linalg.cholesky(torch.linalg.inv(H), upper=True), H


def close(got, H, percdamp):
    U, damped = want(H, percdamp)
    # the factor's error is H's rounding (2^-24 an entry, all columns' sum of it at most) times H's condition number
    limit = 2.0 ** -24 * float(torch.linalg.cond(damped)) * 4
    assert got.dtype == torch.float32 and got.is_contiguous() and not got.tril(-1).any()
    assert float((got.double() - U).norm() / U.norm()) <= limit
    assert float((got.double().t() @ got.double() @ damped - torch.eye(len(H), device=H.device)).norm()) <= limit * len(H) ** 0.5


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("k", [4, 512, 513, 640, 1100])
def test_factor(k, device):
    from deltazip_b200 import compress
    H = hessian(k, device)
    before = H.clone()
    got, dead = compress.hinv_factor(H, 0.05)
    close(got, H, 0.05)
    assert torch.equal(H, before) and dead.nonzero().flatten().tolist() == [3]


@pytest.mark.parametrize("device", DEVICES)
def test_only_the_lower_triangle_counts(device):
    from deltazip_b200 import compress
    H = hessian(640, device)
    got, _ = compress.hinv_factor(H, 0.05)
    other, _ = compress.hinv_factor(H.tril() + torch.full_like(H, float("nan")).triu(1), 0.05)
    assert torch.equal(got, other)


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("precision", ["high", "medium"])
def test_factor_where_products_may_be_reduced(precision, device):
    from deltazip_b200 import compress
    H = hessian(1100, device)
    before = torch.get_float32_matmul_precision()
    torch.set_float32_matmul_precision(precision)
    try:
        got, _ = compress.hinv_factor(H, 0.05)
    finally:
        torch.set_float32_matmul_precision(before)
    close(got, H, 0.05)


def _derivatives(H, direction):
    """What a trace and the forms of differentiation say of the factor: a trace, forward mode twice, backward mode twice
    (which torch refuses above 512 columns, where the joined halves are written in place)."""
    from deltazip_b200 import compress
    factor = lambda h: compress.hinv_factor(h, 0.05)[0]
    yield torch.fx.experimental.proxy_tensor.make_fx(factor)(H + torch.eye(len(H), dtype=H.dtype, device=H.device))(H)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(H, direction)
        tangent = torch.autograd.forward_ad.unpack_dual(factor(dual)).tangent
        yield tangent.clone()
    yield torch.func.jvp(factor, (H,), (direction,))[1]
    if len(H) > 512:
        return
    yield torch.func.grad(lambda h: (factor(h) * direction).sum())(H)
    leaf = H.clone().requires_grad_()
    yield torch.autograd.grad((factor(leaf) * direction).sum(), leaf)[0]


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("k", [96, 256, 640])
def test_derivatives_and_traces(k, device):
    H = hessian(k, "cpu").double() + 0.1 * torch.eye(k, dtype=torch.float64)       # well conditioned, no dead column
    direction = torch.randn((k, k), generator=torch.Generator().manual_seed(k), dtype=torch.float64)
    direction = direction + direction.T
    got = list(_derivatives(H.to(device), direction.to(device)))

    def factor(h):                                 # (a damped H in terms of which torch differentiates the textbook's form)
        h = h + 0.05 * h.diag().mean() * torch.eye(k, dtype=torch.float64)
        return torch.linalg.cholesky(torch.linalg.inv(h), upper=True)
    slope = torch.func.jvp(factor, (H,), (direction,))[1]
    for tangent in got[1:3]:
        torch.testing.assert_close(tangent.cpu(), slope, rtol=1e-7, atol=1e-9)      # 64 bits throughout
    back = torch.func.grad(lambda h: (factor(h) * direction).sum())(H)
    for gradient in got[3:]:                      # (only the lower triangle is read: its gradient along a symmetric direction)
        torch.testing.assert_close((gradient.cpu() * direction).sum(), (back * direction).sum(), rtol=1e-7, atol=1e-9)
    torch.testing.assert_close(got[0].cpu(), factor(H), rtol=1e-9, atol=1e-11)


@pytest.mark.parametrize("k", [300, 1024, 1500, 2048, 2200])
def test_joined_halves(k):
    """Pairs of equal halves in a batch, large ones with a quarter of each factor left out, a last one of any size."""
    from deltazip_b200 import compress
    g = torch.Generator().manual_seed(k)
    R = (torch.randn((k, k), generator=g, dtype=torch.float64) / k ** 0.5).triu(1) + 2 * torch.eye(k, dtype=torch.float64)
    X = torch.zeros_like(R)
    for b in range(0, k, 128):
        e = min(b + 128, k)
        X[b:e, b:e] = torch.linalg.solve_triangular(R[b:e, b:e], torch.eye(e - b, dtype=torch.float64), upper=True)
    compress._join_inverses(X, R, 128)
    assert not X.tril(-1).any()
    # products of at most k terms, one level above the other, with an inverse whose norm is below one
    torch.testing.assert_close(X @ R, torch.eye(k, dtype=torch.float64), rtol=0, atol=k * 2.0 ** -50)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [100, 640, 1536, 2200, 2944])
def test_factor_to_the_last_bit_or_so(k):
    """On the GPU all of it is in 64 bits, and what is off is the rounding of the result: half a unit of the last place."""
    from deltazip_b200 import compress
    H = hessian(k, "cuda")
    H.diagonal().add_(0.05)                        # (damped beforehand: a mean of the diagonal is a sum in 32 bits)
    got, _ = compress.hinv_factor(H, 0.0)
    want = torch.linalg.cholesky(H.flip(0, 1).double()).flip(0, 1)
    want = torch.linalg.solve_triangular(want, torch.eye(k, dtype=torch.float64, device="cuda"), upper=True)
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -24


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("k", [64, 640])
def test_a_hessian_of_16_bits_is_refused(k, dtype, device):
    from deltazip_b200 import compress
    with pytest.raises(RuntimeError, match="not implemented"):
        compress.hinv_factor((torch.eye(k) * 2).to(device, dtype))


@pytest.mark.parametrize("device", DEVICES)
def test_no_columns(device):
    from deltazip_b200 import compress
    factor, dead = compress.hinv_factor(torch.empty((0, 0), device=device))
    assert factor.shape == (0, 0) and dead.shape == (0,)


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="two GPUs")
def test_factor_on_a_gpu_that_is_not_the_current_one():
    from deltazip_b200 import compress
    H = hessian(300, "cuda:1")
    got, _ = compress.hinv_factor(H, 0.05)
    close(got, H, 0.05)

"""The factor of H^-1 that error feedback goes by, on the CPU and on the GPU, against 64 bits: sizes around the halves
and levels of the triangular inverse, a Hessian whose other triangle is not kept up, reduced-precision products."""
import pytest
import torch

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

"""Delta compression on the GPU: 2:4 pruning + symmetric low-bit quantisation with SparseGPT's
error feedback, then packing -- the producer of the tensors the SBMM path serves.

Follows deltazip/core/sparsegpt.py (`SparseGPT.add_batch` :25-43, `fasterprune` :45-196 with
prunen:prunem = 2:4, no activation ordering) and `QuantLinear.pack`
(deltazip/nn_modules/qlinear.py:83-183).  The per-column loop of a block -- mask, quantise,
propagate the error inside the block -- is one kernel launch per 128 columns (dz_sparsegpt_block_strided,
rows in parallel); the dense linear algebra around it (the Cholesky factorisation of H, the products that
join the inverse's blocks, the rank-128 update of the columns behind a block) are library calls on operands
that kernels here prepare.
"""
from __future__ import annotations

import math
from typing import Optional, Tuple

import torch
import torch.autograd.forward_ad as forward_ad
from torch.utils._python_dispatch import _get_current_dispatch_mode

from ._lib import check, lib


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


class HessianAccumulator:
    """Running H = (2 / n) sum x x^T over calibration inputs of a linear layer (sparsegpt.py:25-43)."""

    def __init__(self, columns: int, device="cuda"):
        self.H = torch.zeros((columns, columns), dtype=torch.float32, device=device)
        self.nsamples = 0

    def add_batch(self, inp: torch.Tensor) -> None:
        if inp.dim() == 2:
            inp = inp.unsqueeze(0)
        batch = inp.shape[0]
        x = inp.reshape(-1, inp.shape[-1]).t().float()
        self.H *= self.nsamples / (self.nsamples + batch)
        self.nsamples += batch
        x = math.sqrt(2 / self.nsamples) * x
        self.H += x.matmul(x.t())


def _upper_inverse(R: torch.Tensor) -> torch.Tensor:
    """Inverse of an upper triangular matrix, by halves: the corner of a pair of inverted halves is two products,
    which run at the rate of a GEMM."""
    k = R.shape[0]
    if k <= 512:
        return torch.linalg.solve_triangular(R, torch.eye(k, dtype=R.dtype, device=R.device), upper=True)
    h = -(-k // 256) * 128                                   # whole multiples of 128 first
    out = torch.zeros((k, k), dtype=R.dtype, device=R.device)
    out[:h, :h] = _upper_inverse(R[:h, :h])
    out[h:, h:] = _upper_inverse(R[h:, h:])
    out[:h, h:] = (out[:h, :h] @ R[:h, h:]) @ -out[h:, h:]
    return out


def _join_inverses(X: torch.Tensor, R: torch.Tensor, h: int) -> None:
    """X holds the inverses of R's diagonal blocks of h columns (the last may be smaller); pairs of them are joined
    until one is left."""
    k = R.shape[0]
    while h < k:
        first = 0
        if h < 1024:                                         # pairs of two whole halves: one batched product
            pairs = k // (2 * h)

            def tiles(m, offset):
                return m.as_strided((pairs, h, h), (2 * h * (k + 1), k, 1), offset)
            if pairs:
                left = torch.bmm(tiles(X, 0), tiles(R, h))
                tiles(X, h).baddbmm_(left, tiles(X, h * (k + 1)), beta=0, alpha=-1)
            first = pairs * 2 * h
        for i in range(first, k - h, 2 * h):                 # large pairs, and a last one of unequal halves
            end, g = min(i + 2 * h, k), h // 2
            A, B, C, D = X[i:i + h, i:i + h], R[i:i + h, i + h:end], X[i + h:end, i + h:end], X[i:i + h, i + h:end]
            left = torch.empty(B.shape, dtype=B.dtype, device=B.device)
            torch.mm(A[:g], B, out=left[:g])                 # (a quarter of a triangular factor is zero)
            torch.mm(A[g:, g:], B[g:], out=left[g:])
            c = min(g, end - i - h)
            D[:, :c].addmm_(left[:, :c], C[:c, :c], beta=0, alpha=-1)
            if c < end - i - h:
                D[:, c:].addmm_(left, C[:, c:], beta=0, alpha=-1)
        h *= 2


def _upper_inverse_cuda(R: torch.Tensor) -> torch.Tensor:
    """The same on the GPU for R in 64 bits: blocks of 128 by one launch, joined by products in 64 bits.  4096 columns
    1.44 ms, 11008 21.6; as `_upper_inverse` in 32 bits 2.69 and 21.2, where the error against 64 bits is 3.7e-7 and 6.2e-7
    (here that of rounding the result, 2.6e-8).  Joined in 32 bits above 512 columns 1.06 and 13.8 ms, but with a larger error
    than that form's from about 2500 columns on (2944: 3.4e-7 and 3.3e-7, 11008: 6.7e-7)."""
    k = R.shape[0]
    R = R.contiguous()
    X = torch.zeros_like(R)
    with torch.cuda.device(R.device):                        # (any, as for the library's calls)
        check(lib().dz_triangular_inverse_blocks(R.data_ptr(), k, k, X.data_ptr(), k, _stream()), "dz_triangular_inverse_blocks")
    _join_inverses(X, R, 128)
    return X


def _only_values(t: torch.Tensor) -> bool:
    """Whether nothing is asked of `t` but its values: no gradient, tangent or level of torch.func, no subclass, mode or
    trace that follows the operations.  A kernel behind a pointer shows itself to none of those."""
    return (type(t) is torch.Tensor and not t.requires_grad and not torch._C._functorch.is_functorch_wrapped_tensor(t)
            and forward_ad.unpack_dual(t).tangent is None and _get_current_dispatch_mode() is None
            and not torch.jit.is_tracing() and not torch.compiler.is_compiling())


def _products_are_reduced(t: torch.Tensor) -> bool:
    """Whether the program lets 32-bit products of such matrices run at a lower precision (TF32, bf16)."""
    backend = torch.backends.cuda if t.is_cuda else torch.backends.mkldnn
    return t.dtype == torch.float32 and backend.matmul.fp32_precision in ("tf32", "bf16")


def hinv_factor(H: torch.Tensor, percdamp: float = 0.01) -> Tuple[torch.Tensor, torch.Tensor]:
    """Upper Cholesky factor of the damped H^-1 and the mask of dead columns (sparsegpt.py:69-88).

    With J the reversal of rows and columns and J H J = L L^T, R = J L J is upper triangular and H = R R^T, so
    H^-1 = (R^-1)^T R^-1: the factor is R^-1.  One factorisation and a triangular inverse in place of two
    factorisations and an inverse of H.  Only H's lower triangle is read.  The factorisation is in 64 bits (0.4 ms more at
    4096 columns): its rounding in 32 turned more codes that lie between two values than the two factorisations did (loss of
    a 3072-column layer against 64 bits, ten of them: those 1.2e-4, 32 bits 3.0e-4, so 9e-5; 4096 columns 2.7e-4, 3.0e-4,
    2.4e-4).  So is the inverse on the GPU (`_upper_inverse_cuda`); on the CPU, and where more than values is asked for, it is
    in H's type, but in 64 bits where 32-bit products may be TF32, which also reaches the triangular solve (factor off by
    1e-3)."""
    H = H.clone()
    dead = torch.diag(H) == 0
    H[dead, dead] = 1
    damp = percdamp * torch.mean(torch.diag(H))
    idx = torch.arange(H.shape[0], device=H.device)
    H[idx, idx] += damp
    R = torch.linalg.cholesky(H.mT.flip(0, 1).double()).flip(0, 1)
    if R.is_cuda and R.numel() and _only_values(R) and H.dtype in (torch.float32, torch.float64):
        inverse = _upper_inverse_cuda(R)
    else:
        inverse = _upper_inverse(R if _products_are_reduced(H) else R.to(H.dtype))
    return inverse.to(H.dtype).contiguous(), dead


def find_params(W: torch.Tensor, bits: int) -> Tuple[torch.Tensor, torch.Tensor]:
    """Per-row symmetric grid (scale [N], zero [N]) of W [N, K] float32."""
    n, k = W.shape
    scale = torch.empty(n, dtype=torch.float32, device=W.device)
    zero = torch.empty(n, dtype=torch.float32, device=W.device)
    check(lib().dz_quant_find_params(W.data_ptr(), n, k, bits, scale.data_ptr(), zero.data_ptr(),
                                     _stream()), "dz_quant_find_params")
    return scale, zero


def _feed_back(later: torch.Tensor, errors: torch.Tensor, U: torch.Tensor, left: torch.Tensor, right: torch.Tensor) -> None:
    """later -= errors @ U for the columns behind a block, as one product of bf16 parts (dz_split_update_rows) with sums in
    32 bits and a smaller error than a 32-bit product's; `left`, `right`: room for the parts.  4096 columns, all blocks:
    1.4 ms as 32-bit products of 512 columns, 0.7 so."""
    (n, count), c = errors.shape, later.shape[1]
    check(lib().dz_split_update_rows(errors.data_ptr(), errors.stride(0), n, count, U.data_ptr(), U.stride(0), c,
                                     later.data_ptr(), later.stride(0), left.data_ptr(), right.data_ptr(), _stream()),
          "dz_split_update_rows")
    torch.addmm(later, left[:6 * n * count].view(n, 6 * count), right[:6 * count * c].view(6 * count, c),
                alpha=-1, out_dtype=torch.float32, out=later)


def _without_slope(result: torch.Tensor, *inputs: torch.Tensor) -> torch.Tensor:
    """`result` as a function of `inputs` that is constant around them, as a value on the quantisation grid is: gradients
    of zero for those that carry one, which the kernels' writes through a pointer would not give by themselves."""
    if not torch.is_grad_enabled() or not any(t.requires_grad for t in inputs):
        return result
    tied = result + sum(t.sum() for t in inputs if t.requires_grad)
    return tied.copy_(result)


def sparsegpt_2_4(delta: torch.Tensor, bits: int, H: Optional[torch.Tensor] = None,
                  percdamp: float = 0.01, blocksize: int = 128, hinv: Optional[torch.Tensor] = None):
    """2:4-pruned, `bits`-bit quantised delta with SparseGPT error feedback.

    delta: [N, K] float32 CUDA (target weight minus base weight); H: [K, K] Hessian from
    HessianAccumulator (None = identity: no error feedback, the "keep the two largest of four"
    rule); `hinv` supplies the upper Cholesky factor of the damped H^-1 directly.  Returns (Wq float32 [N, K] on the quantisation grid, scale [N], zero [N], loss [N])."""
    if not delta.is_cuda or delta.dtype != torch.float32 or delta.dim() != 2:
        raise ValueError("delta must be a 2-D float32 CUDA tensor")
    if blocksize > 128 or blocksize % 4:
        raise ValueError("blocksize must be a multiple of 4, at most 128")
    n, k = delta.shape
    if k % 4:
        raise ValueError("K must be a multiple of 4")
    W = delta.detach().clone().contiguous()
    scale, zero = find_params(W, bits)
    if hinv is None:
        if H is None:
            H = torch.eye(k, dtype=torch.float32, device=W.device)
        hinv, dead = hinv_factor(H.to(W.device, torch.float32), percdamp)
        W[:, dead] = 0
    else:
        if hinv.shape != (k, k):
            raise ValueError(f"hinv must be [{k}, {k}]")
        hinv = hinv.to(W.device, torch.float32).contiguous()
    loss = torch.zeros(n, dtype=torch.float32, device=W.device)
    L, factor = lib(), hinv.detach()
    errors = torch.empty((n, blocksize), dtype=torch.float32, device=W.device)
    left = torch.empty(6 * n * blocksize, dtype=torch.bfloat16, device=W.device)
    right = torch.empty(6 * blocksize * k, dtype=torch.bfloat16, device=W.device)
    for i1 in range(0, k, blocksize):
        i2 = min(i1 + blocksize, k)
        count = i2 - i1
        # the quantised block takes the place of the block
        check(L.dz_sparsegpt_block_strided(
            W.data_ptr() + 4 * i1, k, factor.data_ptr() + 4 * (i1 * k + i1), k, scale.data_ptr(), zero.data_ptr(), bits,
            n, count, W.data_ptr() + 4 * i1, k, errors.data_ptr(), blocksize, loss.data_ptr(),
            _stream()), "dz_sparsegpt_block_strided")
        if i2 < k:
            _feed_back(W[:, i2:], errors[:, :count], factor[i1:i2, i2:], left, right)
    return _without_slope(W, delta, hinv), scale, zero, loss


def pack_gptq(Wq: torch.Tensor, scale: torch.Tensor, zero: torch.Tensor, bits: int):
    """(qweight int32 [K*bits/32, N], qzeros int32 [1, N*bits/32], scales fp16 [1, N])."""
    n, k = Wq.shape
    per = 32 // bits
    qweight = torch.empty((k // per, n), dtype=torch.int32, device=Wq.device)
    qzeros = torch.empty((1, n // per), dtype=torch.int32, device=Wq.device)
    scales = torch.empty((1, n), dtype=torch.float16, device=Wq.device)
    check(lib().dz_pack_gptq(Wq.contiguous().data_ptr(), scale.data_ptr(), zero.data_ptr(), n, k, bits,
                             qweight.data_ptr(), qzeros.data_ptr(), scales.data_ptr(), _stream()),
          "dz_pack_gptq")
    return qweight, qzeros, scales


def compress_delta(delta: torch.Tensor, bits: int, H: Optional[torch.Tensor] = None,
                   percdamp: float = 0.01):
    """delta [N, K] float32 -> GPTQ-layout tensors of the compressed delta (and the per-row
    loss); `ops.convert_from_gptq` turns them into slot layout."""
    Wq, scale, zero, loss = sparsegpt_2_4(delta, bits, H, percdamp)
    return pack_gptq(Wq, scale, zero, bits) + (loss,)

"""The slab-fed tcgen05 GEMM of long overlapping views, at its edges.

fp32 sums of exact bf16 products (K / 16 tensor-core additions, each within
2^-22 of the magnitudes summed), rounded to bf16 (2^-8 of the value)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
FIRST = 512 * 148          # rows from which the slab kernel is taken on 148 SMs


@pytest.mark.parametrize("M", [FIRST, FIRST + 1, FIRST + 129, FIRST + 255, 3 * FIRST + 300])
@pytest.mark.parametrize("lda,taps", [(256, 5), (64, 2), (128, 9), (192, 3)])
def test_slab_gemm_matches_64_bit_rows(M, lda, taps):
    from sseqs_b200 import _lib, learned
    g = torch.Generator(device="cuda")
    g.manual_seed(M + lda + taps)
    K, N = lda * taps, 256
    X = torch.randn(M + taps - 1, lda, generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    res = torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device="cuda")
    mask = (torch.rand(M, generator=g, device="cuda") > 0.2).to(torch.uint8)
    plain = torch.full((M + 1, N), 3, dtype=torch.bfloat16, device="cuda")
    fused, Z = (torch.zeros(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    learned._gemm(0, 0, learned._EPI_BF16, M, N, K, X.data_ptr(), lda, B.data_ptr(), K,
                  plain.data_ptr(), N)
    learned._gemm(0, 0, learned._EPI_BIAS_GELU_RES, M, N, K, X.data_ptr(), lda, B.data_ptr(), K,
                  fused.data_ptr(), N, Z.data_ptr(), bias, None, mask, res.data_ptr())
    torch.cuda.synchronize()
    flag = ctypes.c_int(-1)
    _lib.check(_lib.lib().sseqs_gemm_error(ctypes.byref(flag)))
    assert flag.value == 0
    assert (plain[M] == 3).all()                       # nothing past the last row
    # rows of the first, some middle and the last tiles
    rows = torch.cat([torch.arange(0, 700), torch.arange(M // 2, M // 2 + 700),
                      torch.arange(M - 700, M)]).cuda()
    A = torch.as_strided(X, (M, K), (lda, 1))[rows].double()
    exp = A @ B.double().T
    size = A.abs() @ B.double().abs().T
    tol = 2.0 ** -8 * exp.abs() + K / 16 * 2.0 ** -22 * size
    assert ((plain[rows].double() - exp).abs() <= tol).all()
    z = torch.where(mask[rows].bool()[:, None], exp + bias.double(), 0.0)
    assert ((Z[rows].double() - z).abs() <= tol + 2.0 ** -8 * (z.abs() + 1e-30)).all()
    zb = Z[rows].float()
    y = torch.nn.functional.gelu(zb, approximate="tanh") + res[rows].float()
    y = torch.where(mask[rows].bool()[:, None], y, 0.0)
    # tanh.approx is within 2^-10.9 of tanh; the sum is rounded to bf16
    assert ((fused[rows].float() - y).abs() <= 2.0 ** -8 * y.abs() + 2.0 ** -11 * zb.abs() +
            1e-6).all()


@pytest.mark.parametrize("M", [1000, FIRST + 129])
@pytest.mark.parametrize("lda,K", [(128, 192), (64, 64), (192, 256), (0, 128), (8, 320)])
def test_other_row_views_match_64_bits(M, lda, K):
    """Views whose last row ends inside its slab (the operand ends with the
    buffer), one row for every output (lda = 0), rows 8 elements apart."""
    from sseqs_b200 import learned
    g = torch.Generator(device="cuda")
    g.manual_seed(M + lda + K)
    X = torch.randn((M - 1) * lda + K, generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn(256, K, generator=g, device="cuda").to(torch.bfloat16)
    C = torch.zeros(M, 256, dtype=torch.bfloat16, device="cuda")
    learned._gemm(0, 0, learned._EPI_BF16, M, 256, K, X.data_ptr(), lda, B.data_ptr(), K,
                  C.data_ptr(), 256)
    A = torch.as_strided(X, (M, K), (lda, 1)).double()
    exp, size = A @ B.double().T, A.abs() @ B.double().abs().T
    tol = 2.0 ** -8 * exp.abs() + K / 16 * 2.0 ** -22 * size
    assert ((C.double() - exp).abs() <= tol).all()


def _gelu_and_grad(z):
    """GELU (tanh form) and its derivative of z, with bounds on what a tanh within
    2^-10.9 moves them by."""
    z = z.double()
    t = torch.tanh(0.7978845608 * (z + 0.044715 * z ** 3))
    slope = 0.7978845608 * (1 + 0.134145 * z * z)
    dt = 2.0 ** -10.9
    return (0.5 * z * (1 + t), 0.5 * z.abs() * dt,
            0.5 * (1 + t) + 0.5 * z * (1 - t * t) * slope, dt * (0.5 + z.abs() * slope))


@pytest.mark.parametrize("M", [FIRST + 129, 2 * FIRST])
@pytest.mark.parametrize("epi", [2, 3, 5, 6])
def test_slab_gemm_epilogues_match_64_bit_rows(M, epi):
    """Every fused epilogue of the slab kernel, at the embedder's K = 5 x 256: GELU
    (2), GELU with residual (5) and the two gradients (3, 6), with masked rows.  A
    second output that the epilogue rounds first (2, 5, 6) is checked against 64
    bits, and what follows from it against its own values."""
    from sseqs_b200 import _lib, learned
    g = torch.Generator(device="cuda")
    g.manual_seed(M + epi)
    lda, taps, N = 256, 5, 256
    K = lda * taps
    X = (0.2 * torch.randn(M + taps - 1, lda, generator=g, device="cuda")).to(torch.bfloat16)
    B = (0.2 * torch.randn(N, K, generator=g, device="cuda")).to(torch.bfloat16)
    res, aux = (torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    bias = torch.randn(N, generator=g, device="cuda")
    mask = (torch.rand(M, generator=g, device="cuda") > 0.2).to(torch.uint8)
    C, C2 = (torch.full((M + 1, N), 3, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    learned._gemm(0, 0, epi, M, N, K, X.data_ptr(), lda, B.data_ptr(), K, C.data_ptr(), N,
                  None if epi == 3 else C2.data_ptr(), bias if epi in (2, 5) else None,
                  aux.data_ptr() if epi in (3, 6) else None, mask,
                  res.data_ptr() if epi in (5, 6) else None)
    torch.cuda.synchronize()
    flag = ctypes.c_int(-1)
    _lib.check(_lib.lib().sseqs_gemm_error(ctypes.byref(flag)))
    assert flag.value == 0
    assert (C[M] == 3).all() and (C2[M] == 3).all()
    rows = torch.cat([torch.arange(0, 700), torch.arange(M // 2, M // 2 + 700),
                      torch.arange(M - 700, M)]).cuda()
    keep = mask[rows].bool()[:, None]
    A = torch.as_strided(X, (M, K), (lda, 1))[rows].double()
    acc = A @ B.double().T
    acc_tol = K / 16 * 2.0 ** -22 * (A.abs() @ B.double().abs().T)
    got = C[rows].double()
    if epi == 3:
        _, _, gg, gg_tol = _gelu_and_grad(aux[rows])
        exp, tol = acc * gg, acc.abs() * gg_tol + acc_tol * (gg.abs() + gg_tol)
    else:
        first = acc + (res[rows].double() if epi == 6 else bias.double())
        z = C2[rows].double()
        assert ((z - torch.where(keep, first, 0.0)).abs()
                <= acc_tol + 2.0 ** -8 * first.abs() + 1e-30).all()
        if epi == 6:
            _, _, gg, gg_tol = _gelu_and_grad(aux[rows])
            exp, tol = z * gg, z.abs() * gg_tol
        else:
            exp, tol, _, _ = _gelu_and_grad(z)
            if epi == 5:
                exp = exp + res[rows].double()
    exp = torch.where(keep, exp, 0.0)
    assert ((got - exp).abs() <= tol + 2.0 ** -8 * exp.abs() + 1e-6).all()

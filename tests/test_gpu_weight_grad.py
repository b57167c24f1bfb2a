"""The tcgen05 weight-gradient GEMM and the first layer's gradients.

Products of bf16 values are exact in fp32; what can be off is the order and
rounding of the additions: tensor-core sums of 16 products, K / 16 of them a
split, then at most 148 splits, each within 2^-23 of the magnitudes summed."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,lda,K", [
    (1280, 256, 64), (1280, 256, 96), (1280, 256, 4128), (1280, 256, 20_000), (640, 128, 1056),
    (320, 64, 352), (256, 256, 64), (8, 8, 64), (264, 272, 9504), (40, 48, 160),
])
def test_weight_gradient_matches_64_bits(M, lda, K):
    """Plain [K][M] operands (lda >= M) and the convolutions' overlapping
    rows (lda < M); ragged M and K; added to what C holds."""
    from sseqs_b200 import learned
    g = torch.Generator(device="cuda")
    g.manual_seed(M + K)
    rows = K + (M - 1) // lda + 1
    buf = torch.randn(rows, lda, generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn(K, 256, generator=g, device="cuda").to(torch.bfloat16)
    C0 = torch.randn(M, 256, generator=g, device="cuda")
    C = C0.clone()
    learned._gemm(1, 1, learned._EPI_F32_ADD, M, 256, K, buf.data_ptr(), lda, B.data_ptr(), 256,
                  C.data_ptr(), 256)
    A = torch.as_strided(buf, (K, M), (lda, 1)).double()
    exp = C0.double() + A.T @ B.double()
    size = C0.double().abs() + A.abs().T @ B.double().abs()
    tol = (K / 16 + 150) * 2.0 ** -23 * size
    assert ((C.double() - exp).abs() <= tol).all()


@pytest.mark.parametrize("P", [1, 2, 63, 64, 65, 2049, 50_000])
def test_first_layer_gradients_match_64_bits(P):
    from sseqs_b200 import _lib
    g = torch.Generator(device="cuda")
    g.manual_seed(P)
    cin = 32
    cls = torch.randint(0, 24, (P,), generator=g, device="cuda", dtype=torch.uint8)
    cls[cls >= 21] = 255
    dZ = torch.randn(P, 256, generator=g, device="cuda").to(torch.bfloat16)
    E = torch.randn(21, cin, generator=g, device="cuda").to(torch.bfloat16)
    W = torch.randn(256, 5, cin, generator=g, device="cuda").to(torch.bfloat16)
    Wf = W.flip(1).permute(2, 1, 0).contiguous()
    G = torch.empty(5 * 21 * 256, device="cuda")
    dWT = torch.zeros(5 * cin, 256, device="cuda")
    dE = torch.zeros(21, cin, device="cuda")
    _lib.check(_lib.lib().sseqs_embed_conv1_grad(
        _lib.ptr(cls), P, _lib.ptr(dZ), 256, _lib.ptr(E), cin, _lib.ptr(Wf), _lib.ptr(G),
        _lib.ptr(dWT), _lib.ptr(dE), _lib.stream_ptr()))
    pad = torch.full((2,), 255, dtype=torch.uint8, device="cuda")
    c = torch.cat([pad, cls, pad]).long()
    one = torch.nn.functional.one_hot(c.clamp(max=21), 22)[:, :21].double()
    exp_w, size_w = [], []
    exp_e = torch.zeros(21, cin, dtype=torch.float64, device="cuda")
    size_e = torch.zeros_like(exp_e)
    for t in range(5):
        h, z = one[t:t + P], dZ.double()            # cls[p - 2 + t]
        S, A = h.T @ z, h.T @ z.abs()               # [21, 256]
        exp_w.append(E.double().T @ S)
        size_w.append(E.double().abs().T @ A)
        exp_e += S @ W[:, t].double()
        size_e += A @ W[:, t].double().abs()
    # P additions to a class, the blocks' sums, then 21 or 1280 products
    rel = (P + 300) * 2.0 ** -24
    assert ((dWT.double() - torch.cat(exp_w)).abs()
            <= (rel + 21 * 2.0 ** -23) * torch.cat(size_w)).all()
    assert ((dE.double() - exp_e).abs() <= (rel + 1280 * 2.0 ** -23) * size_e).all()


@pytest.mark.parametrize("M,lda,K", [(72, 64, 64), (136, 128, 96), (320, 256, 1056), (64, 0, 96),
                                     (256, 8, 128)])
def test_other_row_views_match_64_bits(M, lda, K):
    """Views whose last row ends inside its slab (the operand ends with the
    buffer, which holds no byte more), one row for every position (lda = 0), and
    rows 8 elements apart."""
    from sseqs_b200 import learned
    g = torch.Generator(device="cuda")
    g.manual_seed(M + lda + K)
    buf = torch.randn((K - 1) * lda + M, generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn(K, 256, generator=g, device="cuda").to(torch.bfloat16)
    C = torch.zeros(M, 256, device="cuda")
    learned._gemm(1, 1, learned._EPI_F32_ADD, M, 256, K, buf.data_ptr(), lda, B.data_ptr(), 256,
                  C.data_ptr(), 256)
    A = torch.as_strided(buf, (K, M), (lda, 1)).double()
    exp, size = A.T @ B.double(), A.abs().T @ B.double().abs()
    assert ((C.double() - exp).abs() <= (K / 16 + 150) * 2.0 ** -23 * size).all()

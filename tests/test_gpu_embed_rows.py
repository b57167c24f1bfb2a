"""Row kernels of the embedder at the edges of their blocks: the 256-channel
forms against the general ones of the same entry points (taken for operands
that are not 16-byte aligned) and against 64-bit sums."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
D = 256


def _off(t, shift):
    """A copy of ``t`` that starts ``shift`` elements into its allocation."""
    buf = torch.empty(t.numel() + 64, dtype=t.dtype, device="cuda")
    v = buf[shift:shift + t.numel()].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("P", [1, 2, 31, 32, 33, 512, 513, 40_000])
@pytest.mark.parametrize("masked", [False, True])
def test_conv1_table_forms_agree(P, masked):
    from sseqs_b200 import _lib
    g = torch.Generator(device="cuda")
    g.manual_seed(P)
    cls = torch.randint(0, 23, (P,), generator=g, device="cuda", dtype=torch.uint8)
    cls[cls >= 21] = 255
    T = torch.randn(5, 21, D, generator=g, device="cuda")
    bias = torch.randn(D, generator=g, device="cuda")
    mask = (torch.rand(P, generator=g, device="cuda") > 0.3).to(torch.uint8) if masked else None
    outs = []
    for shift in (0, 1):            # a bias off the 16-byte grid takes the general form
        b = _off(bias, shift)
        Y = torch.full((P, D), 7, dtype=torch.bfloat16, device="cuda")
        Z = torch.full((P, D), 7, dtype=torch.bfloat16, device="cuda")
        _lib.check(_lib.lib().sseqs_embed_conv1_table(
            _lib.ptr(cls), P, _lib.ptr(T), _lib.ptr(b), _lib.ptr(mask), D, _lib.ptr(Y),
            _lib.ptr(Z), _lib.stream_ptr()))
        outs.append((Y, Z))
    # the same sums in the same order
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


LENS = [0, 1, 7, 8, 9, 31, 32, 33, 100, 1000, 2048]


def _rows(seed):
    lens = torch.tensor(LENS, dtype=torch.int32, device="cuda")
    start = torch.cumsum(lens.to(torch.int64) + 2, 0) - lens
    P = int(start[-1]) + LENS[-1] + 2
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return lens, start, P, g


@pytest.mark.parametrize("shift", [0, 1])
def test_pool_normalize_sums_rows(shift):
    from sseqs_b200 import _lib
    lens, start, P, g = _rows(1)
    Y = _off(torch.randn(P, D, generator=g, device="cuda").to(torch.bfloat16), shift)
    S = lens.numel()
    pooled, emb = (torch.empty(S, D, device="cuda") for _ in range(2))
    inv = torch.empty(S, device="cuda")
    _lib.check(_lib.lib().sseqs_pool_normalize(
        _lib.ptr(Y), D, _lib.ptr(start), _lib.ptr(lens), S, _lib.ptr(pooled), _lib.ptr(emb),
        _lib.ptr(inv), _lib.stream_ptr()))
    for s, n in enumerate(LENS):
        y = Y[int(start[s]):int(start[s]) + n].double()
        exp = y.sum(0) / max(n, 1)
        # n additions in 32 bits, one division
        tol = (n + 2) * 2.0 ** -24 * y.abs().sum(0) / max(n, 1) + 1e-12
        assert ((pooled[s].double() - exp).abs() <= tol).all(), n


@pytest.mark.parametrize("with_g", [False, True])
def test_pool_backward_forms_agree(with_g):
    from sseqs_b200 import _lib
    lens, start, P, g = _rows(2)
    S = lens.numel()
    Z = torch.randn(P, D, generator=g, device="cuda").to(torch.bfloat16)
    emb, dE = (torch.randn(S, D, generator=g, device="cuda") for _ in range(2))
    inv = torch.rand(S, generator=g, device="cuda")
    outs = []
    for shift in (0, 1):
        z = _off(Z, shift)
        dZ, G = (torch.zeros(P, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        _lib.check(_lib.lib().sseqs_pool_backward(
            _lib.ptr(emb), _lib.ptr(dE), _lib.ptr(inv), _lib.ptr(start), _lib.ptr(lens), S, D,
            _lib.ptr(z), _lib.ptr(dZ), _lib.ptr(G) if with_g else None, _lib.stream_ptr()))
        outs.append((dZ, G))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("P,D,both", [(1, 256, True), (31, 256, False), (33, 8, True),
                                      (5000, 256, True)])
def test_zero_rows(P, D, both):
    from sseqs_b200 import _lib
    g = torch.Generator(device="cuda")
    g.manual_seed(P)
    mask = (torch.rand(P, generator=g, device="cuda") > 0.4).to(torch.uint8)
    a, b = (torch.ones(P + 1, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    _lib.check(_lib.lib().sseqs_zero_rows(_lib.ptr(mask), P, D, _lib.ptr(a),
                                          _lib.ptr(b) if both else None, _lib.stream_ptr()))
    want = torch.cat([mask, mask.new_ones(1)])[:, None].expand(P + 1, D).to(torch.bfloat16)
    assert torch.equal(a, want)
    assert torch.equal(b, want if both else torch.ones_like(b))

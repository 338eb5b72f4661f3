"""Linear layers of more than 256 rows on pairs of CTAs (gemm_pair.cu): ragged rows, a last weight tile that is mostly padding,
few pairs with tiles cut along K, two bands of token tiles; against 64 bits.  fp32 sums of K products in some order: 8 K ulp of
2^-24 of the sum of magnitudes; half a bf16 step (2^-9, relative) for the store.  The gated form rounds both projections to bf16
first, and one on the edge of a step may go to its other side, 2^-8 relative: the gate's moves the product by at most
2^-8 |gate| max|silu'| |up| (max|silu'| < 1.1), the up projection's by 2^-8 of it; store and approximate exponential stay within
another 2^-8.  A projection near zero carries the sums' absolute error instead."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 31 + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    return x, w, torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("M,N,K,grid", [
    (257, 256, 64, 0), (257, 129, 128, 0), (300, 1000, 512, 0), (333, 2048, 2048, 0), (511, 768, 192, 3), (513, 256, 4096, 0),
    (1000, 4608, 1024, 37), (777, 5120, 448, 0), (2049, 4096, 64, 0), (4100, 1280, 256, 0), (1024, 1280, 11008, 0)])
def test_product(M, N, K, grid):
    import cpmcu.C as C
    x, w, b = operands(M, N, K)
    ref = x.double() @ w.double().t()
    room = 8 * K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    for bias in (None, b):
        want = ref if bias is None else ref + bias.double()
        for _ in range(2):   # the counters of cut tiles are left as they were found
            y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
            C.call("cpmcu_linear_bf16", ptr(x), ptr(w), ptr(bias), ptr(y), M, N, K, grid)
            assert bool(((y.double() - want).abs() <= room + 2.0 ** -8 * want.abs()).all())


@pytest.mark.parametrize("M,inter,K", [(257, 128, 64), (600, 1408, 576), (1500, 8192, 256), (4096, 2944, 128)])
def test_gated_product(M, inter, K):
    import cpmcu.C as C
    x, w, _ = operands(M, 2 * inter, K)
    y = torch.full((M, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    C.call("cpmcu_linear_swiglu_bf16", ptr(x), ptr(w), ptr(y), M, inter, K, 0)
    p = (x.double() @ w.double().t()).to(torch.bfloat16).double()
    gate, up = p[:, :inter], p[:, inter:]
    ref = gate * torch.sigmoid(gate) * up
    room = 8 * K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    room = room[:, :inter] * 1.1 * up.abs() + room[:, inter:] * gate.abs()
    assert bool(((y.double() - ref).abs() <= room + 2.0 ** -8 * (1.1 * (gate * up).abs() + 2 * ref.abs())).all())

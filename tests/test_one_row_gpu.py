"""Products of one token row (one_row.cu) at the sizes where the division of the rows and of K changes, against 64 bits.

The kernel's sums are fp32 products in some order: 8 K ulp of 2^-24 of the sum of magnitudes bounds that, the bf16 store adds
half a step (2^-9 relative).  The gated form rounds both projections to bf16 first (as the tensor-core path does), and one on the
edge of a step may go to its other side, 2^-8 relative: the gate's moves the product by at most 2^-8 |gate| max|silu'| |up|
(max|silu'| < 1.1), the up projection's by 2^-8 of it; store and approximate exponential stay within another 2^-8.  A projection near zero carries the sums' absolute error instead."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def operands(rows, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(rows, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    return x, w, torch.randn(rows, generator=g, device="cuda").to(torch.bfloat16)


def check(y, x, w, bias=None):
    ref = w.double() @ x.double()
    room = 8 * x.numel() * 2.0 ** -24 * (w.double().abs() @ x.double().abs())
    if bias is not None:
        ref = ref + bias.double()
    assert bool(((y.double() - ref).abs() <= room + 2.0 ** -8 * ref.abs()).all())


@pytest.mark.parametrize("N", [1, 5, 127, 129, 1476, 1484, 2964, 5920, 5936, 73448])
@pytest.mark.parametrize("K", [64, 448, 512, 576, 2112])
def test_product(N, K):
    import cpmcu.C as C
    x, w, b = operands(N, K, N * 7 + K)
    for bias in (None, b):
        y = torch.full((N,), float("nan"), dtype=torch.bfloat16, device="cuda")
        C.call("cpmcu_linear_bf16", ptr(x), ptr(w), ptr(bias), ptr(y), 1, N, K, 0)
        check(y, x, w, bias)


# where the tiles keep up (three CTAs on some SMs, two on others, long rows), and just beside that
@pytest.mark.parametrize("N,K", [(5120, 13824), (5376, 11008), (5632, 11072), (4900, 11008), (5888, 11008), (5376, 10944), (9472, 256), (9473, 256), (4736, 128), (4737, 128)])
def test_product_of_few_and_many_ctas(N, K):
    test_product(N, K)


@pytest.mark.parametrize("inter", [64, 192, 1472, 2944, 3008])
@pytest.mark.parametrize("K", [64, 576, 1024])
def test_gated_product(inter, K):
    import cpmcu.C as C
    x, w, _ = operands(2 * inter, K, inter + K)
    y = torch.full((inter,), float("nan"), dtype=torch.bfloat16, device="cuda")
    C.call("cpmcu_linear_swiglu_bf16", ptr(x), ptr(w), ptr(y), 1, inter, K, 0)
    p = (w.double() @ x.double()).to(torch.bfloat16).double()
    ref = p[:inter] * torch.sigmoid(p[:inter]) * p[inter:]
    room = 8 * K * 2.0 ** -24 * (w.double().abs() @ x.double().abs())
    room = room[:inter] * 1.1 * p[inter:].abs() + room[inter:] * p[:inter].abs()
    assert bool(((y.double() - ref).abs() <= room + 2.0 ** -8 * (1.1 * (p[:inter] * p[inter:]).abs() + 2 * ref.abs())).all())


@pytest.mark.parametrize("n,N,N_s", [(1, 64, 0), (4, 256, 64), (3, 200, 72), (4, 1536, 64)])
def test_grouped_product(n, N, N_s):
    import cpmcu.C as C
    K, ldy = 320, max(N, N_s)
    g = torch.Generator(device="cuda").manual_seed(n + N)
    x = torch.randn(n + (N_s > 0), K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n * N + N_s, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    y = torch.full((x.shape[0], ldy), float("nan"), dtype=torch.bfloat16, device="cuda")
    C.call("cpmcu_grouped_linear", x.data_ptr(), w.data_ptr(), n, N, N_s, K, 1, ldy, y.data_ptr())
    for i in range(n):
        check(y[i, :N], x[i], w[i * N:(i + 1) * N])
    if N_s > 0:
        check(y[n, :N_s], x[n], w[n * N:])

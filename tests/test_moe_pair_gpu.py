"""Grouped products on pairs of CTAs (moe.cu: groups of 128 or 256 rows, an even number of 128-feature tiles per matrix) at the row counts
where the halves of a group change (columns are rounded up to 32, each CTA fetches half of them in boxes of 64), with an odd tile of
the extra matrix, and beside them matrices of an odd number of tiles (single CTAs); against 64 bits.

Sums of fp32 products in some order are within 8 K ulp of 2^-24 of the sum of magnitudes, the bf16 store adds half a step."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,N,N_s", [(4, 256, 64), (2, 512, 0), (3, 200, 300), (2, 384, 64), (1, 2048, 72)])
@pytest.mark.parametrize("rows", [65, 72, 88, 128, 129, 137, 255, 256, 257, 385, 520])
def test_grouped_product(n, N, N_s, rows):
    import cpmcu.C as C
    K, ldy = 448, (max(N, N_s) + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(n + N + rows)
    parts = n + (N_s > 0)
    x = torch.randn(parts * rows, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n * N + N_s, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    y = torch.full((parts * rows, ldy), float("nan"), dtype=torch.bfloat16, device="cuda")
    C.call("cpmcu_grouped_linear", x.data_ptr(), w.data_ptr(), n, N, N_s, K, rows, ldy, y.data_ptr())
    for i in range(parts):
        xi, wi = x[i * rows:(i + 1) * rows].double(), w[i * N:i * N + (N if i < n else N_s)].double()
        got, ref = y[i * rows:(i + 1) * rows, :wi.shape[0]].double(), xi @ wi.t()
        room = 8 * K * 2.0 ** -24 * (xi.abs() @ wi.abs().t()) + 2.0 ** -8 * ref.abs()
        assert bool(((got - ref).abs() <= room).all()), i
        assert bool(y[i * rows:(i + 1) * rows, wi.shape[0]:].isnan().all())   # nothing beyond a matrix's own outputs

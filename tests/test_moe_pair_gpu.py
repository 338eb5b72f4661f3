"""Grouped products on pairs of CTAs (moe.cu: groups of 128 or 256 rows, an even number of 128-feature tiles per matrix, enough of them) at the row
counts where the halves of a group change (columns are rounded up to 32, each CTA fetches half of them in boxes of 64), with an odd tile of
the extra matrix, and beside them launches that stay with single CTAs: an odd number of tiles, short rows; against 64 bits.

Sums of fp32 products in some order are within 8 K ulp of 2^-24 of the sum of magnitudes, the bf16 store adds half a step."""
import ctypes

import pytest
import torch

from oracle import tipetar as T
from test_tipetar_gpu import gen, pad64, padded, spec_of
from tipetar_cases import attn, model, moe

pytestmark = pytest.mark.gpu


def on_pairs(tile, n_tiles, kblocks, tiles):
    import cpmcu.C as C
    return C.call("cpmcu_debug_moe_pairs", tile, n_tiles, kblocks, tiles, torch.cuda.get_device_properties(0).multi_processor_count) == 1


def product(n, N, N_s, K, rows, pairs):
    import cpmcu.C as C
    tile = next(t for t in (16, 32, 64, 128, 256) if t >= min(rows, 256))
    groups, n_tiles = -(-rows // tile), -(-N // 128)
    assert on_pairs(tile, n_tiles, K // 64, groups * (n * n_tiles + -(-N_s // 128))) == pairs
    ldy = (max(N, N_s) + 7) // 8 * 8
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


@pytest.mark.parametrize("n,N,N_s", [(4, 256, 64), (2, 512, 0), (3, 200, 300), (2, 384, 64), (1, 2048, 72)])
@pytest.mark.parametrize("rows", [65, 72, 88, 128, 129, 137, 255, 256, 257, 385, 520])
def test_grouped_product(n, N, N_s, rows):
    product(n, N, N_s, 448, rows, False)


@pytest.mark.parametrize("n,N,N_s", [(4, 5120, 64), (2, 9728, 0), (1, 19200, 300)])
@pytest.mark.parametrize("rows", [129, 137, 160, 255, 256, 257, 288, 289, 385, 520])
def test_grouped_product_on_pairs(n, N, N_s, rows):
    product(n, N, N_s, 1088, rows, True)


@pytest.mark.parametrize("rows", [65, 72, 88, 96, 97, 127, 128])
def test_grouped_product_small_groups(rows):
    product(5, 16384, 72, 4160, rows, True)


@pytest.mark.parametrize("width,mlp,rows,tile", [(1280, moe(4, 2, 2048, identity=1, shared=1088), 1500, 256), (1280, moe(3, 3, 2176), 640, 256),
                                                 (4096, moe(8, 1, 2816, shared=64), 800, 128)])
def test_mixture_on_pairs(width, mlp, rows, tile):
    """Gate/up with the SwiGLU epilogue, and down, on pairs, as test_mixture of the layer's other sizes but with the oracle's 64 bits on the GPU."""
    import cpmcu.C as C
    r, ff, ld, eps, m = mlp["router"], mlp["expert"]["ff"], pad64(width), 1e-3, 0.8
    slots = rows * min(r["top"], r["experts"])
    entries = min(slots, slots // tile + r["experts"])
    assert on_pairs(tile, pad64(ff) // 64, ld // 64, entries * (pad64(ff) // 64))
    cfg = model(width, 16, [(attn(1, 1, 8, 8, 4), mlp)])
    w = {k: v.cuda() for k, v in T.random_weights(cfg, seed=rows).items() if ".mlp." in k or "norm2" in k}
    x = torch.randn(rows, width, generator=gen(rows + width)).bfloat16().double().cuda()
    y = T.mixture(x, mlp, w, "l0.mlp")
    ref = x + m * T.norm_around_one(y, w["l0.norm2"], eps)
    names = [f"e{e}" for e in range(r["experts"])] + (["shared"] if mlp["shared"] else [])
    gu = torch.cat([torch.cat([w[f"l0.mlp.{n}.gate"], w[f"l0.mlp.{n}.up"]]).flatten() for n in names]).bfloat16()
    dn = torch.cat([w[f"l0.mlp.{n}.down"].flatten() for n in names]).bfloat16()
    xc, xh = padded(x, ld, torch.float32), padded(x, ld, torch.bfloat16)
    rt, nw = padded(w["l0.mlp.router"], ld, torch.bfloat16), padded(w["l0.norm2"], ld, torch.bfloat16)
    cc = w["l0.mlp.correction"].float()
    C.call("cpmcu_layer_mixture", ctypes.byref(spec_of(mlp=mlp)), xc.data_ptr(), xh.data_ptr(), rt.data_ptr(), cc.data_ptr(), gu.data_ptr(),
           dn.data_ptr(), m, nw.data_ptr(), rows, width, ld, eps)
    got = xc[:, :width].double()
    corr = w.get("l0.mlp.correction")
    clear = T.choice_margin((x @ w["l0.mlp.router"].T).cpu(), None if corr is None else corr.cpu(), r).cuda() > 1e-3   # not decided by a score's last bits
    assert clear.double().mean() > 0.5
    assert (got - ref)[clear].abs().max() < 0.06, (got - ref)[clear].abs().max()
    assert (got - ref)[clear].pow(2).mean().sqrt() < 0.006
    assert torch.equal(xh, xc.bfloat16())

"""The q, k, v product of one token row with rotation and cache append in its epilogue (one_row.cu), against the plain product and
the rotation in 64 bits: 8 and 16 rows per CTA (up to and beyond 4736 outputs), one key
head and many, positions far out, a cache without room and a
row that is not valid.  The product is the same kernel's (equal sums); the angle is the fp32 product of position and frequency, sine, cosine and
the two products are fp32 (1e-6), the result one bf16 step of the larger operand (2^-8)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("hq,hkv,K,pos", [(1, 1, 64, 0), (2, 1, 256, 5), (16, 4, 2048, 1999), (33, 2, 576, 30000), (40, 4, 320, 777), (64, 64, 128, 1 << 20)])
def test_qkv_rope_row(hq, hkv, K, pos):
    import cpmcu.C as C
    g = torch.Generator(device="cuda").manual_seed(hq + K)
    N, rows, at = (hq + 2 * hkv) * 128, 64, 37
    x = torch.randn(1, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    inv_freq = (10000.0 ** (-torch.arange(0, 128, 2, device="cuda", dtype=torch.float64) / 128)).float()
    p, n = (torch.tensor([v], dtype=torch.int32, device="cuda") for v in (pos, at + 3))
    plain = torch.empty(1, N, dtype=torch.bfloat16, device="cuda")
    C.call("cpmcu_linear_bf16", ptr(x), ptr(w), None, ptr(plain), 1, N, K, 0)
    before = plain.double().view(hq + 2 * hkv, 128)
    angle = (p.float() * inv_freq).double()
    lo, hi = before[:hq + hkv, :64], before[:hq + hkv, 64:]
    ref = torch.cat([lo * angle.cos() - hi * angle.sin(), hi * angle.cos() + lo * angle.sin()], dim=-1)
    room = 2.0 ** -8 * ref.abs() + 1e-6 * (lo.abs() + hi.abs()).repeat(1, 2)

    def run(valid, cache_rows, kc, vc):
        q = torch.full((hq * 128,), float("nan"), dtype=torch.bfloat16, device="cuda")
        C.call("cpmcu_qkv_rope_row", ptr(x), ptr(w), K, hq, hkv, ptr(inv_freq), ptr(p), ptr(n), -3, ptr(valid), cache_rows, ptr(q), ptr(kc), ptr(vc))
        assert bool(((q.double().view(hq, 128) - ref[:hq]).abs() <= room[:hq]).all())

    def caches():
        return [torch.zeros(rows, hkv, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2)]

    for valid in (None, torch.tensor([1], dtype=torch.int32, device="cuda")):
        kc, vc = caches()
        run(valid, at + 1, kc, vc)
        assert bool(((kc[at].double() - ref[hq:]).abs() <= room[hq:]).all()) and torch.equal(vc[at].double(), before[hq + hkv:])
        kc[at] = vc[at] = 0
        assert float(kc.abs().max()) == 0.0 and float(vc.abs().max()) == 0.0
    kc, vc = caches()
    run(torch.tensor([0], dtype=torch.int32, device="cuda"), rows, kc, vc)
    assert float(kc.abs().max()) == 0.0 and float(vc.abs().max()) == 0.0
    # beyond the cache: the error word says so, and nothing is stored (the caches hold 64 rows, so a stray row would lie in them)
    kc, vc = caches()
    with pytest.raises(RuntimeError, match="error flags 8 "):
        run(None, at, kc, vc)
    assert float(kc.abs().max()) == 0.0 and float(vc.abs().max()) == 0.0

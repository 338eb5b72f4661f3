"""Rotation and cache append at the sizes where a row's elements are dealt differently: fewer items than a head has angles, one more
than a CTA's threads, several per thread; and a key cache that 16-byte stores do not fit.  The angle is the fp32 product of position
and frequency; sine, cosine and the two products are fp32 (1e-6), the result one bf16 step of the larger operand (2^-8)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("rows,hq,hkv,shift", [(1, 1, 1, 0), (3, 4, 1, 0), (60, 32, 2, 0), (7, 63, 1, 0), (5, 64, 1, 0), (2, 120, 24, 0), (9, 32, 2, 2)])
def test_rope_append(rows, hq, hkv, shift):
    import cpmcu.C as C
    d, budget, start = 128, 256, 37
    g = torch.Generator(device="cuda").manual_seed(rows + hq)
    qkv = torch.randn(rows, (hq + 2 * hkv) * d, generator=g, device="cuda").to(torch.bfloat16)
    before = qkv.double().view(rows, -1, d)
    inv_freq = (10000.0 ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d)).float()
    pos = torch.randint(0, 30000, (rows,), generator=g, device="cuda", dtype=torch.int32)
    kc = torch.zeros(budget * hkv * d + 8, dtype=torch.bfloat16, device="cuda")[shift:]
    vc = torch.zeros(budget, hkv * d, dtype=torch.bfloat16, device="cuda")
    kv_len = torch.tensor([start + 3], dtype=torch.int32, device="cuda")
    C.call("cpmcu_rope_append", ptr(qkv), rows, hq, hkv, ptr(inv_freq), ptr(pos), ptr(kc), ptr(vc), ptr(kv_len), -3)
    angle = (pos.float()[:, None] * inv_freq).double()[:, None]
    lo, hi = before[:, :hq + hkv, :d // 2], before[:, :hq + hkv, d // 2:]
    ref = torch.cat([lo * angle.cos() - hi * angle.sin(), hi * angle.cos() + lo * angle.sin()], dim=-1)
    room = 2.0 ** -8 * ref.abs() + 1e-6 * (lo.abs() + hi.abs()).repeat(1, 1, 2)
    assert bool(((qkv.double().view(rows, -1, d)[:, :hq] - ref[:, :hq]).abs() <= room[:, :hq]).all())
    cache = kc[:budget * hkv * d].view(budget, hkv, d)
    assert bool(((cache[start:start + rows].double() - ref[:, hq:]).abs() <= room[:, hq:]).all())
    assert torch.equal(vc[start:start + rows].view(rows, hkv, d).double(), before[:, hq + hkv:])
    assert float(cache[:start].abs().max()) == 0.0 and float(cache[start + rows:].abs().max()) == 0.0

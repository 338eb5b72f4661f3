"""Prefill attention with two query tiles per CTA (pair_attn.cu; taken by launches of at least 222 such CTAs on the GPU's 148 SMs):
odd numbers of tiles, ragged last tiles, windows, unused rows, block selection, every head width; against plain attention in
32 bits or more.  Tolerance as for the one-tile kernel: P and the output are rounded to bf16, |out| <= ~4."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import tipetar as T
from test_tipetar_gpu import attn, qkv, run_attention

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def reference(q, k, v, vis):
    """q [T, H, d], k / v [n, G, d]; vis [T, n] or [G, T, n]; rows that see nothing give 0."""
    tq, hq, d = q.shape
    grp = hq // k.shape[1]
    out = torch.zeros(tq, hq, d, device="cuda")
    for h in range(hq):
        s = (q[:, h].float() @ k[:, h // grp].float().t()) / d ** 0.5
        s = s.masked_fill(~(vis if vis.dim() == 2 else vis[h // grp]), float("-inf"))
        out[:, h] = torch.nan_to_num(torch.softmax(s, dim=-1)) @ v[:, h // grp].float()
    return out


def operands(tq, hq, hkv, kv_total, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    budget = (kv_total + 127) // 128 * 128
    q = torch.randn(tq, (hq + 2 * hkv) * 128, generator=g, device="cuda").to(torch.bfloat16)
    k, v = (torch.randn(budget, hkv * 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    return q, k, v, budget


def views(q, k, v, tq, hq, hkv, n):
    return q[:, :hq * 128].reshape(tq, hq, 128), k[:n].view(n, hkv, 128), v[:n].view(n, hkv, 128)


@pytest.mark.parametrize("tq,hq,hkv,L,window,valid", [
    (1769, 32, 2, 0, 0, None), (1777, 32, 2, 63, 0, None), (3545, 16, 1, 333, 0, None), (1800, 32, 32, 200, 0, None),
    (7200, 8, 4, 1000, 0, None), (3545, 16, 1, 700, 512, None), (3545, 16, 1, 0, 0, 3), (3553, 16, 1, 500, 0, 650)])
def test_causal(tq, hq, hkv, L, window, valid):
    import cpmcu.C as C
    rows = tq if valid is None else valid
    kv_total = L + rows
    q, k, v, budget = operands(tq, hq, hkv, kv_total, tq + L)
    at = torch.arange(kv_total, device="cuda")
    t = torch.arange(tq, device="cuda")
    vis = (at[None] < L + t[:, None] + 1) & (t[:, None] < rows)
    if window:
        lo = ((L + t // 64 * 64 + 127) // 128 - window // 128).clamp(min=0) * 128
        vis &= at[None] >= lo[:, None]
    out = torch.full((tq, hq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    kv_len = torch.tensor([kv_total - 5], dtype=torch.int32, device="cuda")
    n_valid = None if valid is None else torch.tensor([valid], dtype=torch.int32, device="cuda")
    C.call("cpmcu_tree_attention", ptr(q), q.shape[1], ptr(k), ptr(v), budget, tq, hq, hkv, ptr(kv_len), 5, ptr(n_valid), None, 0, window, 1,
           ptr(out), hq * 128)
    ref = reference(*views(q, k, v, tq, hq, hkv, kv_total), vis)
    assert float((out.float().view(tq, hq, 128) - ref).abs().max()) < 3e-2


@pytest.mark.parametrize("tq,hq,hkv,L,window,density", [
    (1769, 32, 2, 3000, 8, 0.1), (1790, 32, 2, 4500, 2, 0.0), (3545, 16, 1, 0, 3, 0.3), (7090, 8, 1, 517, 1, 0.02)])
def test_block_selection(tq, hq, hkv, L, window, density):
    import cpmcu.C as C
    kv_total = L + tq
    q, k, v, budget = operands(tq, hq, hkv, kv_total, tq + L)
    nblk = (kv_total + 63) // 64
    words = (nblk + 63) // 64
    bits = np.random.default_rng(L).random((hkv, tq, words * 64)) < density
    bits[:, :, nblk:] = False
    mask = (bits.reshape(hkv, tq, words, 64).astype(np.uint64) << np.arange(64, dtype=np.uint64)).sum(-1, dtype=np.uint64)
    t = torch.arange(tq, device="cuda")
    at = torch.arange(kv_total, device="cuda")
    seen = torch.from_numpy(bits).cuda()[:, :, :nblk] | (torch.arange(nblk, device="cuda")[None] >= ((t + L + 63) // 64 - window)[:, None])[None]
    vis = seen.repeat_interleave(64, dim=2)[:, :, :kv_total] & (at[None] < L + t[:, None] + 1)[None]
    out = torch.full((tq, hq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    kv_len = torch.tensor([kv_total], dtype=torch.int32, device="cuda")
    bm = torch.from_numpy(mask.view(np.int64)).cuda()
    C.call("cpmcu_sparse_attention", ptr(q), q.shape[1], ptr(k), ptr(v), budget, tq, hq, hkv, ptr(kv_len), 0, None, 0, ptr(bm), words, window, 1,
           ptr(out), hq * 128)
    ref = reference(*views(q, k, v, tq, hq, hkv, kv_total), vis)
    assert float((out.float().view(tq, hq, 128) - ref).abs().max()) < 3e-2


# heads, key heads, key width, value width, window: groups that do not divide 128, widths that are padded to 64 or 128 columns
@pytest.mark.parametrize("mix,tq,before", [
    (attn(20, 4, 40, 56, 200), 2790, 70), (attn(20, 4, 64, 64, None), 2800, 0), (attn(24, 8, 128, 64, 1000), 2360, 300),
    (attn(24, 8, 64, 128, 65), 2345, 1), (attn(16, 4, 128, 128, 1024), 3570, 900)], ids=["g5", "narrow", "g3", "wide values", "g4"])
def test_layered(mix, tq, before):
    q, k, v = qkv(mix, tq, before + tq, seed=tq)
    ref = T.attention(q, k, v, mix["scale"], T.mask_size(mix), before)
    assert (run_attention(mix, q, k, v, 1, False) - ref).abs().max() < 0.03

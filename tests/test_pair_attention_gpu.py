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


# A row's output depends on no value beyond the 128-key tiles that some row of its query tile sees (the tiles of the one-tile
# kernel): a NaN there stays there, also where the other tile of the pair sees it.
def reached(vis, tok, at):
    """vis [T, n] bool -> [T] bool: some row of the query tile of `tok` tokens sees a key of the 128-key tile of key `at`."""
    block = vis[:, at // 128 * 128:at // 128 * 128 + 128].any(1)
    rows = torch.zeros((len(block) + tok - 1) // tok * tok, dtype=torch.bool, device=block.device)
    rows[:len(block)] = block
    return rows.view(-1, tok).any(1).repeat_interleave(tok)[:len(block)]


@pytest.mark.parametrize("tq,hq,hkv,L,window", [(1792, 32, 2, 120, 0), (1769, 32, 2, 0, 0), (3545, 16, 1, 56, 512), (7200, 8, 4, 96, 0)])
def test_values_of_the_other_tile(tq, hq, hkv, L, window):
    import cpmcu.C as C
    kv_total, tok = L + tq, 128 * hkv // hq
    q, k, v, budget = operands(tq, hq, hkv, kv_total, tq + L)
    at, t = torch.arange(kv_total, device="cuda"), torch.arange(tq, device="cuda")
    vis = at[None] < L + t[:, None] + 1
    if window:
        first = t // tok * tok   # the window's first key is the same for all rows of a query tile
        vis &= at[None] >= (((L + first // 64 * 64 + 127) // 128 - window // 128).clamp(min=0) * 128)[:, None]
    kv_len = torch.tensor([kv_total], dtype=torch.int32, device="cuda")

    def run(v):
        out = torch.full((tq, hq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
        C.call("cpmcu_tree_attention", ptr(q), q.shape[1], ptr(k), ptr(v), budget, tq, hq, hkv, ptr(kv_len), 0, None, None, 0, window, 1, ptr(out), hq * 128)
        return out

    clean = run(v)
    for p in (128, 130, 640, kv_total // 2 // 128 * 128, kv_total - 1):
        bad = v.clone()
        bad[p] = float("nan")
        far = ~reached(vis, tok, p)
        out = run(bad)
        assert torch.equal(out[far], clean[far]), p
        assert bool(torch.isnan(out[vis[:, p]].float()).all())


def test_values_of_the_other_tiles_blocks():
    import cpmcu.C as C
    tq, hq, hkv, L, window = 1792, 32, 2, 3000, 2
    kv_total, tok = L + tq, 8
    q, k, v, budget = operands(tq, hq, hkv, kv_total, 5)
    nblk = (kv_total + 63) // 64
    # tiles of eight tokens choose different blocks: tile i the blocks 2 (i % 20) and 2 (i % 20) + 1
    t = torch.arange(tq, device="cuda")
    blocks = torch.arange(nblk, device="cuda")
    bits = (blocks[None] // 2) == (t[:, None] // tok % 20)
    words = (nblk + 63) // 64
    m = torch.zeros(tq, words, dtype=torch.int64, device="cuda")
    for b in range(nblk):
        m[:, b // 64] |= bits[:, b].long() << (b % 64)
    bm = m[None].repeat(hkv, 1, 1).contiguous()
    seen = bits | (blocks[None] >= ((t + L + 63) // 64 - window)[:, None])
    vis = seen.repeat_interleave(64, dim=1)[:, :kv_total] & (torch.arange(kv_total, device="cuda")[None] < L + t[:, None] + 1)
    kv_len = torch.tensor([kv_total], dtype=torch.int32, device="cuda")

    def run(v):
        out = torch.full((tq, hq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
        C.call("cpmcu_sparse_attention", ptr(q), q.shape[1], ptr(k), ptr(v), budget, tq, hq, hkv, ptr(kv_len), 0, None, 0, ptr(bm), words, window, 1, ptr(out),
               hq * 128)
        return out

    clean = run(v)
    for p in (0, 200, 128 * 7 + 70, 128 * 19, L + 100):
        bad = v.clone()
        bad[p] = float("nan")
        far = ~reached(vis, tok, p)
        out = run(bad)
        assert torch.equal(out[far], clean[far]), p
        assert bool(torch.isnan(out[vis[:, p]].float()).all())


def test_exact_windows_and_values_of_others():
    """Sliding windows that begin at an odd block, rows of the cache nobody sees at its end."""
    import ctypes as ct

    import cpmcu.C as C
    from test_tipetar_gpu import padded, spec_of
    mix = attn(16, 4, 128, 128, 300)
    tq, before = 3570, 64 + 900
    keys, tok = tq + before, 32
    q, k, v = qkv(mix, tq, keys, seed=2)
    budget = (keys + 127) // 128 * 128 + 256
    kc, vc = (torch.zeros(budget, 4, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    kc[:keys], vc[:keys] = k.to(torch.bfloat16), v.to(torch.bfloat16)
    qc = padded(q.cuda(), 128, torch.bfloat16)
    sp = spec_of(mix)

    def run(v):
        out = torch.zeros(tq, 16 * 128, dtype=torch.bfloat16, device="cuda")
        C.call("cpmcu_layer_attention", ct.byref(sp), qc.data_ptr(), kc.data_ptr(), v.data_ptr(), budget, tq, keys, 1, 0, out.data_ptr())
        return out

    clean = run(vc)
    at, t = torch.arange(budget, device="cuda"), torch.arange(tq, device="cuda")
    vis = (at[None] <= before + t[:, None]) & (at[None] > before + t[:, None] - 300)
    for p in (700, 767, 1024, 1500, keys - 1, (keys + 127) // 128 * 128, budget - 1):
        bad = vc.clone()
        bad[p] = float("nan")
        far = ~reached(vis, tok, p)
        out = run(bad)
        assert torch.equal(out[far], clean[far]), p


# A tree mask reaches this kernel only through the C entry, with key heads enough: 64 tokens, 56 key heads.
def test_tree_mask():
    import cpmcu.C as C
    tq, hq, hkv, L = 64, 16 * 56, 56, 700
    kv_total = L + tq
    q, k, v, budget = operands(tq, hq, hkv, kv_total, 9)
    parent = np.random.default_rng(4).integers(0, np.maximum(np.arange(tq), 1))
    bits = np.zeros((tq, tq), dtype=bool)
    for i in range(tq):
        bits[i] = bits[parent[i]] if i else False
        bits[i, i] = True
    mask = (bits.astype(np.uint64) << np.arange(64, dtype=np.uint64)).sum(-1, dtype=np.uint64)
    vis = torch.ones(tq, kv_total, dtype=torch.bool, device="cuda")
    vis[:, L:] = torch.from_numpy(bits).cuda()
    out = torch.full((tq, hq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    kv_len = torch.tensor([kv_total], dtype=torch.int32, device="cuda")
    m = torch.from_numpy(mask.view(np.int64)).cuda()
    C.call("cpmcu_tree_attention", ptr(q), q.shape[1], ptr(k), ptr(v), budget, tq, hq, hkv, ptr(kv_len), 0, None, ptr(m), tq, 0, 1, ptr(out), hq * 128)
    ref = reference(*views(q, k, v, tq, hq, hkv, kv_total), vis)
    assert float((out.float().view(tq, hq, 128) - ref).abs().max()) < 3e-2

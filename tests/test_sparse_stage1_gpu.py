"""Prefill-sized stage-1 scores (sparse_stage1.cu: more than 64 query rows, 16 query heads per key head): ragged last token tile, ragged
last chunks of compressed keys, both kinds of log-sum-exp keys, caches of several sizes, up to one that is full; the checks of
the decode-sized kernels."""
import pytest
import torch

from test_sparse_gpu import test_block_selection_matches_oracle as check_selection

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,hq,hkv,L,top,sink,window,lse,budget", [
    (65, 16, 1, 5000, 64, 1, 4, True, None), (100, 32, 2, 3000, 16, 1, 8, False, None), (131, 32, 2, 2064, 8, 2, 2, True, 65536),
    (72, 16, 1, 8256, 30, 1, 2, True, 131072), (67, 16, 1, 2048, 7, 0, 1, False, None), (80, 48, 3, 16300, 64, 1, 32, True, 16384 + 128),
    # caches beyond 131072 rows: few CTAs go to the decode-sized kernels where the log-sum-exp has keys of its own
    (95, 16, 1, 9000, 32, 1, 8, True, 196608), (95, 16, 1, 9000, 32, 1, 8, False, 196608), (96, 16, 1, 9000, 32, 1, 8, True, 196608)])
def test_block_selection(T, hq, hkv, L, top, sink, window, lse, budget):
    check_selection(T, hq, hkv, L, top, sink, window, lse, budget)


def test_scores_below_the_smallest_normal_number():
    """A head so peaked that the far blocks score between 2^-130 and 2^-123, later blocks higher: the bf16 scores, exact to a step
    of 2^-133 or 2^-8 of the value (store) and 2^-6 (exponent of up to 133 from a score in fp32: 133 * 2^-16 * ln 2 and the
    exponential's last places), and so the choice, as 64 bits give them and as the decode-sized kernels make it."""
    import cpmcu.C as C
    T, hq, L, top, window = 80, 16, 4096, 6, 4
    budget, words, ld = 4224, 2, 384
    q = torch.zeros(T, (hq + 2) * 128)
    q[:, 0:hq * 128:128] = 64.0
    k = torch.zeros(budget, 128)
    blocks = torch.arange(L // 64)
    # score in powers of two: -64 * b / sqrt(128) * log2(e) = -8.16 b; b falls from 16 3/8 to 15 5/8 over the blocks
    b = 16.375 - (blocks * 7 // len(blocks)).float() * 0.125
    k[64:L, 0] = -b.repeat_interleave(64)[64:]
    q, k = q.to(torch.bfloat16).cuda(), k.to(torch.bfloat16).cuda()
    kv_len = torch.tensor([L], dtype=torch.int32, device="cuda")

    def select(rows):
        scores = torch.zeros(1, rows, ld, dtype=torch.bfloat16, device="cuda")
        bm = torch.zeros(1, rows, words, dtype=torch.int64, device="cuda")
        c1 = torch.zeros(budget // 16, 128, dtype=torch.bfloat16, device="cuda")
        p = [t.data_ptr() for t in (q, k, kv_len, c1, scores, bm)]
        C.call("cpmcu_sparse_select", p[0], q.shape[1], rows, hq, 1, p[1], budget, p[2], 0, 1, window, top, 256, 0, p[3], None, p[4], ld, p[5], words)
        return scores[0].double(), bm[0], c1

    scores, bm, c1 = select(T)
    n1 = (L - 16) // 16
    s = 64.0 * c1[:n1, 0].double() / 128 ** 0.5
    want = 16 * torch.exp(s - s.max()) / torch.exp(s - s.max()).sum()
    assert bool((want < 2.0 ** -126).any()) and bool(((scores[:, :n1] - want).abs() <= 2.0 ** -133 + 2.0 ** -6 * want).all())
    # every row alike: block 0 (sink) and the highest of those before the window, the last ones first come first
    few, bm_few, _ = select(64)
    assert torch.equal(bm[:64], bm_few)
    assert bool(((few - scores[:64]).abs() <= 2.0 ** -133 + 2.0 ** -6 * few).all())

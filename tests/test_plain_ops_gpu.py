"""Plain attention and the fp32 products of layered models at the sizes where their ways of dividing the work change:
a token alone (keys dealt to warps and to the CTAs of a cluster), a few rows, tiles with remainders; against the plain
implementation in 64 bits."""
import pytest
import torch

from oracle import tipetar as T
from test_tipetar_gpu import attn, case, open_case, qkv, run_attention, tokens_of

pytestmark = pytest.mark.gpu


# sums of up to 3000 fp32 products of magnitude one, in another order than the reference's: 2e-5 as for the other shapes
@pytest.mark.parametrize("mix", [attn(3, 1, 72, 72, None), attn(12, 4, 64, 40, 1500), attn(8, 1, 128, 128, 33), attn(20, 1, 40, 64, None),
                                 attn(4, 2, 300, 500, None, scale=0.05)], ids=["g3", "window", "narrow", "g20", "wide"])
@pytest.mark.parametrize("tq,keys", [(1, 31), (1, 33), (1, 1025), (1, 3000), (2, 2000), (11, 700), (33, 64), (130, 600)])
def test_attention_divisions(mix, tq, keys):
    q, k, v = qkv(mix, tq, keys, seed=tq + keys)
    ref = T.attention(q.double(), k.double(), v.double(), mix["scale"], T.mask_size(mix), keys - tq).float()
    assert (run_attention(mix, q, k, v, 0, True) - ref).abs().max() < 2e-5
    assert (run_attention(mix, q, k, v, 0, False) - ref).abs().max() < 0.03


# A row's output does not depend on values it may not see, infinities and NaN among them: those of later tokens, those before
# its window.  Query rows of one launch share key tiles; with 1 or 11 rows the keys are dealt to warps and CTAs.
@pytest.mark.parametrize("mix", [attn(3, 1, 72, 72, None), attn(12, 4, 64, 40, 50), attn(8, 1, 128, 128, 33), attn(4, 2, 300, 500, 200, scale=0.05)],
                         ids=["g3", "window", "narrow", "wide"])
@pytest.mark.parametrize("tq,keys", [(1, 700), (11, 700), (130, 600), (300, 300)])
def test_values_that_a_row_may_not_see(mix, tq, keys):
    q, k, v = qkv(mix, tq, keys, seed=tq)
    window = T.mask_size(mix) or keys + 1
    i = torch.arange(keys - tq, keys)
    for fp32 in (True, False):
        clean = run_attention(mix, q, k, v, 0, fp32)
        for p, value in ((keys - 1, float("nan")), (keys - 1 - tq // 2, float("inf")), (keys - 40, float("nan")), (keys - 2 - window, float("-inf"))):
            if not 0 <= p < keys:
                continue
            bad = v.clone()
            bad[p] = value
            out = run_attention(mix, q, k, bad, 0, fp32)
            sees = (i >= p) & (i - p < window)
            assert torch.equal(out[~sees], clean[~sees]), (p, value)
            assert not bool(torch.isfinite(out[sees]).any())


@pytest.mark.parametrize("name", ["mixed", "odd"])
def test_products_of_every_row_count(name):
    import cpmcu.C as C
    cfg = case(name)
    w = T.random_weights(cfg, seed=2)
    llm = open_case(cfg, w, torch.float32)
    toks = tokens_of(cfg, 200, seed=6)
    ref = T.forward(cfg, w, toks)
    for n in (1, 2, 3, 4, 5, 8, 9, 16, 31, 32, 33, 64, 65, 97, 200):
        got = llm.extend(toks[:n], 0, list(range(n))).double().cpu()
        assert (got - ref[:n]).abs().max() < 2e-5 * float(ref.std()) * 10, n
    C.release()

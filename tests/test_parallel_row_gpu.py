"""One token of layers with attention beside a recurrence, whose launches overlap in pairs (queries and keys beside the recurrence's product, the
merge of the attention's splits beside the recurrence's step): more CTAs in the product than the GPU holds at once and a handful, one
split and many, query rows read 16 bytes and 2 bytes at a time, attention on and off the tensor cores.  The same tokens twice give the same bits
(a row, a cache line or a partial result of the layer before would show), and the logits agree with the plain model's as in the checks of whole models."""
import pytest
import torch

from fabulix_cases import dense, left, model, parallel
from oracle import fabulix as F
from test_fabulix_gpu import check, open_case, tokens_of

pytestmark = pytest.mark.gpu

LAYERS = {
    "wide": [parallel(left(8, 2, 128, 128, 64), 48, 64, 0.9, 0.7, dense(256, 2.0)), parallel(left(4, 4, 64, 64, 32), 24, 128, 0.5, 0.8)],
    "narrow": [parallel(left(6, 2, 9, 7, 6, scale=0.4), 2, 16, 0.7, 1.2), parallel(left(200, 200, 8, 8, 8), 3, 24, 0.6, 0.9, dense(100, 0.9))],
    "untiled": [parallel(left(2, 1, 136, 144, 64, scale=0.1), 5, 40, 0.8, 0.6), parallel(left(8, 1, 64, 64, 16), 2, 64, 0.8, 0.6)],
}


@pytest.mark.parametrize("name", sorted(LAYERS))
def test_tokens_repeat(name):
    import cpmcu.C as C
    cfg = model(1024 if name == "wide" else 192, 200, LAYERS[name], side=24)
    w = F.random_weights(cfg, seed=5)
    toks = tokens_of(cfg, 150, seed=6)
    llm = open_case(cfg, w, torch.bfloat16)
    try:
        runs = []
        for _ in range(2):
            got = [llm.extend(toks[:110], 0, [109])]
            got += [llm.extend([t], 110 + i, [0]) for i, t in enumerate(toks[110:])]
            runs.append(torch.cat(got).cpu())
        assert torch.equal(runs[0], runs[1])
        check(runs[0], F.forward(cfg, w, toks)[109:], torch.bfloat16)
    finally:
        C.release()

"""One token: the shared expert's gate/up product runs beside the router (one_row.cu), and the sum over the experts asks for the router's choice
before its wait (layered_ops.cu).  More CTAs than the GPU holds at once, fewer, a choice without any expert, more experts than the sum
has in flight, and a wide row, against the plain mixture with the tolerances of the other mixtures; then whole passes, where the row, the
activations and the cache lines of the layer before must not be seen: the same tokens twice give the same bits, and the logits agree
with the plain model's as in the checks of whole models."""
import pytest
import torch

from oracle import tipetar as T
from test_tipetar_gpu import check, open_case, test_mixture as mixture, tokens_of
from tipetar_cases import attn, model, moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,mlp", [(1024, moe(3, 2, 128, identity=1, shared=5200)), (512, moe(2, 1, 64, identity=6, shared=4800)),
                                       (64, moe(1, 1, 64, identity=7, shared=64)), (4096, moe(2, 2, 8, shared=16)),
                                       (256, moe(40, 11, 64, identity=3, shared=64)), (4200, moe(3, 2, 16, identity=2, shared=16))])
def test_mixture_of_one_row(width, mlp):
    mixture(width, mlp, 1)


def test_passes_repeat():
    import cpmcu.C as C
    layers = [(attn(4, 2, 64, 64, 100), moe(6, 2, 128, identity=2, shared=5200)), (attn(8, 1, 128, 64, None), moe(3, 3, 64, shared=64)),
              (attn(4, 2, 64, 64, 100), moe(2, 1, 64, identity=6, shared=4800))]
    cfg = model(768, 300, layers, mult=0.8)
    w = T.random_weights(cfg, seed=3)
    toks = tokens_of(cfg, 90, seed=4)
    margins = []
    ref = T.forward(cfg, w, toks, margins_out=margins)
    llm = open_case(cfg, w, torch.bfloat16)
    try:
        runs = []
        for _ in range(2):
            got = [llm.extend(toks[:5], 0, [4])]
            got += [llm.extend([t], 5 + i, [0]) for i, t in enumerate(toks[5:])]
            runs.append(torch.cat(got).cpu())
        assert torch.equal(runs[0], runs[1])
        check(runs[0], ref[4:], torch.bfloat16, torch.stack(margins).min(0).values[4:])
    finally:
        C.release()

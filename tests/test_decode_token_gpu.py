"""One token by value (cpmcu_decode_token): ids and positions that are refused leave the sequence as it was, and the logits in the caller's
buffer are those of extend(), in the first pass of a model (launch by launch) and in replayed ones, for models of both kinds."""
import pytest
import torch

from oracle import fabulix as F
from oracle import tipetar as T
from test_llama_passes_gpu import open_llm, tokens_of

pytestmark = pytest.mark.gpu


def open_model(kind):
    if kind == "llama":
        return open_llm()[0], tokens_of(12)
    if kind == "tipetar":
        from test_tipetar_gpu import open_case, tokens_of as toks
        from tipetar_cases import attn, model, moe
        cfg = model(192, 300, [(attn(4, 2, 64, 64, 100), moe(6, 2, 128, identity=2, shared=128))], mult=0.8)
        return open_case(cfg, T.random_weights(cfg, seed=3), torch.bfloat16), toks(cfg, 12, seed=4)
    from fabulix_cases import dense, left, model, parallel
    from test_fabulix_gpu import open_case, tokens_of as toks
    cfg = model(192, 200, [parallel(left(4, 2, 64, 64, 32), 2, 64, 0.9, 0.7, dense(100, 0.9))], side=24)
    return open_case(cfg, F.random_weights(cfg, seed=5), torch.bfloat16), toks(cfg, 12, seed=6)


@pytest.mark.parametrize("kind", ["llama", "tipetar", "fabulix"])
def test_refusals_and_buffers(kind):
    import cpmcu.C as C
    llm, toks = open_model(kind)
    try:
        vocab, budget = llm.config.vocab_size, (llm.max_total_length + 127) // 128 * 128
        llm.extend(toks[:8], 0, [7])
        ref = [llm.extend([t], 8 + i, [0]) for i, t in enumerate(toks[8:])]
        llm.extend(toks[:8], 0, [7])
        buffers = [torch.full((1, vocab), float("nan"), dtype=llm.dtype, device="cuda") for _ in range(2)]
        for i, t in enumerate(toks[8:]):
            for bad in (-1, vocab, 2**31 - 1):
                with pytest.raises(RuntimeError, match="vocabulary"):
                    llm.extend([bad], 8 + i, [0])
            with pytest.raises(OverflowError):
                llm.extend([2**32 + t], 8 + i, [0])
            for position in (-1, budget):
                with pytest.raises(RuntimeError, match="KV budget"):
                    C.decode_token(t, position, llm.logits.data_ptr(), buffers[0].data_ptr(), True)
            out = buffers[i % 2]
            C.decode_token(t, 8 + i, llm.logits.data_ptr(), out.data_ptr(), True)
            assert torch.equal(out, ref[i])
            out.fill_(float("nan"))
    finally:
        C.release()

"""Ids outside the vocabulary in the device's hands: prompts and decode passes of a Llama-format model take token 0 in their place and report
them (they once read outside the embedding), launched one by one and replayed; what follows is as without them."""
import pytest
import torch

from test_llama_passes_gpu import Passes, open_llm, tokens_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [-1, 4096, 2**31 - 1])
def test_prompts_and_passes(bad):
    llm, C = open_llm()
    try:
        toks = tokens_of(200)
        want = llm.extend(toks, 0, [199])
        for at in (0, 149, 150, 199):   # both chunks' ends
            with pytest.raises(RuntimeError, match="flags 16 "):
                llm.extend(toks[:at] + [bad] + toks[at + 1:], 0, [199])
        assert torch.equal(llm.extend(toks, 0, [199]), want)
        run = Passes(llm, C)
        ref = run(5, False, 5)
        for _ in range(3):
            ids, pos = torch.tensor(tokens_of(5, 5), dtype=torch.int32, device="cuda"), torch.arange(40, 45, dtype=torch.int32, device="cuda")
            ids[3] = bad
            with pytest.raises(RuntimeError, match="flags 16 "):
                llm.decode(ids, pos, torch.tensor([40], dtype=torch.int32, device="cuda"))
            assert torch.equal(run(5, False, 5), ref)
    finally:
        C.release()

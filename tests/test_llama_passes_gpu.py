"""Passes of a Llama-format model through the Python class: the logits of several prompt tokens at once, and decode passes that are
captured and replayed (every shape's first pass runs launch by launch; so does every pass while per-launch timing is on)."""
import ctypes
import os

import numpy as np
import pytest
import torch

from helpers import hf_config, tiny_configs
from oracle.model import make_weights

pytestmark = pytest.mark.gpu


def open_llm(which="a", chunk=150, tokens=1024, base=None, **kw):
    import cpmcu.C as C
    from cpmcu.llm import LLM
    cfg = tiny_configs(which)
    hf = hf_config(cfg)
    if base:
        hf.dim_model_base = base   # the head's input is scaled by base / hidden_size
    w, _ = make_weights(cfg, 3, None)
    os.environ["CPMCU_MAX_TOKENS"] = str(tokens)
    try:
        llm = LLM(None, config=hf, dtype=torch.bfloat16, chunk_length=chunk, memory_limit=0.3, **kw)
        llm.init_storage()
    finally:
        os.environ["CPMCU_MAX_TOKENS"] = "4096"
    llm.load_state_dict_tensors({k: v.to(torch.bfloat16) for k, v in w.items()})
    return llm, C


def tokens_of(n, seed=0):
    return np.random.default_rng(seed).integers(0, 4096, n).tolist()


def test_logits_of_several_prompt_tokens():
    """Rows asked for together against rows asked for alone.  The hidden states are the same; both are bf16 stores (a step of
    2^-8) of fp32 sums of 256 products in two orders (8 * 256 * 2^-24 of the sum of magnitudes, which is below 40 here)."""
    toks = tokens_of(400)
    llm, C = open_llm()
    alone = {w: llm.extend(toks, 0, [w])[0].double() for w in (0, 3, 63, 64, 65, 127, 128, 148, 149, 150, 213, 214, 299, 300, 363, 364, 398, 399)}
    close = lambda got, ref: bool(((got.double() - ref).abs() <= 2.0 ** -7 * ref.abs() + 5e-3).all())  # noqa: E731
    every = llm.extend(toks, 0, list(range(400)))   # chunks of 150, 150 and 100 rows: groups of 64 and what is left of them
    assert all(close(every[w], ref) for w, ref in alone.items())
    mixed = [399, 3, 3, 150, 149, 0, 399, 64, 300]
    got = llm.extend(toks, 0, mixed)
    assert all(close(got[i], alone[w]) for i, w in enumerate(mixed))
    only_last_chunk = llm.extend(toks, 0, [398, 399])
    assert all(close(only_last_chunk[i], alone[w]) for i, w in enumerate([398, 399]))
    # any collection with a length will do, and none at all
    assert close(llm.extend(toks, 0, {64})[0], alone[64]) and close(llm.extend(toks, 0, dict.fromkeys((3, 399)))[1], alone[399])
    assert llm.extend(toks, 0, []).shape == (0, 4096)
    # one token behind others
    two = llm.extend(toks[399:], 399, [0, 0])
    assert two.shape == (2, 4096) and torch.equal(two[0], two[1])
    C.release()
    # a scale of 1 / 4 in front of the head is exact: the logits are a quarter of the others, bit for bit
    llm, C = open_llm(base=64)
    scaled = llm.extend(toks, 0, list(range(400)))
    C.release()
    assert torch.equal(scaled.float() * 4, every.float())


class Passes:
    """Decode passes over fresh buffers behind a prompt of 40 tokens."""

    def __init__(self, llm, C):
        self.llm, self.C = llm, C
        p = torch.tensor(tokens_of(40, 1), dtype=torch.int32, device="cuda")
        llm.prefill(p, torch.arange(40, dtype=torch.int32, device="cuda"))

    def __call__(self, n, masked, seed):
        g = np.random.default_rng(seed)
        ids = torch.tensor(tokens_of(n, seed), dtype=torch.int32, device="cuda")
        depth = np.sort(g.integers(0, 4, n)) if masked else np.arange(n)
        pos = torch.tensor(40 + depth, dtype=torch.int32, device="cuda")
        length = torch.tensor([40], dtype=torch.int32, device="cuda")
        mask = None
        if masked:
            bits = np.tril(g.random((n, n)) < 0.4) | np.eye(n, dtype=bool)
            words = (bits.astype(np.uint64) << np.arange(n, dtype=np.uint64)).sum(-1, dtype=np.uint64)
            mask = torch.from_numpy(words.view(np.int64)).cuda()
        return self.llm.decode(ids, pos, length, mask)

    def plain(self, *a):
        self.C.call("cpmcu_profile", 1, None, None)
        out = self(*a)
        self.C.call("cpmcu_profile", 0, None, None)
        return out


def test_replayed_passes_of_many_shapes():
    """Forty shapes, more than are kept as graphs, masked and unmasked passes of a size in turn; the inputs of a replay are not those
    of its capture, nor where they were.  The kernels and their order of summing are the same: equal bit for bit."""
    llm, C = open_llm()
    run = Passes(llm, C)
    shapes = [(n, masked) for n in (1, 2, 3, 5, 8, 15, 16, 17, 31, 32, 33, 48, 60, 61, 62, 63, 64, 20, 21, 22) for masked in (False, True)]
    want = {(n, m, s): run.plain(n, m, s) for n, m in shapes for s in (n, 100 + n)}
    for k in range(4):
        for n, m in shapes:
            s = n if k % 2 == 0 else 100 + n
            assert torch.equal(run(n, m, s), want[n, m, s]), (k, n, m)
    # a shape that came too late gets a graph once another has not been used for a while, and that one runs without again
    late, early = (22, True), (1, False)
    for _ in range(300):
        last = run(*late, 22)
    assert torch.equal(last, want[late + (22,)]) and torch.equal(run(*late, 122), want[late + (122,)])
    assert all(torch.equal(run(*early, s), want[early + (s,)]) for s in (1, 101, 1))
    # a new sequence in between
    again = Passes(llm, C)
    assert torch.equal(again(3, True, 3), want[3, True, 3])
    C.release()


def test_replayed_passes_with_block_selection():
    llm, C = open_llm(tokens=2048, apply_sparse=True, sink_window_size=1, block_window_size=2, sparse_topk_k=3, sparse_switch=256,
                      apply_compress_lse=True)
    prompt = tokens_of(900, 5)
    line = tokens_of(70, 6)

    def steps(plain):
        llm.extend(prompt, 0, [899])
        if plain:
            C.call("cpmcu_profile", 1, None, None)
        out = [llm.extend([t], 900 + i, [0])[0] for i, t in enumerate(line)]
        if plain:
            C.call("cpmcu_profile", 0, None, None)
        return torch.stack(out)

    want = steps(True)
    assert torch.equal(steps(False), want) and torch.equal(steps(False), want)
    C.release()

"""The work users of this framework have it do, as cases that can be timed and compared.

A case is one request (or one replay of given tokens) on one model, through the Python classes:

  generate  LLM_with_eagle.generate: prompt in, tokens out, speculative decoding with a draft tree
  verify    LLM.prefill, then LLM.decode on trees of tokens with a tree mask (the reference's verify call)
  replay    LLM.extend as bin/trace_run calls it: a prompt in portions, logits of chosen places, then single tokens

The library holds one model per process, so the model of a case is built once, by the case's sizes alone, and kept until a
case of another model is prepared; what `seed` makes is the request.  The weights are random, with the spread of trained
ones where it matters: the stream keeps the token's embedding, every sublayer adds a little, the head prefers one next token
for every token (so that greedy streams do not hang on the last bit), and the drafter knows that token for about 70 % of
the vocabulary (so that a step accepts about three tokens, as the reference's transcript shows).
"""
import functools
import math
import os
import sys
import types
import zlib

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "cpm.cu_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "cpm.cu_b200"))

F64 = torch.float64
EPS, THETA = 1e-5, 10000.0
SIGNAL = 16.0        # logit of a token's own successor; the others have a spread of one
KNOWN = 0.7          # share of the tokens whose successor the drafter predicts
DECAY_RANK = 64      # inner width of a time mix's decay


# ------------------------------------------------------------------------------------------------ cases
def _llama(hidden, layers, hq, hkv, inter, vocab, **more):
    return dict({"family": "llama", "hidden": hidden, "layers": layers, "hq": hq, "hkv": hkv, "inter": inter, "vocab": vocab,
                 "w4": False, "sparse": False, "frspec": 0, "window": 0, "mup": False, "iters": 0, "topk": 0, "tree": 0,
                 "dtype": "bf16", "chunk": 4096}, **more)


def _8b(**more):
    return _llama(4096, 32, 32, 2, 16384, 73448, iters=6, topk=10, tree=60, **more)


def _tipetar(width, layers, heads, kv_heads, dim, window, experts, top, ff, identity, groups, keep, shared, **more):
    return dict({"family": "tipetar", "hidden": width, "layers": layers, "hq": heads, "hkv": kv_heads, "dim": dim, "attn_window": window,
                 "experts": experts, "top": top, "ff": ff, "identity": identity, "groups": groups, "keep": keep, "shared": shared,
                 "vocab": 32768, "dtype": "bf16", "chunk": 4096}, **more)


def _fabulix(width, layers, left, right, light, ff, side, **more):
    return dict({"family": "fabulix", "hidden": width, "layers": layers, "hq": left[0], "hkv": left[1], "dim": left[2], "rec_heads": right[0],
                 "rec_dim": right[1], "light_heads": light[0], "light_dim": light[1], "ff": ff, "side": side, "vocab": 32768,
                 "dtype": "bf16", "chunk": 4096}, **more)


def _request(mode, prompt, steps, portion=0, want=1, temperature=0.0):
    return {"mode": mode, "prompt": prompt, "steps": steps, "portion": portion, "want": want, "temperature": temperature}


def _case(name, model, request):
    return dict(model, name=name, **request)


def listed():
    return [
        # the smallest call: a short prompt and a few tokens on a model of the tests' size; latency and launches count
        _case("tiny_chat", _llama(256, 2, 2, 1, 704, 4096, chunk=1024), _request("replay", 16, 4)),
        # scoring and continuing a text on a small model: many logits wanted, ragged portions, then single tokens
        _case("llama_2k_score", _llama(2048, 8, 16, 4, 8192, 32768, chunk=1024), _request("replay", 1500, 24, want=64)),
        # the headline model's verify calls: 60-node trees behind a 4096-token prompt, logits of every node
        _case("verify_8b", _8b(), _request("verify", 4096, 6)),
        # the headline: speculative decoding behind a 4096-token prompt
        _case("eagle_8b", _8b(), _request("generate", 4096, 64)),
        # the reduced draft vocabulary (drafter with input norms) on a short chat turn, decoding dominates
        _case("eagle_8b_frspec", _8b(frspec=32768), _request("generate", 333, 96)),
        # int4 target with MiniCPM scales, sampled
        _case("eagle_8b_w4", _8b(w4=True, mup=True, chunk=1024), _request("generate", 1024, 64, temperature=0.6)),
        # long context: block-sparse target, windowed drafter, chunks of 2048
        _case("eagle_8b_sparse_32k", _8b(sparse=True, window=1024, chunk=2048), _request("generate", 32768, 24)),
        # mixture of experts, windowed attention: a long prompt in one chunk
        _case("tipetar_2k_prompt", _tipetar(2048, 8, 16, 4, 128, 1024, 60, 6, 1024, 4, 8, 4, 2048), _request("replay", 4096, 0, want=4)),
        # the same design, wider: a ragged prompt and its continuation token by token
        _case("tipetar_4k_chat", _tipetar(4096, 6, 32, 8, 128, 2048, 30, 4, 2048, 2, 4, 3, 4096, chunk=1024), _request("replay", 777, 32)),
        # recurrences beside attention: a long prompt in one chunk
        _case("fabulix_2k_prompt", _fabulix(2048, 9, (16, 4, 128), (32, 64), (16, 128), 5632, 128), _request("replay", 4096, 0, want=4)),
        # narrow heads: a prompt that arrives in portions, then token by token
        _case("fabulix_3k_chat", _fabulix(3072, 9, (48, 12, 64), (48, 64), (24, 128), 8192, 192, chunk=1024),
              _request("replay", 1405, 24, portion=333)),
        # 32-bit activations, odd widths
        _case("tipetar_fp32", _tipetar(1000, 3, 12, 4, 72, 200, 14, 3, 328, 2, 4, 3, 504, dtype="fp32", chunk=1024), _request("replay", 300, 8)),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["replay", "verify", "generate", "generate", "tipetar", "fabulix"])
    if kind in ("replay", "verify", "generate"):
        hidden = rng.choice([256, 512, 1024, 1536, 2048, 3072, 4096])
        hq = hidden // 128
        sparse = kind == "generate" and hidden >= 512 and rng.random() < 0.25
        w4 = not sparse and rng.random() < 0.3
        # a tile of the attention holds 128 rows: query heads per key head divide it (16 at most with block selection)
        hkv = rng.choice([g for g in (1, 2, 3, 4, 6, 8, 12, 24) if hq % g == 0 and hq // g in (1, 2, 4, 8, 16)])
        step = 256 if w4 else 64
        inter = max(1, int(hidden * rng.uniform(2, 4)) // step) * step
        model = _llama(hidden, rng.randint(2, 8), hq, hkv, inter, rng.choice([4096, 5000, 32768, 73448]), w4=w4, sparse=sparse,
                       mup=rng.random() < 0.3, chunk=rng.choice([512, 1024, 2048, 4096]))
        prompt = _log_uniform(rng, 9000, 20000) if sparse else _log_uniform(rng, 8, 8192)
        if kind != "replay":
            model["topk"] = rng.randint(4, 10)
            model["iters"] = rng.randint(2, 6)
            model["tree"] = rng.randint(12, 60) if model["topk"] * (1 + model["topk"] * (model["iters"] - 1)) >= 60 else 12
        if sparse:
            model["window"] = 1024
        elif kind == "generate" and rng.random() < 0.3:
            model["frspec"] = model["vocab"] // 2 // 64 * 64
        if kind == "replay":
            return dict(model, **_request("replay", prompt, rng.randint(0, 32), portion=_log_uniform(rng, 8, 2048), want=_log_uniform(rng, 1, min(64, prompt))))
        if kind == "verify":
            return dict(model, **_request("verify", prompt, rng.randint(2, 8)))
        return dict(model, **_request("generate", prompt, rng.randint(8, 64), temperature=rng.choice([0.0, 0.0, 0.6])))
    fp32 = rng.random() < 0.25
    width = rng.randint(96, 1024) if fp32 else rng.choice([512, 1000, 1024, 2048, 3072, 4096])
    prompt = _log_uniform(rng, 1, 512) if fp32 else _log_uniform(rng, 4, 6000)
    request = _request("replay", prompt, rng.randint(0, 24), portion=_log_uniform(rng, 8, 4096), want=_log_uniform(rng, 1, min(16, prompt)))
    dim = rng.choice([40, 64, 96, 128])
    kv = rng.choice([1, 2, 4])
    heads = kv * rng.randint(1, max(1, min(8, width // dim // kv)))
    if kind == "tipetar":
        keep, groups = rng.choice([(1, 1), (2, 4), (4, 8)])
        outputs = groups * rng.randint(4, 8)
        identity = rng.randint(0, 2)
        model = _tipetar(width, rng.randint(2, 6), heads, kv, dim, rng.randint(100, 4096), outputs - identity, rng.randint(1, 4),
                         max(2, int(width * rng.uniform(0.25, 0.75))), identity, groups, keep, rng.choice([0, width // 2, width]))
    else:
        model = _fabulix(width, rng.randint(2, 7), (heads, kv, dim), (max(1, width // 128), rng.choice([32, 64, 128])),
                         (max(1, width // 192), rng.choice([64, 96, 128])), int(width * rng.uniform(1, 3)), rng.choice([32, 72, 128, 256]))
    return dict(model, dtype="fp32" if fp32 else "bf16", chunk=rng.choice([512, 1024, 4096]), **request)


# ------------------------------------------------------------------------------------------------ weights
MODEL_KEYS = ("family", "hidden", "layers", "hq", "hkv", "inter", "vocab", "w4", "sparse", "frspec", "window", "mup", "iters", "topk", "tree",
              "dtype", "chunk", "dim", "attn_window", "experts", "top", "ff", "identity", "groups", "keep", "shared", "rec_heads", "rec_dim",
              "light_heads", "light_dim", "side")


def _budget(c):
    """Rows the K/V cache is asked to hold: a power of two, so that requests of one model share it."""
    return 1 << max(10, math.ceil(math.log2(c["prompt"] + c["steps"] + 192)))


def _model_key(c):
    return tuple(c.get(k) for k in MODEL_KEYS) + (c["temperature"], _budget(c))


def _rnd(tag, *shape, std, mean=0.0):
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(tag.encode()))
    return (torch.randn(*shape, device="cuda", dtype=torch.bfloat16, generator=g) * std + mean).to(torch.bfloat16)


@functools.lru_cache(maxsize=4)
def _successors(vocab, common):
    """(next token of every token, whether the drafter knows it): the first `common` tokens follow one another."""
    g = np.random.default_rng(7)
    nxt = np.empty(vocab, dtype=np.int64)
    for lo, hi in ((0, common), (common, vocab)):
        order = lo + g.permutation(hi - lo)
        nxt[order] = np.roll(order, -1)
    return nxt, g.random(vocab) < KNOWN


def _mup(c):
    """(embedding scale, residual scale, LM-head input scale) of a model with MiniCPM's scales."""
    return (12.0, 1.4 / math.sqrt(c["layers"]), 0.5) if c["mup"] else (1.0, 1.0, 1.0)


def llama_embed(c):
    """Rows of spread one (before the embedding scale); a token whose successor the drafter does not know lives in the other half
    of the dimensions."""
    H = c["hidden"]
    e = _rnd("embed", c["vocab"], H, std=math.sqrt(2.0) / _mup(c)[0])
    known = torch.from_numpy(_successors(c["vocab"], c["frspec"] or c["vocab"])[1]).cuda()
    e[known, H // 2:] = 0
    e[~known, :H // 2] = 0
    return e


def llama_head(c):
    nxt, _ = _successors(c["vocab"], c["frspec"] or c["vocab"])
    scale = _mup(c)
    head = _rnd("head", c["vocab"], c["hidden"], std=c["hidden"] ** -0.5 / scale[2])
    before = torch.from_numpy(np.argsort(nxt)).cuda()
    head += (llama_embed(c)[before] * (SIGNAL * scale[0] / scale[2] / c["hidden"])).to(torch.bfloat16)
    return head


def _llama_shapes(c):
    H, I, nq, nk = c["hidden"], c["inter"], c["hq"] * 128, c["hkv"] * 128
    return {"self_attn.q_proj": (nq, H), "self_attn.k_proj": (nk, H), "self_attn.v_proj": (nk, H), "self_attn.o_proj": (H, nq),
            "mlp.gate_proj": (I, H), "mlp.up_proj": (I, H), "mlp.down_proj": (H, I)}


def _llama_std(c, name):
    """What a sublayer adds has a spread of about 1 / sqrt(2 * layers) of the embedding's (with MiniCPM's scales the residual
    scale does that)."""
    add = 1.0 if c["mup"] or not ("o_proj" in name or "down" in name) else (2 * c["layers"]) ** -0.5
    return add * _llama_shapes(c)[name][1] ** -0.5


def llama_matrix(c, layer, name):
    return _rnd("%s.%s" % (layer, name), *_llama_shapes(c)[name], std=_llama_std(c, name))


FUSED = {"self_attn.qkv_proj": ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj"), "self_attn.o_proj": ("self_attn.o_proj",),
         "mlp.gate_up_proj": ("mlp.gate_proj", "mlp.up_proj"), "mlp.down_proj": ("mlp.down_proj",)}


def llama_int4(c, layer, fused):
    """(4-bit values [K, N] around 8, scales [K / 128, N]) of a fused linear."""
    shapes = _llama_shapes(c)
    N, K = sum(shapes[p][0] for p in FUSED[fused]), shapes[FUSED[fused][0]][1]
    std = _llama_std(c, FUSED[fused][0])
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(("%s.%s.q" % (layer, fused)).encode()))
    q = torch.randint(1, 16, (K, N), device="cuda", generator=g, dtype=torch.uint8)
    # a group's largest value is 7 scales from zero; 4.32 is the spread of fifteen equally likely values
    scales = (std / 4.32 * (0.8 + 0.4 * torch.rand(K // 128, N, device="cuda", generator=g))).to(torch.bfloat16)
    return q, scales


def dequantised(q, scales):
    K, N = q.shape
    w = (q.to(torch.bfloat16) - 8).view(K // 128, 128, N) * scales[:, None, :]     # one rounding, as the format defines
    return w.view(K, N).t()


@functools.lru_cache(maxsize=1)
def _marlin_orders():
    """Index tables of the GPTQ-Marlin checkpoint layout: 1024 values of four 16 x 16 tiles, and 64 neighbouring scales."""
    values = []
    for lane in range(32):
        col, row = lane // 4, 2 * (lane % 4)
        one = [16 * r + col + 8 * half for half in (0, 1) for r in (row, row + 1, row + 8, row + 9)]
        for tile in range(4):
            values += [256 * tile + one[i] for i in (0, 2, 4, 6, 1, 3, 5, 7)]
    return torch.tensor(values).cuda(), torch.tensor([i + 8 * j for i in range(8) for j in range(8)]).cuda()


def marlin(q, scales):
    """The checkpoint tensors (qweight int32 [K / 16, 2 N], scales) of 4-bit values [K, N]."""
    K, N = q.shape
    values, order = _marlin_orders()
    t = q.view(K // 16, 16, N // 16, 16).permute(0, 2, 1, 3).reshape(-1, 1024)[:, values].view(K // 16, N * 2, 8)
    packed = torch.zeros(K // 16, N * 2, device="cuda", dtype=torch.int64)
    for i in range(8):
        packed |= t[..., i].to(torch.int64) << (4 * i)
    packed = torch.where(packed >= 1 << 31, packed - (1 << 32), packed).to(torch.int32)
    return packed, scales.view(-1, 64)[:, order].reshape(K // 128, N).contiguous()


def llama_weights(c):
    """(class, name, tensor) of everything a checkpoint of this model holds; class "eagle" is the drafter's."""
    H = c["hidden"]
    ones = torch.ones(H, device="cuda", dtype=torch.bfloat16)
    if c["frspec"]:
        yield "eagle", "token_id_remap", torch.arange(c["frspec"], device="cuda", dtype=torch.int32).flip(0)
    yield None, "model.embed_tokens.weight", llama_embed(c)
    yield None, "lm_head.weight", llama_head(c)
    yield None, "model.norm.weight", ones
    for i in range(c["layers"]):
        p = "model.layers.%d." % i
        for fused, parts in FUSED.items():
            if c["w4"]:
                qweight, scales = marlin(*llama_int4(c, i, fused))
                yield None, p + fused + ".qweight", qweight
                yield None, p + fused + ".scales", scales
            else:
                for name in parts:
                    yield None, p + name + ".weight", llama_matrix(c, i, name)
        yield None, p + "input_layernorm.weight", ones
        yield None, p + "post_attention_layernorm.weight", ones
    if not c["iters"]:
        return
    for name in _llama_shapes(c):
        yield "eagle", "layers.0." + name + ".weight", llama_matrix(c, "draft", name) * (0.5 if "o_proj" in name or "down" in name else 1.0)
    yield "eagle", "layers.0.input_layernorm.weight", ones
    yield "eagle", "layers.0.post_attention_layernorm.weight", ones
    # the embedding half of fc keeps the dimensions of known tokens (at spread one), the hidden-state half adds a little
    fc = torch.zeros(H, 2 * H, device="cuda", dtype=torch.bfloat16)
    fc[:, :H].diagonal()[:H // 2] = 1.0
    fc[:, H:] = _rnd("fc", H, H, std=0.2 * H ** -0.5)
    yield "eagle", "fc.weight", fc
    yield "eagle", "fc.bias", torch.zeros(H, device="cuda", dtype=torch.bfloat16)
    if _input_norm(c):
        yield "eagle", "input_norm1.weight", ones
        yield "eagle", "input_norm2.weight", ones


def _input_norm(c):
    return bool(c["frspec"] or c["window"])


def tipetar_config(c):
    layers = []
    for i in range(c["layers"]):
        mix = {"heads": c["hq"], "kv_heads": c["hkv"], "dim": c["dim"], "vdim": c["dim"], "scale": c["dim"] ** -0.5, "mask": {"size": c["attn_window"]}}
        if i >= (c["layers"] + 1) // 2:      # the second half of the layers shares one cache
            mix["kv_from"] = (c["layers"] + 1) // 2 - 1
        mlp = {"kind": "moe", "expert": {"ff": c["ff"]}, "shared": {"ff": c["shared"]} if c["shared"] else None,
               "router": {"experts": c["experts"], "top": c["top"], "identity": c["identity"], "groups": {"count": c["groups"], "keep": c["keep"]},
                          "scale": 2.0}}
        layers.append({"type": "attention", "mixer": mix, "mlp": mlp})
    return {"architecture": "Tipetar", "width": c["hidden"], "vocab": c["vocab"], "norm": {"eps": EPS}, "residual_mult": 0.5, "layers": layers}


def tipetar_weights(c):
    W, nq, nk = c["hidden"], c["hq"] * c["dim"], c["hkv"] * c["dim"]

    def mat(name, *shape, std=None, mean=0.0):
        return name, _rnd("tipetar." + name, *shape, std=std or shape[-1] ** -0.5, mean=mean)

    yield mat("embed", c["vocab"], W, std=1.0)
    yield mat("head", c["vocab"], W)
    yield mat("final.norm", W, std=0.1)
    for i, layer in enumerate(tipetar_config(c)["layers"]):
        p = "l%d." % i
        yield mat(p + "mix.q", nq, W)
        yield mat(p + "mix.q.norm", nq, std=0.1, mean=1.0)
        if layer["mixer"].get("kv_from") is None:
            yield mat(p + "mix.k", nk, W)
            yield mat(p + "mix.k.norm", nk, std=0.1, mean=1.0)
            yield mat(p + "mix.v", nk, W)
        yield mat(p + "mix.o", W, nq)
        yield mat(p + "norm1", W, std=0.1)
        yield mat(p + "norm2", W, std=0.1)
        n = c["experts"] + c["identity"]
        yield mat(p + "mlp.router", n, W, std=3.0 * W ** -0.5)
        yield mat(p + "mlp.correction", n, std=0.01)
        for who, ff in [("e%d" % e, c["ff"]) for e in range(c["experts"])] + ([("shared", c["shared"])] if c["shared"] else []):
            yield mat("%smlp.%s.gate" % (p, who), ff, W)
            yield mat("%smlp.%s.up" % (p, who), ff, W)
            yield mat("%smlp.%s.down" % (p, who), W, ff)


def fabulix_config(c):
    layers = []
    for i in range(c["layers"]):
        if i % 3 == 0:                        # every third layer is a lightning layer without feed-forward
            n = c["light_heads"]
            layers.append({"type": "lightning", "mlp": None, "mixer": {"heads": n, "dim": c["light_dim"], "vdim": c["light_dim"],
                                                                       "decay": [0.9 + 0.099 * h / n for h in range(n)]}})
            continue
        layers.append({"type": "parallel", "mlp": {"kind": "dense", "ff": c["ff"], "limit": 7.0},
                       "mixer": {"left": {"heads": c["hq"], "kv_heads": c["hkv"], "dim": c["dim"], "vdim": c["dim"], "scale": c["dim"] ** -0.5,
                                          "rot": {"base": 500000.0, "dims": c["dim"]}},
                                 "right": {"heads": c["rec_heads"], "dim": c["rec_dim"]}, "left_scale": 0.7, "right_scale": 0.6}})
    return {"architecture": "Fabulix", "width": c["hidden"], "vocab": c["vocab"], "norm": {"eps": EPS}, "embedding": {"scale": 1.0},
            "token_side": {"dim": c["side"]}, "layers": layers}


def fabulix_weights(c):
    W, side = c["hidden"], c["side"]

    def mat(name, *shape, std=None, mean=0.0):
        return name, _rnd("fabulix." + name, *shape, std=std or shape[-1] ** -0.5, mean=mean)

    def norm(name):
        yield mat(name, W, std=0.1, mean=1.0)
        yield mat(name + ".b", W, std=0.1)
        yield name + ".alpha", torch.tensor(0.5, dtype=torch.bfloat16, device="cuda")

    yield mat("embed", c["vocab"], W, std=1.0)
    yield mat("side.embed", c["vocab"], c["layers"] * side, std=1.0)
    yield from norm("final.norm")
    for i, layer in enumerate(fabulix_config(c)["layers"]):
        p = "l%d." % i
        yield from norm(p + "norm1")
        yield from norm(p + "norm1b")
        if layer["type"] == "lightning":
            n = c["light_heads"] * c["light_dim"]
            for part in "qkvg":
                yield mat("%smix.%s" % (p, part), n, W)
            yield mat(p + "mix.o", W, n)
            yield mat(p + "mix.norm", n, std=0.1, mean=1.0)
        else:
            n = c["rec_heads"] * c["rec_dim"]
            for part, rows in (("q", c["hq"] * c["dim"]), ("k", c["hkv"] * c["dim"]), ("v", c["hkv"] * c["dim"])):
                yield mat("%smix.left.%s" % (p, part), rows, W)
            yield mat(p + "mix.left.o", W, c["hq"] * c["dim"])
            for part in "rkvg":
                yield mat("%smix.right.%s" % (p, part), n, W)
            for part in "rkvgw":
                yield mat("%smix.right.mu.%s" % (p, part), W, std=0.2, mean=0.5)
            yield mat(p + "mix.right.w1", DECAY_RANK, W)
            yield mat(p + "mix.right.w2", n, DECAY_RANK)
            yield mat(p + "mix.right.w0", n, std=1.0, mean=-3.0)
            yield mat(p + "mix.right.u", c["rec_heads"], c["rec_dim"], std=0.3)
            yield mat(p + "mix.right.norm", n, std=0.1, mean=1.0)
            yield mat(p + "mix.right.o", W, n)
            yield from norm(p + "norm2")
            yield from norm(p + "norm2b")
            yield mat(p + "mlp.gate", c["ff"], W)
            yield mat(p + "mlp.up", c["ff"], W)
            yield mat(p + "mlp.down", W, c["ff"])
        yield mat(p + "side.gate", side, W)
        yield mat(p + "side.proj", W, side)
        yield mat(p + "side.norm", W, std=0.1, mean=0.2)


# ------------------------------------------------------------------------------------------------ preparing, running
_open = {"key": None, "llm": None}


def _model(c):
    """The model of a case, loaded; the library holds one at a time."""
    key = _model_key(c)
    if _open["key"] == key:
        return _open["llm"]
    import cpmcu.C as C
    C.release()
    _open.update(key=None, llm=None)
    os.environ["CPMCU_MAX_TOKENS"] = str(_budget(c))
    common = dict(dtype=torch.bfloat16 if c["dtype"] == "bf16" else torch.float32, chunk_length=c["chunk"], memory_limit=0.6)
    if c["family"] == "llama":
        llm = _open_llama(c, dict(common, temperature=c["temperature"], random_seed=11))
        weights = llama_weights(c)
    elif c["family"] == "tipetar":
        from cpmcu.tipetar import TipetarLLM
        llm, weights = TipetarLLM(config=tipetar_config(c), **common), ((None,) + w for w in tipetar_weights(c))
    else:
        from cpmcu.fabulix import FabulixLLM
        ranks = {"l%d.mix.right.w1" % i: (DECAY_RANK, c["hidden"]) for i in range(c["layers"])}
        llm, weights = FabulixLLM(config=fabulix_config(c), shapes=ranks, **common), ((None,) + w for w in fabulix_weights(c))
    llm.init_storage()
    for cls, name, tensor in weights:
        llm._load(name, tensor, cls=cls)
    if c["family"] == "llama":
        llm._load("model.rotary_emb.inv_freq", llm._rope_inv_freq(), dtype=torch.float32)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    _open.update(key=key, llm=llm)
    return llm


def _open_llama(c, common):
    from cpmcu.llm import LLM
    from cpmcu.llm_w4a16_gptq_marlin import W4A16GPTQMarlinLLM
    from cpmcu.speculative.eagle import LLM_with_eagle
    from cpmcu.speculative.eagle_base_quant.eagle_base_w4a16_marlin_gptq import W4A16GPTQMarlinLLM_with_eagle
    hf = dict(vocab_size=c["vocab"], num_hidden_layers=c["layers"], hidden_size=c["hidden"], intermediate_size=c["inter"],
              num_attention_heads=c["hq"], num_key_value_heads=c["hkv"], head_dim=128, rms_norm_eps=EPS, rope_theta=THETA,
              torch_dtype=torch.bfloat16)
    scales = {}
    if c["mup"]:
        scales = dict(scale_emb=12.0, scale_depth=1.4, dim_model_base=c["hidden"] / 2)
    if c["w4"]:
        hf["quantization_config"] = {"group_size": 128, "bits": 4}
    hf = types.SimpleNamespace(**hf, **scales)
    if c["sparse"]:
        # blocks of 64: the 64 best, the first one and a window of 2048 tokens, from 8192 tokens on
        common = dict(common, apply_sparse=True, sink_window_size=1, block_window_size=32, sparse_topk_k=64, sparse_switch=8192,
                      apply_compress_lse=True)
    if not c["iters"]:
        return (W4A16GPTQMarlinLLM if c["w4"] else LLM)(None, config=hf, **common)
    cls = W4A16GPTQMarlinLLM_with_eagle if c["w4"] else LLM_with_eagle
    return cls(None, None, num_iter=c["iters"], topk_per_iter=c["topk"], tree_size=c["tree"], eagle_window_size=c["window"],
               frspec_vocab_size=c["frspec"], use_input_norm=_input_norm(c), eagle_config=dict(num_hidden_layers=1, **scales), config=hf, **common)


def _zipf(rng, vocab, n):
    p = 1.0 / np.arange(1, vocab + 1, dtype=np.float64) ** 1.1
    return np.searchsorted(np.cumsum(p) / p.sum(), rng.random(n)).clip(0, vocab - 1)


def _tree(rng, n):
    """(depth of every node, ancestors and itself as bits): a draft tree at most six deep."""
    depth, bits = [0], [1]
    while len(depth) < n:
        p = int(rng.integers(0, len(depth)))
        if depth[p] < 6:
            bits.append(bits[p] | 1 << len(depth))
            depth.append(depth[p] + 1)
    return depth, bits


def _inputs(c, seed):
    """The request, on the host: tokens (prompt, then what follows), the places whose logits are wanted, trees."""
    rng = np.random.default_rng(seed)
    P, G = c["prompt"], c["steps"]
    out = {"tokens": _zipf(rng, c["vocab"], P + (G if c["mode"] == "replay" else 0)).tolist()}
    if c["mode"] == "replay":
        out["want"] = sorted({P - 1, *rng.choice(P, size=min(P, c["want"]) - 1, replace=False).tolist()})
    if c["mode"] == "verify":
        out["trees"] = [dict(zip(("depth", "bits"), _tree(rng, c["tree"])), ids=_zipf(rng, c["vocab"], c["tree"]).tolist()) for _ in range(G)]
    return out


def prepare(case, seed):
    c, req = case, _inputs(case, seed)
    s = {"case": c, "llm": _model(c), "key": _model_key(c)}
    if c["mode"] == "replay":
        # portions as they arrive, then single tokens: (tokens, how many came before, wanted places among them)
        at, P = [], c["prompt"]
        step = c["portion"] or P
        for a in range(0, P, step):
            b = min(P, a + step)
            at.append((req["tokens"][a:b], a, [w - a for w in req["want"] if a <= w < b]))
        at += [([req["tokens"][P + i]], P + i, [0]) for i in range(c["steps"])]
        s["portions"] = at
        return s
    s["prompt"] = torch.tensor(req["tokens"], dtype=torch.int32, device="cuda")
    if c["mode"] == "verify":
        s["positions"] = torch.arange(c["prompt"], dtype=torch.int32, device="cuda")
        s["length"] = torch.tensor([c["prompt"]], dtype=torch.int32, device="cuda")
        s["trees"] = []
        for t in req["trees"]:
            mask = torch.tensor(np.array(t["bits"], dtype=np.uint64), device="cuda")
            s["trees"].append((torch.tensor(t["ids"], dtype=torch.int32, device="cuda"),
                               torch.tensor([c["prompt"] + d for d in t["depth"]], dtype=torch.int32, device="cuda"), mask))
    return s


def run(s):
    c, llm = s["case"], s["llm"]
    if _open["key"] != s["key"]:
        raise RuntimeError("another model has been loaded since this state was prepared")
    if c["mode"] == "replay":
        return {"logits": torch.cat([x for x in (llm.extend(*p) for p in s["portions"]) if x.shape[0]])}
    if c["mode"] == "verify":
        first = llm.prefill(s["prompt"], s["positions"])
        return {"first": first, "nodes": torch.cat([llm.decode(ids, pos, s["length"], mask_2d=mask) for ids, pos, mask in s["trees"]])}
    tokens, accepted, _, _ = llm.generate(s["prompt"], c["steps"] + 1)
    accepted += [0] * (c["steps"] - len(accepted))
    return {"logits": llm.logits[:1].clone(), "tokens": torch.tensor(tokens), "accepted": torch.tensor(accepted)}


# ------------------------------------------------------------------------------------------------ what a pass needs
def _params(c):
    """(multiply-adds of a token without the head, weight elements a single token's pass reads, bytes per element)."""
    W = c["hidden"]
    if c["family"] == "llama":
        n = c["layers"] * sum(a * b for a, b in _llama_shapes(c).values())
        return n, n, 0.5 + 2 / 128 if c["w4"] else 2.0
    if c["family"] == "tipetar":
        nq, nk = c["hq"] * c["dim"], c["hkv"] * c["dim"]
        own = (c["layers"] + 1) // 2
        n = c["layers"] * (2 * W * nq + 3 * W * (c["top"] * c["ff"] + c["shared"])) + own * 2 * W * nk
        return n, n, 2.0
    light = (c["layers"] + 2) // 3
    nl, nr, nq, nk = c["light_heads"] * c["light_dim"], c["rec_heads"] * c["rec_dim"], c["hq"] * c["dim"], c["hkv"] * c["dim"]
    n = c["layers"] * 2 * W * c["side"] + light * 5 * W * nl
    n += (c["layers"] - light) * (2 * W * nq + 2 * W * nk + 5 * W * nr + DECAY_RANK * (W + nr) + 3 * W * c["ff"])
    return n, n, 2.0


def _all_weights(c):
    """Weight elements a long prompt reads: with experts, all of them."""
    n = _params(c)[1]
    if c["family"] == "tipetar":
        n += c["layers"] * 3 * c["hidden"] * c["ff"] * (c["experts"] - c["top"])
    return n


def _attention(c, rows, context):
    """Multiply-adds of `rows` queries behind `context` keys that include them."""
    heads = c["hq"] * (128 if c["family"] == "llama" else c["dim"])
    layers = c["layers"] if c["family"] != "fabulix" else c["layers"] - (c["layers"] + 2) // 3
    most = c.get("attn_window") or (64 * 64 + 2048 + 64 if c.get("sparse") and context >= 8192 else context)
    keys = min(most, context)
    pairs = rows * (context - rows / 2) if keys >= context else rows * keys
    return 2 * layers * heads * pairs


def work(case):
    c = case
    P, G, V, H = c["prompt"], c["steps"], c["vocab"], c["hidden"]
    mac, read, size = _params(c)
    d = 128 if c["family"] == "llama" else c["dim"]
    attending = c["layers"] if c["family"] != "fabulix" else c["layers"] - (c["layers"] + 2) // 3
    row = 2 * attending * c["hkv"] * d * (4 if c["dtype"] == "fp32" else 2)
    out = 4 if c["dtype"] == "fp32" else 2
    pieces = [min(c["portion"], P - a) for a in range(0, P, c["portion"])] if c["mode"] == "replay" and c["portion"] else [P]
    wants = min(P, c["want"])
    flops = 2 * (mac * P + _attention(c, P, P) + wants * V * H)
    nbytes = sum(_all_weights(c) * min(1.0, 0.1 + p / 64) if c["family"] == "tipetar" else read for p in pieces) * size
    nbytes += P * row + V * H * 2 + wants * V * out
    if c["mode"] == "replay":
        flops += G * 2 * (mac + V * H) + 2 * _attention(c, 1, P) * G
        nbytes += G * (read * size + V * H * 2 + P * row + V * out)
    elif c["mode"] == "verify":
        flops += G * 2 * (c["tree"] * (mac + V * H) + _attention(c, c["tree"], P))
        nbytes += G * (read * size + V * H * 2 + P * row + c["tree"] * V * out)
    else:
        share = KNOWN
        steps = G / (1 + sum(share ** i for i in range(1, c["iters"] + 1)))
        draft = 2 * H * H + sum(a * b for a, b in _llama_shapes(c).values())
        head = (c["frspec"] or V) * H
        flops += 2 * draft * P + steps * 2 * (c["tree"] * (mac + V * H) + _attention(c, c["tree"], P) + c["iters"] * c["topk"] * (draft + head))
        nbytes += 2 * draft + steps * (read * size + V * H * 2 + P * row * min(1.0, 6208 / P if c["sparse"] else 1.0) + c["iters"] * 2 * (draft + head))
    return {"bytes": int(nbytes), "flops": int(flops)}


def tolerance(case):
    # measured against 64 bits: 1e-6 with 32-bit activations; 0.003 to 0.014 in bf16, growing with the depth
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.03, "max": 0.3, "differ": 0.01}


# ------------------------------------------------------------------------------------------------ 64 bits
def _rms(x):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + EPS)


def _attend(q, k, v, scale, seen, bias=None, sink=False):
    """q [rows, H, d], k [keys, G, d], v [keys, G, dv], seen [rows, keys] or one for each key head -> [rows, H * dv]."""
    rows, H, _ = q.shape
    G = k.shape[1]
    out = []
    for h in range(H):
        g = h // (H // G)
        score = (q[:, h] @ k[:, g].t()) * scale
        if bias is not None:
            score -= bias(h)
        score.masked_fill_(~(seen[g] if isinstance(seen, list) else seen), float("-inf"))
        if sink:
            score = torch.cat([score, score.new_zeros(rows, 1)], dim=1)
        p = torch.softmax(score, dim=-1)
        out.append((p[:, :-1] if sink else p) @ v[:, g])
    return torch.cat(out, dim=1)


def _rotate(x, pos, base, dims):
    half = dims // 2
    freq = base ** (-2.0 * torch.arange(half, dtype=F64, device="cuda") / dims)
    angle = pos.to(F64)[:, None, None] * freq
    a, b, rest = x[..., :half], x[..., half:dims], x[..., dims:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), rest], dim=-1)


def _blocks(q, k, before, rows):
    """Keys that each of `rows` queries of a chunk behind `before` cached keys may see by the block choice, for each key head;
    None while too few are cached."""
    n1, n2 = max((before - 16) // 16, 0), max((before - 64) // 64, 0)
    if n2 * 64 < 8192:
        return None

    def means(stride, n):
        s = torch.cat([k.new_zeros(1, *k.shape[1:]), k[:before].cumsum(0)])
        at = torch.arange(n, device="cuda") * stride
        return (s[at + 2 * stride] - s[at]) / (2 * stride)

    c1, c2 = means(16, n1), means(64, n2)
    H, G = q.shape[1], k.shape[1]
    blocks = (before + 63) // 64
    total = before + rows
    t = torch.arange(rows, device="cuda")[:, None]
    b = torch.arange(blocks, device="cuda")[None, :]
    key_block = torch.arange(total, device="cuda")[None, :] // 64
    seen = []
    for g in range(G):
        score = q.new_zeros(rows, 4 * blocks + 8)
        for h in range(g * (H // G), (g + 1) * (H // G)):
            low = (q[:, h] @ c2[:, g].t()) * 128 ** -0.5
            score[:, 1:1 + n1] += torch.exp((q[:, h] @ c1[:, g].t()) * 128 ** -0.5 - torch.logsumexp(low, dim=-1, keepdim=True))
        # block b: the best of the five means that begin in it or one before (column 0 of `score` stands for place -1)
        pool = torch.stack([score[:, i:i + 4 * blocks:4] for i in range(5)]).amax(0)
        pool = pool.masked_fill(b > (t + before) // 64 - 32, float("-inf")).masked_fill(b < 1, float("inf"))
        pick = torch.zeros(rows, (total + 63) // 64 + 1, dtype=torch.bool, device="cuda")
        pick.scatter_(1, pool.sort(dim=1, descending=True, stable=True).indices[:, :64], True)
        seen.append(torch.gather(pick, 1, key_block.expand(rows, -1)) | (key_block >= (t + before + 63) // 64 - 32))
    return seen


def exact_llama(c, ids, pos, seen, places):
    """Logits at `places`; seen: which rows each row may attend to."""
    scale_e, scale_r, scale_l = _mup(c)
    ids, pos, n, hq, hkv = ids.cuda(), pos.cuda(), len(ids), c["hq"], c["hkv"]
    x = llama_embed(c)[ids].to(F64) * scale_e
    for i in range(c["layers"]):
        if c["w4"]:
            w = {f: dequantised(*llama_int4(c, i, f)) for f in FUSED}
            parts = {"mlp.down_proj": w["mlp.down_proj"], "self_attn.o_proj": w["self_attn.o_proj"]}
            for f in ("self_attn.qkv_proj", "mlp.gate_up_proj"):
                parts.update(zip(FUSED[f], w[f].split([_llama_shapes(c)[p][0] for p in FUSED[f]])))
        else:
            parts = {name: llama_matrix(c, i, name) for name in _llama_shapes(c)}

        def mul(y, name):
            return y @ parts[name].to(F64).t()

        h = _rms(x)
        q = _rotate(mul(h, "self_attn.q_proj").view(n, hq, 128), pos, THETA, 128)
        k = _rotate(mul(h, "self_attn.k_proj").view(n, hkv, 128), pos, THETA, 128)
        v = mul(h, "self_attn.v_proj").view(n, hkv, 128)
        if c["sparse"]:
            parts_a = []
            for a in range(0, n, c["chunk"]):
                b = min(n, a + c["chunk"])
                causal = seen[a:b, :b]
                chosen = _blocks(q[a:b], k, a, b - a)
                parts_a.append(_attend(q[a:b], k[:b], v[:b], 128 ** -0.5, causal if chosen is None else [m & causal for m in chosen]))
            att = torch.cat(parts_a)
        else:
            att = _attend(q, k, v, 128 ** -0.5, seen)
        x = x + mul(att, "self_attn.o_proj") * scale_r
        h = _rms(x)
        x = x + mul(torch.nn.functional.silu(mul(h, "mlp.gate_proj")) * mul(h, "mlp.up_proj"), "mlp.down_proj") * scale_r
    return (_rms(x[places]) * scale_l) @ llama_head(c).to(F64).t()


def exact_tipetar(c, ids, places):
    w, n = dict(tipetar_weights(c)), len(ids)
    x = w["embed"][ids.cuda()].to(F64)
    at = torch.arange(n, device="cuda")
    dist = (at[:, None] - at[None, :]).to(F64)
    seen = (dist >= 0) & (dist < c["attn_window"])

    def mul(y, name):
        return y @ w[name].to(F64).t()

    def gated(y, p):
        return mul(torch.nn.functional.silu(mul(y, p + ".gate")) * mul(y, p + ".up"), p + ".down")

    def add(x, y, name):
        return x + 0.5 * _rms(y) * (1 + w[name].to(F64))

    kv = {}
    for i, layer in enumerate(tipetar_config(c)["layers"]):
        mix, p = layer["mixer"], "l%d." % i
        q = (_rms(mul(x, p + "mix.q")) * w[p + "mix.q.norm"].to(F64)).view(n, c["hq"], c["dim"])
        source = mix.get("kv_from")
        if source is None:
            kv[i] = ((_rms(mul(x, p + "mix.k")) * w[p + "mix.k.norm"].to(F64)).view(n, c["hkv"], c["dim"]), mul(x, p + "mix.v").view(n, c["hkv"], c["dim"]))
        k, v = kv[i if source is None else source]
        a = _attend(q, k, v, mix["scale"], seen, bias=lambda h: 2.0 ** (-8.0 * (h + 1) / c["hq"]) * dist)
        x = add(x, mul(a, p + "mix.o"), p + "norm1")
        s = torch.softmax(mul(x, p + "mlp.router"), dim=-1)
        choice = s + w[p + "mlp.correction"].to(F64)
        best = choice.view(n, c["groups"], -1).amax(-1).topk(c["keep"], dim=-1).indices
        open_ = torch.zeros(n, c["groups"], dtype=torch.bool, device="cuda").scatter_(1, best, True)
        choice = choice.masked_fill(~open_.repeat_interleave(s.shape[1] // c["groups"], dim=1), float("-inf"))
        chosen = choice.topk(c["top"], dim=-1).indices
        wt = s.gather(1, chosen)
        wt = wt / (wt.sum(dim=-1, keepdim=True) + 1e-20) * 2.0
        y = x * (wt * (chosen >= c["experts"])).sum(dim=-1, keepdim=True)
        for e in range(c["experts"]):
            rows, slot = (chosen == e).nonzero(as_tuple=True)
            if rows.numel():
                y[rows] += wt[rows, slot, None] * gated(x[rows], "%smlp.e%d" % (p, e))
        if c["shared"]:
            y = y + gated(x, p + "mlp.shared")
        x = add(x, y, p + "norm2")
    return (_rms(x[places]) * (1 + w["final.norm"].to(F64))) @ w["head"].to(F64).t()


def exact_fabulix(c, ids, places):
    w, n, cfg = dict(fabulix_weights(c)), len(ids), fabulix_config(c)
    ids = ids.cuda()
    x = w["embed"][ids].to(F64)
    pos = torch.arange(n, device="cuda")
    seen = pos[None, :] <= pos[:, None]

    def get(name):
        return w[name].to(F64)

    def mul(y, name):
        return y @ get(name).t()

    def norm(y, name):
        return torch.tanh(get(name + ".alpha") * y) * get(name) + get(name + ".b")

    for i, layer in enumerate(cfg["layers"]):
        p, mix = "l%d." % i, layer["mixer"]
        h = norm(x, p + "norm1")
        if layer["type"] == "lightning":
            H, d = mix["heads"], mix["dim"]
            q, k, v = (torch.nn.functional.silu(mul(h, p + "mix." + s)).view(n, H, d) for s in "qkv")
            keep = torch.tensor(mix["decay"], dtype=F64, device="cuda")[:, None, None]
            S, o = x.new_zeros(H, d, d), torch.empty(n, H, d, dtype=F64, device="cuda")
            for t in range(n):
                S = torch.baddbmm(S * keep, k[t].unsqueeze(2), v[t].unsqueeze(1))
                o[t] = torch.bmm(q[t].unsqueeze(1), S).squeeze(1)
            y = mul(_rms(o.reshape(n, H * d)) * get(p + "mix.norm") * torch.sigmoid(mul(h, p + "mix.g")), p + "mix.o")
        else:
            a, d = mix["left"], mix["left"]["dim"]
            q, k, v = (mul(h, "%smix.left.%s" % (p, s)).view(n, -1, d) for s in "qkv")
            q, k = (_rotate(u, pos, a["rot"]["base"], d) for u in (q, k))
            y = mix["left_scale"] * mul(_attend(q, k, v, a["scale"], seen, sink=True), p + "mix.left.o")
            r_, H, d = p + "mix.right.", mix["right"]["heads"], mix["right"]["dim"]
            before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
            m = {s: h + (before - h) * get(r_ + "mu." + s) for s in "rkvgw"}
            r, k, v = (mul(m[s], r_ + s).view(n, H, d) for s in "rkv")
            keep = torch.exp(-torch.exp(mul(torch.tanh(mul(m["w"], r_ + "w1")), r_ + "w2") + get(r_ + "w0"))).view(n, H, d, 1)
            bonus = get(r_ + "u")
            S, o = x.new_zeros(H, d, d), torch.empty(n, H, d, dtype=F64, device="cuda")
            for t in range(n):
                o[t] = torch.bmm(r[t].unsqueeze(1), S).squeeze(1)
                S = torch.baddbmm(S * keep[t], k[t].unsqueeze(2), v[t].unsqueeze(1))
            o += (r * bonus * k).sum(dim=-1, keepdim=True) * v
            o = _rms(o).reshape(n, H * d) * get(r_ + "norm") * torch.nn.functional.silu(mul(m["g"], r_ + "g"))
            y = y + mix["right_scale"] * mul(o, r_ + "o")
        x = x + norm(y, p + "norm1b")
        if layer["mlp"]:
            h = norm(x, p + "norm2")
            g, u = mul(h, p + "mlp.gate").clamp(max=7.0), mul(h, p + "mlp.up").clamp(-7.0, 7.0)
            x = x + norm(mul(g * torch.sigmoid(1.702 * g) * (u + 1), p + "mlp.down"), p + "norm2b")
        own = get("side.embed")[ids][:, i * c["side"]:(i + 1) * c["side"]]
        side = torch.nn.functional.gelu(mul(x, p + "side.gate"), approximate="tanh") * own
        x = x + _rms(mul(side, p + "side.proj")) * get(p + "side.norm")
    return norm(x[places], "final.norm") @ get("embed").t()


def exact(case, seed):
    c, req = case, _inputs(case, seed)
    # 64-bit tensor throughput makes the long-context 8B case a matter of minutes
    if c["family"] == "llama" and (c["layers"] * c["hidden"] ** 2 * 12 + c["layers"] * c["hq"] * 256 * c["prompt"]) * 2 * c["prompt"] > 2e14:
        return None
    ids = torch.tensor(req["tokens"])
    P, n = c["prompt"], len(ids)
    places = req["want"] + list(range(P, n)) if c["mode"] == "replay" else [P - 1]
    with torch.no_grad():
        if c["family"] != "llama":
            return {"logits": (exact_tipetar if c["family"] == "tipetar" else exact_fabulix)(c, ids, places)}
        if c["mode"] != "verify":
            at = torch.arange(n, device="cuda")
            got = exact_llama(c, ids, torch.arange(n), at[None, :] <= at[:, None], places)
            return {"logits": got} if c["mode"] == "replay" else {"logits": got, "tokens": None, "accepted": None}
        # every tree behind the same prompt: its nodes see the prompt and their own ancestors
        T, G = c["tree"], c["steps"]
        n = P + T * G
        at = torch.arange(n, device="cuda")
        seen = at[None, :] <= at[:, None]
        seen[P:, P:] = False
        pos = list(range(P))
        for j, t in enumerate(req["trees"]):
            bits = torch.tensor([[b >> i & 1 for i in range(T)] for b in t["bits"]], dtype=torch.bool)
            seen[P + j * T:P + (j + 1) * T, P + j * T:P + (j + 1) * T] = bits.cuda()
            pos += [P + d for d in t["depth"]]
            ids = torch.cat([ids, torch.tensor(t["ids"])])
        got = exact_llama(c, ids, torch.tensor(pos), seen, [P - 1] + list(range(P, n)))
        return {"first": got[:1], "nodes": got[1:]}

"""The work users give this framework, as measurable cases: the standalone packed linear, greedy and sampled
generation, concurrent decode streams, log-likelihood scoring, and the imported Llama decoder.

Every case runs on a model or weight that a program loads once and keeps; what changes from call to call are the
token ids (or activations) and the sampler's seed. Model shapes are the named ones of ferrum_cpu_b200.synth. Weights
are drawn N(0, 0.02^2) on the GPU and stored as GGML Q8_0 blocks; biases and LayerNorm vectors are drawn too, so that
every term of the forward pass takes part.
"""
import ctypes as C
import math
from collections import OrderedDict

import numpy as np
import torch

from ferrum_cpu_b200 import _lib, engine, llama, synth

FP32, BF16X3 = _lib.FC_MATH_FP32, _lib.FC_MATH_BF16X3
#: The import precision of a Llama model: Q8_0 as stored, or every Linear packed to one scale per row.
PRECISIONS = {"q8_0": None, "int8": _lib.FC_Q_INT8, "int4": _lib.FC_Q_INT4}


# ------------------------------------------------------------------------------------------------ weights
class _Draws:
    """Seeded normal draws on the GPU, handed to the library as host memory that stays alive with this object."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.keep = []

    def _host(self, t):
        a = t.cpu().numpy()
        self.keep.append(a)
        return a.ctypes.data

    def q8_0(self, n, k):
        """An [n][k] matrix N(0, 0.02^2) as raw Q8_0 blocks: f16 scale = amax / 127, 32 int8 levels."""
        w = torch.randn((n * k // 32, 32), generator=self.gen, device="cuda") * 0.02
        d = (w.abs().amax(dim=1, keepdim=True) / 127.0).to(torch.float16)
        q = torch.round(w / d.float().clamp_min(1e-12)).clamp_(-127, 127).to(torch.int8)
        return self._host(torch.cat([d.view(torch.uint8), q.view(torch.uint8)], dim=1).reshape(-1))

    def vec(self, n, base, scale):
        return self._host(base + scale * torch.randn(n, generator=self.gen, device="cuda"))


def _gpt2(shape, math_mode):
    n_layer, d, n_head, F, ctx, V = synth.SHAPES[shape]
    w = _Draws(20)
    table = (_lib.FcLayerWeights * n_layer)()
    for L in table:
        L.attn_qkv_q8, L.attn_out_q8, L.ffn_up_q8, L.ffn_down_q8 = w.q8_0(3 * d, d), w.q8_0(d, d), w.q8_0(F, d), w.q8_0(d, F)
        L.attn_qkv_b, L.attn_out_b, L.ffn_up_b, L.ffn_down_b = w.vec(3 * d, 0, 0.02), w.vec(d, 0, 0.02), w.vec(F, 0, 0.02), w.vec(d, 0, 0.02)
        L.ln1_g, L.ln1_b, L.ln2_g, L.ln2_b = w.vec(d, 1, 0.1), w.vec(d, 0, 0.05), w.vec(d, 1, 0.1), w.vec(d, 0, 0.05)
    weights = _lib.FcWeights(w.q8_0(V, d), w.vec(ctx * d, 0, 0.02), C.cast(table, C.POINTER(_lib.FcLayerWeights)),
                             w.vec(d, 1, 0.1), w.vec(d, 0, 0.05), None)
    return engine.CudaSlm(_lib.FcConfig(n_layer, d, n_head, F, ctx, V, 1, math_mode), weights)


def _llama(shape, math_mode, prec):
    V, d, n_layer, n_head, n_kv, hd, F, ctx = synth.LLAMA_SHAPES[shape]
    w = _Draws(21)
    qd, kvd = n_head * hd, n_kv * hd
    table = (_lib.FcLlamaLayer * n_layer)()
    for L in table:
        L.attn_norm, L.ffn_norm = w.vec(d, 1, 0.1), w.vec(d, 1, 0.1)
        L.wq_q8, L.wk_q8, L.wv_q8, L.wo_q8 = w.q8_0(qd, d), w.q8_0(kvd, d), w.q8_0(kvd, d), w.q8_0(d, qd)
        L.gate_q8, L.up_q8, L.down_q8 = w.q8_0(F, d), w.q8_0(F, d), w.q8_0(d, F)
    config = _lib.FcLlamaConfig(V, d, n_layer, n_head, n_kv, hd, F, hd, 10000.0, _lib.FC_ROPE_NORM, 1.0, 1e-6, ctx, 1, math_mode)
    weights = _lib.FcLlamaWeights(w.q8_0(V, d), C.cast(table, C.POINTER(_lib.FcLlamaLayer)), w.vec(d, 1, 0.1), None, None)
    return llama.CudaLlama(config, weights, prec=PRECISIONS[prec])


#: Models and weights a program keeps for its lifetime (the most recent ones; a model's caches go with it).
_kept = OrderedDict()


def _keep(key, make):
    if key not in _kept:
        while len(_kept) >= 4:
            _kept.popitem(last=False)
        _kept[key] = make()
    _kept.move_to_end(key)
    return _kept[key]


def _gpt2_of(case):
    key = ("gpt2", case["shape"], case["math"])
    return _keep(key, lambda: _gpt2(case["shape"], BF16X3 if case["math"] == "bf16x3" else FP32))


def _llama_of(case):
    def make():
        m = _llama(case["shape"], BF16X3 if case["math"] == "bf16x3" else FP32, case["prec"])
        return m, m.new_cache()
    return _keep(("llama", case["shape"], case["math"], case["prec"]), make)


def _linear_of(case):
    n, k = case["n"], case["k"]

    def make():
        w = _Draws(22)
        w.q8_0(n, k)
        return engine.QWeight(w.keep[0], n, k), 0.02 * torch.randn(n, generator=w.gen, device="cuda")
    return _keep(("linear", n, k), make)


# ---------------------------------------------------------------------------------------- the listed cases
def listed():
    return [
        # the packed-weight seam under Linear::forward: one decode row of GPT-2-small's down projection, device pointers
        {"name": "linear-row", "kind": "linear", "m": 1, "k": 3072, "n": 768, "math": "fp32"},
        # the same entry as a prefill product, in the tensor-core math mode
        {"name": "linear-prefill", "kind": "linear", "m": 4096, "k": 1024, "n": 4096, "math": "bf16x3"},
        # a short interactive completion on the smallest model: prompt and 64 greedy tokens
        {"name": "generate-tiny", "kind": "generate", "shape": "tiny", "math": "fp32", "prompt": 16, "new": 64, "sampled": False},
        # GPT-2-small completion, batch 1: the headline decode
        {"name": "generate-small", "kind": "generate", "shape": "small", "math": "fp32", "prompt": 32, "new": 256, "sampled": False},
        # a served chat-style completion: an odd prompt length, temperature / top-k / top-p / repetition penalty on the device
        {"name": "generate-sampled", "kind": "generate", "shape": "small", "math": "fp32", "prompt": 101, "new": 48, "sampled": True},
        # a handful of concurrent completions on the small model
        {"name": "streams-small", "kind": "streams", "shape": "small", "math": "fp32", "streams": 8, "prompt": 64, "new": 64},
        # a full serving batch on the medium model: 64 concurrent streams
        {"name": "streams-medium", "kind": "streams", "shape": "medium", "math": "fp32", "streams": 64, "prompt": 64, "new": 32},
        # full-window log-likelihood scoring, the throughput mode
        {"name": "score-small", "kind": "score", "shape": "small", "math": "bf16x3", "seqs": 64, "len": 1024},
        # the same on the medium model: the largest case
        {"name": "score-medium", "kind": "score", "shape": "medium", "math": "bf16x3", "seqs": 64, "len": 1024},
        # an evaluation server's queue: requests of mixed, odd lengths answered together, in the default math mode
        {"name": "score-requests", "kind": "requests", "shape": "small", "math": "fp32", "requests": 24, "longest": 700},
        # the imported decoder on the 1B-class shape: a completion, weights as stored
        {"name": "llama-generate", "kind": "llama-generate", "shape": "llama-1b", "math": "fp32", "prec": "q8_0", "prompt": 33, "new": 64},
        # the imported decoder packed to one int8 scale per row, as the reference's importer does
        {"name": "llama-int8", "kind": "llama-generate", "shape": "llama-narrow", "math": "fp32", "prec": "int8", "prompt": 33, "new": 64},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "generate", "streams", "score", "requests", "llama-generate"])
    math_mode = rng.choice(["fp32", "bf16x3"])
    if kind == "linear":
        return {"kind": kind, "m": rng.choice([1, _log(rng, 2, 4096)]), "k": rng.choice([128, 512, 768, 1024, 2048, 3072, 4096]),
                "n": _log(rng, 512, 4096), "math": math_mode}
    if kind == "generate":
        shape = rng.choice(["tiny", "small", "medium"])
        # tiny: prompt + completion may outgrow its 128 positions, as long completions do (the stream re-primes itself)
        return {"kind": kind, "shape": shape, "math": "fp32", "prompt": _log(rng, 3, 100 if shape == "tiny" else 500),
                "new": _log(rng, 8, 192), "sampled": rng.choice([False, True])}
    if kind == "streams":
        return {"kind": kind, "shape": rng.choice(["tiny", "small", "medium"]), "math": "fp32", "streams": _log(rng, 2, 64),
                "prompt": _log(rng, 5, 72), "new": _log(rng, 8, 32)}
    if kind == "score":
        shape = rng.choice(["tiny", "small", "medium"])
        return {"kind": kind, "shape": shape, "math": math_mode, "seqs": _log(rng, 1, 64 if math_mode == "bf16x3" else 8),
                "len": _log(rng, 24, 128 if shape == "tiny" else 1024)}
    if kind == "requests":
        return {"kind": kind, "shape": rng.choice(["tiny", "small", "medium"]), "math": math_mode, "requests": _log(rng, 1, 32),
                "longest": _log(rng, 16, 800)}
    prec = rng.choice(["q8_0", "int8", "int4"])
    return {"kind": kind, "shape": rng.choice(["llama-1b", "llama-narrow"]) if prec == "q8_0" else "llama-narrow", "math": "fp32",
            "prec": prec, "prompt": _log(rng, 4, 400), "new": _log(rng, 8, 96)}


# ------------------------------------------------------------------------------------- inputs of one state
def _request_lengths(case):
    """Lengths from 5 ids to the longest, evenly over the logarithm, every one odd or even as it falls."""
    n, top = case["requests"], case["longest"]
    return [int(round(5 * (top / 5) ** (i / max(1, n - 1)))) if n > 1 else top for i in range(n)]


def prepare(case, seed):
    rng = np.random.RandomState(seed % (1 << 32))
    kind = case["kind"]
    if kind == "linear":
        w, bias = _linear_of(case)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        x = torch.randn((case["m"], case["k"]), generator=gen, device="cuda")
        return {"case": case, "w": w, "bias": bias, "x": x, "y": torch.empty((case["m"], case["n"]), device="cuda")}
    if kind == "llama-generate":
        m, cache = _llama_of(case)
        V = synth.LLAMA_SHAPES[case["shape"]][0]
        return {"case": case, "model": m, "cache": cache, "ids": rng.randint(0, V, case["prompt"]).astype(np.int32),
                "params": engine.sampling(temperature=0.0)}
    m = _gpt2_of(case)
    V = synth.SHAPES[case["shape"]][5]
    s = {"case": case, "model": m}
    if kind == "generate":
        s.update(ids=rng.randint(0, V, case["prompt"]).astype(np.int32), params=engine.sampling(0.8, 40, 0.95, 1.1),
                 rng=_lib.lib().fc_rng_seed(seed))
    elif kind == "streams":
        s.update(ids=rng.randint(0, V, (case["streams"], case["prompt"])).astype(np.int32))
    elif kind == "score":
        s.update(ids=rng.randint(0, V, (case["seqs"], case["len"])).astype(np.int32))
    else:
        # score(context, continuation): the last third of the ids is the continuation
        s.update(requests=[(rng.randint(0, V, n).astype(np.int32), max(1, n - n // 3)) for n in _request_lengths(case)])
    return s


def _scores(scores):
    return np.array([(s.logprob, s.n_tokens, s.greedy) for s in scores])


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "linear":
        state["w"].linear_dev(state["x"].data_ptr(), state["bias"].data_ptr(), state["y"].data_ptr(), case["m"],
                              BF16X3 if case["math"] == "bf16x3" else FP32)
        return state["y"]
    if kind == "llama-generate":
        return state["model"].generate(state["ids"], case["new"], state["params"], cache=state["cache"])[0]
    m = state["model"]
    if kind == "generate":
        if case["sampled"]:
            return m.generate_sampled(state["ids"], case["new"], state["params"], state["rng"])[0]
        return m.generate_tokens(state["ids"], case["new"])[0]
    if kind == "streams":
        return m.decode_batch(state["ids"], case["new"])
    if kind == "score":
        scores, lp = m.score_sequences(state["ids"])
        return {"scores": _scores(scores), "logprobs": lp}
    return _scores(m.score_requests(state["requests"]))


# ------------------------------------------------------------------- the work a pass cannot do without
def _gpt2_size(shape):
    n_layer, d, _, F, ctx, V = synth.SHAPES[shape]
    blocks, head = n_layer * (4 * d * d + 2 * d * F), d * V
    return n_layer, d, ctx, V, blocks, head


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": n * k * 34 / 32 + 4 * (m * k + n + m * n), "flops": 2 * m * n * k}
    if kind == "llama-generate":
        V, d, n_layer, n_head, n_kv, hd, F, ctx = synth.LLAMA_SHAPES[case["shape"]]
        width = 2 * n_kv * hd
        blocks, head = n_layer * (2 * d * n_head * hd + d * width + 3 * d * F), d * V
        per_weight = {"q8_0": 34 / 32, "int8": 1.0, "int4": 0.5}[case["prec"]]
        streams, att = 1, n_layer * 4 * n_head * hd
    else:
        n_layer, d, ctx, V, blocks, head = _gpt2_size(case["shape"])
        width, per_weight, streams, att = 2 * d, 34 / 32, case.get("streams", 1), n_layer * 4 * d
    if kind in ("score", "requests"):
        lens = [case["len"]] * case["seqs"] if kind == "score" else _request_lengths(case)
        lens = [min(n, ctx) for n in lens]
        flops = sum(2 * n * (blocks + head) + att * n * (n + 1) / 2 for n in lens)
        return {"bytes": (blocks + head) * per_weight + 8 * sum(lens), "flops": flops}
    # generation: the prompt once, then every matrix once for each new token (all streams of a step together), and the
    # f32 key / value rows of the positions before it (of the window, where the completion outgrows the context)
    p, new = case["prompt"], case["new"]
    rows = [min(p + i, ctx) for i in range(new)]
    bytes_ = (blocks + head) * per_weight * new + streams * sum(4 * n_layer * width * r for r in rows)
    flops = streams * (2 * blocks * (p + new - 1) + 2 * head * new + att * (p * (p + 1) / 2 + sum(rows)))
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # token ids are whole numbers: greedy picks and seeded draws are decided by f32 logits
    if case["kind"] in ("generate", "streams", "llama-generate"):
        return {"rel": 0.0, "differ": 0.01}
    # f32 sums against f32 sums in another order; the three-term bf16 product drops terms of 2^-16 of a product.
    # Log-probabilities are that same error against values of about ln V.
    return {"rel": 1e-5 if case["math"] == "fp32" else 5e-5, "differ": 0.01}

"""The work a user of this package has it do, as measurable cases.

Five kinds, each through the public entry points:

  decode    token steps of a LLaMA-architecture model with a context in the KV cache (``Llama.decode``)
  prefill   a prompt, or a further turn of a chat, into the KV cache (``Llama.prefill``)
  linears   one layer's quantized linears (and the output projection) one by one (``tlc_linear``)
  script    the forward pass as a TL script composes it from the builtins (rms_norm, linear, rope, ...)
  matmul    the dense ``matmul`` builtin (``tlc_matmul``)

A case is a dict of plain values; ``prepare`` builds what a program keeps between calls (weights in HBM, the
runner with its cache, buffers), ``run`` makes one pass.  Weights are synthetic with the generators' distributions
and random in the seed; contexts are random rows already in the cache, as in the repository's benchmark.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from tensorlogic_b200 import _lib, synth
from tensorlogic_b200.api import Device, KVCache, QTensor, add, embedding, linear, mul, rms_norm, rope, silu
from tensorlogic_b200.model import (LLAMA2_7B, TINYLLAMA, Llama, LlamaArch, Model, get_tensor, split_for,
                                    weight_scale_log2)

TYPES = {"q4_0": _lib.TYPE_Q4_0, "q8_0": _lib.TYPE_Q8_0, "q6_k": 14, "f16": _lib.TYPE_F16}
BYTES_PER_WEIGHT = {"q4_0": 18 / 32, "q8_0": 34 / 32, "q6_k": 210 / 256, "f16": 2.0}

# The benchmark's model shapes; the last is what one of eight GPUs holds of the 70B shape.
MODELS = {
    "tinyllama": TINYLLAMA,
    "llama2_7b": LLAMA2_7B,
    "llama2_70b_rank_of_8": LlamaArch(80, 8192, 8, 1, 128, 28672 // 8, 32000 // 8),
}


def listed():
    return [
        # Chat with the small model on stock settings: one sequence, greedy, the tokens come back one by one.
        dict(name="decode_tiny_q4_b1", kind="decode", model="tinyllama", qtype="q4_0", out="q4_0", batch=1,
             context=512, gap=0, steps=16, read="tokens", temperature=0.0),
        # A few concurrent chats of different lengths whose host program samples from the logits itself.
        dict(name="decode_tiny_q8_b5_logits", kind="decode", model="tinyllama", qtype="q8_0", out="q8_0", batch=5,
             context=1100, gap=97, steps=8, read="logits", temperature=0.0),
        # A served 7B file as quantizers write it (output.weight in Q6_K), a full batch, temperature sampling.
        dict(name="decode_7b_q4_b32_q6k_out", kind="decode", model="llama2_7b", qtype="q4_0", out="q6_k", batch=32,
             context=768, gap=11, steps=4, read="tokens", temperature=0.8),
        # One GPU's share of the 70B shape (one KV head, narrow shards), long contexts.
        dict(name="decode_70b_rank_q4_b8", kind="decode", model="llama2_70b_rank_of_8", qtype="q4_0", out="q4_0",
             batch=8, context=2048, gap=0, steps=2, read="tokens", temperature=0.0),
        # The benchmark's prompt.
        dict(name="prefill_tiny_q4_512", kind="prefill", model="tinyllama", qtype="q4_0", out="q4_0", tokens=512,
             pos0=0),
        # A further turn of a chat: a short ragged prompt behind a context.
        dict(name="prefill_tiny_q8_77_turn", kind="prefill", model="tinyllama", qtype="q8_0", out="q6_k", tokens=77,
             pos0=391),
        # A long document into the 7B shape: the largest case.
        dict(name="prefill_7b_q4_2048", kind="prefill", model="llama2_7b", qtype="q4_0", out="q4_0", tokens=2048,
             pos0=0),
        # The decode linears of the small model on their own: the smallest products.
        dict(name="linears_tiny_q4_m1", kind="linears", qtype="q4_0", rows=1, d=2048, kv=256, ffn=5632, vocab=32000),
        # A small batch against the 7B layer in 8 bits.
        dict(name="linears_7b_q8_m16", kind="linears", qtype="q8_0", rows=16, d=4096, kv=4096, ffn=11008, vocab=0),
        # A file left in f16, a prompt of ordinary length.
        dict(name="linears_f16_m128", kind="linears", qtype="f16", rows=128, d=2048, kv=256, ffn=5632, vocab=0),
        # A token the way a TL script computes it, builtin by builtin: launches and host calls count.
        dict(name="script_tiny_q4_m1", kind="script", qtype="q4_0", rows=1, pos0=500, layers=6),
        # The general matrix product of the language, with sizes nothing divides.
        dict(name="matmul_1000x1030x777", kind="matmul", m=1000, k=1030, n=777),
    ]


def _log(rng, lo, hi, step=1):
    """A size between lo and hi, even in its logarithm, a multiple of step."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, min(int(hi), int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "linears", "linears", "script", "matmul"))
    if kind == "decode":
        model = rng.choice(("tinyllama", "tinyllama", "llama2_7b", "llama2_70b_rank_of_8"))
        batch = _log(rng, 1, 32)
        context = _log(rng, 64, 1000 if model == "llama2_7b" else 2048)
        if model == "llama2_7b":  # the caches of three states stay within the card
            context = max(64, min(context, 24576 // batch))
        steps = {"tinyllama": _log(rng, 4, 16), "llama2_7b": rng.randint(1, 4), "llama2_70b_rank_of_8": rng.randint(1, 2)}
        return dict(kind=kind, model=model, qtype=rng.choice(("q4_0", "q4_0", "q8_0")),
                    out=rng.choice(("q4_0", "q8_0", "q6_k")), batch=batch, context=context,
                    gap=rng.randint(0, context // (2 * batch)), steps=steps[model],
                    read=rng.choice(("tokens", "tokens", "logits")), temperature=rng.choice((0.0, 0.0, 0.8)))
    if kind == "prefill":
        model = rng.choice(("tinyllama", "tinyllama", "llama2_7b"))
        tokens = _log(rng, 2, 2048)
        return dict(kind=kind, model=model, qtype=rng.choice(("q4_0", "q4_0", "q8_0")),
                    out=rng.choice(("q4_0", "q8_0", "q6_k")), tokens=tokens,
                    pos0=rng.choice((0, rng.randint(0, 2048 - tokens))))
    if kind == "linears":
        qtype = rng.choice(("q4_0", "q4_0", "q8_0", "q8_0", "q6_k", "f16"))
        step = 256 if qtype == "q6_k" else 32
        d = _log(rng, 1024, 8192, step)
        return dict(kind=kind, qtype=qtype, rows=_log(rng, 1, 2048 if qtype in ("q4_0", "q8_0") else 256), d=d,
                    kv=_log(rng, 64, d, 32), ffn=max(step, int(d * rng.uniform(2.0, 3.5)) // step * step),
                    vocab=rng.choice((0, 0, rng.randint(8000, 33000))))
    if kind == "script":
        rows = rng.choice((1, _log(rng, 1, 512)))
        return dict(kind=kind, qtype=rng.choice(("q4_0", "q8_0")), rows=rows, pos0=rng.randint(0, 2048 - rows),
                    layers=rng.randint(2, 8))
    return dict(kind=kind, m=_log(rng, 64, 4096), k=_log(rng, 256, 4096), n=_log(rng, 64, 4096))


# ---- what a program has in hand ---------------------------------------------------------------------------

_device = None


def _dev() -> Device:
    global _device
    if _device is None:
        _device = Device()
    return _device


class _Span:
    """f16 device memory of the library under torch's eyes, without a copy."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f2", data=(int(ptr), False), version=3)


def _view(ptr, shape, owner):
    return torch.as_tensor(_Span(ptr, shape, owner), device="cuda")


def _normal(seed, tag, *shape):
    """f16 N(0, 1) on the GPU: activations."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1009 + tag)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).half()


def _q6k_blocks(seed, tag, rows, cols):
    """Random Q6_K super-blocks: every 6-bit value and scale, d such that a weight is about 0.02 in size."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1013 + tag)
    raw = torch.randint(0, 256, (rows * cols // 256, 210), generator=g, device="cuda", dtype=torch.uint8)
    d = (torch.rand(raw.shape[0], 1, generator=g, device="cuda") + 0.5) * 1.5e-5
    raw[:, 208:210] = d.half().view(torch.uint8).reshape(-1, 2)
    return raw.cpu().numpy()


def _weight(dev, qtype, name, rows, cols, seed, scale_log2):
    if qtype == "q6_k":
        return QTensor.from_blocks(dev, TYPES[qtype], rows, cols, _q6k_blocks(seed, rows % 997, rows, cols))
    if qtype == "f16":
        return QTensor.normal_f16(dev, rows, cols, seed, synth.tensor_id(name), 0.0, 0.02)
    return QTensor.synthetic(dev, TYPES[qtype], rows, cols, seed, synth.tensor_id(name), scale_log2=scale_log2)


def _model(dev, arch, qtype, out, seed):
    m = Model(dev)
    for name, (rows, cols) in arch.tensor_shapes().items():
        if name.endswith("norm.weight"):
            t = QTensor.normal_f16(dev, 1, cols, seed, synth.tensor_id(name), 1.0, 0.02)
        elif name == "token_embd.weight":
            t = QTensor.normal_f16(dev, rows, cols, seed, synth.tensor_id(name), 0.0, 0.02)
        else:
            q = out if name == "output.weight" else qtype
            scale = weight_scale_log2(TYPES[q], cols, split_for(name) == _lib.SPLIT_COLS)
            t = _weight(dev, q, name, rows, cols, seed, scale)
        m.add(name, t)
    return m


def _cache_rows(dev, runner, arch, max_seq, batch, first, gap, count):
    """Views of the cache rows that a pass writes: [layers, batch, count, kv_heads * head_dim], sequence i from
    position first - gap * i on."""
    k, v = ctypes.c_void_p(), ctypes.c_void_p()
    _lib.check(dev.lib.tlc_kvcache_layer_ptrs(dev.lib.tlc_llama_cache(runner.handle), 0, ctypes.byref(k),
                                              ctypes.byref(v)))
    row = arch.n_kv_heads * arch.head_dim
    views = []
    for p in (k.value, v.value):
        whole = _view(p, (arch.n_layers, batch, max_seq, row), runner)
        views.append(whole.as_strided((arch.n_layers, batch, count, row),
                                      (batch * max_seq * row, (max_seq - gap) * row, row, 1), first * row))
    return views


def prepare(case, seed):
    dev = _dev()
    s = dict(case=case, dev=dev)
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        arch = MODELS[case["model"]]
        decode = kind == "decode"
        first, count = (case["context"], case["steps"]) if decode else (case["pos0"], case["tokens"])
        batch, gap = (case["batch"], case["gap"]) if decode else (1, 0)
        max_seq = first + count
        s["model"] = _model(dev, arch, case["qtype"], case["out"], seed)
        s["llama"] = Llama(dev, s["model"], arch, max_seq=max_seq, max_batch=batch,
                           max_prefill=1 if decode else count)
        if first:
            s["llama"].fill_cache_random(seed)
        s["rows"] = _cache_rows(dev, s["llama"], arch, max_seq, batch, first, gap, count)
        s["ids"] = synth.token_ids(seed, "ids", batch * count, arch.vocab).reshape(count, batch)
        if decode:
            s["positions"] = np.array([first - gap * i for i in range(batch)], np.int32)
            s["llama"].set_sampling(case["temperature"], seed)
    elif kind == "linears":
        d, kv, ffn, m = case["d"], case["kv"], case["ffn"], case["rows"]
        shapes = [("q", d, d), ("k", kv, d), ("v", kv, d), ("o", d, d), ("gate", ffn, d), ("up", ffn, d),
                  ("down", d, ffn)] + ([("out", case["vocab"], d)] if case["vocab"] else [])
        x = {c: _normal(seed, c, m, c) for c in {d, ffn}}
        s["calls"] = []
        for i, (name, rows, cols) in enumerate(shapes):
            w = _weight(dev, case["qtype"], name, rows, cols, seed * 16 + i, 0)
            s["calls"].append((w, x[cols], torch.empty(m, rows, dtype=torch.float16, device="cuda")))
    elif kind == "script":
        arch = LlamaArch(n_layers=case["layers"])
        m = s["model"] = _model(dev, arch, case["qtype"], case["qtype"], seed)
        s["arch"] = arch
        s["table"] = get_tensor(m, "token_embd.weight").dequantize()
        s["out_norm"] = get_tensor(m, "output_norm.weight").dequantize().reshape((arch.d_model,))
        s["out"] = get_tensor(m, "output.weight")
        s["layers"] = []
        for l in range(arch.n_layers):
            w = {n: get_tensor(m, f"blk.{l}.{n}.weight")
                 for n in ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")}
            for n in ("attn_norm", "ffn_norm"):
                w[n] = get_tensor(m, f"blk.{l}.{n}.weight").dequantize().reshape((arch.d_model,))
            s["layers"].append(w)
        s["cache"] = KVCache(dev, arch.n_layers, arch.n_kv_heads, arch.head_dim, max_seq=case["pos0"] + case["rows"])
        row = arch.n_kv_heads * arch.head_dim
        context = _normal(seed, 7, 2, case["pos0"], row)
        torch.cuda.synchronize()
        for l in range(arch.n_layers if case["pos0"] else 0):  # a context in the cache
            k, v = ctypes.c_void_p(), ctypes.c_void_p()
            _lib.check(dev.lib.tlc_kvcache_layer_ptrs(s["cache"].handle, l, ctypes.byref(k), ctypes.byref(v)))
            for p, rows in zip((k.value, v.value), context):
                _view(p, (case["pos0"], row), s["cache"]).copy_(rows)
        s["ids"] = synth.token_ids(seed, "ids", case["rows"], arch.vocab)
    else:
        m, k, n = case["m"], case["k"], case["n"]
        s["a"], s["b"] = _normal(seed, 1, m, k), _normal(seed, 2, k, n)
        s["y"] = torch.empty(m, n, dtype=torch.float16, device="cuda")
    return s


# ---- one pass ---------------------------------------------------------------------------------------------

def run(s):
    return RUN[s["case"]["kind"]](s)


def _run_decode(s):
    """Given continuations (so that a pass computes the same whatever a tie in the logits would decide): the logits
    of every step, or of the last one where the program takes the sampled tokens, and the cache rows written."""
    llama, ids, case = s["llama"], s["ids"], s["case"]
    llama.set_state(ids[0], s["positions"])
    logits = []
    for i, step in enumerate(ids):
        read = case["read"] == "logits" or i + 1 == len(ids)
        row = llama.decode(step, return_logits=read)[1]
        if read:
            logits.append(row)
    return {"logits": logits, "k": s["rows"][0], "v": s["rows"][1]}


def _run_prefill(s):
    _, logits = s["llama"].prefill(s["ids"].reshape(-1), s["case"]["pos0"])
    return {"logits": logits, "k": s["rows"][0], "v": s["rows"][1]}


def _run_linears(s):
    dev = s["dev"]
    for w, x, y in s["calls"]:
        _lib.check(dev.lib.tlc_linear(dev.handle, w.handle, x.data_ptr(), x.shape[0], x.shape[1], y.data_ptr(), None))
    return [y for _, _, y in s["calls"]]


def _run_script(s):
    """The forward pass of the TL chat script: about 20 builtins a layer, logits read back."""
    a, cache, pos0, m = s["arch"], s["cache"], s["case"]["pos0"], s["case"]["rows"]
    x = embedding(s["table"], s["ids"])
    for l, w in enumerate(s["layers"]):
        h = rms_norm(x, w["attn_norm"], a.rms_eps)
        q = rope(linear(h, w["attn_q"]).reshape((m, a.n_heads, a.head_dim)), pos0)
        k = rope(linear(h, w["attn_k"]).reshape((m, a.n_kv_heads, a.head_dim)), pos0)
        v = linear(h, w["attn_v"])
        cache.lengths[l] = pos0  # the same turn again
        cache.append(l, k, v)
        o = cache.attention(l, q, a.n_heads, q_pos0=pos0)
        x = add(x, linear(o.reshape((m, a.d_model)), w["attn_output"]))
        h = rms_norm(x, w["ffn_norm"], a.rms_eps)
        x = add(x, linear(mul(silu(linear(h, w["ffn_gate"])), linear(h, w["ffn_up"])), w["ffn_down"]))
    return linear(rms_norm(x, s["out_norm"], a.rms_eps), s["out"]).numpy()


def _run_matmul(s):
    dev, (m, k), (k2, n) = s["dev"], s["a"].shape, s["b"].shape
    _lib.check(dev.lib.tlc_matmul(dev.handle, s["a"].data_ptr(), s["b"].data_ptr(), s["y"].data_ptr(), m, k, k2, n))
    return s["y"]


RUN = {"decode": _run_decode, "prefill": _run_prefill, "linears": _run_linears, "script": _run_script,
       "matmul": _run_matmul}


# ---- what a pass cannot do without, and how far its results may be off --------------------------------------

def _layer_weights(a):
    qd, kvd = a.n_heads * a.head_dim, a.n_kv_heads * a.head_dim
    return a.d_model * (2 * qd + 2 * kvd) + 3 * a.d_model * a.ffn_dim


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prefill", "script"):
        a = LlamaArch(n_layers=case["layers"]) if kind == "script" else MODELS[case["model"]]
        qd, kv_row = a.n_heads * a.head_dim, 2 * a.n_kv_heads * a.head_dim * 2  # bytes of K and V of a position
        layers, out = a.n_layers * _layer_weights(a), a.vocab * a.d_model
        weight_bytes = layers * BYTES_PER_WEIGHT[case["qtype"]] + out * BYTES_PER_WEIGHT[case.get("out", case["qtype"])]
        nbytes = flops = 0.0
        if kind == "decode":
            B = case["batch"]
            for i in range(case["steps"]):
                keys = sum(case["context"] - case["gap"] * b + i + 1 for b in range(B))
                nbytes += weight_bytes + a.n_layers * kv_row * (keys + B) + B * a.d_model * 2
                nbytes += B * a.vocab * 2 if case["read"] == "logits" or i + 1 == case["steps"] else 0
                flops += 2.0 * B * (layers + out) + 4.0 * a.n_layers * qd * keys
        else:
            n = case["tokens"] if kind == "prefill" else case["rows"]
            rows = 1 if kind == "prefill" else n  # rows of logits
            keys = n * case["pos0"] + n * (n + 1) / 2
            nbytes = weight_bytes + a.n_layers * kv_row * (case["pos0"] + 2 * n) + n * a.d_model * 2 + rows * a.vocab * 2
            flops = 2.0 * n * layers + 2.0 * rows * out + 4.0 * a.n_layers * qd * keys
        return {"bytes": nbytes, "flops": flops}
    if kind == "linears":
        d, kv, ffn, m = case["d"], case["kv"], case["ffn"], case["rows"]
        weights = 2 * d * d + 2 * kv * d + 3 * d * ffn + case["vocab"] * d
        outputs = 3 * d + 2 * kv + 2 * ffn + case["vocab"]
        return {"bytes": weights * BYTES_PER_WEIGHT[case["qtype"]] + 2 * m * (d + ffn + outputs),
                "flops": 2.0 * m * weights}
    m, k, n = case["m"], case["k"], case["n"]
    return {"bytes": 2.0 * (m * k + k * n + m * n), "flops": 2.0 * m * k * n}


def tolerance(case):
    # f16 tensors between operations, f32 sums: a product is off by its f16 rounding, and by the rounding of each
    # dequantized weight where an implementation keeps them in f16; a whole model by what its layers add up to.
    if case["kind"] == "matmul":
        return {"rel": 1e-3}
    if case["kind"] == "linears":
        return {"rel": 2e-3}
    return {"rel": 1e-2}

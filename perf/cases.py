"""The work that a user of this framework has it do, as measured cases.

Whole calls go through `uzu_b200.binding.Engine` on synthetic checkpoints (the presets of `uzu_b200.synth` with fewer layers, cached in shared
memory); blocks go through the C ABI's `uzu_*_encode` entries inside a command buffer, as a host program that brings its own graph calls them.

  decode     a chat answer: tokens one by one after a prompt that is kept as a snapshot, each step read back by the host
  prompt     a prompt taken in by a fresh sequence, up to its last row's logits
  batch      several users' prompts, then their answers through shared weight passes
  verify     a speculation pass over a tree of proposed tokens, with every node's logits
  linears    the four quantised projections of a layer on a few dozen rows: a short turn, the tail of a chunk
  attention  attention of a prompt chunk over the cache behind it (grouped heads; 64, 128 and 256 channels)
  sampling   seeded sampling with temperature, top-k, top-p and min-p over a vocabulary
  delta      the generalized delta rule of a prompt, state carried in and out
  latent     attention over a shared latent cache, a prompt's rows or a decoded one
  mlp        a dense bf16 gated feed-forward on f32 rows, one token or a prompt's
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import json
import math
import os
import struct
from pathlib import Path

import numpy as np
import torch

from uzu_b200 import binding as B
from uzu_b200 import synth

F64 = torch.float64


def listed():
    return [
        # an answer of an 8B model at a few thousand tokens of context: bound by the weights of each step
        {"name": "decode-llama-int4", "kind": "decode", "model": "llama3-8b", "layers": 4, "bits": 4, "group": 64, "method": "zero", "vocab": 128256, "context": 2048, "steps": 8},
        # an answer of a small hybrid model: launches and latency count
        {"name": "decode-qwen-int4", "kind": "decode", "model": "qwen3.5-0.8b", "layers": 8, "bits": 4, "group": 64, "method": "zero", "vocab": 248320, "context": 500, "steps": 16},
        # the benchmark's prompt of 2048 tokens
        {"name": "prompt-llama-int4", "kind": "prompt", "model": "llama3-8b", "layers": 4, "bits": 4, "group": 64, "method": "zero", "vocab": 32768, "tokens": 2048},
        # the small hybrid model's prompt, a ragged length
        {"name": "prompt-qwen-int4", "kind": "prompt", "model": "qwen3.5-0.8b", "layers": 8, "bits": 4, "group": 64, "method": "zero", "vocab": 248320, "tokens": 509},
        # eight users at once on an int8 model
        {"name": "batch-llama-int8", "kind": "batch", "model": "llama3-8b", "layers": 2, "bits": 8, "group": 64, "method": "zero", "vocab": 32768, "sequences": 8, "tokens": 256, "steps": 16},
        # a proposal of sixteen nodes
        {"name": "verify-llama-int4", "kind": "verify", "model": "llama3-8b", "layers": 4, "bits": 4, "group": 64, "method": "zero", "vocab": 32768, "context": 2048, "nodes": 16},
        # a short user turn
        {"name": "linears-llama-m40", "kind": "linears", "model": "llama3-8b", "bits": 4, "group": 64, "method": "zero", "rows": 40},
        # the second chunk of a long prompt on wide heads
        {"name": "attention-d256", "kind": "attention", "heads": 8, "groups": 2, "dim": 256, "rows": 1024, "prefix": 1024},
        # eight answers sampled together
        {"name": "sampling-8", "kind": "sampling", "rows": 8, "vocab": 128256, "temperature": 0.7, "top_k": 50, "top_p": 0.95, "min_p": 0.0},
        # mixers of a dense family at width 2048
        {"name": "delta-prompt", "kind": "delta", "heads": 16, "dim": 128, "rows": 1024},
        {"name": "latent-prompt", "kind": "latent", "heads": 16, "rank": 512, "rot": 64, "rows": 1024, "prefix": 0},
        # the feed-forward of one decoded token of a dense family at width 4096
        {"name": "mlp-decode", "kind": "mlp", "width": 4096, "ff": 14336, "rows": 1},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def _quant(rng):
    return {"bits": rng.choice([4, 4, 8]), "group": rng.choice([64, 64, 128, 32]), "method": rng.choice(["zero", "zero", "symmetric", "mlx"])}


def draw(rng):
    kind = rng.choice(["decode", "prompt", "batch", "verify", "linears", "attention", "sampling", "delta", "latent", "mlp"])
    if kind == "decode":
        if rng.random() < 0.5:
            return {"kind": kind, "model": "qwen3.5-0.8b", "layers": rng.choice([4, 8]), **_quant(rng), "vocab": 248320, "context": _log(rng, 16, 2048), "steps": 16}
        return {"kind": kind, "model": "llama3-8b", "layers": rng.choice([1, 2, 4]), **_quant(rng), "vocab": 32768, "context": _log(rng, 16, 6000), "steps": 8}
    if kind == "prompt":
        if rng.random() < 0.5:
            return {"kind": kind, "model": "qwen3.5-0.8b", "layers": rng.choice([4, 8]), **_quant(rng), "vocab": 248320, "tokens": _log(rng, 16, 1024)}
        return {"kind": kind, "model": "llama3-8b", "layers": rng.choice([1, 2, 4]), **_quant(rng), "vocab": 32768, "tokens": _log(rng, 16, 2048)}
    if kind == "batch":
        return {"kind": kind, "model": "llama3-8b", "layers": 1, **_quant(rng), "vocab": 32768, "sequences": rng.randint(2, 16), "tokens": _log(rng, 16, 300), "steps": 16}
    if kind == "verify":
        return {"kind": kind, "model": "llama3-8b", "layers": rng.choice([1, 2, 4]), **_quant(rng), "vocab": 32768, "context": _log(rng, 16, 4096), "nodes": rng.randint(2, 16)}
    if kind == "linears":
        return {"kind": kind, "model": rng.choice(["llama3-8b", "qwen3.5-0.8b"]), **_quant(rng), "rows": _log(rng, 2, 1024)}
    if kind == "attention":
        heads, groups, dim = rng.choice([(32, 8, 128), (8, 2, 256), (32, 8, 64)])
        return {"kind": kind, "heads": heads, "groups": groups, "dim": dim, "rows": _log(rng, 16, 1024), "prefix": _log(rng, 1, 3072)}
    if kind == "sampling":
        return {"kind": kind, "rows": rng.randint(1, 16), "vocab": rng.choice([32768, 128256, 248320]), "temperature": rng.choice([0.7, 1.0]), "top_k": rng.choice([0, 20, 50]),
                "top_p": rng.choice([0.0, 0.9, 0.95]), "min_p": rng.choice([0.0, 0.05])}
    if kind == "delta":
        return {"kind": kind, "heads": rng.choice([8, 16, 32]), "dim": rng.choice([64, 128, 128]), "rows": _log(rng, 1, 1024)}
    if kind == "latent":
        if rng.random() < 0.3:
            return {"kind": kind, "heads": rng.choice([8, 16, 32]), "rank": 512, "rot": 64, "rows": 1, "prefix": _log(rng, 16, 8000)}
        return {"kind": kind, "heads": rng.choice([8, 16]), "rank": rng.choice([256, 512]), "rot": 64, "rows": _log(rng, 16, 1024), "prefix": rng.choice([0, 0, _log(rng, 1, 500)])}
    width = rng.choice([1024, 2048, 4096])
    return {"kind": kind, "width": width, "ff": {1024: 4096, 2048: 8192, 4096: 14336}[width], "rows": rng.choice([1, 1, _log(rng, 128, 1024)])}


# ---- the models -------------------------------------------------------------------------------------------------------------------------
def _quant_spec(c):
    return synth.QuantSpec("mlx" if c["method"] == "mlx" else "int", c["bits"], c["group"], c["method"] == "symmetric")


def _spec(c):
    s = synth.PRESETS[c["model"]](bits=c["bits"], group_size=c["group"], layers=c["layers"])
    return dataclasses.replace(s, quant=_quant_spec(c), vocab_size=c["vocab"])


def _checkpoint(c):
    name = "-".join(str(c[k]) for k in ("model", "layers", "bits", "group", "method", "vocab"))
    base = Path(os.environ.get("UZU_MODEL_CACHE", "/dev/shm/uzu_b200_models")) / f"cases-{name}"
    if not (base / ".done").exists():
        tmp = base.with_name(f"{base.name}.{os.getpid()}")
        synth.write_model(_spec(c), tmp, seed=1)
        (tmp / ".done").write_text("ok")
        try:
            tmp.rename(base)
        except OSError:          # another process was first
            return base if (base / ".done").exists() else tmp
    return base


_context = None


def _ctx():
    global _context
    if _context is None:
        _context = B.Context(0)
    return _context


class _EngineState:
    """A loaded model with the tokens of this request."""

    def __init__(self, c, max_context):
        self.case = c
        self.engine = B.Engine(_ctx(), _checkpoint(c), max_context_length=max_context)

    def __del__(self):
        if getattr(self, "engine", None) is not None:
            self.engine.close()


class _BlockState:
    """Device tensors and the encoder of one command buffer; the buffer of the last pass is retired by the next one."""

    def __init__(self, c, encode, tensors, outputs):
        self.case, self.encode, self.tensors, self.outputs, self.pending = c, encode, tensors, outputs, None

    def run(self):
        lib = _ctx().lib
        self.retire()
        h = C.c_void_p()
        B._check(lib.uzu_command_buffer_create(_ctx().h, b"case", C.byref(h)))
        self.pending = h
        B._check(lib.uzu_command_buffer_start_encoding(h))
        self.encode(lib, h)
        B._check(lib.uzu_command_buffer_end_encoding(h))
        B._check(lib.uzu_command_buffer_submit(h))
        return self.outputs

    def retire(self):
        if self.pending is not None:
            h, self.pending = self.pending, None
            lib = _ctx().lib
            B._check(lib.uzu_command_buffer_wait_until_completed(h))
            lib.uzu_command_buffer_destroy(h)

    def __del__(self):
        self.retire()


def _bf16_of(bits):
    return torch.from_numpy(np.ascontiguousarray(bits).view(np.int16)).view(torch.bfloat16)


def _tokens(c, seed):
    rng = np.random.default_rng(seed)
    k = c["kind"]
    if k == "prompt":
        return {"prompt": rng.integers(0, c["vocab"], c["tokens"])}
    if k == "batch":     # every user's prompt has a length of its own
        lengths = [max(1, int(c["tokens"] * f)) for f in rng.uniform(0.5, 1.0, c["sequences"])]
        return {"prompts": [rng.integers(0, c["vocab"], n) for n in lengths], "steps": rng.integers(0, c["vocab"], (c["steps"], c["sequences"]))}
    if k == "decode":
        return {"prompt": rng.integers(0, c["vocab"], c["context"]), "steps": rng.integers(0, c["vocab"], c["steps"])}
    n = c["nodes"]
    heights = [0]
    for _ in range(n - 1):
        heights.append(int(rng.integers(1, heights[-1] + 2)))
    ends = []
    for i in range(n):
        j = i
        while j + 1 < n and heights[j + 1] > heights[i]:
            j += 1
        ends.append(j)
    nodes = np.array([[i, ends[i], heights[i]] for i in range(n)], dtype=np.uint32)
    return {"prompt": rng.integers(0, c["vocab"], c["context"]), "tokens": rng.integers(0, c["vocab"], n), "nodes": nodes}


# ---- blocks: inputs ------------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, std=1.0):
    return torch.randn(*shape, device="cuda", generator=g) * std


def _layer_shapes(model):
    if model == "llama3-8b":
        return [("qkv", 6144, 4096), ("out", 4096, 4096), ("up", 28672, 4096), ("down", 4096, 14336)]
    return [("qkv", 3072, 1024), ("out", 1024, 2048), ("up", 7168, 1024), ("down", 1024, 3584)]


def _linears_inputs(c, seed):
    g = _gen(seed)
    out, n_codes = [], 1 << c["bits"]
    for _, n, k in _layer_shapes(c["model"]):
        groups = k // c["group"]
        m = {"n": n, "k": k, "codes": torch.randint(0, 256, (n, k * c["bits"] // 8), device="cuda", generator=g, dtype=torch.uint8)}
        base = 1.0 / math.sqrt(k) / (n_codes / math.sqrt(6.0))
        m["scales"] = ((torch.rand(n, groups, device="cuda", generator=g) + 0.5) * base).bfloat16()
        if c["method"] == "mlx":
            m["biases"] = (-m["scales"].float() * torch.randint(0, n_codes, (n, groups), device="cuda", generator=g)).bfloat16()
        elif c["method"] == "zero":
            m["zero"] = torch.randint(0, 256, (n, -(-groups // 2) if c["bits"] == 4 else groups), device="cuda", generator=g, dtype=torch.uint8)
        m["x"] = _randn(g, c["rows"], k).bfloat16()
        m["y"] = torch.zeros(c["rows"], n, device="cuda", dtype=torch.bfloat16)
        out.append(m)
    return out


def _attention_inputs(c, seed):
    g, D, n = _gen(seed), c["dim"], c["prefix"] + c["rows"]
    return {"q": _randn(g, c["heads"], c["rows"], D).bfloat16(), "k": _randn(g, n, c["groups"], D).bfloat16(), "v": _randn(g, n, c["groups"], D).bfloat16(),
            "out": torch.zeros(c["rows"], c["heads"], D, device="cuda", dtype=torch.bfloat16)}


def _delta_inputs(c, seed):
    g, hd, T = _gen(seed), c["heads"] * c["dim"], c["rows"]
    t = {n: _randn(g, T, hd) for n in ("r", "k", "v", "rate", "decay")}
    t["rate_bias"], t["decay_bias"] = _randn(g, hd, std=0.5), _randn(g, hd, std=1.5) - 1.0
    t["state0"] = _randn(g, c["heads"], c["dim"], c["dim"], std=0.5)
    for n in ("rate", "decay"):      # the kernel works in place on these; a program's projections write them anew for each pass
        t[n + "_work"] = torch.empty_like(t[n])
    t["state"], t["unit"], t["out"] = torch.empty_like(t["state0"]), torch.empty(T, hd, device="cuda"), torch.zeros(T, hd, device="cuda")
    return t


def _latent_inputs(c, seed):
    g, n, w = _gen(seed), c["prefix"] + c["rows"], c["rank"] + c["rot"]
    splits = 1
    if c["rows"] < 16:       # as the engine cuts the keys of a decoded row
        splits = max(1, min(-(-n // 32), 2 * 148 // max(1, c["rows"] * -(-c["heads"] // 8)), 64))
    return {"q": _randn(g, c["rows"], c["heads"], w, std=0.7), "cache": _randn(g, n, w).bfloat16(), "splits": splits,
            "partials": torch.empty(c["rows"] * c["heads"] * splits * (c["rank"] + 2), device="cuda"),
            "out": torch.zeros(c["rows"], c["heads"], c["rank"], device="cuda")}


def _mlp_inputs(c, seed):
    g, W, F, m = _gen(seed), c["width"], c["ff"], c["rows"]
    return {"x": _randn(g, m, W), "up": _randn(g, 2 * F, W, std=W ** -0.5).bfloat16(), "down": _randn(g, W, F, std=F ** -0.5).bfloat16(),
            "h": torch.zeros(m, F, device="cuda"), "gate_up": torch.zeros(m, 2 * F if m > 8 else 1, device="cuda"),
            "work": torch.empty(m, max(W, F), device="cuda", dtype=torch.bfloat16), "out": torch.zeros(m, W, device="cuda")}


def _sampling_inputs(c, seed):
    g = _gen(seed)
    return {"logits": _randn(g, c["rows"], c["vocab"], std=2.5).bfloat16(), "out": torch.zeros(c["rows"], device="cuda", dtype=torch.int32),
            "seeds": torch.randint(0, 1 << 62, (c["rows"],), device="cuda", generator=g, dtype=torch.int64)}


# ---- prepare / run ---------------------------------------------------------------------------------------------------------------------------
def prepare(c, seed):
    k = c["kind"]
    if k in ("decode", "prompt", "batch", "verify"):
        t = _tokens(c, seed)
        most = c.get("context", 0) + c.get("steps", 0) + c.get("tokens", 0) + 64
        s = _EngineState(c, -(-most // 1024) * 1024)
        s.tokens = t
        if k in ("decode", "verify"):
            s.engine.prefill(t["prompt"])
            s.engine.snapshot()
        return s
    if k == "linears":
        mats = _linears_inputs(c, seed)
        prologue = {"mlx": B.B_SCALE_BIAS, "zero": B.B_SCALE_ZERO_POINT, "symmetric": B.B_SCALE_SYMMETRIC}[c["method"]]
        args = [B.MatmulArgs(a=m["x"].data_ptr(), b=m["codes"].data_ptr(), b_scales=m["scales"].data_ptr(), b_zero_points=m["zero"].data_ptr() if "zero" in m else 0,
                             b_biases=m["biases"].data_ptr() if "biases" in m else 0, d=m["y"].data_ptr(), b_prologue=prologue,
                             b_mode=B.QMODE_U4 if c["bits"] == 4 else B.QMODE_U8, b_group_size=c["group"], b_transpose=1, ab_scale=1.0, m=c["rows"], n=m["n"], k=m["k"],
                             weights_dt=B.DT_BF16, input_dt=B.DT_BF16, output_dt=B.DT_BF16) for m in mats]

        def encode(lib, h):
            for a in args:
                lib.uzu_matmul_encode(h, C.byref(a))
        return _BlockState(c, encode, mats, [m["y"] for m in mats])
    if k == "attention":
        t, D = _attention_inputs(c, seed), c["dim"]
        a = B.AttentionArgs(queries=t["q"].data_ptr(), keys=t["k"].data_ptr(), values=t["v"].data_ptr(), out=t["out"].data_ptr(), gqa_factor=c["heads"] // c["groups"],
                            sequence_length=c["prefix"] + c["rows"], k_head_stride=D, k_seq_stride=c["groups"] * D, v_head_stride=D, v_seq_stride=c["groups"] * D,
                            scale=D ** -0.5, num_heads=c["heads"], suffix_length=c["rows"], head_dim=D, is_causal=1)
        return _BlockState(c, lambda lib, h: lib.uzu_attention_single_pass_encode(h, C.byref(a)), t, t["out"])
    if k == "sampling":
        t = _sampling_inputs(c, seed)
        a = B.UnifiedSamplingArgs(logits=t["logits"].data_ptr(), output=t["out"].data_ptr(), seeds=t["seeds"].data_ptr(), temperature=c["temperature"], top_k=c["top_k"],
                                  top_p=c["top_p"], min_p=c["min_p"], vocab_size=c["vocab"], batch_size=c["rows"], is_stochastic=1, has_temperature=1,
                                  has_top_k=int(c["top_k"] > 0), has_top_p=int(c["top_p"] > 0), has_min_p=int(c["min_p"] > 0))
        return _BlockState(c, lambda lib, h: lib.uzu_unified_sampling_encode(h, C.byref(a)), t, t["out"])
    if k == "delta":
        t = _delta_inputs(c, seed)
        hd = c["heads"] * c["dim"]
        a = B.GeneralDeltaArgs(r=t["r"].data_ptr(), k=t["k"].data_ptr(), v=t["v"].data_ptr(), rate_logit=t["rate_work"].data_ptr(), decay_logit=t["decay_work"].data_ptr(),
                               rate_bias=t["rate_bias"].data_ptr(), decay_bias=t["decay_bias"].data_ptr(), unit=t["unit"].data_ptr(), state=t["state"].data_ptr(),
                               out=t["out"].data_ptr(), r_stride=hd, k_stride=hd, v_stride=hd, rate_stride=hd, decay_stride=hd, rows=c["rows"], heads=c["heads"], dim=c["dim"])

        def encode(lib, h):
            for n, d in (("rate", "rate_work"), ("decay", "decay_work"), ("state0", "state")):
                lib.uzu_command_buffer_encode_copy(h, t[n].data_ptr(), t[d].data_ptr(), t[n].numel() * 4)
            lib.uzu_general_delta_encode(h, C.byref(a))
        return _BlockState(c, encode, t, [t["out"], t["state"]])
    if k == "latent":
        t = _latent_inputs(c, seed)
        a = B.LatentAttentionArgs(query=t["q"].data_ptr(), cache=t["cache"].data_ptr(), out=t["out"].data_ptr(), partials=t["partials"].data_ptr(), rows=c["rows"],
                                  heads=c["heads"], rank=c["rank"], rot_dim=c["rot"], prefix=c["prefix"], cache_dt=B.DT_BF16, scale=192 ** -0.5, splits=t["splits"])
        return _BlockState(c, lambda lib, h: lib.uzu_latent_attention_encode(h, C.byref(a)), t, t["out"])
    t = _mlp_inputs(c, seed)
    W, F, m = c["width"], c["ff"], c["rows"]
    common = dict(m=m, batch=1, weights_dt=B.DT_BF16, scale=1.0, workspace=t["work"].data_ptr() if m >= 128 else 0)
    down = B.DenseLinearArgs(a=t["h"].data_ptr(), w=t["down"].data_ptr(), d=t["out"].data_ptr(), n=W, k=F, lda=F, ldd=W, **common)
    if m <= 8:       # the gated unit as the product's epilogue
        up = B.DenseLinearArgs(a=t["x"].data_ptr(), w=t["up"].data_ptr(), d=t["h"].data_ptr(), n=F, k=W, lda=W, ldd=F, pair_rows=F, glu_kind=1, **common)
    else:
        up = B.DenseLinearArgs(a=t["x"].data_ptr(), w=t["up"].data_ptr(), d=t["gate_up"].data_ptr(), n=2 * F, k=W, lda=W, ldd=2 * F, **common)

    def encode(lib, h):
        lib.uzu_dense_linear_encode(h, C.byref(up))
        if m > 8:
            lib.uzu_silu_glu_encode(h, t["gate_up"].data_ptr(), t["h"].data_ptr(), m, F)
        lib.uzu_dense_linear_encode(h, C.byref(down))
    return _BlockState(c, encode, t, t["out"])


def run(s):
    if isinstance(s, _BlockState):
        return s.run()
    e, t, k = s.engine, s.tokens, s.case["kind"]
    if k == "prompt":
        e.reset()
        e.prefill(t["prompt"])
        return _bf16_of(e.last_logits())
    if k == "decode":
        e.restore()
        for tok in t["steps"]:
            e.step_host(tok)
        return _bf16_of(e.last_logits())
    if k == "batch":
        e.batch_begin(len(t["prompts"]))
        for i, p in enumerate(t["prompts"]):
            e.batch_prefill(i, p)
        for row in t["steps"]:
            e.batch_step(row)
        return _bf16_of(e.batch_logits())
    _, logits = e.trie_pass(t["tokens"], t["nodes"], want_logits=True)
    e.trie_accept([0], int(t["tokens"][0]))
    e.restore()
    return _bf16_of(logits)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------------------
def _matrix_bytes(n, k, bits, group, method):
    groups = k // group
    extra = {"mlx": 2 * groups, "symmetric": 0, "zero": -(-groups // 2) if bits == 4 else groups}[method]
    return n * (k * bits // 8 + 2 * groups + extra)


def _model_work(c):
    """(bytes of the weights of one pass, multiply-adds of a row without readout and attention, bytes of the readout, cache bytes and
    multiply-adds of a row and a cached token, bytes of recurrent state)"""
    s = _spec(c)
    mats, cache, macs, state = [], 0, 0, 0
    for kind in s.layer_kinds:
        if kind == "attn":
            q, kv = s.num_heads * s.head_dim, s.num_groups * s.head_dim
            mats += [(q + 2 * kv, s.model_dim), (s.model_dim, q)] + ([(q, s.model_dim)] if s.attn_gate else [])
            cache += 2 * kv * 2
            macs += 2 * q
        else:
            kd, vd = s.dn_num_groups * s.dn_head_dim, s.dn_num_heads * s.dn_value_head_dim
            mats += [(2 * kd + 2 * vd + 2 * s.dn_num_heads, s.model_dim), (s.model_dim, vd)]
            state += 2 * 4 * vd * s.dn_head_dim
        mats += [(2 * s.hidden_dim, s.model_dim), (s.model_dim, s.hidden_dim)]
    q = (c["bits"], c["group"], c["method"])
    return sum(_matrix_bytes(n, k, *q) for n, k in mats), sum(n * k for n, k in mats), _matrix_bytes(s.vocab_size, s.model_dim, *q), cache, macs, state


def work(c):
    k = c["kind"]
    if k in ("decode", "prompt", "batch", "verify"):
        w, row, head, cache, att, state = _model_work(c)
        head_macs = c["vocab"] * _spec(c).model_dim
        if k == "decode":
            n = c["steps"]
            return {"bytes": n * (w + head + state + cache * (c["context"] + n / 2)), "flops": 2.0 * n * (row + head_macs + att * c["context"])}
        if k == "prompt":
            n = c["tokens"]
            return {"bytes": w + head + state + cache * n, "flops": 2.0 * (n * row + head_macs + att * n * n / 2)}
        if k == "verify":
            n = c["nodes"]
            return {"bytes": w + head + cache * c["context"] + n * c["vocab"] * 2, "flops": 2.0 * n * (row + head_macs + att * c["context"])}
        n, b, p = c["steps"], c["sequences"], c["tokens"] * 0.75
        return {"bytes": (b + n) * (w + head) + n * b * cache * p, "flops": 2.0 * b * (p * row + n * (row + head_macs) + att * p * (p / 2 + n))}
    if k == "linears":
        m = c["rows"]
        return {"bytes": sum(_matrix_bytes(n, kk, c["bits"], c["group"], c["method"]) + 2 * m * (n + kk) for _, n, kk in _layer_shapes(c["model"])),
                "flops": 2.0 * m * sum(n * kk for _, n, kk in _layer_shapes(c["model"]))}
    if k == "attention":
        n, m = c["prefix"] + c["rows"], c["rows"]
        return {"bytes": 2 * c["dim"] * (2 * c["groups"] * n + 2 * c["heads"] * m), "flops": 4.0 * c["heads"] * c["dim"] * m * (c["prefix"] + m / 2)}
    if k == "sampling":
        return {"bytes": c["rows"] * c["vocab"] * 2, "flops": 0}
    if k == "delta":
        hd = c["heads"] * c["dim"]
        return {"bytes": 4 * (6 * c["rows"] * hd + 2 * hd * c["dim"]), "flops": 9.0 * c["rows"] * hd * c["dim"]}
    if k == "latent":
        n, w = c["prefix"] + c["rows"], c["rank"] + c["rot"]
        return {"bytes": 2 * n * w + 4 * c["rows"] * c["heads"] * (w + c["rank"]), "flops": 2.0 * c["heads"] * c["rows"] * (c["prefix"] + c["rows"] / 2) * (w + c["rank"])}
    return {"bytes": 6 * c["width"] * c["ff"] + 8 * c["rows"] * c["width"], "flops": 6.0 * c["rows"] * c["width"] * c["ff"]}


def tolerance(c):
    k = c["kind"]
    if k == "sampling":
        return "exact"
    if k in ("delta", "latent"):                 # f32 sums
        return {"rel": 1e-5, "max": 1e-3}
    if k == "mlp":                               # one token: f32 rows; a prompt: rows rounded to bf16 for the tensor pipe
        return {"rel": 1e-5, "max": 1e-3} if c["rows"] <= 8 else {"rel": 1e-2, "max": 0.1}
    if k in ("linears", "attention"):            # bf16 results of f32 sums
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 0.03, "max": 0.3}             # bf16 logits behind several layers


# ---- 64-bit restatements -------------------------------------------------------------------------------------------------------------------------
def _read(path):
    with open(path / "model.safetensors", "rb") as f:
        (n,) = struct.unpack("<Q", f.read(8))
        header = json.loads(f.read(n))
    data = np.memmap(path / "model.safetensors", dtype=np.uint8, mode="r", offset=8 + n)
    header.pop("__metadata__", None)
    return header, data


def _dequant(codes, scales, zero, biases, bits, group):
    if bits == 4:
        codes = torch.stack([codes & 15, codes >> 4], -1).flatten(-2)
        if zero is not None:
            zero = torch.stack([zero & 15, zero >> 4], -1).flatten(-2)[:, :scales.shape[1]]
    w = codes.to(F64).reshape(codes.shape[0], -1, group)
    if biases is not None:
        return (w * scales.to(F64)[..., None] + biases.to(F64)[..., None]).flatten(1)
    z = zero.to(F64)[..., None] if zero is not None else float(1 << (bits - 1))
    return ((w - z) * scales.to(F64)[..., None]).flatten(1)


class _Model64:
    def __init__(self, c):
        self.c, self.s = c, _spec(c)
        self.header, self.data = _read(_checkpoint(c))

    def raw(self, name):
        if name not in self.header:
            return None
        h = self.header[name]
        t = torch.from_numpy(np.array(self.data[h["data_offsets"][0]:h["data_offsets"][1]])).cuda()
        return t.view({"F32": torch.float32, "BF16": torch.bfloat16, "U8": torch.uint8}[h["dtype"]]).reshape(h["shape"])

    def matrix(self, p, rows=None):
        parts = [self.raw(p + n) for n in (".weights", ".scales", ".zero_points", ".biases")]
        if rows is not None:
            parts = [None if x is None else x[rows] for x in parts]
        return _dequant(*parts, self.c["bits"], self.c["group"])

    def norm(self, x, name, eps, offset):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * (self.raw(name).to(F64) + (offset or 0.0))

    def rope(self, x, pos):
        r = self.s.rope
        d = r["head_dim"]
        inv = r["base"] ** (-torch.arange(0, d, 2, device="cuda", dtype=F64) / d)
        if r["type"] == "LlamaRoPEConfig":
            wave = 2 * math.pi / inv
            low, high = r["original_context_length"] / r["low_frequency_factor"], r["original_context_length"] / r["high_frequency_factor"]
            smooth = (r["original_context_length"] / wave - r["low_frequency_factor"]) / (r["high_frequency_factor"] - r["low_frequency_factor"])
            mixed = smooth * inv + (1 - smooth) * inv / r["scaling_factor"]
            inv = torch.where(wave < high, inv, torch.where(wave > low, inv / r["scaling_factor"], mixed))
        a = pos.to(F64)[:, None] * inv
        co, si = a.cos()[:, None, :], a.sin()[:, None, :]
        x1, x2, rest = x[..., :d // 2], x[..., d // 2:d], x[..., d:]
        return torch.cat([x1 * co - x2 * si, x2 * co + x1 * si, rest], -1)

    def attention(self, x, p, pos, mask):
        s, m = self.s, x.shape[0]
        qd, kd = s.num_heads * s.head_dim, s.num_groups * s.head_dim
        y = x @ self.matrix(p + "qkv_projection.weights").T
        q, k, v = y[:, :qd].reshape(m, -1, s.head_dim), y[:, qd:qd + kd].reshape(m, -1, s.head_dim), y[:, qd + kd:].reshape(m, -1, s.head_dim)
        if s.qk_norm:
            q, k = (self.norm(t, p + n + "_norm.scales", 1e-6, s.qk_norm_scale_offset) for t, n in ((q, "query"), (k, "key")))
        q, k = self.rope(q, pos), self.rope(k, pos)
        out, per = torch.empty_like(q), s.num_heads // s.num_groups
        for h in range(s.num_heads):
            a = (q[:, h] @ k[:, h // per].T * s.head_dim ** -0.5).masked_fill(~mask, -math.inf)
            out[:, h] = torch.softmax(a, -1) @ v[:, h // per]
        out = out.flatten(1)
        if s.attn_gate:
            out = out * torch.sigmoid(x @ self.matrix(p + "gate_projection.weights").T)
        return out @ self.matrix(p + "out_projection.weights").T

    def delta_net(self, x, p):
        s, m = self.s, x.shape[0]
        G, Hv, Dk, Dv, taps = s.dn_num_groups, s.dn_num_heads, s.dn_head_dim, s.dn_value_head_dim, s.dn_kernel_size
        kd, vd = G * Dk, Hv * Dv
        y = x @ self.matrix(p + "in_proj.weights").T
        u, z, b, a = y[:, :2 * kd + vd], y[:, 2 * kd + vd:2 * kd + 2 * vd], y[:, 2 * kd + 2 * vd:2 * kd + 2 * vd + Hv], y[:, 2 * kd + 2 * vd + Hv:]
        w = self.raw(p + "conv.weights").to(F64)
        padded = torch.cat([torch.zeros(taps - 1, u.shape[1], device="cuda", dtype=F64), u])
        u = torch.nn.functional.silu(sum(padded[j:j + m] * w[:, j] for j in range(taps)))
        q, k, v = u[:, :kd].reshape(m, G, Dk), u[:, kd:2 * kd].reshape(m, G, Dk), u[:, 2 * kd:].reshape(m, Hv, Dv)
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)    # noqa: E731
        q, k = unit(q).repeat_interleave(Hv // G, 1) * Dk ** -0.5, unit(k).repeat_interleave(Hv // G, 1)
        beta = torch.sigmoid(b)
        g = torch.exp(-torch.exp(self.raw(p + "a_log").to(F64)) * torch.nn.functional.softplus(a + self.raw(p + "dt_bias").to(F64)))
        S, o = torch.zeros(Hv, Dv, Dk, device="cuda", dtype=F64), torch.empty(m, Hv, Dv, device="cuda", dtype=F64)
        for t in range(m):
            S = S * g[t, :, None, None]
            S = S + (beta[t, :, None] * (v[t] - (S @ k[t, :, :, None])[..., 0]))[..., None] * k[t, :, None, :]
            o[t] = (S @ q[t, :, :, None])[..., 0]
        o = self.norm(o, p + "norm.scales", 1e-6, None) * torch.nn.functional.silu(z).reshape(m, Hv, Dv)
        return o.flatten(1) @ self.matrix(p + "out_proj.weights").T

    def logits(self, tokens, rows, pos=None, mask=None):
        s, m = self.s, len(tokens)
        tokens = torch.as_tensor(np.asarray(tokens, np.int64), device="cuda")
        pos = torch.arange(m, device="cuda") if pos is None else pos
        mask = torch.ones(m, m, device="cuda", dtype=torch.bool).tril() if mask is None else mask
        e = "decoder.embedding." + ("embedding" if s.tied_embeddings else "input_embedding")
        x = self.matrix(e, tokens)
        for i, kind in enumerate(s.layer_kinds):
            p = f"decoder.transformer.layers.{i}."
            h = self.norm(x, p + "pre_mixer_norm.scales", s.norm_eps, s.norm_scale_offset)
            x = x + (self.attention(h, p + "mixer.", pos, mask) if kind == "attn" else self.delta_net(h, p + "mixer."))
            up = self.norm(x, p + "pre_mlp_norm.scales", s.norm_eps, s.norm_scale_offset) @ self.matrix(p + "mlp.up_projection.weights").T
            x = x + (up[:, :s.hidden_dim] * torch.nn.functional.silu(up[:, s.hidden_dim:])) @ self.matrix(p + "mlp.down_projection.weights").T
        x = self.norm(x[rows], "decoder.transformer.output_norm.scales", s.norm_eps, s.norm_scale_offset)
        head, out = "decoder.embedding." + ("embedding" if s.tied_embeddings else "output_embedding"), []
        for v0 in range(0, s.vocab_size, 32768):
            out.append(x @ self.matrix(head, slice(v0, v0 + 32768)).T)
        return torch.cat(out, -1)


def exact(c, seed):
    k = c["kind"]
    if k == "sampling":
        return None
    if k in ("decode", "prompt", "batch", "verify"):
        t, model = _tokens(c, seed), _Model64(c)
        if k == "prompt":
            return model.logits(t["prompt"], [-1])
        if k == "decode":
            return model.logits(np.concatenate([t["prompt"], t["steps"]]), [-1])
        if k == "batch":
            return torch.cat([model.logits(np.concatenate([p, t["steps"][:, i]]), [-1]) for i, p in enumerate(t["prompts"])])
        P, n = c["context"], c["nodes"]
        heights = torch.as_tensor(t["nodes"][:, 2].astype(np.int64), device="cuda")
        mask = torch.ones(P + n, P + n, device="cuda", dtype=torch.bool).tril()
        for j in range(n):            # node j is seen by its own subtree only
            mask[P:, P + j] = False
            mask[P + j:P + int(t["nodes"][j, 1]) + 1, P + j] = True
        pos = torch.cat([torch.arange(P, device="cuda"), P + heights])
        return model.logits(np.concatenate([t["prompt"], t["tokens"]]), list(range(P, P + n)), pos, mask)
    if k == "linears":
        return [m["x"].to(F64) @ _dequant(m["codes"], m["scales"], m.get("zero"), m.get("biases"), c["bits"], c["group"]).T for m in _linears_inputs(c, seed)]
    if k == "attention":
        t, per = _attention_inputs(c, seed), c["heads"] // c["groups"]
        mask = torch.arange(c["prefix"] + c["rows"], device="cuda")[None, :] <= c["prefix"] + torch.arange(c["rows"], device="cuda")[:, None]
        out = torch.empty(c["rows"], c["heads"], c["dim"], device="cuda", dtype=F64)
        for h in range(c["heads"]):
            a = (t["q"][h].to(F64) @ t["k"][:, h // per].to(F64).T * c["dim"] ** -0.5).masked_fill(~mask, -math.inf)
            out[:, h] = torch.softmax(a, -1) @ t["v"][:, h // per].to(F64)
        return out
    if k == "delta":
        t, H, D, T = {n: x.to(F64) for n, x in _delta_inputs(c, seed).items()}, c["heads"], c["dim"], c["rows"]
        r, kk, v = (t[n].reshape(T, H, D) for n in ("r", "k", "v"))
        d = torch.exp(-math.exp(-0.5) * torch.sigmoid(t["decay"] + t["decay_bias"])).reshape(T, H, D)
        a = torch.sigmoid(t["rate"] + t["rate_bias"]).reshape(T, H, D)
        u = kk / torch.sqrt((kk * kk).sum(-1, keepdim=True) + 1e-6)
        S, out = t["state0"], torch.empty(T, H, D, device="cuda", dtype=F64)
        for i in range(T):
            S = d[i][..., None] * S - (a[i] * u[i])[..., None] * (u[i][:, None, :] @ S) + kk[i][..., None] * v[i][:, None, :]
            out[i] = (r[i][:, None, :] @ S)[:, 0]
        return [out.reshape(T, H * D), S]
    if k == "latent":
        t, n = _latent_inputs(c, seed), c["prefix"] + c["rows"]
        cache = t["cache"].to(F64)
        mask = torch.arange(n, device="cuda")[None, :] <= c["prefix"] + torch.arange(c["rows"], device="cuda")[:, None]
        out = torch.empty(c["rows"], c["heads"], c["rank"], device="cuda", dtype=F64)
        for h in range(c["heads"]):
            out[:, h] = torch.softmax((t["q"][:, h].to(F64) @ cache.T * 192 ** -0.5).masked_fill(~mask, -math.inf), -1) @ cache[:, :c["rank"]]
        return out
    t, F = _mlp_inputs(c, seed), c["ff"]
    y = t["x"].to(F64) @ t["up"].to(F64).T
    return (torch.nn.functional.silu(y[:, :F]) * y[:, F:]) @ t["down"].to(F64).T

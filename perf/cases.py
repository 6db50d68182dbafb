"""What a user of this framework has it do, as measurable cases.

Every case goes through the public entry points: the C ABI (tensormark_b200.lib, include/cuda_shim.h) for single
projections and for decode attention, the chain driver (tensormark_b200.chain, include/llama_chain.h) for whole models.

  gemv       y = W x, device pointers: the same projection of `layers` layers of one decoded token, one call each
  gemv_host  the same through the host-pointer entry, x and y in page-locked host memory (the per-tensor hook of a host program)
  gemm       C = A W^T for a batch of tokens, device pointers: one projection of a prompt
  attn       decode attention of one token over a K/V cache, device pointers
  decode     a prompt through the batched layer stack, then greedy tokens on the GPU
  prompt     a prompt through the batched layer stack up to the model's first token
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from tensormark_b200 import chain, lib, synth

DTYPES = {"Q8_0": synth.Q8_0, "Q4_0": synth.Q4_0, "Q4_1": synth.Q4_1, "Q5_K": synth.Q5_K, "Q6_K": synth.Q6_K, "Q4_K": synth.Q4_K,
          "GGUF_Q4_0": synth.GGUF_Q4_0, "F16": synth.F16, "BF16": synth.BF16}

# Two model geometries. 4096 positions of K/V cache: what a serving program reserves, not what one request uses.
MODELS = {
    "llama3_8b": dict(synth.LLAMA3_8B, ctx=4096),                                  # Q4_0 projections, Q6_K head
    "tinyllama": dict(L=22, D=2048, H=32, KVH=4, dh=64, F=5632, V=32000, ctx=4096, theta=10000.0, eps=1e-5,
                      dt_proj=synth.Q8_0, dt_head=synth.Q8_0, dt_embed=synth.Q8_0),
}


def listed():
    return [
        # the K projection of a small model's layers: the smallest call there is, all launch and latency
        {"name": "gemv_q4_0_256x2048_x8", "op": "gemv", "dtype": "Q4_0", "n": 256, "k": 2048, "layers": 8},
        # a small model's LM head, the widest format: pure streaming
        {"name": "gemv_q8_0_32000x2048", "op": "gemv", "dtype": "Q8_0", "n": 32000, "k": 2048, "layers": 1},
        # the down projection of an 8B model: long rows, few of them, a K-quant
        {"name": "gemv_q5_k_4096x14336", "op": "gemv", "dtype": "Q5_K", "n": 4096, "k": 14336, "layers": 1},
        # rows whose byte length is no multiple of 16 (eleven super-blocks) and an odd number of them
        {"name": "gemv_q6_k_5119x2816", "op": "gemv", "dtype": "Q6_K", "n": 5119, "k": 2816, "layers": 1},
        # the gate projection as a host program's per-tensor hook calls it, once per tensor and token
        {"name": "gemv_host_q4_1_5632x2048", "op": "gemv_host", "dtype": "Q4_1", "n": 5632, "k": 2048},
        # a long prompt against a small model's gate projection
        {"name": "gemm_q4_0_2000x5632x2048", "op": "gemm", "dtype": "Q4_0", "m": 2000, "n": 5632, "k": 2048},
        # the same prompt against the LM head: the largest single contraction
        {"name": "gemm_q6_k_2000x32000x2048", "op": "gemm", "dtype": "Q6_K", "m": 2000, "n": 32000, "k": 2048},
        # a short prompt or a handful of sequences: few, odd tokens, the weights are the traffic
        {"name": "gemm_q4_0_17x4096x4096", "op": "gemm", "dtype": "Q4_0", "m": 17, "n": 4096, "k": 4096},
        # decode attention of an 8B model late in a long conversation
        {"name": "attn_f16_32x8x128_8191", "op": "attn", "heads": 32, "kv_heads": 8, "dh": 128, "allow": 8191, "half": True},
        # a question and its answer: 512 tokens in, 128 out
        {"name": "decode_llama3_8b_512_128", "op": "decode", "model": "llama3_8b", "prompt": 512, "steps": 128},
        # a small model, short prompt: every layer is a few microseconds of work
        {"name": "decode_tinyllama_33_64", "op": "decode", "model": "tinyllama", "prompt": 33, "steps": 64},
        # time to the first token of a document
        {"name": "prompt_llama3_8b_1500", "op": "prompt", "model": "llama3_8b", "prompt": 1500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["gemv", "gemv_host", "gemm", "attn", "decode", "prompt"], [6, 1, 5, 2, 2, 2])[0]
    if op in ("gemv", "gemv_host"):
        dtype = rng.choice([d for d in DTYPES if op == "gemv" or d not in ("F16", "BF16")])
        be = synth.BLOCK_ELEMS.get(DTYPES[dtype], 32)
        # most rows are a multiple of 256 long, some any number of blocks
        step = 256 if be == 256 or rng.random() < 0.7 else be
        k = max(1, _log(rng, 256, 14336) // step) * step
        top = 430e6 if op == "gemv" else 70e6
        n = max(1, min(_log(rng, 64, 131072), int(top / _row_bytes(dtype, k))))
        if op == "gemv_host":
            return {"op": op, "dtype": dtype, "n": n, "k": k}
        # short calls come in numbers: a token has one of them for every layer
        return {"op": op, "dtype": dtype, "n": n, "k": k, "layers": 8 if n * _row_bytes(dtype, k) < 8e6 else 1}
    if op == "gemm":
        dtype = rng.choice([d for d in DTYPES if d not in ("F16", "BF16")])
        be = synth.BLOCK_ELEMS[DTYPES[dtype]]
        step = 256 if be == 256 or rng.random() < 0.7 else be
        k = max(1, _log(rng, 256, 14336) // step) * step
        m = _log(rng, 2, 2048)
        n = min(_log(rng, 128, 32768), int(262e9 / (2 * m * k)))
        return {"op": "gemm", "dtype": dtype, "m": m, "n": max(64, n), "k": k}
    if op == "attn":
        heads, kv_heads, dh = rng.choice([(32, 8, 128), (32, 4, 64), (32, 32, 128), (16, 8, 64)])
        return {"op": "attn", "heads": heads, "kv_heads": kv_heads, "dh": dh, "allow": _log(rng, 64, 32768), "half": rng.random() < 0.75}
    model = rng.choice(sorted(MODELS))
    if op == "decode":
        return {"op": "decode", "model": model, "prompt": _log(rng, 3, 512), "steps": _log(rng, 8, 128)}
    return {"op": "prompt", "model": model, "prompt": _log(rng, 16, 2000)}


# ---- inputs --------------------------------------------------------------------------------------------------
def _row_bytes(dtype, k):
    dt = DTYPES[dtype]
    return 2 * k if dt in (synth.F16, synth.BF16) else synth.weight_bytes(dt, 1, k)


def _blocks(dt, n, k, gen):
    """Random blocks of an n x k tensor on the GPU, flat uint8: the field distributions of synth.make_weights."""
    if dt in (synth.F16, synth.BF16):
        w = torch.randn(n * k, generator=gen, device="cuda") * 0.05
        return w.to(torch.float16 if dt == synth.F16 else torch.bfloat16).view(torch.uint8)
    nb, bb = n * (k // synth.BLOCK_ELEMS[dt]), synth.BLOCK_BYTES[dt]
    out = torch.randint(0, 256, (nb, bb), generator=gen, device="cuda", dtype=torch.uint8)

    def half(scale, signed=False):
        v = torch.randn(nb, generator=gen, device="cuda") * scale
        return (v if signed else v.abs()).half().view(torch.uint8).view(nb, 2)

    if dt == synth.Q8_0:
        out[:, 2:] = torch.randint(-127, 128, (nb, 32), generator=gen, device="cuda", dtype=torch.int8).view(torch.uint8)
        out[:, 0:2] = half(0.005)
    elif dt == synth.Q6_K:
        out[:, 192:208] = torch.randint(-32, 32, (nb, 16), generator=gen, device="cuda", dtype=torch.int8).view(torch.uint8)
        out[:, 208:210] = half(0.001)
    elif dt in (synth.Q5_K, synth.Q4_K):
        out[:, 0:2] = half(0.001)
        out[:, 2:4] = half(0.001)
    else:
        out[:, 0:2] = half(0.02)
        if dt == synth.Q4_1:
            out[:, 2:4] = half(0.05, signed=True)
    return out.view(-1)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _device_weights(dt, n, k, gen):
    """The blocks with the 32 spare bytes behind them that every weight buffer has."""
    b = _blocks(dt, n, k, gen)
    out = torch.zeros(b.numel() + 32, dtype=torch.uint8, device="cuda")
    out[:b.numel()] = b
    return out


# Weights that a program loads once and keeps. The library knows host tensors by their address, so they live as long as the process.
_host_tensors = {}
_model = {"name": None, "chain": None, "weights": None}


def _host_weights(dtype, n, k):
    key = (dtype, n, k)
    if key not in _host_tensors:
        _host_tensors[key] = _blocks(DTYPES[dtype], n, k, _gen(11)).cpu()
    return _host_tensors[key]


def _make_weights(cfg, gen):
    """A random-init model, every tensor inside one host mapping, as synth.make_llama lays it out."""
    L, D, F, V = cfg["L"], cfg["D"], cfg["F"], cfg["V"]
    qd, kvd = cfg["H"] * cfg["dh"], cfg["KVH"] * cfg["dh"]
    specs = [("embed", cfg["dt_embed"], V, D), ("head", cfg["dt_head"], V, D)]
    for l in range(L):
        for name, n, k in (("q", qd, D), ("k", kvd, D), ("v", kvd, D), ("o", D, qd), ("gate", F, D), ("up", F, D), ("down", D, F)):
            specs.append((f"l{l}.{name}", cfg["dt_proj"], n, k))
    size = sum((synth.weight_bytes(dt, n, k) + 15) // 16 * 16 for _, dt, n, k in specs) + 64
    blob = torch.zeros(size, dtype=torch.uint8)
    host, out, at = blob.numpy(), {}, 0
    out["blob"] = host
    for name, dt, n, k in specs:
        nb = synth.weight_bytes(dt, n, k)
        blob[at:at + nb] = _blocks(dt, n, k, gen)
        out[name] = host[at:at + nb].reshape(n, -1)
        at += (nb + 15) // 16 * 16
    for name in ["rmsf"] + [f"l{l}.rms{i}" for l in range(L) for i in (1, 2)]:
        out[name] = (1.0 + 0.02 * torch.randn(D, generator=gen, device="cuda")).cpu().numpy()
    return out


def _chain(name):
    """The loaded model. A process has one decode lane, so it holds one model at a time."""
    if _model["name"] != name:
        if _model["chain"] is not None:
            _model["chain"].close()
        cfg = MODELS[name]
        _model["weights"] = _make_weights(cfg, _gen(5))
        _model["chain"] = chain.Chain(cfg, _model["weights"])
        _model["chain"].prefill_prepare(2048)
        _model["name"] = name
    return _model["chain"]


def prepare(case, seed):
    cuda = lib.load()
    lib.check(cuda.tm_cuda_init(torch.cuda.current_device()), "tm_cuda_init")
    op, gen = case["op"], _gen(seed)
    ptr = lambda t: C.c_void_p(t.data_ptr())                                       # noqa: E731
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if op == "gemv":
        n, k, dt, layers = case["n"], case["k"], DTYPES[case["dtype"]], case["layers"]
        w = [_device_weights(dt, n, k, gen) for _ in range(layers)]
        x = [torch.randn(k, generator=gen, device="cuda") for _ in range(layers)]
        y = [torch.empty(n, device="cuda") for _ in range(layers)]
        args = [(ptr(x[i]), ptr(w[i]), ptr(y[i]), n, k, dt, stream) for i in range(layers)]
        return {"call": cuda.tm_cuda_gemv_q_dev, "args": args, "out": y, "keep": (w, x)}
    if op == "gemv_host":
        n, k, dt = case["n"], case["k"], DTYPES[case["dtype"]]
        w = _host_weights(case["dtype"], n, k)
        x = torch.randn(k, generator=gen, device="cuda").cpu().pin_memory()
        y = torch.empty(n).pin_memory()
        return {"call": cuda.tm_cuda_gemv_q, "args": [(ptr(x), ptr(w), ptr(y), n, k, dt)], "out": y, "keep": (w, x)}
    if op == "gemm":
        m, n, k, dt = case["m"], case["n"], case["k"], DTYPES[case["dtype"]]
        w = _device_weights(dt, n, k, gen)
        a = torch.randn(m, k, generator=gen, device="cuda")
        c = torch.empty(m, n, device="cuda")
        need = cuda.tm_cuda_sgemm_q_workspace(m, n, k, dt)
        ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
        base = C.c_void_p((ws.data_ptr() + 255) // 256 * 256)
        return {"call": cuda.tm_cuda_sgemm_q_dev, "args": [(ptr(a), ptr(w), ptr(c), m, n, k, dt, base, need, stream)], "out": c, "keep": (w, a, ws)}
    if op == "attn":
        h, kvh, dh, allow = case["heads"], case["kv_heads"], case["dh"], case["allow"]
        ctx = (allow + 255) // 256 * 256
        kv = torch.float16 if case["half"] else torch.float32
        q = torch.randn(h * dh, generator=gen, device="cuda")
        kc, vc = (torch.randn(kvh * ctx * dh, generator=gen, device="cuda").to(kv) for _ in range(2))
        need = cuda.tm_cuda_attn_decode_scratch(h, kvh, dh, ctx, allow)
        scratch = torch.empty(need // 4 + 4, device="cuda")
        out = torch.empty(h * dh, device="cuda")
        return {"call": cuda.tm_cuda_attn_decode_dev,
                "args": [(ptr(q), ptr(kc), ptr(vc), ptr(scratch), need, ptr(out), h, kvh, dh, ctx, allow, 1.0 / math.sqrt(dh), int(case["half"]), stream)],
                "out": out, "keep": (q, kc, vc, scratch)}
    m = _chain(case["model"])
    rng = np.random.default_rng(int(seed))
    prompt = rng.integers(0, MODELS[case["model"]]["V"], size=case["prompt"]).astype(np.int32)
    return {"chain": m, "prompt": prompt, "steps": case.get("steps", 1)}


def run(state):
    if "call" in state:
        for args in state["args"]:
            lib.check(state["call"](*args), "the call")
        return state["out"]
    m = state["chain"]
    m.seen = 0                                                                     # a new conversation
    first = m.prefill(state["prompt"])
    tokens, logits = m.greedy(first, state["steps"])
    return {"first": first, "tokens": tokens, "logits": logits}


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _model_work(cfg, prompt, steps):
    qd, kvd = cfg["H"] * cfg["dh"], cfg["KVH"] * cfg["dh"]
    weights = cfg["L"] * ((qd + 2 * kvd) * cfg["D"] + cfg["D"] * qd + 3 * cfg["F"] * cfg["D"])
    layer_bytes = weights // 32 * synth.weight_bytes(cfg["dt_proj"], 1, 256) // 8
    head_bytes = synth.weight_bytes(cfg["dt_head"], cfg["V"], cfg["D"])
    kv = 2 * cfg["L"] * kvd * 2                                                    # bytes of one position's K and V rows
    # the prompt's layers read the weights once; its last token's logits, then every step, read all of them and the cache
    nbytes = layer_bytes + prompt * kv + head_bytes + sum(layer_bytes + head_bytes + (prompt + i + 1) * kv for i in range(steps))
    attn = 4 * cfg["L"] * qd                                                       # operations per (query, key) pair
    flops = 2 * weights * (prompt + steps) + 2 * cfg["V"] * cfg["D"] * (1 + steps)
    flops += attn * (prompt * (prompt + 1) // 2 + sum(prompt + i + 1 for i in range(steps)))
    return {"bytes": nbytes, "flops": flops}


def work(case):
    op = case["op"]
    if op in ("gemv", "gemv_host"):
        n, k, calls = case["n"], case["k"], case.get("layers", 1)
        return {"bytes": calls * (n * _row_bytes(case["dtype"], k) + 4 * (n + k)), "flops": calls * 2 * n * k}
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": n * _row_bytes(case["dtype"], k) + 4 * m * (n + k), "flops": 2 * m * n * k}
    if op == "attn":
        rows = case["kv_heads"] * case["allow"] * case["dh"]
        return {"bytes": 2 * rows * (2 if case["half"] else 4) + 8 * case["heads"] * case["dh"], "flops": 4 * case["heads"] * case["dh"] * case["allow"]}
    return _model_work(MODELS[case["model"]], case["prompt"], case.get("steps", 1))


def tolerance(case):
    op = case["op"]
    if op in ("gemv", "gemv_host"):
        # block formats: activations as 15-bit block floating point; 16-bit rows: fp32 sums
        return {"rel": 1e-5 if case["dtype"] in ("F16", "BF16") else 1e-4}
    if op == "gemm":
        return {"rel": 1e-3}                                                       # fp16 operands, fp32 sums
    if op == "attn":
        return {"rel": 2e-5}                                                       # fp32 arithmetic on the cache's rows
    return {"rel": 5e-3, "differ": 0.01}                                           # fp16 operands and K/V rows through every layer

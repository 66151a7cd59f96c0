"""What a program built on this library has it do, as cases that can be timed one by one.

Seven kinds of work, each called as its users call it:

  attention_host   ops on numpy arrays through grilly_core (flash_attention2, float32: the default of the API)
  linear_host      linear on numpy arrays through grilly_core (float32: the default of the API)
  prefill          flash_attention2 on bf16 DeviceTensors (the prompt of a batch of sequences)
  fill             grl_kv_append of a whole prompt into the paged cache
  decode           one generation step: grl_kv_append of the new token, then grl_gqa_decode over the cache
  project          grl_linear on bf16 device buffers (the projections around attention)
  backward         grl_attention_backward on float32 device buffers (training)

The sizes are those of this repository's configurations, tests and benchmark, or round figures near them; draw() gives
more of each kind over the whole range, odd sizes and every option among them.
"""
import ctypes as C
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "grilly-next_b200", "python"))
import grilly_core as core  # noqa: E402
from grilly_next import cabi  # noqa: E402

THETA = 10000.0
ROPE = {"none": cabi.ROPE_NONE, "interleaved": cabi.ROPE_INTERLEAVED, "half": cabi.ROPE_HALF}


def listed():
    return [
        # A short float32 attention call on numpy arrays: batch 1, 4 heads, 256 tokens, head_dim 64, causal.  The smallest
        # call of the public op; what counts is the trip through the whole op, host arrays in, host array out.
        {"name": "attention_host_fp32", "kind": "attention_host", "batch": 1, "heads": 4, "seq": 256, "dim": 64, "causal": True,
         "mask": "none", "rope": "none"},
        # A float32 projection on numpy arrays: 4 x 128 tokens of width 768 to 3072, with bias.
        {"name": "linear_host_fp32", "kind": "linear_host", "rows": 512, "k": 768, "n": 3072, "bias": True},
        # One chat prompt of odd length: too little work to fill the GPU, launch and latency count.
        {"name": "prefill_prompt", "kind": "prefill", "batch": 1, "heads": 32, "seq": 333, "dim": 128, "causal": True,
         "rope": "half", "ragged": False},
        # The batch prefill of the benchmark: 4 x 32 heads x 2048 tokens, head_dim 128, causal, RoPE.
        {"name": "prefill_batch", "kind": "prefill", "batch": 4, "heads": 32, "seq": 2048, "dim": 128, "causal": True,
         "rope": "interleaved", "ragged": False},
        # The padded batch of the benchmark: 8 sequences of 512 to 4096 tokens, causal and length masks, RoPE.
        {"name": "prefill_ragged", "kind": "prefill", "batch": 8, "heads": 32, "seq": 4096, "dim": 128, "causal": True,
         "rope": "interleaved", "ragged": True},
        # The cache fill behind a prefill: 4 prompts of 2048 tokens, 8 kv heads, RoPE on the keys.
        {"name": "fill_prompt", "kind": "fill", "batch": 4, "new": 2048, "kv_heads": 8, "dim": 128, "page": 64, "quant": False,
         "rope": "interleaved"},
        # A single user generating text: batch 1, about a thousand cached tokens.  Latency.
        {"name": "decode_single", "kind": "decode", "batch": 1, "kv_heads": 8, "group": 4, "dim": 128, "tokens": 1001, "page": 64,
         "quant": False, "rope": "interleaved", "ragged": False},
        # The decode step of the benchmark: 32 sequences, 32 query / 8 kv heads, 4096 cached tokens each.
        {"name": "decode_batch", "kind": "decode", "batch": 32, "kv_heads": 8, "group": 4, "dim": 128, "tokens": 4096, "page": 64,
         "quant": False, "rope": "interleaved", "ragged": False},
        # Long context: one sequence of 131072 tokens over the quantised cache, the storage long contexts are kept in.
        {"name": "decode_long_quant", "kind": "decode", "batch": 1, "kv_heads": 8, "group": 4, "dim": 128, "tokens": 131072, "page": 64,
         "quant": True, "rope": "interleaved", "ragged": False},
        # The projection of a prompt batch: 4096 tokens, 4096 wide (the benchmark's linear line).
        {"name": "project_prompt", "kind": "project", "rows": 4096, "k": 4096, "n": 4096, "bias": True},
        # The packed Q/K/V projection of a decode step: 32 rows, 4096 wide, 3 x 32 heads x 128.
        {"name": "project_step", "kind": "project", "rows": 32, "k": 4096, "n": 12288, "bias": True},
        # The backward pass of a small training batch in float32.
        {"name": "backward_fp32", "kind": "backward", "batch": 4, "heads": 12, "seq": 512, "dim": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["attention_host", "linear_host", "prefill", "fill", "decode", "project", "backward"])
    if kind == "attention_host":
        return {"kind": kind, "batch": rng.randint(1, 2), "heads": rng.randint(1, 8), "seq": _log(rng, 16, 512),
                "dim": rng.choice([32, 64, 128]), "causal": rng.random() < 0.6, "mask": rng.choice(["none", "key", "full"]),
                "rope": rng.choice(["none", "interleaved", "half"])}
    if kind == "linear_host":
        return {"kind": kind, "rows": _log(rng, 1, 512), "k": _log(rng, 64, 768), "n": _log(rng, 64, 3072),
                "bias": rng.random() < 0.8}
    if kind == "prefill":
        while True:
            c = {"kind": kind, "batch": rng.randint(1, 8), "heads": rng.choice([4, 8, 12, 16, 32]), "seq": _log(rng, 64, 4096),
                 "dim": rng.choice([64, 128, 128]), "causal": rng.random() < 0.8,
                 "rope": rng.choice(["none", "interleaved", "half"]), "ragged": rng.random() < 0.4}
            if work(c)["flops"] <= work(listed()[4])["flops"]:
                return c
    if kind == "fill":
        return {"kind": kind, "batch": rng.randint(1, 4), "new": _log(rng, 16, 2048), "kv_heads": rng.choice([2, 4, 8]),
                "dim": rng.choice([64, 128]), "page": rng.choice([16, 32, 64]), "quant": rng.random() < 0.3,
                "rope": rng.choice(["none", "interleaved", "half"])}
    if kind == "decode":
        while True:
            quant = rng.random() < 0.35
            c = {"kind": kind, "batch": _log(rng, 1, 64), "kv_heads": rng.choice([2, 4, 8]), "group": rng.choice([1, 2, 3, 4, 8]),
                 "dim": 128 if quant else rng.choice([64, 128, 128]), "tokens": _log(rng, 32, 131072),
                 "page": rng.choice([16, 32, 64, 64]), "quant": quant, "rope": rng.choice(["interleaved", "half"]),
                 "ragged": rng.random() < 0.4}
            if c["batch"] * c["kv_heads"] * c["tokens"] * c["dim"] <= 32 * 8 * 4096 * 128:
                return c
    if kind == "project":
        while True:
            c = {"kind": kind, "rows": _log(rng, 1, 4096), "k": 8 * _log(rng, 8, 1024), "n": _log(rng, 64, 12288),
                 "bias": rng.random() < 0.7}
            if c["rows"] * c["k"] * c["n"] <= 4096 ** 3:
                return c
    while True:
        c = {"kind": kind, "batch": rng.randint(1, 4), "heads": rng.randint(1, 12), "seq": _log(rng, 32, 1024),
             "dim": rng.choice([32, 64, 128])}
        if work(c)["flops"] <= work(listed()[11])["flops"]:
            return c


def _lengths(case, lo, hi):
    """Ragged lengths of a batch: fixed by the case, so that every seed has the same work."""
    rng = random.Random(case["batch"] * 1000003 + hi)
    return [rng.randint(lo, hi) for _ in range(case["batch"])]


def _prefill_lengths(case):
    s = case["seq"]
    return _lengths(case, max(1, s // 8), s) if case["ragged"] else [s] * case["batch"]


def _decode_lengths(case):
    t = case["tokens"]
    return _lengths(case, max(1, t // 2), t) if case["ragged"] else [t] * case["batch"]


def _token_bytes(case):
    """Bytes one cached token takes for one kv head, keys and values."""
    d = case["dim"]
    return d + d // 2 + d // 16 if case["quant"] else 4 * d


def work(case):
    k = case["kind"]
    if k in ("attention_host", "prefill"):
        d, heads, s = case["dim"], case["heads"], case["seq"]
        lens = [s] * case["batch"] if k == "attention_host" else _prefill_lengths(case)
        pairs = sum(n * (n + 1) // 2 if case["causal"] else n * n for n in lens)
        masks = {"none": 0, "key": case["batch"] * s, "full": case["batch"] * heads * s * s}[case.get("mask", "none")]
        each = 4 if k == "attention_host" else 2
        return {"flops": 4.0 * d * heads * pairs, "bytes": 3.0 * each * sum(lens) * heads * d + 4.0 * case["batch"] * s * heads * d + 4 * masks}
    if k in ("linear_host", "project"):
        m, kk, n = case["rows"], case["k"], case["n"]
        each = 4 if k == "linear_host" else 2
        return {"flops": 2.0 * m * kk * n, "bytes": each * float(m * kk + kk * n) + 4.0 * m * n + (4 * n if case["bias"] else 0)}
    if k == "fill":
        rows = case["batch"] * case["new"] * case["kv_heads"]
        return {"flops": 3.0 * rows * case["dim"] * (case["rope"] != "none"), "bytes": rows * (8.0 * case["dim"] + _token_bytes(case))}
    if k == "decode":
        tokens, hq = sum(n + 1 for n in _decode_lengths(case)), case["kv_heads"] * case["group"]
        small = case["batch"] * case["dim"] * 4.0 * (2 * case["kv_heads"] + 3 * hq)
        return {"flops": 4.0 * tokens * hq * case["dim"], "bytes": tokens * case["kv_heads"] * float(_token_bytes(case)) + small}
    bh, s, d = case["batch"] * case["heads"], case["seq"], case["dim"]
    return {"flops": 8.0 * bh * s * s * d, "bytes": 4.0 * bh * (7 * s * d + s * s)}


def tolerance(case):
    if case["kind"] in ("attention_host", "linear_host", "backward"):
        return {"rel": 2e-5, "max": 1e-3}       # float32 sums in another order
    if case["kind"] == "project":
        return {"rel": 1e-4, "max": 1e-2}       # float32 sums of bf16 products
    if case["kind"] == "fill":
        return {"rel": 2e-3, "max": 2e-2, "differ": 1e-3}   # a rotated key may round to its bf16 (or 8-bit) neighbour
    # probabilities in bf16 or float16; the cache holds one new token, whose bytes may round to their neighbours
    return {"rel": 1e-2, "max": 2e-1, "differ": 1e-4}


# ---------------------------------------------------------------------------------------------- preparation
@functools.lru_cache(maxsize=None)
def _device():
    """The device object a program opens once."""
    return core.Device()


@functools.lru_cache(maxsize=None)
def _abi():
    return cabi.Device(0)


class _Shared:
    """torch's view of a DeviceTensor's memory (kept alive by the view)."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.__cuda_array_interface__ = {"shape": tuple(tensor.shape), "typestr": "<f4" if tensor.dtype == "fp32" else "<i2",
                                         "data": (tensor.data_ptr, False), "version": 2}


def _view(tensor):
    v = torch.as_tensor(_Shared(tensor), device="cuda")
    return v if tensor.dtype == "fp32" else v.view(torch.bfloat16)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _layout(case, k_pages, v_pages, scales, table, lens):
    kv = cabi.KVLayout()
    kv.k_pages, kv.v_pages = k_pages.data_ptr(), v_pages.data_ptr()
    kv.scales = scales.data_ptr() if scales is not None else None
    kv.cache_dtype = cabi.FP8_INT4 if case["quant"] else cabi.BF16
    kv.block_table, kv.seq_lens = table.data_ptr(), lens.data_ptr()
    kv.batch, kv.num_kv_heads, kv.head_dim = case["batch"], case["kv_heads"], case["dim"]
    kv.page_tokens, kv.max_pages, kv.num_pages = case["page"], table.shape[1], table.numel()
    return kv


def _pages(case, tokens, g):
    """Page pools for `tokens` tokens a sequence, pages handed out in no order."""
    max_pages = -(-tokens // case["page"])
    n = max_pages * case["batch"]
    table = torch.randperm(n, generator=g, device="cuda").to(torch.int32).reshape(case["batch"], max_pages).contiguous()
    rows, d = n * case["kv_heads"] * case["page"], case["dim"]
    if case["quant"]:
        pools = [torch.zeros(rows, d, dtype=torch.uint8, device="cuda"), torch.zeros(rows, d // 2, dtype=torch.uint8, device="cuda"),
                 torch.zeros(rows, d // 32, dtype=torch.int16, device="cuda")]
    else:
        pools = [torch.zeros(rows, d, dtype=torch.bfloat16, device="cuda"), torch.zeros(rows, d, dtype=torch.bfloat16, device="cuda"), None]
    return pools, table


def _append_params(case, kv, k_new, v_new, q=None, q_out=None, rope="none"):
    p = cabi.AppendParams()
    p.kv, p.k_new, p.v_new = kv, k_new.data_ptr(), v_new.data_ptr()
    p.n_new = k_new.shape[1]
    if q is not None:
        p.q_in, p.q_out, p.num_q_heads = q.data_ptr(), q_out.data_ptr(), q.shape[2]
    p.rope_mode, p.rope_theta, p.rope_scaling = ROPE[rope], THETA, 1.0
    p.update_lens = 0        # the program keeps the lengths itself
    return p


def _prepare_attention_host(case, seed):
    r = np.random.default_rng(seed)
    b, h, s, d = case["batch"], case["heads"], case["seq"], case["dim"]
    q, k, v = (r.standard_normal((b, h, s, d), dtype=np.float32) for _ in range(3))
    kw = {"causal": case["causal"]}
    if case["mask"] == "key":
        kw["mask"] = (np.arange(s)[None, :] < r.integers(max(1, s // 2), s + 1, (b, 1))).astype(np.float32)
    elif case["mask"] == "full":
        m = (r.random((b, h, s, s)) < 0.8).astype(np.float32)
        m[..., 0] = 1.0
        kw["mask"] = m
    if case["rope"] != "none":
        kw.update(rope_theta=THETA, rope_mode=case["rope"])
    return {"args": (_device(), q, k, v), "kw": kw}


def _prepare_linear_host(case, seed):
    r = np.random.default_rng(seed)
    x = r.standard_normal((case["rows"], case["k"]), dtype=np.float32)
    w = r.standard_normal((case["n"], case["k"]), dtype=np.float32) / np.float32(math.sqrt(case["k"]))
    bias = r.standard_normal(case["n"], dtype=np.float32) if case["bias"] else None
    return {"args": (_device(), x, w, bias)}


def _prepare_prefill(case, seed):
    dev, g = _device(), _generator(seed)
    shape = [case["batch"], case["heads"], case["seq"], case["dim"]]
    q, k, v = (core.DeviceTensor.empty(dev, shape, "bf16") for _ in range(3))
    for t in (q, k, v):
        _view(t).normal_(generator=g)
    out = core.DeviceTensor.empty(dev, shape, "fp32")
    kw = {"causal": case["causal"], "out": out}
    if case["ragged"]:
        kw["seq_lens"] = np.array(_prefill_lengths(case), np.int32)
    if case["rope"] != "none":
        kw.update(rope_theta=THETA, rope_mode=case["rope"])
    return {"args": (dev, q, k, v), "kw": kw, "out": _view(out)}


def _prepare_fill(case, seed):
    g = _generator(seed)
    shape = (case["batch"], case["new"], case["kv_heads"], case["dim"])
    k_new, v_new = (torch.randn(shape, generator=g, device="cuda") for _ in range(2))
    pools, table = _pages(case, case["new"], g)
    lens = torch.zeros(case["batch"], dtype=torch.int32, device="cuda")
    p = _append_params(case, _layout(case, *pools, table, lens), k_new, v_new, rope=case["rope"])
    return {"p": p, "keep": (k_new, v_new, table, lens), "pools": [t for t in pools if t is not None]}


def _prepare_decode(case, seed):
    g, dev = _generator(seed), _abi()
    b, hkv, hq, d = case["batch"], case["kv_heads"], case["kv_heads"] * case["group"], case["dim"]
    lens = _decode_lengths(case)
    pools, table = _pages(case, max(lens) + 1, g)
    # the program's own length arrays: before the step (where the token goes) and after it (what attention reads)
    before = torch.tensor(lens, dtype=torch.int32, device="cuda")
    after = before + 1
    if case["quant"]:        # the cache of such a program was filled by the library
        empty = torch.zeros(b, dtype=torch.int32, device="cuda")
        n, part = max(lens), 16384
        for t0 in range(0, n, part):
            old = [torch.randn((b, min(part, n - t0), hkv, d), generator=g, device="cuda") for _ in range(2)]
            offset = empty + t0
            fill = _append_params(case, _layout(case, *pools, table, offset), *old)
            torch.cuda.synchronize()
            cabi.check(dev.L.grl_kv_append(dev.h, C.byref(fill)))
            dev.sync()
    else:
        for t in pools[:2]:
            t.normal_(generator=g)
    k_new, v_new = (torch.randn((b, 1, hkv, d), generator=g, device="cuda") for _ in range(2))
    q = torch.randn((b, 1, hq, d), generator=g, device="cuda")
    q_rot, out = torch.empty_like(q), torch.empty_like(q)
    append = _append_params(case, _layout(case, *pools, table, before), k_new, v_new, q, q_rot, case["rope"])
    p = cabi.DecodeParams()
    p.kv, p.q, p.out, p.num_q_heads = _layout(case, *pools, table, after), q_rot.data_ptr(), out.data_ptr(), hq
    p.max_seq_len = max(lens) + 1
    splits, size = C.c_int(), C.c_size_t()
    cabi.check(dev.L.grl_decode_pick_splits(dev.h, C.byref(p), C.byref(splits)))
    cabi.check(dev.L.grl_decode_workspace_bytes(C.byref(p), splits, C.byref(size)))
    space = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = space.data_ptr(), size.value
    return {"append": append, "p": p, "keep": (table, before, after, k_new, v_new, q, space),
            "out": [out, q_rot] + [t for t in pools if t is not None]}


def _prepare_project(case, seed):
    g = _generator(seed)
    m, k, n = case["rows"], case["k"], case["n"]
    x = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device="cuda") / math.sqrt(k)).to(torch.bfloat16)
    bias = torch.randn(n, generator=g, device="cuda") if case["bias"] else None
    y = torch.empty((m, n), device="cuda")
    args = (x.data_ptr(), w.data_ptr(), bias.data_ptr() if bias is not None else None, y.data_ptr(), m, k, n, cabi.BF16)
    return {"args": args, "keep": (x, w, bias), "out": y}


def _prepare_backward(case, seed):
    g = _generator(seed)
    b, h, s, d = case["batch"], case["heads"], case["seq"], case["dim"]
    go, q, k, v = (torch.randn((b, h, s, d), generator=g, device="cuda") for _ in range(4))
    attn = torch.softmax(q @ k.transpose(-1, -2) / math.sqrt(d), -1)
    grads = [torch.empty_like(q) for _ in range(3)]
    scratch = torch.empty_like(attn)
    args = [t.data_ptr() for t in (go, q, k, v, attn, *grads, scratch)] + [b, h, s, d, 0.0]
    return {"args": args, "keep": (go, q, k, v, attn, scratch), "out": grads}


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


# ---------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "attention_host":
        return core.flash_attention2(*state["args"], **state["kw"])
    if kind == "linear_host":
        return core.linear(*state["args"])
    if kind == "prefill":
        core.flash_attention2(*state["args"], **state["kw"])
        return state["out"]
    dev = _abi()
    if kind == "fill":
        cabi.check(dev.L.grl_kv_append(dev.h, C.byref(state["p"])))
        return state["pools"]
    if kind == "decode":
        cabi.check(dev.L.grl_kv_append(dev.h, C.byref(state["append"])))
        cabi.check(dev.L.grl_gqa_decode(dev.h, C.byref(state["p"])))
        return state["out"]
    if kind == "project":
        cabi.check(dev.L.grl_linear(dev.h, *state["args"]))
        return state["out"]
    cabi.check(dev.L.grl_attention_backward(dev.h, *state["args"]))
    return state["out"]

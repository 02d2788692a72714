"""Workloads of the attention forward path, as programs that use the package call it.

Each case is one call of ``flash_attn_cute`` (or of ``flash_attn_cute_host`` for operands in pinned host
memory).  ``listed()`` names the workloads, ``draw(rng)`` gives further ones from the ranges they stand for,
``prepare`` makes what a program holds before the call, ``run`` makes the call, ``work`` counts what it cannot
do without, and ``exact`` restates it in 64 bits.
"""
import math

import torch

from fray_b200.jit_kernels import flash_attn_cute, flash_attn_cute_host


def _case(B, H, Sq, D, name=None, Hkv=None, Sk=None, causal=False, dtype="fp16", lse=False, layout="bhsd",
          values="normal", memory="device"):
    case = {"B": B, "H": H, "Hkv": Hkv or H, "Sq": Sq, "Sk": Sk or Sq, "D": D, "causal": causal, "dtype": dtype,
            "lse": lse, "layout": layout, "values": values, "memory": memory}
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the smallest call, where launch and host latency count: four heads of a short sequence
        _case(1, 4, 256, 64, "tiny"),
        # a short-context batch of a small model: many short ragged causal slices at head dim 64
        _case(6, 12, 333, 64, "short_ragged_causal", causal=True),
        # a medium encoder call
        _case(2, 16, 2048, 128, "encode_2k"),
        # causal prefill or training forward of a 4k context
        _case(4, 32, 4096, 128, "causal_4k", causal=True),
        # causal prefill of one long prompt
        _case(1, 32, 16384, 128, "causal_16k", causal=True),
        # many 1k sequences with large logits; q is a transposed view of a [B, S, H, D] projection
        _case(16, 16, 1024, 64, "short_1k_large_logits", layout="q_bshd", values="large"),
        # the benchmark's default workload: full attention over 4k tokens
        _case(4, 32, 4096, 128, "full_4k"),
        # prefill with grouped K/V heads in bf16, ragged length, log-sum-exp kept for a later merge
        _case(2, 32, 3000, 128, "grouped_bf16_lse", Hkv=8, causal=True, dtype="bf16", lse=True),
        # one new query per sequence against a long cache with grouped K/V heads
        _case(8, 32, 1, 128, "decode_8k", Hkv=8, Sk=8192, dtype="bf16"),
        # a chunk of new queries against a longer cache, partial result to be merged through its log-sum-exp
        _case(2, 16, 513, 128, "chunk_on_cache", Hkv=4, Sk=6000, lse=True),
        # operands in pinned host memory, copies and kernel overlapped by the call
        _case(4, 16, 1024, 128, "host_buffers", memory="host"),
    ]


_MOST_FLOPS = 2.2e12  # the largest listed case


def _spread(rng, low, high):
    """A whole number from low..high, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    while True:
        kind = rng.choice(["full", "full", "causal", "causal", "short", "grouped", "decode", "chunk", "host"])
        D = rng.choice([64, 128, 128])
        dtype = rng.choice(["fp16", "fp16", "bf16"])
        layout = rng.choice(["bhsd", "bhsd", "q_bshd", "bshd"])
        values = rng.choice(["normal", "normal", "normal", "large"])
        if kind in ("full", "causal"):
            case = _case(rng.randint(1, 4), rng.choice([8, 12, 16, 32]), _spread(rng, 700, 9000), D, causal=kind == "causal",
                         dtype=dtype, layout=layout, values=values, lse=rng.random() < 0.25)
        elif kind == "short":
            case = _case(rng.randint(1, 16), rng.choice([4, 8, 12, 16]), _spread(rng, 60, 1100), D,
                         causal=rng.random() < 0.5, dtype=dtype, layout=layout, values=values)
        elif kind == "grouped":
            kv = rng.choice([1, 2, 4, 8])
            case = _case(rng.randint(1, 3), kv * rng.choice([2, 4, 8]), _spread(rng, 500, 6000), D, Hkv=kv,
                         causal=rng.random() < 0.75, dtype=dtype, layout=layout, lse=rng.random() < 0.5)
        elif kind == "decode":
            kv = rng.choice([2, 4, 8])
            case = _case(_spread(rng, 1, 16), kv * rng.choice([1, 4, 8]), rng.choice([1, 1, 2, 4]), D, Hkv=kv,
                         Sk=_spread(rng, 500, 16384), dtype=dtype, lse=rng.random() < 0.25)
        elif kind == "chunk":
            kv = rng.choice([2, 4, 8])
            case = _case(rng.randint(1, 4), kv * rng.choice([1, 2, 4]), _spread(rng, 30, 1200), D, Hkv=kv,
                         Sk=_spread(rng, 1300, 12000), dtype=dtype, lse=rng.random() < 0.5)
        else:
            case = _case(rng.randint(1, 4), rng.choice([4, 8, 16]), _spread(rng, 200, 2000), D, causal=rng.random() < 0.5,
                         dtype=dtype, memory="host")
        if work(case)["flops"] <= _MOST_FLOPS:
            return case


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.half


def _inputs(case, seed):
    """q, k, v on the GPU, contiguous [B, H, S, D], from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(1000 + seed)
    tensors = []
    for heads, length in ((case["H"], case["Sq"]), (case["Hkv"], case["Sk"]), (case["Hkv"], case["Sk"])):
        t = torch.randn(case["B"], heads, length, case["D"], generator=gen, device="cuda", dtype=torch.float32)
        if case["values"] == "large" and len(tensors) < 2:
            # large logits: wide scores, and one entry in a hundred at +-16
            t.mul_(4.0)
            u = torch.rand(t.shape, generator=gen, device="cuda")
            t = torch.where(u < 0.005, 16.0, torch.where(u < 0.01, -16.0, t))
        tensors.append(t.to(_dtype(case)))
        del t
    return tensors


def prepare(case, seed):
    q, k, v = _inputs(case, seed)
    state = {"causal": case["causal"], "memory": case["memory"], "lse": None}
    if case["memory"] == "host":
        state["qkv"] = tuple(t.cpu().pin_memory() for t in (q, k, v))
        state["out"] = torch.zeros(q.shape, dtype=q.dtype).pin_memory()
        return state

    def as_bshd(t):  # the logical [B, H, S, D] view of a [B, S, H, D] buffer
        return t.transpose(1, 2).contiguous().transpose(1, 2)

    if case["layout"] == "bshd":
        q, k, v = as_bshd(q), as_bshd(k), as_bshd(v)
    elif case["layout"] == "q_bshd":
        q = as_bshd(q)
    state["qkv"] = (q, k, v)
    state["out"] = torch.empty_like(q) if case["layout"] == "bshd" else torch.empty(q.shape, dtype=q.dtype, device="cuda")
    if case["lse"]:
        state["lse"] = torch.empty(q.shape[:3], dtype=torch.float32, device="cuda")
    return state


def run(state):
    q, k, v = state["qkv"]
    if state["memory"] == "host":
        flash_attn_cute_host(q, k, v, state["out"], causal=state["causal"])
    else:
        flash_attn_cute(q, k, v, state["out"], causal=state["causal"], lse=state["lse"])
    if state["lse"] is not None:
        return {"out": state["out"], "lse": state["lse"]}
    return {"out": state["out"]}


def _pairs(case):
    """(query, key) pairs of one head that count."""
    sq, sk = case["Sq"], case["Sk"]
    if not case["causal"]:
        return sq * sk
    full = min(sq, sk)  # query i sees keys 0..i
    return full * (full + 1) // 2 + (sq - full) * sk


def work(case):
    rows, keys = case["B"] * case["H"] * case["Sq"], case["B"] * case["Hkv"] * case["Sk"]
    return {"bytes": 2 * case["D"] * (2 * rows + 2 * keys) + (4 * rows if case["lse"] else 0),
            "flops": 4 * case["D"] * case["B"] * case["H"] * _pairs(case)}


def tolerance(case):
    # 16-bit outputs of fp32 sums over 16-bit probabilities, about four times the relative error seen
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 1.3e-3}


def exact(case, seed):
    q, k, v = _inputs(case, seed)
    B, H, Sq, Sk = case["B"], case["H"], case["Sq"], case["Sk"]
    group, scale = H // case["Hkv"], 1.0 / math.sqrt(case["D"])
    out = torch.empty(B, H, Sq, case["D"], dtype=torch.float64)
    lse = torch.empty(B, H, Sq, dtype=torch.float64)
    block = 2048
    for b in range(B):
        for h in range(H):
            kd, vd = k[b, h // group].double(), v[b, h // group].double()
            for r0 in range(0, Sq, block):
                r1 = min(Sq, r0 + block)
                last = min(Sk, r1) if case["causal"] else Sk
                s = (q[b, h, r0:r1].double() @ kd[:last].T) * scale
                if case["causal"]:
                    rows = torch.arange(r0, r1, device=s.device).unsqueeze(1)
                    s.masked_fill_(torch.arange(last, device=s.device).unsqueeze(0) > rows, float("-inf"))
                lse[b, h, r0:r1] = torch.logsumexp(s, -1).cpu()
                out[b, h, r0:r1] = (torch.softmax(s, -1) @ vd[:last]).cpu()
    return {"out": out, "lse": lse} if case["lse"] else {"out": out}

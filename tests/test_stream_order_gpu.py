"""Launches may be set up while the stream's previous kernel still runs: a call that reads what the call before it writes has to
wait for that one's end, whichever kinds follow each other, eagerly and in a captured graph."""
import ctypes
import importlib
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


def runtimes(D, monkeypatch):
    """One library per kernel kind with overlapped launches, and one kind that is launched plainly."""
    from fray_b200.jit import build, cpp_format, generate
    monkeypatch.delenv("FRAY_ATTN_FORCE", raising=False)
    points = {p["KIND"]: p for p in reversed((*op.tuning_space(D), *op.few_query_space()))}
    kinds = (op.KIND_SIMPLE, op.KIND_TWO_TILES, op.KIND_ALTERNATING, op.KIND_ONE_TILE, op.KIND_FEW_QUERIES, op.KIND_ROW_PAIRS)
    made = {}
    for kind in kinds:
        keys = {"D": D, **points[kind]}
        code = generate(op.includes, op.arg_defs, cpp_format(op.template, keys), cpp_format(op.epilogue, keys))
        made[kind] = build("flash_attn_cute", op.arg_defs, code)
    return made


def launch(runtime, q, k, v, o):
    strides = tuple(int(t.stride(i)) for t in (q, k, v, o) for i in range(3))
    no_lse = torch.empty(0, dtype=torch.float32, device="cuda")
    assert runtime(q, k, v, o, q.shape[0], q.shape[1], q.shape[2], *strides, k.shape[1], k.shape[2], no_lse, False,
                   1.0 / math.sqrt(q.shape[3]), torch.cuda.current_stream()) == 0


def chain(kinds, made, x, rest, bufs, role):
    """x -> kernel -> kernel -> ...: every call's operand number `role` is the output of the call before it."""
    for kind, out in zip(kinds, bufs):
        operands = [rest[0], rest[1], rest[2]]
        operands[role] = x
        launch(made[kind], *operands, out)
        x = out
    return x


# rows: a tile of the few-query kernel on many heads, so that launches are long enough to overlap and the successor's CTAs find
# room while the predecessor drains
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("role", [0, 1, 2])
def test_a_call_reads_the_finished_output_of_the_call_before_it(D, role, monkeypatch):
    made = runtimes(D, monkeypatch)
    g = torch.Generator(device="cuda").manual_seed(101)
    B, H, S = 3, 100, 128
    x, *rest = (torch.randn(B, H, S, D, generator=g, device="cuda").half() for _ in range(4))
    kinds = list(made)
    order = [a for first in kinds for second in kinds for a in (first, second)]  # every kind behind every kind
    bufs = [torch.empty_like(x) for _ in order]

    step = x
    want = []
    for kind, out in zip(order, bufs):  # the same calls, each finished before the next is queued
        step = chain([kind], made, step, rest, [out], role)
        torch.cuda.synchronize()
        want.append(step.clone())

    def compare():
        torch.cuda.synchronize()
        for n, (a, b) in enumerate(zip(bufs, want)):
            assert torch.equal(a, b), f"call {n}: kind {order[n]} behind kind {order[n - 1] if n else None}"

    for _ in range(5):
        for b in bufs:
            b.fill_(float("nan"))
        chain(order, made, x, rest, bufs, role)
        compare()

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(order, made, x, rest, bufs, role)
    for _ in range(3):
        for b in bufs:
            b.fill_(float("nan"))
        graph.replay()
        compare()
    for kind, runtime in made.items():
        status = (ctypes.c_int * 4)()
        assert runtime.symbol("fray_attn_status")(status, ctypes.c_int(1)) == 0 and status[0] == 0, f"kind {kind}"


def test_calls_between_torch_kernels_in_a_graph():
    """Through the public op: the operand is written by a torch kernel just before the call, the output read just after it."""
    from fray_b200.jit_kernels import flash_attn_cute, flash_attn_status
    g = torch.Generator(device="cuda").manual_seed(103)
    x = torch.randn(2, 24, 400, 64, generator=g, device="cuda").half()
    dec = torch.randn(2, 24, 1, 64, generator=g, device="cuda").half()
    k, v = (torch.randn(2, 6, 2048, 64, generator=g, device="cuda").half() for _ in range(2))

    def step():
        y, z, w = torch.empty_like(x), torch.empty_like(dec), torch.empty_like(dec)
        a = x * 0.5
        flash_attn_cute(a, x, x, y, causal=True)
        b = y[:, :, :1] + dec
        flash_attn_cute(b, k, v, z)
        flash_attn_cute(z, k, v, w)
        return y, z, w + z

    want = [t.clone() for t in step()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    for _ in range(3):
        for t in got:
            t.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    assert flash_attn_status()[0] == 0

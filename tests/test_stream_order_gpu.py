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
    """One library per kernel kind with overlapped launches and, at head dim 128, the kind that is launched plainly."""
    from fray_b200.jit import build, cpp_format, generate
    monkeypatch.delenv("FRAY_ATTN_FORCE", raising=False)
    points = {p["KIND"]: p for p in reversed((*op.tuning_space(D), *op.few_query_space()))}
    kinds = (op.KIND_SIMPLE, op.KIND_TWO_TILES, op.KIND_ALTERNATING, op.KIND_ONE_TILE, op.KIND_FEW_QUERIES, op.KIND_ROW_PAIRS,
             *((op.KIND_PAIRED,) if D == 128 else ()))
    made = {}
    for kind in kinds:
        keys = {"D": D, **points[kind]}
        code = generate(op.includes, op.arg_defs, cpp_format(op.template, keys), cpp_format(op.epilogue, keys))
        made[kind] = build("flash_attn_cute", op.arg_defs, code)
    return made


def form(runtime, x, causal):
    """(mode, CTAs per work item) of a row-pair launch whose operands all have x's shape and layout."""
    layout = op._AttnLayout(*op._launch_args(x, x, x, x, may_fold=False)[4:], int(causal), 1.0)
    mode, parts = ctypes.c_int(-1), ctypes.c_int(-1)
    assert runtime.symbol("fray_attn_form")(ctypes.byref(layout), ctypes.byref(mode), ctypes.byref(parts)) == 0
    return mode.value, parts.value


def launch(runtime, q, k, v, o, causal):
    strides = tuple(int(t.stride(i)) for t in (q, k, v, o) for i in range(3))
    no_lse = torch.empty(0, dtype=torch.float32, device="cuda")
    assert runtime(q, k, v, o, q.shape[0], q.shape[1], q.shape[2], *strides, k.shape[1], k.shape[2], no_lse, causal,
                   1.0 / math.sqrt(q.shape[3]), torch.cuda.current_stream()) == 0


def chain(kinds, made, x, rest, bufs, role, causal):
    """x -> kernel -> kernel -> ...: every call's operand number `role` is the output of the call before it."""
    for kind, out in zip(kinds, bufs):
        operands = [rest[0], rest[1], rest[2]]
        operands[role] = x
        launch(made[kind], *operands, out, causal)
        x = out
    return x


def compare_chains(made, order, x, rest, role, causal):
    bufs = [torch.empty_like(x) for _ in order]
    step = x
    want = []
    for kind, out in zip(order, bufs):  # the same calls, each finished before the next is queued
        step = chain([kind], made, step, rest, [out], role, causal)
        torch.cuda.synchronize()
        want.append(step.clone())

    def compare():
        torch.cuda.synchronize()
        for n, (a, b) in enumerate(zip(bufs, want)):
            assert torch.equal(a, b), f"call {n}: kind {order[n]} behind kind {order[n - 1] if n else None}"

    for _ in range(5):
        for b in bufs:
            b.fill_(float("nan"))
        chain(order, made, x, rest, bufs, role, causal)
        compare()

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(order, made, x, rest, bufs, role, causal)
    for _ in range(3):
        for b in bufs:
            b.fill_(float("nan"))
        graph.replay()
        compare()
    for kind, runtime in made.items():
        status = (ctypes.c_int * 4)()
        assert runtime.symbol("fray_attn_status")(status, ctypes.c_int(1)) == 0 and status[0] == 0, f"kind {kind}"


def operands(B, H, S, D):
    g = torch.Generator(device="cuda").manual_seed(101)
    return [torch.randn(B, H, S, D, generator=g, device="cuda").half() for _ in range(4)]


# rows: a tile of the few-query kernel on many heads, so that launches are long enough to overlap and the successor's CTAs find
# room while the predecessor drains
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("role", [0, 1, 2])
def test_a_call_reads_the_finished_output_of_the_call_before_it(D, role, monkeypatch):
    made = runtimes(D, monkeypatch)
    x, *rest = operands(3, 100, 128, D)
    kinds = list(made)
    order = [a for first in kinds for second in kinds for a in (first, second)]  # every kind behind every kind
    compare_chains(made, order, x, rest, role, causal=False)


# The row-pair kernel's other two forms in front of and behind every kind and themselves: keys split over clusters (two heads of
# 8 items; results by plain stores), and causal items matched by twos (400 heads).
@pytest.mark.parametrize("mode,B,H,S,causal", [(1, 1, 2, 2048, False), (2, 8, 50, 1280, True)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("role", [0, 1, 2])
def test_calls_in_front_of_and_behind_the_other_forms_of_the_row_pair_kernel(mode, B, H, S, causal, D, role, monkeypatch):
    made = runtimes(D, monkeypatch)
    x, *rest = operands(B, H, S, D)
    assert form(made[op.KIND_ROW_PAIRS], x, causal)[0] == mode
    order = [op.KIND_ROW_PAIRS] + [a for kind in made for a in (kind, op.KIND_ROW_PAIRS)]
    compare_chains(made, order, x, rest, role, causal)


# At head dim 64 the row-pair kernel's launcher has two kernels: four streams per CTA (300 items of 128 rows above too), and two
# threads per row for many short items of whole steps.
@pytest.mark.parametrize("B,H,S,streams", [(3, 100, 128, 1), (4, 100, 256, 0)])
@pytest.mark.parametrize("role", [0, 1, 2])
def test_calls_in_front_of_and_behind_both_kernels_of_head_dim_64(B, H, S, streams, role, monkeypatch):
    made = runtimes(64, monkeypatch)
    x, *rest = operands(B, H, S, 64)
    layout = op._AttnLayout(*op._launch_args(x, x, x, x, may_fold=False)[4:], 0, 1.0)
    assert made[op.KIND_ROW_PAIRS].symbol("fray_attn_four_streams")(ctypes.byref(layout)) == streams
    order = [op.KIND_ROW_PAIRS] + [a for kind in made for a in (kind, op.KIND_ROW_PAIRS)]
    compare_chains(made, order, x, rest, role, causal=False)


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

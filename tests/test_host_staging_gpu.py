"""The host-buffer call from several streams and threads at once, and in a captured graph: all share one shape's staging buffers."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(seed, B=6, H=4, S=700, D=128):
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(B, H, S, D, generator=g).half().pin_memory() for _ in range(3))
    return q, k, v, torch.zeros(B, H, S, D, dtype=torch.half).pin_memory()


def wanted(q, k, v, causal):
    from fray_b200.jit_kernels import flash_attn_cute_host
    out = torch.zeros_like(q).pin_memory()
    flash_attn_cute_host(q, k, v, out, causal=causal, chunks=6)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("causal", [False, True])
def test_calls_on_several_streams_at_once(causal):
    from fray_b200.jit_kernels import flash_attn_cute_host
    sets = [operands(n) for n in range(4)] + [operands(9, S=300)]  # the last shape takes the buffers away from the others
    want = [wanted(*t[:3], causal) for t in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    for order in ((0, 1, 2, 3, 4), (4, 3, 0, 2, 1), (0, 1, 4, 0, 1)):
        for t in sets:
            t[3].zero_()
        for n in order:
            with torch.cuda.stream(streams[n]):
                flash_attn_cute_host(*sets[n], causal=causal, chunks=6)
        torch.cuda.synchronize()
        for n in set(order):
            assert torch.equal(sets[n][3], want[n])


def test_calls_from_several_threads_at_once():
    from fray_b200.jit_kernels import flash_attn_cute_host
    sets = [operands(20 + n) for n in range(4)]
    want = [wanted(*t[:3], False) for t in sets]

    def work(n):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                flash_attn_cute_host(*sets[n], chunks=6)

    threads = [threading.Thread(target=work, args=(n,)) for n in range(len(sets))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    for t, w in zip(sets, want):
        assert torch.equal(t[3], w)


def test_captured_call_beside_eager_ones():
    from fray_b200.jit_kernels import flash_attn_cute_host
    a, b = operands(40), operands(41)
    want = [wanted(*t[:3], False) for t in (a, b)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        flash_attn_cute_host(*a, chunks=6)
    side = torch.cuda.Stream()
    for _ in range(4):
        a[3].zero_(), b[3].zero_()
        graph.replay()
        with torch.cuda.stream(side):
            flash_attn_cute_host(*b, chunks=6)
        torch.cuda.synchronize()
        assert torch.equal(a[3], want[0]) and torch.equal(b[3], want[1])

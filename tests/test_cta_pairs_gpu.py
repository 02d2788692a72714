"""The row-pair kernel on CTA pairs (head dim 128): items of 512 rows, and items of 256 rows of two heads of a group."""
import ctypes
import importlib

import pytest
import torch

from tests.test_split_keys_gpu import bound, exact
from tests.test_stream_order_gpu import compare_chains, operands, runtimes

pytestmark = pytest.mark.gpu

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")
SINGLE, ROWS, HEADS = 0, 1, 2


def forced(monkeypatch):
    point = next(p for p in op.tuning_space(128) if p["KIND"] == op.KIND_ROW_PAIRS)
    monkeypatch.setenv("FRAY_ATTN_FORCE", ",".join(f"{k}={v}" for k, v in point.items()))
    op._fast_path.clear()  # a layout launched before would go straight to the kernel it was tuned to


def pair(q, k, v, out, causal):
    """Whether the launcher puts CTA pairs to the items of a call."""
    from fray_b200.jit import build, cpp_format, generate
    bf16 = q.dtype is torch.bfloat16
    arg_defs = op.arg_defs_bf16 if bf16 else op.arg_defs
    keys = {"D": q.shape[3], **op.split_keys_space()[0]}
    library = build("flash_attn_cute", arg_defs, generate(op.includes_bf16 if bf16 else op.includes, arg_defs,
                                                          cpp_format(op.template, keys), cpp_format(op.epilogue, keys)))
    layout = op._AttnLayout(*op._launch_args(q, k, v, out, may_fold=not causal)[4:], int(causal), 1.0)
    return library.symbol("fray_attn_pair")(ctypes.byref(layout))


# By rows: a last item of six rows (the second CTA's tiles and both tiles 1 empty), one whose tile 1 is empty, keys that end inside a
# step, items that end with a tile's last row.  By heads: ragged ends, a last pair of tiles without a second one, heaviest of all
# slices first and matched by twos, more queries than keys, heads that do not follow each other (no mask).
@pytest.mark.parametrize("form,B,H,Hkv,Sq,Sk,causal,strided", [
    (ROWS, 1, 60, 60, 1030, 3072, False, False), (ROWS, 1, 74, 74, 600, 4090, False, True), (ROWS, 16, 16, 16, 1024, 1024, False, False),
    (HEADS, 4, 64, 16, 1300, 1300, True, False), (HEADS, 1, 64, 32, 3000, 3000, True, True), (HEADS, 8, 64, 32, 2048, 2048, True, False),
    (HEADS, 2, 60, 10, 2100, 2000, True, False), (HEADS, 2, 74, 37, 600, 2100, False, True)])
@pytest.mark.parametrize("dtype,gain", [(torch.half, 1.0), (torch.half, 6.0), (torch.bfloat16, 1.0)])
def test_pairs(form, B, H, Hkv, Sq, Sk, causal, strided, dtype, gain, monkeypatch):
    forced(monkeypatch)
    g = torch.Generator(device="cuda").manual_seed(107)
    q = (gain * torch.randn(B, H, Sq, 128, generator=g, device="cuda")).to(dtype)  # gain 6: offsets move during a row
    if strided:
        q = q.transpose(1, 2).contiguous().transpose(1, 2)
    k, v = (torch.randn(B, Hkv, Sk, 128, generator=g, device="cuda").to(dtype) for _ in range(2))
    guard = torch.full((B, H, Sq + 1, 128), 7.0, dtype=dtype, device="cuda")
    out, lse = guard[:, :, :Sq], torch.zeros(B, H, Sq, device="cuda")
    assert pair(q, k, v, out, causal) == form
    op.flash_attn_cute(q, k, v, out, causal=causal, lse=lse)
    torch.cuda.synchronize()
    assert op.flash_attn_status()[0] == 0
    assert (guard[:, :, Sq:] == 7.0).all()
    group = H // Hkv
    for b, kv in {(0, 0), (B // 2, Hkv // 2), (B - 1, Hkv - 1)}:
        heads = slice(kv * group, (kv + 1) * group)
        want, want_lse, weighted, total = exact(q[b:b + 1, heads], k[b:b + 1, kv:kv + 1], v[b:b + 1, kv:kv + 1], causal)
        assert ((out[b:b + 1, heads].double() - want).abs() <= bound(want, weighted, total, dtype)).all()
        assert (lse[b:b + 1, heads].double() - want_lse).abs().max().item() <= 2e-4
        del want, weighted
    again = torch.empty_like(out)
    op.flash_attn_cute(q, k, v, again, causal=causal)
    assert torch.equal(out, again)


@pytest.mark.parametrize("role", [0, 1, 2])
def test_calls_in_front_of_and_behind_pairs(role, monkeypatch):
    made = runtimes(128, monkeypatch)
    x, *rest = operands(16, 16, 1024, 128)
    layout = op._AttnLayout(*op._launch_args(x, *rest[:2], torch.empty_like(x), may_fold=False)[4:], 0, 1.0)
    assert made[op.KIND_ROW_PAIRS].symbol("fray_attn_pair")(ctypes.byref(layout)) == ROWS
    order = [op.KIND_ROW_PAIRS] + [a for kind in made for a in (kind, op.KIND_ROW_PAIRS)]
    compare_chains(made, order, x, rest, role, causal=False)

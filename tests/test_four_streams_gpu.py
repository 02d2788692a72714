"""Head dim 64 with four independent streams per CTA (what the row-pair kernel's launcher gives most of its calls to)."""
import ctypes
import importlib

import pytest
import torch

from tests.test_split_keys_gpu import bound, exact

pytestmark = pytest.mark.gpu

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


def four_streams(q, k, v, out, causal):
    """Whether the launcher gives a call to this kernel."""
    from fray_b200.jit import build, cpp_format, generate
    bf16 = q.dtype is torch.bfloat16
    arg_defs = op.arg_defs_bf16 if bf16 else op.arg_defs
    keys = {"D": q.shape[3], **op.split_keys_space()[0]}
    library = build("flash_attn_cute", arg_defs, generate(op.includes_bf16 if bf16 else op.includes, arg_defs,
                                                          cpp_format(op.template, keys), cpp_format(op.epilogue, keys)))
    layout = op._AttnLayout(*op._launch_args(q, k, v, out, may_fold=not causal)[4:], int(causal), 1.0)
    return library.symbol("fray_attn_four_streams")(ctypes.byref(layout))


# Items of one step (the second group has none), of two, of an odd number of steps without and with a mask, over several rounds
# per CTA; a second tile that is empty in every item, in the last one of a slice, or holds a single row; tiles whose steps differ by
# two or, clipped by the keys, by one or none; more queries than keys and the reverse; dealt slice by slice, heaviest first and
# matched by twos over one slice and over two; more than 255 items per SM (more CTAs than run at a time).
# TWO_THREADS: so many short items of whole steps that the other kernel has them; the same steps with fewer items are here.
TWO_THREADS = {(2, 200, 50, 257, 100, False), (1, 160, 160, 513, 321, False)}


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,causal", [
    (2, 200, 200, 300, 40, False), (2, 200, 50, 257, 100, False), (2, 92, 23, 257, 100, False), (2, 150, 150, 129, 190, False),
    (1, 160, 160, 513, 321, False), (1, 120, 120, 513, 321, False), (3, 70, 70, 100, 1100, False), (2, 90, 45, 513, 3000, False),
    (1, 200, 200, 64, 64, True), (3, 60, 20, 333, 333, True), (2, 80, 80, 700, 500, True), (1, 100, 100, 1500, 640, True),
    (2, 40, 40, 300, 900, True), (4, 40, 40, 1300, 1300, True), (8, 50, 50, 1280, 1280, True), (8, 37, 37, 1800, 1800, True),
    (220, 200, 200, 40, 50, True)])
@pytest.mark.parametrize("dtype,gain", [(torch.half, 1.0), (torch.half, 6.0), (torch.bfloat16, 1.0)])
def test_four_streams(B, H, Hkv, Sq, Sk, causal, dtype, gain, monkeypatch):
    point = next(p for p in op.tuning_space(64) if p["KIND"] == op.KIND_ROW_PAIRS)
    monkeypatch.setenv("FRAY_ATTN_FORCE", ",".join(f"{k}={v}" for k, v in point.items()))
    op._fast_path.clear()  # a layout launched before would go straight to the kernel it was tuned to
    g = torch.Generator(device="cuda").manual_seed(109)
    q = (gain * torch.randn(B, Sq, H, 64, generator=g, device="cuda")).to(dtype).transpose(1, 2)  # gain 6: offsets move during a row
    k, v = (torch.randn(B, Hkv, Sk, 64, generator=g, device="cuda").to(dtype) for _ in range(2))
    guard = torch.full((B, H, Sq + 1, 64), 7.0, dtype=dtype, device="cuda")
    out, lse = guard[:, :, :Sq], torch.zeros(B, H, Sq, device="cuda")
    assert four_streams(q, k, v, out, causal) == ((B, H, Hkv, Sq, Sk, causal) not in TWO_THREADS)
    op.flash_attn_cute(q, k, v, out, causal=causal, lse=lse)
    torch.cuda.synchronize()
    assert op.flash_attn_status()[0] == 0
    assert (guard[:, :, Sq:] == 7.0).all()
    group = H // Hkv
    for b, kv in {(0, 0), (B // 2, Hkv // 2), (B - 1, Hkv - 1), (B - 1, 0)}:
        heads = slice(kv * group, (kv + 1) * group)
        want, want_lse, weighted, total = exact(q[b:b + 1, heads], k[b:b + 1, kv:kv + 1], v[b:b + 1, kv:kv + 1], causal)
        # both groups round P against offsets of their own, each within the bound for its keys
        assert ((out[b:b + 1, heads].double() - want).abs() <= bound(want, weighted, total, dtype)).all()
        assert (lse[b:b + 1, heads].double() - want_lse).abs().max().item() <= 2e-4
        del want, weighted
    again = torch.empty_like(out)
    for _ in range(2):
        op.flash_attn_cute(q, k, v, again, causal=causal)
        assert torch.equal(out, again)

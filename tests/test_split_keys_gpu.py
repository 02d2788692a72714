"""The row-pair kernel with the keys of its work items split over clusters, and folded groups of query heads."""
import ctypes
import importlib
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")
DEALT, SPLIT, MATCHED = 0, 1, 2


def exact(q, k, v, causal):
    """Output and log-sum-exp in 64 bits, and what bounds the error of each output: sum p |v| and sum |v|."""
    group = q.shape[1] // k.shape[1]
    ke, ve = (t.repeat_interleave(group, 1).double() for t in (k, v))
    s = q.double() @ ke.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        s.masked_fill_(torch.arange(k.shape[2], device=s.device) > torch.arange(q.shape[2], device=s.device)[:, None], float("-inf"))
    p = torch.softmax(s, -1)
    return p @ ve, torch.logsumexp(s, -1), p @ ve.abs(), ve.abs().sum(-2, keepdim=True)


def bound(want, weighted, total, dtype):
    """What 16-bit P and outputs may be off by, value by value.  Every P is rounded to within u of itself (fp16 below 2^-14: to
    within 2^-25, at row sums of 1 and more), which the products carry to at most u * sum p |v| (2^-25 * sum |v|), and the
    output is rounded to within u of itself.  Scores and exponentials are fp32, good to 2^-13 of a weight (the coarsest
    exponential is a cubic, 9e-5)."""
    u = 2.0 ** -11 if dtype is torch.half else 2.0 ** -8
    return u * (weighted + want.abs()) + 2.0 ** -13 * weighted + (2.0 ** -25 * total if dtype is torch.half else 0.0)


def form(q, k, v, out, causal):
    """(mode, CTAs per work item) that the row-pair kernel's launcher chooses for a call."""
    from fray_b200.jit import build, cpp_format, generate
    bf16 = q.dtype is torch.bfloat16
    arg_defs = op.arg_defs_bf16 if bf16 else op.arg_defs
    keys = {"D": q.shape[3], **op.split_keys_space()[0]}
    library = build("flash_attn_cute", arg_defs, generate(op.includes_bf16 if bf16 else op.includes, arg_defs,
                                                          cpp_format(op.template, keys), cpp_format(op.epilogue, keys)))
    layout = op._AttnLayout(*op._launch_args(q, k, v, out, may_fold=not causal)[4:], int(causal), 1.0)
    mode, parts = ctypes.c_int(-1), ctypes.c_int(-1)
    assert library.symbol("fray_attn_form")(ctypes.byref(layout), ctypes.byref(mode), ctypes.byref(parts)) == 0
    return mode.value, parts.value


def check(B, H, Hkv, Sq, Sk, D, causal, gain, dtype, parts, folded=False):
    g = torch.Generator(device="cuda").manual_seed(91)
    q = (gain * torch.randn(B, Sq, H, D, generator=g, device="cuda")).to(dtype).transpose(1, 2)  # strided q and output
    if folded:
        q = q.contiguous()
    k, v = (torch.randn(B, Hkv, Sk, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    guard = torch.full((B, H, Sq + (not folded), D), 7.0, dtype=dtype, device="cuda")
    out = guard[:, :, :Sq]
    mode, n = form(q, k, v, out, causal)
    assert mode == SPLIT and n in parts
    # leaves NaN in the shared memory that parts without any step do not write
    op.flash_attn_cute(q, k, torch.full_like(v, float("nan")), torch.empty_like(q), causal=causal)
    lse = torch.zeros(B, H, Sq, device="cuda")
    op.flash_attn_cute(q, k, v, out, causal=causal, lse=lse)
    torch.cuda.synchronize()
    assert op.flash_attn_status()[0] == 0
    want, want_lse, weighted, total = exact(q, k, v, causal)
    assert ((out.double() - want).abs() <= bound(want, weighted, total, dtype)).all()
    assert (lse.double() - want_lse).abs().max().item() <= 2e-4
    assert (guard[:, :, Sq:] == 7.0).all()
    again = torch.zeros_like(out)
    op.flash_attn_cute(q, k, v, again, causal=causal)
    assert torch.equal(again, out)  # with and without lse, and from call to call


# items of 256 rows (1 to 37) that are given 8 to 3 CTAs, one and two tiles in the last item, keys around the 128-key tile and
# the number of parts, causal items with fewer steps than parts, wide scores (parts with different offsets)
CASES = [(1, 1, 1, 129, 1024, 64, False, 1.0), (1, 2, 2, 300, 1025, 128, False, 4.0), (1, 4, 2, 200, 4095, 128, False, 4.0),
         (2, 3, 1, 513, 3000, 64, False, 6.0), (1, 5, 5, 1000, 2049, 128, False, 1.0), (1, 37, 37, 256, 3100, 64, False, 1.0),
         (1, 1, 1, 2048, 2048, 128, True, 4.0), (1, 2, 2, 4000, 4000, 64, True, 1.0), (2, 4, 4, 1000, 1000, 64, True, 1.0),
         (1, 3, 1, 2500, 1600, 128, True, 4.0), (1, 1, 1, 1300, 5000, 64, True, 1.0)]


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,causal,gain", CASES)
@pytest.mark.parametrize("dtype", [torch.half, torch.bfloat16])
def test_split_keys(B, H, Hkv, Sq, Sk, D, causal, gain, dtype):
    assert op._split_keys(B * H, Sq, Sk, causal, 148, D)
    check(B, H, Hkv, Sq, Sk, D, causal, gain, dtype, range(3, 9))


# More items, to which the launcher gives two CTAs each where the search (or a forced kernel) takes it: 50, 72, 74 items, one and
# two tiles in the last one, an odd number of steps, a last step of a single key, folded groups, causal items of up to 16 steps
@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,causal,gain", [
    (1, 50, 50, 256, 2500, False, 1.0), (2, 16, 4, 513, 6000, False, 4.0), (2, 37, 37, 200, 2561, False, 4.0),
    (1, 74, 74, 129, 5889, False, 1.0), (1, 8, 8, 2048, 2048, True, 4.0), (2, 4, 2, 1537, 1700, True, 1.0)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.half, torch.bfloat16])
def test_two_parts(B, H, Hkv, Sq, Sk, D, causal, gain, dtype, monkeypatch):
    monkeypatch.setenv("FRAY_ATTN_FORCE", ",".join(f"{k}={v}" for k, v in op.split_keys_space()[0].items()))
    op._fast_path.clear()  # a layout launched before would go straight to the kernel it was tuned to
    check(B, H, Hkv, Sq, Sk, D, causal, gain, dtype, (2,), folded=Hkv < H and not causal)


# what is not split: items for more than half of the SMs, items of four steps, and causal problems that are dealt by twos
@pytest.mark.parametrize("B,H,Sq,Sk,causal,mode", [(1, 75, 256, 6000, False, DEALT), (1, 4, 256, 512, False, DEALT),
                                                   (1, 40, 512, 4096, True, DEALT), (8, 50, 1280, 1280, True, MATCHED)])
def test_forms_of_other_calls(B, H, Sq, Sk, causal, mode):
    q, k = torch.empty(B, H, Sq, 64, dtype=torch.half, device="cuda"), torch.empty(B, H, Sk, 64, dtype=torch.half, device="cuda")
    assert form(q, k, k, q, causal) == (mode, 1)


# heads that follow each other as rows do (contiguous), do not (one row between them), and few and many rows per head
@pytest.mark.parametrize("Sq", [2, 33, 300])
@pytest.mark.parametrize("gap", [0, 1])
@pytest.mark.parametrize("B,H,Hkv,Sk,D", [(2, 8, 2, 700, 128), (1, 6, 3, 129, 64), (1, 4, 1, 3000, 64)])
def test_groups_of_heads_as_one_sequence(B, H, Hkv, Sk, D, gap, Sq):
    g = torch.Generator(device="cuda").manual_seed(93)
    q = torch.randn(B, H, Sq + gap, D, generator=g, device="cuda").half()[:, :, :Sq]
    k, v = (torch.randn(B, Hkv, Sk, D, generator=g, device="cuda").half() for _ in range(2))
    out, lse = torch.zeros(B, H, Sq + gap, D, device="cuda").half()[:, :, :Sq], torch.zeros(B, H, Sq, device="cuda")
    for causal in (False, True):  # a causal row's place in its head counts: not folded
        for _ in range(2):        # the checked and the warm call
            out.zero_()
            op.flash_attn_cute(q, k, v, out, causal=causal, lse=lse)
            want, want_lse, weighted, total = exact(q, k, v, causal)
            assert ((out.double() - want).abs() <= bound(want, weighted, total, torch.half)).all()
            assert (lse.double() - want_lse).abs().max().item() <= 2e-4

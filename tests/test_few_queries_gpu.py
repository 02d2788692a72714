"""The few-query kernel (all rows of a K/V head's group in one tile, keys split over a cluster) and the rule that
sends calls to it."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def exact(q, k, v):
    group = q.shape[1] // k.shape[1]
    ke, ve = (t.repeat_interleave(group, 1).double() for t in (k, v))
    s = q.double() @ ke.transpose(-1, -2) / math.sqrt(q.shape[-1])
    return torch.softmax(s, -1) @ ve, torch.logsumexp(s, -1)


# rows = group * Sq around the edges of the row placement (32, 64, 128); keys around the 128-key tile and the number
# of splits; more units than SMs; wide scores, so that offsets move inside a split and differ between splits
@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,gain", [
    (1, 1, 1, 1, 512, 64, 1.0), (1, 4, 1, 1, 513, 128, 1.0), (1, 8, 1, 4, 639, 128, 4.0), (2, 3, 1, 11, 1025, 64, 4.0),
    (1, 4, 2, 32, 4096, 128, 4.0), (2, 5, 1, 13, 1000, 128, 1.0), (1, 1, 1, 127, 515, 64, 4.0), (1, 2, 1, 64, 2049, 128, 4.0),
    (80, 4, 2, 1, 600, 64, 4.0), (8, 32, 8, 1, 8192, 128, 1.0), (1, 16, 2, 8, 16000, 128, 6.0),
    (40, 8, 2, 25, 700, 64, 4.0)])
@pytest.mark.parametrize("dtype", [torch.half, torch.bfloat16])
def test_few_queries(B, H, Hkv, Sq, Sk, D, gain, dtype):
    from fray_b200.jit_kernels import flash_attn_cute, flash_attn_status
    g = torch.Generator(device="cuda").manual_seed(71)
    q = (gain * torch.randn(B, Sq, H, D, generator=g, device="cuda")).to(dtype).transpose(1, 2)  # strided q and output
    k, v = (torch.randn(B, Hkv, Sk, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    guard = torch.full((B, H, Sq + 1, D), 7.0, dtype=dtype, device="cuda")
    out = guard[:, :, :Sq]
    lse = torch.zeros(B, H, Sq, device="cuda")
    flash_attn_cute(q, k, v, out, lse=lse)
    torch.cuda.synchronize()
    assert flash_attn_status()[0] == 0
    want, want_lse = exact(q, k, v)
    # P and the output are rounded to 16 bits (relative step u = 2^-11 or 2^-8): every output is a convex sum of values
    # |v| <= 6 with weights off by u/2, rounded once more
    u = 2.0 ** -11 if dtype is torch.half else 2.0 ** -8
    assert (out.double() - want).abs().max().item() <= 6 * u
    assert (lse.double() - want_lse).abs().max().item() <= 2e-4
    assert (guard[:, :, Sq:] == 7.0).all()
    again = torch.zeros_like(out)
    flash_attn_cute(q, k, v, again)
    assert torch.equal(again, out)  # with and without lse, and from call to call


def test_few_queries_non_finite_values_stay_in_their_rows():
    from fray_b200.jit_kernels import flash_attn_cute
    g = torch.Generator(device="cuda").manual_seed(73)
    q, k, v = (torch.randn(1, 4, s, 128, generator=g, device="cuda").half() for s in (3, 700, 700))
    want = torch.zeros_like(q)
    flash_attn_cute(q, k, v, want)
    q[0, 2, 1] = float("nan")
    out = torch.zeros_like(q)
    flash_attn_cute(q, k, v, out)
    assert torch.isnan(out[0, 2, 1]).all()
    out[0, 2, 1] = want[0, 2, 1]
    assert torch.equal(out, want)


# every row placement (rows = 4, 32, 44, 64, 100) and infinities in every quarter of a step, in several splits and in the
# ragged last step: a key's value reaches the sums of its own weights only, never a product with another copy's zero
@pytest.mark.parametrize("H,Sq", [(4, 1), (4, 8), (4, 11), (4, 16), (4, 25)])
@pytest.mark.parametrize("Sk", [600, 3000])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.half, torch.bfloat16])
def test_few_queries_infinite_values_stay_in_their_columns(H, Sq, Sk, D, dtype):
    from fray_b200.jit_kernels import flash_attn_cute, flash_attn_status
    g = torch.Generator(device="cuda").manual_seed(79)
    q, k, v = (torch.randn(2, h, s, D, generator=g, device="cuda").to(dtype) for h, s in ((H, Sq), (1, Sk), (1, Sk)))
    want = torch.zeros_like(q)
    flash_attn_cute(q, k, v, want)
    for column, key in enumerate((5, 40, 70, 101, 300, 511, Sk - 1)):
        v[0, 0, key, 3 * column] = float("inf")
        v[0, 0, key, 3 * column + 1] = float("-inf")
        want[0, :, :, 3 * column] = float("inf")  # weights of normal scores stay above the smallest 16-bit number
        want[0, :, :, 3 * column + 1] = float("-inf")
    v[0, 0, 200, 40], v[0, 0, 330, 40], v[0, 0, 450, 41] = float("inf"), float("-inf"), float("nan")
    want[0, :, :, 40:42] = float("nan")
    out = torch.zeros_like(q)
    flash_attn_cute(q, k, v, out)
    torch.cuda.synchronize()
    assert flash_attn_status()[0] == 0
    no_number = torch.isnan(want)
    assert torch.equal(torch.isnan(out), no_number) and torch.equal(out[~no_number], want[~no_number])


# one, two, three and more steps per split, each call behind other kernels (whose code takes the instruction cache): however
# long a warp is held up between its last P and the epilogue, it finds the last product's barrier phase
def test_few_queries_between_other_kernels():
    from fray_b200.jit_kernels import flash_attn_cute, flash_attn_status
    g = torch.Generator(device="cuda").manual_seed(97)
    calls = []
    for H, Hkv, Sq, Sk, D in ((8, 2, 1, 1024, 128), (8, 2, 1, 2048, 64), (8, 2, 13, 2900, 128), (8, 1, 9, 8192, 64), (4, 4, 300, 300, 128)):
        q, k, v = (torch.randn(1, h, s, D, generator=g, device="cuda").half() for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
        out = torch.zeros_like(q)
        flash_attn_cute(q, k, v, out)
        calls.append((q, k, v, out.clone(), out))
    for n in range(400):
        for q, k, v, want, out in calls[n % 2:] + calls[:n % 2]:
            flash_attn_cute(q, k, v, out)
        torch.softmax(calls[0][1].float(), -1)
    torch.cuda.synchronize()
    assert flash_attn_status()[0] == 0
    for q, k, v, want, out in calls:
        assert torch.equal(out, want)

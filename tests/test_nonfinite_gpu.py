"""Infinite and NaN operands through the row-pair kernel's forms: they stay in the rows (columns, slices) that they belong to."""
import importlib

import pytest
import torch

from tests.test_cta_pairs_gpu import HEADS, ROWS, SINGLE, pair
from tests.test_four_streams_gpu import four_streams
from tests.test_split_keys_gpu import bound, exact

pytestmark = pytest.mark.gpu

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")
STREAMS = "streams"

# four streams with a group that has no step, an odd number of steps, steps above the diagonal; two threads per row; single CTAs
# and pairs at head dim 128
CASES = [(STREAMS, 2, 200, 200, 300, 40, 64, False), (STREAMS, 2, 90, 45, 513, 3000, 64, False), (STREAMS, 3, 60, 20, 333, 333, 64, True),
         (SINGLE, 4, 100, 50, 256, 256, 64, False), (SINGLE, 2, 60, 60, 300, 700, 128, True), (ROWS, 1, 74, 74, 600, 4090, 128, False),
         (HEADS, 4, 64, 16, 1300, 1300, 128, True)]


def call(case, monkeypatch, spoil=None):
    """Operands (spoilt), output and log-sum-exp of a call that takes the case's form."""
    form, B, H, Hkv, Sq, Sk, D, causal = case
    point = next(p for p in op.tuning_space(D) if p["KIND"] == op.KIND_ROW_PAIRS)
    monkeypatch.setenv("FRAY_ATTN_FORCE", ",".join(f"{k}={v}" for k, v in point.items()))
    op._fast_path.clear()  # a layout launched before would go straight to the kernel it was tuned to
    g = torch.Generator(device="cuda").manual_seed(113)
    q = torch.randn(B, Sq, H, D, generator=g, device="cuda").half().transpose(1, 2)  # strided: groups are not folded
    k, v = (torch.randn(B, Hkv, Sk, D, generator=g, device="cuda").half() for _ in range(2))
    k[0, 0, :, 0] = k[0, 0, :, 0].abs() + 0.1
    if spoil:
        spoil(q, k, v)
    out, lse = torch.full_like(q, 7.0), torch.zeros(B, H, Sq, device="cuda")
    if form == STREAMS:
        assert four_streams(q, k, v, out, causal) == 1
    else:
        assert pair(q, k, v, out, causal) == form and four_streams(q, k, v, out, causal) == 0
    op.flash_attn_cute(q, k, v, out, causal=causal, lse=lse)
    torch.cuda.synchronize()
    assert op.flash_attn_status()[0] == 0
    return q, k, v, out, lse


@pytest.mark.parametrize("case", CASES)
def test_scores(case, monkeypatch):
    """A NaN query, a query whose scores are all -inf (no key counts: zeros), a key with infinite scores: NaN for the queries that
    score it +inf, no weight for those that score it -inf."""
    _, _, H, Hkv, _, Sk, _, causal = case
    group = H // Hkv

    def spoil(q, k, v):
        q[0, 0, 5, 3] = float("nan")
        q[0, 0, 9, 0] = float("-inf")
        q[0, 0, 9, 1] = -1.0
        k[0, 0, Sk // 2, 1] = float("inf")

    q, k, v, out, lse = call(case, monkeypatch, spoil)
    want, want_lse, weighted, total = exact(q[:1, :group], k[:1, :1], v[:1, :1], causal)
    got, got_lse = out[:1, :group].double(), lse[:1, :group].double()
    assert (got[0, 0, 9] == 0).all() and got_lse[0, 0, 9] == float("-inf")
    want[0, 0, 9], weighted[0, 0, 9] = 0.0, 0.0
    bad = want.isnan()
    assert bad[0, 0, 5].all() and 0 < bad.sum() < bad.numel() and bad.any(-1).equal(bad.all(-1))
    assert got.isnan().equal(bad) and not got_lse[bad[..., 0]].isfinite().any()
    assert ((got - want).abs() <= bound(want, weighted, total, torch.half))[~bad].all()
    fine = ~bad[..., 0]
    fine[0, 0, 9] = False
    assert (got_lse - want_lse)[fine].abs().max().item() <= 2e-4
    *_, clean, clean_lse = call(case, monkeypatch)
    assert torch.equal(out[1:], clean[1:]) and torch.equal(out[:, group:], clean[:, group:])
    assert torch.equal(lse[1:], clean_lse[1:]) and torch.equal(lse[:, group:], clean_lse[:, group:])


@pytest.mark.parametrize("case", CASES)
def test_values(case, monkeypatch):
    """An infinite value, whatever weight it has: its column is infinite or NaN for the queries that see it, the others as they were."""
    _, _, H, Hkv, Sq, Sk, D, causal = case
    group, key = H // Hkv, min(Sq, Sk) - 1 if causal else Sk - 1

    def spoil(q, k, v):
        v[0, 0, key, 2] = float("inf")

    *_, out, lse = call(case, monkeypatch, spoil)
    *_, clean, clean_lse = call(case, monkeypatch)
    others = [d for d in range(D) if d != 2]
    assert torch.equal(out[..., others], clean[..., others]) and torch.equal(lse, clean_lse) and clean.isfinite().all()
    assert torch.equal(out[1:], clean[1:]) and torch.equal(out[:, group:], clean[:, group:])
    first = key if causal else 0  # queries from here on see the key; up to 127 before share a tile with one that does
    assert not out[0, :group, first:, 2].isfinite().any()
    assert torch.equal(out[0, :group, :max(0, first - 127), 2], clean[0, :group, :max(0, first - 127), 2])

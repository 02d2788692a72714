"""The rule that sends calls to the row-pair kernel with split keys, at its edges, and which groups of heads are folded."""
import ctypes
import importlib

import pytest
import torch

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


def split(slices, sq, sk, causal=False, d=128):
    return op._split_keys(slices, sq, sk, causal, 148, d)


def test_calls_the_rule_takes():
    # measured on 148 SMs: the kernel's time over the best other one's
    assert split(1, 256, 12000) and split(8, 1024, 6000) and split(36, 256, 3000)  # 0.37, 0.68, 0.92
    assert split(24, 256, 1536) and split(30, 256, 2048) and split(12, 256, 1024)  # 0.97, 0.94, 1.00
    assert split(32, 256, 1024, d=64) and split(1, 3000, 3000, causal=True)        # 1.00, 0.67


def test_calls_the_rule_leaves():
    assert not split(36, 256, 2048) and not split(48, 256, 6000)     # 1.17, 1.05: no room for four parts, for three
    assert not split(16, 256, 1024) and not split(12, 256, 768)      # 1.01, 1.15: the merge costs what the split saves
    assert not split(36, 256, 1024, d=64) and not split(1, 256, 512, d=64)
    assert not split(1, 256, 12000, causal=True)                     # a causal item of 256 rows has two steps
    assert not split(4, 3000, 3000, causal=True)                     # 48 items, 1.08


def test_heads_that_follow_each_other_as_rows_do():
    t = torch.empty(2, 4, 10, 64)
    assert op._folds(t) and not op._folds(t[:, :, :9]) and not op._folds(torch.empty(2, 10, 4, 64).transpose(1, 2))


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    """The launcher's rules, which are host code: parts(items, steps, causal, sms, active) and may_split(items, steps, sms)."""
    from fray_b200.jit import build, generate
    args = (("n", int),)
    code = generate(op.includes, args, "\n__return_code = 0;\n", """
extern "C" EXPORT_API int parts(int items, int steps, int causal, int sms, const int* active) {
    return fray::sm100::duo_parts(items, steps, causal != 0, sms, *reinterpret_cast<const int (*)[fray::kMaxClusterCtas + 1]>(active));
}
extern "C" EXPORT_API int may_split(int items, int steps, int sms) { return fray::sm100::duo_may_split(items, steps, sms); }
""")
    with pytest.MonkeyPatch.context() as patch:
        patch.setenv("FRAY_CACHE_DIR", str(tmp_path_factory.mktemp("rules")))
        lib = build("split_rules", args, code)
    parts, may_split = lib.symbol("parts"), lib.symbol("may_split")
    return (lambda items, steps, causal, sms, active: parts(items, steps, causal, sms, (ctypes.c_int * 9)(*active))), may_split


# clusters of 1 to 8 CTAs that run at the same time on 148 SMs: as many as the SMs allow at best, and as on a device whose GPCs
# leave some over
PLACES = [(0, 148, 74, 49, 37, 29, 24, 21, 18), (0, 148, 74, 47, 35, 27, 22, 18, 16), (0, 148, 70, 40, 30, 0, 0, 0, 0)]


@pytest.mark.parametrize("places", PLACES)
def test_calls_that_are_not_looked_at_would_not_be_split(rules, places):
    parts, may_split = rules
    for items in range(1, 200):
        for steps in range(1, 60):
            for causal in (0, 1):
                n = parts(items, steps, causal, 148, places)
                assert 1 <= n <= min(8, steps)
                if not may_split(items, steps, 148):
                    assert n == 1 or 2 * items > 148  # two CTAs per item do not fit
                if causal and n > 1:
                    assert items <= places[n]


def test_parts_of_some_calls(rules):
    parts, may_split = rules
    assert not may_split(4, 2, 148) and not may_split(75, 47, 148) and may_split(74, 5, 148)
    first = PLACES[0]
    assert [parts(n, 47, 0, 148, first) for n in (1, 18, 37, 38, 50, 72, 74)] == [8, 8, 4, 3, 2, 2, 2]
    assert [parts(n, 20, 0, 148, first) for n in (50, 72)] == [2, 2] and parts(64, 32, 1, 148, first) == 2
    assert parts(71, 32, 1, 148, PLACES[2]) == 1  # causal: a second round is not looked at

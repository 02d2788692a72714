"""The rule that sends calls to the few-query kernel, at its edges."""
import importlib

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


def few(group, sq, sk, units, causal=False, d=128):
    return op._few_queries(group, sq, sk, causal, units, 148, d)


def test_calls_the_rule_takes_and_leaves():
    assert few(4, 1, 8192, 64) and few(1, 64, 512, 74) and few(8, 16, 512, 1000)
    assert not few(4, 1, 8192, 64, causal=True)      # rows see different keys
    assert not few(4, 33, 8192, 64)                  # 132 rows: more than a tile
    assert not few(4, 1, 511, 64)                    # too few keys to split
    assert not few(1, 1, 2048, 149)                  # nothing to share, and the units fill the chip
    assert few(1, 1, 8192, 149) and few(1, 1, 4096, 296) and few(1, 1, 4096, 149, d=64)


def test_calls_whose_other_kernels_are_faster_are_left_to_them():
    # measured on 148 SMs: the few-query kernel's time over the best other one's is in the comment
    assert not few(1, 128, 512, 148)                                     # 1.46: a K/V head per query head, keys not split
    assert not few(1, 128, 4096, 260) and not few(1, 128, 8192, 1000)    # 1.17, 1.10
    assert not few(1, 64, 1536, 90) and not few(1, 64, 1536, 90, d=64)   # 1.36, 1.16
    assert not few(1, 16, 4096, 150)                                     # 1.11
    assert not few(2, 64, 512, 40) and not few(2, 64, 1024, 200)         # 1.20, 1.20
    assert not few(3, 42, 512, 149) and not few(4, 32, 512, 37)          # 1.27, 1.18


def test_calls_the_kernel_is_for_stay_with_it():
    assert few(1, 1, 8192, 8) and few(1, 128, 8192, 8) and few(2, 64, 8192, 40)      # 0.20, 0.29, 0.57: keys split
    assert few(8, 1, 8192, 1000) and few(4, 32, 1024, 148) and few(2, 1, 512, 1000)  # 0.17, 0.55, 0.77: one reading per group
    assert few(1, 32, 1024, 100) and few(1, 32, 2048, 100, d=64)                     # 0.87, 0.72


def test_the_kernel_is_a_library_of_its_own_beside_the_tuned_ones(monkeypatch):
    monkeypatch.delenv("FRAY_ATTN_FORCE", raising=False)
    for d in (64, 128):
        assert op.few_query_space()[0] not in op.tuning_space(d)
    assert sum(point == op.few_query_space()[0] for _, point, _ in op._space_points((64, 128), forced=False)) == 4

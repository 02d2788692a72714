"""The rule that sends calls to the few-query kernel, at its edges."""
import importlib

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


def few(group, sq, sk, units, causal=False):
    return op._few_queries(group, sq, sk, causal, units, 148)


def test_calls_the_rule_takes_and_leaves():
    assert few(4, 1, 8192, 64) and few(1, 128, 512, 148) and few(8, 16, 512, 1000)
    assert not few(4, 1, 8192, 64, causal=True)      # rows see different keys
    assert not few(4, 33, 8192, 64)                  # 132 rows: more than a tile
    assert not few(4, 1, 511, 64)                    # too few keys to split
    assert not few(1, 1, 2048, 149)                  # nothing to share, and the units fill the chip
    assert few(1, 1, 4096, 149)


def test_the_kernel_is_a_library_of_its_own_beside_the_tuned_ones(monkeypatch):
    monkeypatch.delenv("FRAY_ATTN_FORCE", raising=False)
    for d in (64, 128):
        assert op.few_query_space()[0] not in op.tuning_space(d)
    assert sum(point == op.few_query_space()[0] for _, point, _ in op._space_points((64, 128), forced=False)) == 4

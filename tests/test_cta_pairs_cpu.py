"""Which calls the row-pair kernel's launcher gives to CTA pairs: the rule, which is host code, at its edges."""
import importlib

import pytest

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")
SINGLE, ROWS, HEADS = 0, 1, 2


@pytest.fixture(scope="module")
def pair(tmp_path_factory):
    from fray_b200.jit import build, generate
    args = (("n", int),)
    code = generate(op.includes, args, "\n__return_code = 0;\n", """
extern "C" EXPORT_API int pair(int causal, int slices, int group, int seq_len, int steps, int sms) {
    return fray::sm100::duo_pair(causal != 0, slices, group, seq_len, steps, sms);
}
""")
    with pytest.MonkeyPatch.context() as patch:
        patch.setenv("FRAY_CACHE_DIR", str(tmp_path_factory.mktemp("pair")))
        return build("pair_rule", args, code).symbol("pair")


def test_calls_the_rule_takes(pair):
    assert pair(0, 128, 1, 4096, 32, 148) == ROWS and pair(0, 256, 1, 1024, 8, 148) == ROWS   # 0.98, 0.99
    assert pair(1, 64, 4, 3000, 24, 148) == HEADS and pair(1, 160, 2, 2895, 23, 148) == HEADS  # 0.98, 0.95
    assert pair(0, 148, 2, 600, 17, 148) == HEADS  # heads that could not be laid end to end


def test_calls_the_rule_leaves(pair):
    assert pair(1, 128, 1, 4096, 32, 148) == SINGLE and pair(1, 128, 3, 4096, 32, 148) == SINGLE  # causal items by rows: 1.03
    assert pair(0, 40, 1, 2610, 39, 148) == SINGLE   # 240 items of 512 rows on 74 pairs take a fourth round: 1.14
    assert pair(0, 640, 1, 3490, 1, 148) == SINGLE   # 1.06
    assert pair(0, 32, 1, 2048, 16, 148) == SINGLE   # 28 steps per SM: level, and 1.01 on a cooler board


def test_calls_whose_last_round_is_mostly_empty(pair):
    assert pair(0, 12, 1, 6958, 55, 148) == ROWS     # 168 items of 512 rows on three times 74 pairs
    assert pair(0, 16, 1, 4894, 39, 148) == SINGLE   # 160: 1.015 with wide scores
    assert pair(0, 8, 1, 6031, 48, 148) == SINGLE    # 96 on twice 74: 1.05
    assert pair(0, 8, 2, 5861, 46, 148) == SINGLE    # the same by heads, 92: 1.04


def test_fewer_pairs_than_half_of_the_sms(pair, monkeypatch):
    from fray_b200.jit import build, generate
    args = (("n", int),)
    code = generate(op.includes, args, "\n__return_code = 0;\n", """
extern "C" EXPORT_API int pair(int slices, int group, int seq_len, int steps, int sms, int pairs) {
    return fray::sm100::duo_pair(false, slices, group, seq_len, steps, sms, pairs);
}
""")
    of = build("pair_rule_places", args, code).symbol("pair")
    assert of(128, 1, 4096, 32, 148, 74) == ROWS and of(128, 1, 4096, 32, 148, 73) == SINGLE  # 1024 items on 73: 15 rounds for 14
    assert of(128, 2, 4096, 32, 148, 74) == HEADS and of(128, 2, 4096, 32, 148, 70) == SINGLE
    assert of(128, 1, 4096, 32, 148, 0) == SINGLE  # a device that places none


def test_the_longest_folded_sequences(pair):
    longest = 2 ** 31 - 1 - 255  # what folded groups may grow to
    for seq_len in (longest - 256, longest, 2 ** 31 - 1):
        assert pair(0, 2, 1, seq_len, 8, 148) == ROWS and pair(0, 2, 2, seq_len, 8, 148) == HEADS


def test_pairs_never_need_more_rounds(pair):
    for slices in range(2, 400, 2):
        for seq_len in (200, 256, 257, 512, 513, 700, 1024, 1100):
            for group in (1, 2):
                form = pair(0, slices, group, seq_len, 64, 148)
                items = slices * -(-seq_len // 256)
                if form != SINGLE:
                    mine = items // 2 if form == HEADS else slices * -(-seq_len // 512)
                    assert -(-mine // 74) <= -(-items // 148) and (form == HEADS) == (group == 2)
    assert pair(0, 400, 2, 4096, 64, 1) == SINGLE  # a device without a pair of SMs

"""Which causal calls of the row-pair kernel are matched by twos: the rule, which is host code, at its edges."""
import ctypes
import importlib

import pytest

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


@pytest.fixture(scope="module")
def matched(tmp_path_factory):
    from fray_b200.jit import build, generate
    args = (("n", int),)
    code = generate(op.includes, args, "\n__return_code = 0;\n", """
extern "C" EXPORT_API int matched(int causal, int heads, int kv_heads, int rows, int units, int max_deal) {
    const fray::AttnShape shp{1, heads, rows, 128}, shp_kv{1, kv_heads, rows, 128};
    return fray::sm100::duo_matched(causal != 0, shp, shp_kv, (rows + 255LL) / 256 * heads, units, max_deal);
}
""")
    with pytest.MonkeyPatch.context() as patch:
        patch.setenv("FRAY_CACHE_DIR", str(tmp_path_factory.mktemp("matched")))
        lib = build("matched_rule", args, code).symbol("matched")
    lib.argtypes = [ctypes.c_int] * 6
    return lib


@pytest.mark.parametrize("kv_heads,units,taken", [
    (400, 500, 1), (200, 500, 1),  # whole rounds
    (400, 565, 1), (400, 566, 0),  # 1130 and 1132 places for 1000 twos
    (200, 525, 1), (200, 526, 0),  # grouped heads: 1050 and 1052
    (400, 1000, 1), (400, 1001, 0),  # two items a CTA at least
])
def test_last_round(matched, kv_heads, units, taken):
    assert matched(1, 400, kv_heads, 1280, units, 189) == taken
    assert matched(0, 400, kv_heads, 1280, units, 189) == 0


def test_the_deal_has_room(matched):
    assert matched(1, 400, 400, 1280, 10, 201) == 1 and matched(1, 400, 400, 1280, 10, 200) == 0

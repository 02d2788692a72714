"""Which calls of head dim 64 go to four independent streams per CTA: the rule, which is host code, at its edges."""
import importlib

import pytest

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


@pytest.fixture(scope="module")
def quad(tmp_path_factory):
    from fray_b200.jit import build, generate
    args = (("n", int),)
    code = generate(op.includes, args, "\n__return_code = 0;\n", """
extern "C" EXPORT_API int quad(int causal, long long items, int seq_k, int sms) {
    return fray::sm100::duo_quad(causal != 0, items, seq_k, sms);
}
""")
    with pytest.MonkeyPatch.context() as patch:
        patch.setenv("FRAY_CACHE_DIR", str(tmp_path_factory.mktemp("quad")))
        lib = build("quad_rule", args, code).symbol("quad")
    import ctypes
    lib.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return lib


def test_rule(quad):
    assert quad(1, 1024, 1024, 148) and quad(1, 1, 64, 148)          # any causal call
    assert quad(0, 369, 1024, 148) and not quad(0, 370, 1024, 148)   # two and a half rounds of items
    assert quad(0, 1024, 1025, 148) and not quad(0, 1024, 961, 148)  # up to eight steps of 128 keys
    assert quad(0, 1024, 960, 148) and not quad(0, 1024, 897 + 64, 148) and quad(0, 1024, 64, 148) and not quad(0, 1024, 65, 148)


def test_the_kernel_settles_before_its_last_barrier():
    """As every kernel that waits with a limit: it stays for its own copies and products when a wait has run out."""
    import os
    import re

    import fray_b200
    path = os.path.join(os.path.dirname(fray_b200.__file__), "include", "flash_attn", "four_streams_sm100.cuh")
    text = open(path).read()
    end = text.rindex("tmem_dealloc(tmem_base")
    settle = text.rindex("if (*abort_flag == 1u) settle_after_abort();")
    assert settle < end and text[settle:end].count("__syncthreads();") == 1
    assert not re.search(r"mbar_wait|tma_load|mma_", text[settle:end])

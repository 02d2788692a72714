"""Every kernel header brings in what it uses: each compiles as the only one of a translation unit."""
import os
import re
from concurrent.futures import ThreadPoolExecutor

from fray_b200.jit import build, generate

HEADERS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fray_b200", "include", "flash_attn")


def test_each_header_compiles_alone(tmp_path, monkeypatch):
    monkeypatch.setenv("FRAY_CACHE_DIR", str(tmp_path))
    args = (("n", int),)

    def alone(header):
        build("header", args, generate((f'"flash_attn/{header}"',), args, "\n__return_code = 0;\n"))

    headers = sorted(os.listdir(HEADERS))
    assert "fwd_split_sm100.cuh" in headers
    with ThreadPoolExecutor() as pool:
        list(pool.map(alone, headers))


def test_a_kernel_names_one_cta_group():
    """All tcgen05 instructions of a kernel have to name the same cta_group: in kernels that are built for one CTA and for pairs
    each wrapper of one goes by the kernel's number of CTAs, in the others none does."""
    pairs = 0
    for header in sorted(os.listdir(HEADERS)):
        text = re.sub(r"//.*", "", open(os.path.join(HEADERS, header)).read())
        if header == "sm100_ptx.cuh" or "tmem_alloc" not in text:
            continue
        calls = re.findall(r"\b((?:tmem_alloc|tmem_relinquish|tmem_dealloc|mma_ss|mma_ts|mma_commit)\w*[<(][^;]*;)", text)
        by_argument = ["CtaGroup<CTAS>{}" in call or re.match(r"\w+<CTAS>\(", call) is not None for call in calls]
        if "int CTAS" in text:
            pairs += 1
            assert all(by_argument), (header, calls)
        else:
            assert not any(by_argument), (header, calls)
        assert len(calls) >= 6, header
    assert pairs == 2


def test_a_declared_alignment_is_tested_behind_the_compilers_back():
    """Swizzled tiles need a base of 1024 bytes.  Where the declaration promises it, a plain test of the address is folded to true."""
    text = open(os.path.join(HEADERS, "fwd_duo_sm100.cuh")).read()
    declared = re.findall(r"extern __shared__ __align__\(1024\) uint8_t (\w+)\[\];\s*smem = (\w+);\s*fits = ([^;]*);", text)
    assert len(declared) == text.count("__align__(1024)") == 1
    name, base, test = declared[0]
    assert name == base and re.fullmatch(r"\(opaque\(smem_u32\(smem\)\) & 1023u\) == 0", test)

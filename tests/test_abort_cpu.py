"""Every kernel that waits with a limit stays for its own copies and products when a wait has run out, before it gives back its
tensor memory and leaves."""
import glob
import os
import re

import fray_b200

HEADERS = os.path.join(os.path.dirname(fray_b200.__file__), "include", "flash_attn")


def test_every_kernel_settles_before_its_last_barrier():
    seen = 0
    for path in glob.glob(os.path.join(HEADERS, "fwd_*_sm100.cuh")):
        text = open(path).read()
        end = text.rindex("tmem_dealloc(tmem_base")
        settle = text.rindex("if (*abort_flag == 1u) settle_after_abort();")
        assert settle < end and text[settle:end].count("__syncthreads();") == 1, path
        assert not re.search(r"mbar_wait|tma_load|mma_", text[settle:end]), path
        seen += 1
    assert seen == 6


def test_a_warp_of_many_lanes_leaves_its_loop_as_one():
    """The abort flag can go up between two lanes' looks at it: where a whole warp (the issuing one) decides by it, the lanes that
    left would leave the others alone at the next shuffle or election, which has no limit."""
    seen = 0
    for path in glob.glob(os.path.join(HEADERS, "*_sm100.cuh")):
        roles = re.split(r"// =====+ ", open(path).read())
        for role in roles[1:]:
            if not role.startswith("MMA issue"):
                continue
            for line in role.split("if (*abort_flag == 1u)")[0].splitlines():
                if re.search(r"\bif \(.*\*abort_flag|= \*abort_flag", line):
                    assert "__any_sync(0xffffffffu, *abort_flag" in line, (path, line)
            seen += 1
    assert seen == 6

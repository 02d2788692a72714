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

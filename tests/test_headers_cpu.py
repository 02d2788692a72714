"""Every kernel header brings in what it uses: each compiles as the only one of a translation unit."""
import os
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

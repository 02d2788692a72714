"""The structure that carries a warm call's fixed arguments matches the argument table of `launch` and its C++ side."""
import importlib
import os
import re

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


def test_layout_fields_follow_the_argument_table():
    fields = [name for name, _ in op._AttnLayout._fields_]
    table = [name for name, _ in op.arg_defs if name not in ("Q", "K", "V", "O", "Lse", "stream")]
    assert fields == table
    header = os.path.join(os.path.dirname(op.__file__), "..", "include", "flash_attn", "flash_attn_sm100.cuh")
    body = re.search(r"struct AttnLayout \{(.*?)\};", open(header).read(), re.S).group(1)
    members = [m for line in body.split(";") for m in re.sub(r"\b(int|float)\b", "", line).replace(",", " ").split()]
    short = [re.sub(r"^([qkvo])_stride_([bhs])$", r"\1_s\2", f) for f in fields]
    assert members == short

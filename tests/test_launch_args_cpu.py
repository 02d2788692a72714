"""Sizes and strides reach `launch` as they are, or the call is refused: the ABI has 32 bits for each, and ctypes wraps silently.
Tensors of the sizes that matter have no storage here, and the kernel library is faked."""
import importlib
import types

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

op = importlib.import_module("fray_b200.jit_kernels.flashattn_cute")


@pytest.fixture
def launched(monkeypatch):
    """Calls of the op end in this list of argument tuples."""
    calls = []

    class Library:
        path = "fake"

        def __call__(self, *args):
            calls.append(args)
            return 0

        def symbol(self, name):
            return types.SimpleNamespace()

    monkeypatch.delenv("FRAY_ATTN_FORCE", raising=False)
    monkeypatch.setattr(torch.Tensor, "data_ptr", lambda t: 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: None)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda dev: types.SimpleNamespace(multi_processor_count=148))
    monkeypatch.setattr(op.jit_tuner, "compile_and_tune", lambda **k: Library())
    monkeypatch.setattr(op, "_fast_path", op.OrderedDict())
    monkeypatch.setattr(op, "_used_runtimes", {})
    monkeypatch.setattr(op, "_no_lse", {})
    with FakeTensorMode():
        yield calls


def call(B, H, Hkv, S, D, Sk=128, causal=False, view=lambda t: t):
    q, out = (view(torch.empty(B, H, S, D, dtype=torch.half, device="cuda:0")) for _ in range(2))
    k, v = (torch.empty(B, Hkv, Sk, D, dtype=torch.half, device="cuda:0") for _ in range(2))
    op.flash_attn_cute(q, k, v, out, causal=causal)


def sizes(args):
    """(heads, queries, q's strides, out's strides) of a launch; modes of extent 1 are not stepped over."""
    return args[5], args[6], args[7:10], args[16:19]


def test_groups_are_folded_while_their_step_fits(launched):
    call(1, 64, 2, 524280, 128)  # 32 * 524280 * 128 = 2^31 - 32768
    heads, rows, q, out = sizes(launched[0])
    assert (heads, rows) == (2, 32 * 524280) and q == out and q[1:] == (32 * 524280 * 128, 128) and q[1] < 2 ** 31


# (the step from group to group would wrap to 16384, to -2^31, to 2^20 + ...): the query heads stay slices of their own
@pytest.mark.parametrize("H,S", [(64, 1048580), (32, 2 ** 20), (32, 2 ** 20 + 512), (32, 2 ** 21 + 512)])
def test_groups_whose_step_does_not_fit_are_not_folded(launched, H, S):
    call(1, H, 2, S, 128)
    heads, rows, q, out = sizes(launched[0])
    assert (heads, rows) == (H, S) and q == out and q[1:] == (S * 128, 128)


def test_one_group_has_no_step(launched):
    call(1, 32, 1, 2 ** 20, 128)  # 2^32 elements in a single folded slice
    heads, rows, q, _ = sizes(launched[0])
    assert (heads, rows) == (1, 32 * 2 ** 20) and q[2] == 128 and all(0 < s < 2 ** 31 for s in q)


@pytest.mark.parametrize("rows", [2 ** 28 - 32, 2 ** 28 - 8])  # 8 heads of them: 2^31 - 256 and 2^31 - 64
def test_folded_length_leaves_room_for_whole_tiles(launched, rows):
    overlapping = lambda t: t.as_strided(t.shape, (8, 8 * rows, 8, 1))  # noqa: E731
    call(1, 8, 1, rows, 64, view=overlapping)
    heads, n, _, _ = sizes(launched[0])
    assert (heads, n) == ((1, 8 * rows) if 8 * rows + 255 < 2 ** 31 else (8, rows))


# contiguous tensors are handed on as they are, whatever their strides: these wrap to 8 * n, to 0 and to a negative number
@pytest.mark.parametrize("H,S", [(8, 2 ** 22 + 8), (8, 2 ** 22), (8, 2 ** 21)])
@pytest.mark.parametrize("causal", [False, True])
def test_contiguous_strides_that_do_not_fit_are_refused(launched, H, S, causal):
    with pytest.raises(RuntimeError):
        call(2, H, H, S, 128, causal=causal)
    with pytest.raises(RuntimeError):
        call(2, H, H, 64, 128, Sk=S, causal=causal)
    assert not launched


def test_strides_that_fit_are_not_refused(launched):
    call(2, 8, 8, 2 ** 21 - 8, 128, causal=True)
    assert launched[0][7] == 8 * (2 ** 21 - 8) * 128
    call(1, 8, 8, 2 ** 22, 128)  # the batch stride of one batch is not stepped over
    assert sizes(launched[1])[2][1:] == (2 ** 29, 128)

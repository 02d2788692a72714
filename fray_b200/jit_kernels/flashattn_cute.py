"""``flash_attn_cute(Q, K, V, Output)`` - fp16 (or bf16) attention forward written in place.

Drop-in for the reference op (fray/jit_kernels/flashattn_cute.py:15-45): four fp16 CUDA
tensors of identical shape ``[B, H, S, D]``, result stored into ``Output``, launch on
the current stream, nothing returned.  The 4-positional call behaves as in the
reference (non-causal, scale ``1/sqrt(D)``); ``causal``, ``scale`` and ``lse`` are keyword-only
extensions, and K / V may carry fewer heads than Q (grouped-query attention).  Unlike the reference, strided views whose last dimension is contiguous are
consumed and produced through their strides (no hidden copies, and a non-contiguous
``Output`` really receives the result).
"""
import ctypes
import math
import os
import threading
from collections import OrderedDict
from typing import Any, Dict, Optional, Tuple

import torch

from .tuner import jit_tuner

includes = ('"flash_attn/flash_attn_sm100.cuh"',)
# bf16 tensors get libraries of their own: this header, sorted ahead of the other one by the generator,
# switches the operand type of the whole translation unit.
includes_bf16 = ('"flash_attn/bf16_operands.cuh"', *includes)

template = """
// Templated args from Python JIT call
fray::flash_attn_sm100<{KIND}, {D}, {BLOCK_N}, {STAGES}>(
    Q, K, V, O, batch_size, num_heads, seq_len,
    q_stride_b, q_stride_h, q_stride_s, k_stride_b, k_stride_h, k_stride_s,
    v_stride_b, v_stride_h, v_stride_s, o_stride_b, o_stride_h, o_stride_s,
    num_kv_heads, seq_len_kv, Lse, causal, scale, stream, __return_code);
"""

# Exported next to `launch`: blocking read (and optional clear) of the device status words.
epilogue = """
extern "C" EXPORT_API int fray_attn_status(int* out4, int clear) {
    return fray::read_attn_status(out4, clear != 0);
}
extern "C" EXPORT_API void fray_attn_kernel_info(int* out4) {
    out4[0] = {KIND}; out4[1] = {D}; out4[2] = {BLOCK_N}; out4[3] = {STAGES};
}
extern "C" EXPORT_API int fray_attn_operand_is_bf16(void) {
    return fray::kOperandIsBf16;
}
extern "C" EXPORT_API int fray_attn_launch_layout(void* Q, void* K, void* V, void* O, void* Lse, void* stream,
                                                  const fray::AttnLayout* l) {
    int rc = 0;
    fray::flash_attn_layout<{KIND}, {D}, {BLOCK_N}, {STAGES}>(Q, K, V, O, Lse, stream, *l, rc);
    return rc;
}
extern "C" EXPORT_API int fray_attn_form(const fray::AttnLayout* l, int* mode, int* parts) {
    return fray::flash_attn_form<{KIND}, {D}, {STAGES}>(*l, mode, parts);
}
extern "C" EXPORT_API int fray_attn_pair(const fray::AttnLayout* l) { return fray::flash_attn_pair<{KIND}, {D}, {STAGES}>(*l); }
extern "C" EXPORT_API int fray_attn_four_streams(const fray::AttnLayout* l) {
    return fray::flash_attn_four_streams<{KIND}, {D}, {STAGES}>(*l);
}
#ifdef FRAY_ATTN_TRACE
extern "C" EXPORT_API int fray_attn_trace_read(unsigned int* out, int max_words) {
    return fray::sm100::read_attn_trace(out, max_words);
}
#endif
"""

_STRIDE_NAMES = tuple(f"{t}_stride_{d}" for t in "qkvo" for d in "bhs")


class _AttnLayout(ctypes.Structure):
    """fray::AttnLayout (flash_attn/flash_attn_sm100.cuh): the arguments of a launch that a tensor layout fixes."""
    _fields_ = [(n, ctypes.c_int) for n in ("batch_size", "num_heads", "seq_len", *_STRIDE_NAMES, "num_kv_heads",
                                            "seq_len_kv", "causal")] + [("scale", ctypes.c_float)]


arg_defs = (
    ("Q", torch.half), ("K", torch.half), ("V", torch.half), ("O", torch.half),
    ("batch_size", int), ("num_heads", int), ("seq_len", int),
    *((n, int) for n in _STRIDE_NAMES),
    ("num_kv_heads", int), ("seq_len_kv", int), ("Lse", torch.float),
    ("causal", bool), ("scale", float), ("stream", torch.cuda.Stream),
)

# the same argument table with bf16 tensors (the generated `launch` prototype is identical: raw pointers)
arg_defs_bf16 = tuple((n, torch.bfloat16 if t is torch.half else t) for n, t in arg_defs)

SUPPORTED_HEAD_DIMS = (64, 128)

# Return codes of `launch` (flash_attn/host_sm100.cuh).
_RC_TEXT = {
    1: "bad shape", 2: "null or misaligned pointer", 3: "unsupported stride",
    5: "cuTensorMapEncodeTiled not resolvable", 6: "tensor map rejected by the driver",
    7: "could not raise the dynamic shared memory limit", 8: "kernel launch failed",
}
_RC_TENSOR_MAP = 6


# Kernel kinds (flash_attn/flash_attn_sm100.cuh).
KIND_SIMPLE, KIND_TWO_TILES, KIND_ALTERNATING, KIND_PAIRED, KIND_ONE_TILE = 0, 1, 2, 3, 4
KIND_FEW_QUERIES, KIND_ROW_PAIRS = 6, 7

# The few-query kernel holds all rows (queries x query heads per K/V head) of a K/V head in one 128-row tile.  Up to half
# that many are placed several times, and its warps share out the keys of a step.
FEW_QUERY_ROWS = 128
FEW_QUERY_SHARED_STEP_ROWS = 64
# Below this many keys its cluster's start and merge cost more than the split saves (16 heads x 128 queries, head dim
# 128: 11.2 us against 7.3 at 256 keys, 9.5 against 10.8 at 512, 10.6 against 17.2 at 1024).
FEW_QUERY_MIN_KEYS = 512


def few_query_space() -> Tuple[Dict[str, Any], ...]:
    """The one kernel for calls of few queries (see ``_few_queries``); BLOCK_N and STAGES are those of the two-tile
    kernel its library falls back to."""
    return ({"KIND": KIND_FEW_QUERIES, "BLOCK_N": 128, "STAGES": 4},)


def _few_queries(group: int, seq_len: int, seq_len_kv: int, causal: bool, units: int, sms: int, d: int = 128) -> bool:
    """Whether a call goes to the few-query kernel: all rows of a K/V head's group fit one tile, every row sees every
    key, there are many keys (a decoding step, a short chunk of new queries), and the kernel is no slower there than the
    best of the others.  ``units``: batch x K/V heads.

    It gains in two ways: the query heads of a group share one reading of K and V, and while two and more CTAs per unit fit
    the chip they share its keys.  Figures: its time over the best other kernel's, on 148 SMs, for 5100 combinations of 4 to
    1000 units, groups of 1 to 8, 1 to 128 rows and 512 to 8192 keys at both head dims: 0.11 to 1.03 where it is taken.
    """
    rows = group * seq_len
    if causal or rows > FEW_QUERY_ROWS or seq_len_kv < FEW_QUERY_MIN_KEYS:
        return False
    if rows <= FEW_QUERY_SHARED_STEP_ROWS:
        if group > 1 or 2 * units <= sms:  # 0.11-1.01
            return True
        # Nothing is shared and no unit's keys are split: only a step that is short beside its copies gains.
        if units <= sms:  # 32 rows: 0.62-1.00 at head dim 64, 0.64-0.94 up to 1024 keys, beyond that up to 1.13 (4 rows: 1.02)
            return rows <= (32 if d == 64 or seq_len_kv <= 1024 else 4)
        # One whole-SM CTA per unit pays for its start and end on top, and for an incomplete last round: 16 rows, 150 units:
        # 1.11 at 4096 keys and 0.92 at 8192 (head dim 64: 0.88, 0.66), 300 units: 0.87 at 4096.
        return rows <= 16 and seq_len_kv >= (4096 if d == 64 or units >= 2 * sms else 8192)
    # A warp goes through all 128 keys of a step for its rows, as in the one-tile kernels that have two CTAs per SM.
    if group >= 4 and group * units > sms:  # the others need a round and more per head of a group: 0.16-1.02
        return True
    if 2 * units <= sms:  # keys split; 512 keys: 0.78-0.92 at 16 units, 1.2 at 37 (768: 0.92); 60 units 1.10 at 768, 1.03 at 1024
        return seq_len_kv >= (512 if 8 * units <= sms else 768 if 4 * units <= sms else 1024)
    if group == 1:  # 0.94-2.36
        return False
    return seq_len_kv >= (1536 if group == 2 else 1024)  # 2 x 64 rows: 1.44 at 512 keys, 1.20 at 1024, 1.03 at 1536


def split_keys_space() -> Tuple[Dict[str, Any], ...]:
    """The one kernel for calls whose keys are split (see ``_split_keys``); its launcher chooses the number of parts."""
    return ({"KIND": KIND_ROW_PAIRS, "BLOCK_N": 128, "STAGES": 4},)


def _split_keys(slices: int, seq_len: int, seq_len_kv: int, causal: bool, sms: int, d: int = 128) -> bool:
    """Whether a call goes to the row-pair kernel without a search, because its launcher can share the keys of a work item
    (256 query rows of one of ``slices`` heads) among three and more CTAs and gains more by it than any other kernel.

    Figures: its time over the best other kernel's for 700 combinations of 1 to 72 items and 4 to 94 KV steps of the longest
    item at both head dims, with and without a causal mask, on 148 SMs: 0.33 to 1.00 where it is taken.
    """
    items = slices * -(-seq_len // 256)
    steps = -(-seq_len_kv // 128)
    if causal:
        steps = min(steps, 2 * -(-seq_len // 256))
    if 4 * items > sms:  # 48 items: 1.02-1.30 (head dim 64: 0.92-1.27): half of the one-tile kernels' CTAs are enough for them
        return False
    if 9 * items > 2 * sms:  # no room for four parts: 36 items 0.73-0.92 from 24 steps on, up to 1.17 at 16
        return steps >= 24
    # 30 items at 12 steps: 0.95 (head dim 64: 0.85), 16 steps 0.94; at 8 steps 1.09 (1.00); 12 items at 8 steps 1.00, at 6 1.15
    return steps >= (8 if d == 64 or 12 * items <= sms else 12)


# Sizes and element strides cross the C ABI as 32-bit integers, which ctypes fills without a check.
_ABI_INT_MAX = 2 ** 31 - 1


def _folds(t: torch.Tensor, num_kv_heads: int = 1) -> bool:
    """Whether the heads of ``t`` follow each other as further rows do: the query heads of a K/V head's group are then one
    longer sequence of queries to it (without a causal mask, where a query's place in its head counts), as long as its length,
    rounded up to whole tiles, and the step from group to group still fit the ABI."""
    group = t.shape[1] // num_kv_heads
    return (t.stride(1) == t.shape[2] * t.stride(2) and group * t.shape[2] <= _ABI_INT_MAX - 255
            and (num_kv_heads == 1 or group * t.stride(1) <= _ABI_INT_MAX))


def _launch_args(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, out: torch.Tensor, may_fold: bool) -> tuple:
    """The arguments of ``launch`` that the operands fix: ``(q, k, v, out, batch, heads, queries, 12 strides, K/V heads, keys)``.

    With ``may_fold`` there is one slice per K/V head instead of per query head where the layout allows it: fewer tiles that end
    early, and K and V are fetched once for rows that share a tile.  2 x 16/4 x 513 on 6000 x 128: 12 times 256 rows per K/V
    head become 9.
    """
    batch_size, num_heads, seq_len, d = q.shape
    num_kv_heads, seq_len_kv = k.shape[1], k.shape[2]
    group = num_heads // num_kv_heads
    if may_fold and group > 1 and seq_len > 1 and _folds(q, num_kv_heads) and _folds(out, num_kv_heads):
        num_heads, seq_len = num_kv_heads, group * seq_len
        q, out = (t.as_strided((batch_size, num_heads, seq_len, d), (t.stride(0), group * t.stride(1), t.stride(2), 1))
                  for t in (q, out))
    strides = tuple(int(t.stride(i)) if t.shape[i] > 1 else 8 for t in (q, k, v, out) for i in range(3))
    if max(*strides, seq_len, seq_len_kv) > _ABI_INT_MAX:
        raise RuntimeError(f"flash_attn_cute: sizes and strides are limited to {_ABI_INT_MAX} elements (strides {strides}, "
                           f"{seq_len} queries, {seq_len_kv} keys)")
    return (q, k, v, out, int(batch_size), int(num_heads), int(seq_len), *strides, int(num_kv_heads), int(seq_len_kv))


def tuning_space(d: int) -> Tuple[Dict[str, Any], ...]:
    """Candidate kernels for head dim ``d``: kernel kind (which fixes BLOCK_M: one 128-row tile, two tiles per
    CTA, or 256 rows on a CTA pair driven by ``tcgen05.mma.cta_group::2``) x KV tile length x pipeline depth.

    KIND: 0 single-role, 1 warp-specialised with two query tiles per CTA, 2 warp-specialised with one tile per CTA
    and two softmax groups on alternate KV steps, 3 the same on a pair of CTAs (2-CTA MMA; D = 128 only), 4
    warp-specialised with one tile per CTA and two CTAs per SM (a CTA's start and end run beside its neighbour's
    steady state; the kind for short sequences), 7 two query tiles per CTA with two softmax threads per row, as a
    persistent grid of one CTA per SM that walks through the work items.
    BLOCK_N: KV tile (64 or 128 for kind 0, 128 otherwise).  STAGES: K/V ring slots of kinds 1, 4 and 7, K ring
    slots of kinds 2 and 3 (their V tiles use three slots).
    """
    space = [
        {"KIND": KIND_TWO_TILES, "BLOCK_N": 128, "STAGES": 4},
        {"KIND": KIND_TWO_TILES, "BLOCK_N": 128, "STAGES": 3},
        {"KIND": KIND_ROW_PAIRS, "BLOCK_N": 128, "STAGES": 4},
        {"KIND": KIND_ONE_TILE, "BLOCK_N": 128, "STAGES": 2},
        {"KIND": KIND_ALTERNATING, "BLOCK_N": 128, "STAGES": 2 if d == 128 else 4},
        {"KIND": KIND_SIMPLE, "BLOCK_N": 128, "STAGES": 1},
        {"KIND": KIND_SIMPLE, "BLOCK_N": 64, "STAGES": 1},
    ]
    if d == 128:
        space[4:4] = [{"KIND": KIND_PAIRED, "BLOCK_N": 128, "STAGES": 4}, {"KIND": KIND_PAIRED, "BLOCK_N": 128, "STAGES": 6}]
    else:
        space.insert(1, {"KIND": KIND_TWO_TILES, "BLOCK_N": 128, "STAGES": 6})
    forced = _forced_point()
    if forced is not None:
        if forced["KIND"] == KIND_PAIRED and d != 128:
            raise ValueError("FRAY_ATTN_FORCE: the paired kernel (KIND=3) is built for head dim 128 only")
        return (forced,)
    return tuple(space)


def _forced_point() -> Optional[Dict[str, int]]:
    # e.g. "KIND=0,BLOCK_N=64,STAGES=1"; for bring-up: looked at when a layout is first launched, not on warm calls
    forced = os.getenv("FRAY_ATTN_FORCE")
    if not forced:
        return None
    point = {"BLOCK_N": 128, "STAGES": 4}
    point.update({kv.split("=")[0].strip(): int(kv.split("=")[1]) for kv in forced.split(",")})
    return point


def _workload_class(seq_len: int, seq_len_kv: int, units: int, sms: int) -> str:
    """Coarse workload class the tuner memoises on, from what the kinds differ in: how many steps a work item has (bucket of
    the number of keys), whether items of two query tiles fill the chip, and whether there is a second tile at all.  Items for up
    to half of the SMs are apart: an SM for each of their tiles (one-tile kernels), or two and more CTAs for each (row-pair kernel
    with its keys split).  As one class, the call that came first decided: 144 items of 333 causal rows, head dim 64, 8.2 us, or
    16.2 behind 4 items; 48 heads of 256 rows on 2048 keys, head dim 128, 20.1, or 25.1 behind 140."""
    k_bucket = 1 << max(7, (max(seq_len_kv, 1) - 1).bit_length())
    items = units * -(-seq_len // 256)
    fill = "big" if items >= sms else "half" if 2 * items <= sms else "small"
    return f"K{min(k_bucket, 16384)}_{fill}{'_one_tile' if seq_len <= 128 else ''}"


def _usable_strides(t: torch.Tensor) -> bool:
    if t.stride(-1) != 1 and t.shape[-1] > 1:
        return False
    if t.data_ptr() % 16 != 0:
        return False
    return all(t.shape[i] == 1 or (t.stride(i) > 0 and t.stride(i) % 8 == 0 and t.stride(i) < 2 ** 31)
               for i in range(3))


def _space_points(head_dims, forced: bool):
    """(d, point, bf16) for every library of the tuning space (forced: honour FRAY_ATTN_FORCE)."""
    old = None if forced else os.environ.pop("FRAY_ATTN_FORCE", None)
    try:
        few = () if forced else few_query_space()
        return [(d, point, bf16) for d in head_dims for bf16 in (False, True) for point in (*tuning_space(d), *few)]
    finally:
        if old is not None:
            os.environ["FRAY_ATTN_FORCE"] = old


def prebuild(head_dims=SUPPORTED_HEAD_DIMS, prune: bool = False):
    """Compile every point of the tuning space ahead of time (fp16 and bf16 operands) and return the kernel
    directories.

    With ``prune`` the cache directory is also cleared of attention kernels that belong neither to the
    space nor to a point forced through FRAY_ATTN_FORCE (left over from older headers).
    """
    import shutil
    from ..jit import build, cpp_format, generate
    from ..jit.compiler import get_cache_dir

    def build_point(d, point, bf16):
        keys = {"D": d, **point}
        code = generate(includes_bf16 if bf16 else includes, arg_defs_bf16 if bf16 else arg_defs,
                        cpp_format(template, keys), cpp_format(epilogue, keys))
        return build("flash_attn_cute", arg_defs_bf16 if bf16 else arg_defs, code).path

    paths = [build_point(*p) for p in _space_points(head_dims, forced=False)]
    if os.getenv("FRAY_ATTN_FORCE"):
        paths += [build_point(*p) for p in _space_points(head_dims, forced=True)
                  if not (p[1]["KIND"] == KIND_PAIRED and p[0] != 128)]
    if prune:
        for entry in os.listdir(get_cache_dir()):
            full = os.path.join(get_cache_dir(), entry)
            if entry.startswith("kernel.flash_attn_cute.") and full not in paths:
                shutil.rmtree(full, ignore_errors=True)
    return paths


# Every kernel library this process has launched: the device status words are per library.
_used_runtimes: Dict[str, Any] = {}
# Warm-call fast path: (shapes, strides, dtype, device, causal, scale, lse layout) -> (launch symbol, layout,
# the layout's address, device index).  Everything the slow path validates is a function of that key, so a hit only
# has to marshal the pointers and the stream; the other arguments of `launch` wait in the structure behind the address
# (a call of the smallest problem takes 6.0 us of host time, 8.7 with `launch`'s 27 arguments).  Bounded: the oldest
# entries go first.
_fast_path: "OrderedDict[Any, Any]" = OrderedDict()
_FAST_PATH_ENTRIES = 64


def flash_attn_status(clear: bool = True) -> Tuple[int, int, int, int]:
    """Synchronise and return the device status words: ``(0, 0, 0, 0)`` means healthy.

    Every kernel library keeps its own status; this reads all libraries the process has launched,
    returns the first raised one and (with ``clear``) resets them all.  A non-zero first word is the
    code of the first wait that ran out inside a kernel; the other words are the block indices and an
    iteration number.  The status is sticky: until cleared, later launches of that library return
    immediately WITHOUT computing (``launch`` still reports 0), so a caller that cannot rule out a
    preempted or faulty device should check it before trusting an output.
    """
    first = (0, 0, 0, 0)
    for runtime in list(_used_runtimes.values()):
        fn = runtime.symbol("fray_attn_status")
        assert fn is not None, "kernel library does not export fray_attn_status"
        out = (ctypes.c_int * 4)()
        err = fn(out, ctypes.c_int(1 if clear else 0))
        if err != 0:
            raise RuntimeError(f"reading the attention status failed with CUDA error {err}")
        if out[0] != 0 and first[0] == 0:
            first = tuple(out)
    return first


_no_lse: Dict[Any, torch.Tensor] = {}


def flash_attn_cute(Q: torch.Tensor, K: torch.Tensor, V: torch.Tensor, Output: torch.Tensor, *,
                    causal: bool = False, scale: Optional[float] = None, lse: Optional[torch.Tensor] = None) -> None:
    """See the module docstring.  Extensions beyond the reference's call:

    ``K`` and ``V`` may be ``[B, H_kv, S_k, D]`` with ``H_kv`` a divisor of ``H``: query head ``h`` then attends
    to K/V head ``h // (H // H_kv)`` (grouped-query / multi-query attention), and ``S_k`` may differ from the
    number of queries (cross attention, or new queries against a longer cache); with ``causal`` query ``i``
    sees keys ``0..i``, the top-left alignment of torch's ``is_causal``.
    All four tensors may be bf16 instead of fp16 (P is then rounded to bf16 too; accumulation stays fp32).
    ``lse``: optional contiguous fp32 CUDA tensor ``[B, H, S]`` that receives ``log(sum_j exp(scale * q_i.k_j))``
    over the keys row ``i`` may see, the quantity needed to merge partial attention results.

    The launch goes to the current stream of the tensors' device, which must be the current device (as in
    the reference, which takes ``torch.cuda.current_stream()``, fray/jit_kernels/flashattn_cute.py:27).
    A raised device status (see ``flash_attn_status``) turns later launches into no-ops until it is cleared.
    """
    fast_key = (Q.shape, Q.stride(), K.shape, K.stride(), V.shape, V.stride(), Output.shape, Output.stride(),
                Q.dtype, K.dtype, V.dtype, Output.dtype, Q.device, K.device, V.device, Output.device, causal, scale,
                None if lse is None else (lse.shape, lse.stride(), lse.dtype, lse.device))
    hit = _fast_path.get(fast_key)
    if hit is not None:
        launch, _, layout_address, dev_index = hit
        if dev_index == torch.cuda.current_device():
            if launch(Q.data_ptr(), K.data_ptr(), V.data_ptr(), Output.data_ptr(), None if lse is None else lse.data_ptr(),
                      torch._C._cuda_getCurrentRawStream(dev_index), layout_address) == 0:
                return
        # e.g. a misaligned data pointer this time, or another current device: let the checked path deal with it
    assert Q.dim() == 4 and K.dim() == 4, "expected [B, H, S, D] tensors"
    batch_size, num_heads, seq_len, d = Q.shape
    num_kv_heads = K.shape[1]
    assert Q.shape == Output.shape and K.shape == V.shape
    seq_len_kv = K.shape[2]
    assert K.shape == (batch_size, num_kv_heads, seq_len_kv, d), "K and V must match Q in batch and head dim"
    assert num_kv_heads > 0 and num_heads % num_kv_heads == 0, "the number of K/V heads must divide the number of Q heads"
    assert Q.dtype == K.dtype == V.dtype == Output.dtype and Q.dtype in (torch.half, torch.bfloat16)
    bf16 = Q.dtype is torch.bfloat16
    assert Q.device.type == "cuda", "flash_attn_cute has no CPU path"
    assert Q.device == K.device == V.device == Output.device
    assert Q.device.index == torch.cuda.current_device(), \
        "the tensors must live on the current CUDA device (wrap the call in torch.cuda.device(...))"
    if lse is not None:
        assert lse.dtype == torch.float32 and lse.device == Q.device and lse.is_contiguous()
        assert lse.shape == (batch_size, num_heads, seq_len), "lse must be [B, H, S]"
    if d not in SUPPORTED_HEAD_DIMS:
        raise ValueError(f"head dim {d} not supported (supported: {SUPPORTED_HEAD_DIMS})")
    if batch_size == 0 or num_heads == 0 or seq_len == 0:
        return
    assert seq_len_kv > 0, "attention over zero keys is undefined"
    assert batch_size * num_heads <= 65535, "batch * heads is a grid dimension: at most 65535"

    q, k, v = (t if _usable_strides(t) else t.contiguous() for t in (Q, K, V))
    out = Output if _usable_strides(Output) else torch.empty_like(Output, memory_format=torch.contiguous_format)

    sms = torch.cuda.get_device_properties(Q.device).multi_processor_count
    forced = os.getenv("FRAY_ATTN_FORCE", "")
    few = not forced and _few_queries(num_heads // num_kv_heads, seq_len, seq_len_kv, bool(causal), batch_size * num_kv_heads,
                                      sms, d)
    stream = torch.cuda.current_stream(Q.device)
    sm_scale = float(scale) if scale is not None else 1.0 / math.sqrt(d)
    assert sm_scale > 0 and math.isfinite(sm_scale), "the softmax scale must be positive and finite"

    lse_arg = lse
    if lse_arg is None:  # a null pointer for the library: an empty tensor's data pointer is 0
        lse_arg = _no_lse.get(Q.device)
        if lse_arg is None:
            lse_arg = _no_lse[Q.device] = torch.empty(0, dtype=torch.float32, device=Q.device)

    def pack(q, k, v, out):
        return (*_launch_args(q, k, v, out, may_fold=not causal and not few), lse_arg, bool(causal), sm_scale, stream)

    args = pack(q, k, v, out)
    num_heads, seq_len = args[5:7]
    split = not forced and not few and _split_keys(batch_size * num_heads, seq_len, seq_len_kv, bool(causal), sms, d)
    runtime = jit_tuner.compile_and_tune(
        name="flash_attn_cute",
        keys={"D": d, "CAUSAL": int(bool(causal)),
              "CLASS": "few" if few else "split" if split else _workload_class(seq_len, seq_len_kv, batch_size * num_heads, sms),
              "FORCED": forced, **({"BF16": 1} if bf16 else {})},
        space=few_query_space() if few else split_keys_space() if split else tuning_space(d),
        includes=includes_bf16 if bf16 else includes,
        arg_defs=arg_defs_bf16 if bf16 else arg_defs,
        template=template,
        args=args,
        epilogue=epilogue,
    )
    _used_runtimes[runtime.path] = runtime

    rc = runtime(*args)
    if rc == _RC_TENSOR_MAP and not all(t.is_contiguous() for t in (q, k, v, out)):
        # The layout cannot be described to the copy engine: fall back to packed copies.
        q, k, v = (t.contiguous() for t in (q, k, v))
        if not out.is_contiguous():
            out = torch.empty_like(Output, memory_format=torch.contiguous_format)
        rc = runtime(*pack(q, k, v, out))
    if rc != 0:
        raise RuntimeError(f"flash_attn_cute launch failed with code {rc} ({_RC_TEXT.get(rc, 'unknown')})")
    if q is Q and k is K and v is V and out is Output and not forced:
        # no copies were needed: remember how to launch this layout directly
        launch = runtime.symbol("fray_attn_launch_layout")
        launch.argtypes = [ctypes.c_void_p] * 7
        layout = _AttnLayout(*args[4:4 + 3 + 12 + 2], int(bool(causal)), sm_scale)
        _fast_path[fast_key] = (launch, layout, ctypes.addressof(layout), Q.device.index)
        while len(_fast_path) > _FAST_PATH_ENTRIES:
            _fast_path.popitem(last=False)
    if out is not Output:
        Output.copy_(out)


# Device staging buffers of the host-buffer call, one shape at a time, shared by every stream and thread of the process: the
# events say until when a buffer set is in use, the lock covers the queueing of a whole call.
_host_staging: Dict[Any, Any] = {}
_host_staging_lock = threading.Lock()


# From here on the staging buffers (two slices) are kept at a quarter of the operands, as five slices' would be two thirds (2.5 GB).
# Five slices against nine and eight equal ones, us: 0.5 GB of operands 8030, 8240, 8340; 1 GB 15700, 15930, 16200; 2 GB 31060,
# 31330, 31930; 3.9 GB 59860, 60200, 61600.  Where the device has no room for them, eight equal slices.
_LARGE_HOST_CALL_BYTES = 4 << 30


def _slice_bounds(units: int, chunks: Optional[int], nbytes: int = 0) -> list:
    """Where the slices of a host-buffer call begin and end: ``chunks`` equal ones, or by default five that get smaller (nine for
    large operands, ``nbytes``).  A copy costs the link 3.7 us beside its bytes, so few slices; what follows the last copy-in is
    one slice's kernel and copy-out, so the last one is small.  4 x 16 x 1024 x 128, with eight equal slices before: 1269 -> 1180
    us, 2 x 16 x 512 594 -> 396, 4 x 32 x 4096 8420 -> 8070 (the nine: 8310).
    """
    if chunks:
        n = max(1, min(units, chunks))
        return [(units * c) // n for c in range(n + 1)]
    parts = (6, 12, 16, 18, 19) if nbytes < _LARGE_HOST_CALL_BYTES else (2, 4, 6, 8, 10, 12, 14, 15, 16)
    return sorted({0, *((2 * units * c + parts[-1]) // (2 * parts[-1]) for c in parts)})


def _drop_host_staging() -> None:
    """Gives the staging buffers back once everything queued on them, on whatever stream, has run."""
    for st in _host_staging.values():
        for event in (*st["computed"], *st["drained"]):
            if event is not None:
                st["s_in"].wait_event(event)
        for buf in (*st["bufs"][0], *st["bufs"][1]):
            buf.record_stream(st["s_in"])
    _host_staging.clear()


def flash_attn_cute_host(Q: torch.Tensor, K: torch.Tensor, V: torch.Tensor, Output: torch.Tensor, *,
                         causal: bool = False, scale: Optional[float] = None, lse: Optional[torch.Tensor] = None,
                         chunks: Optional[int] = None) -> None:
    """``flash_attn_cute`` for operands in pinned HOST memory: result written to the pinned ``Output``.

    No counterpart in the reference (its op asserts CUDA tensors, fray/jit_kernels/flashattn_cute.py:17-20);
    this is the call a host-side caller of the C ABI makes.  Same operands as the device op: fp16 or bf16,
    ``K``/``V`` with ``H_kv | H`` heads and their own length, optional pinned fp32 ``lse`` ``[B, H, S]``.  The
    B * H_kv independent (batch, K/V head) units (each with its group of query heads) are cut into ``chunks``
    slices (by default five to nine of falling size) that move through two sets of device staging buffers on three streams of the current
    device: while slice c is computed, slice c+1 is copied in and slice c-1 is copied out, so the two
    directions of the host link run at the same time and the kernel hides behind them.  Work is ordered
    after the current stream's earlier work, and the current stream waits for the last copy-out: as with the
    device op, the result is valid for work queued on the current stream afterwards (or after a
    synchronize), not at return.  Calls may come from several streams and threads: they share the staging
    buffers, one after the other on the device, and queue one at a time; a captured call has its own.
    """
    tensors = (Q, K, V, Output) + ((lse,) if lse is not None else ())
    assert all(t.device.type == "cpu" and t.is_pinned() for t in tensors), "operands must be pinned host tensors"
    assert Q.dim() == 4 and K.dim() == 4 and Q.shape == Output.shape and K.shape == V.shape
    assert Q.dtype == K.dtype == V.dtype == Output.dtype and Q.dtype in (torch.half, torch.bfloat16)
    assert all(t.is_contiguous() for t in tensors), "host operands must be contiguous"
    B, H, Sq, D = Q.shape
    Hkv, Sk = K.shape[1], K.shape[2]
    assert K.shape == (B, Hkv, Sk, D) and Hkv > 0 and H % Hkv == 0
    if lse is not None:
        assert lse.dtype == torch.float32 and lse.shape == (B, H, Sq)
    group = H // Hkv
    dev = torch.device("cuda", torch.cuda.current_device())
    units = B * Hkv                                    # one unit = one K/V head with its `group` query heads
    Qu, Ou = (t.view(units, group, Sq, D) for t in (Q, Output))
    Ku, Vu = (t.view(units, 1, Sk, D) for t in (K, V))
    Lu = lse.view(units, group, Sq) if lse is not None else None
    bounds = _slice_bounds(units, chunks, sum(t.numel() * t.element_size() for t in tensors))
    rows = max(b1 - b0 for b0, b1 in zip(bounds, bounds[1:]))
    equal = _slice_bounds(units, chunks or 8)
    key = (dev, rows, group, Sq, Sk, D, Q.dtype, lse is not None)
    with _host_staging_lock:
        # A graph being captured gets buffers of its own (from its pool): it runs whenever it is replayed, and events of calls
        # outside it cannot be waited for in it.
        capturing = torch.cuda.is_current_stream_capturing()
        st = None if capturing else _host_staging.get(key)
        if st is None:
            def make_set(rows):
                bufs = [torch.empty((rows, group, Sq, D), dtype=Q.dtype, device=dev),
                        torch.empty((rows, 1, Sk, D), dtype=Q.dtype, device=dev),
                        torch.empty((rows, 1, Sk, D), dtype=Q.dtype, device=dev),
                        torch.empty((rows, group, Sq, D), dtype=Q.dtype, device=dev)]
                if lse is not None:
                    bufs.append(torch.empty((rows, group, Sq), dtype=torch.float32, device=dev))
                return bufs
            if not capturing:
                _drop_host_staging()  # one shape at a time: the buffers are as large as the operands' slices
            fewer = -(-units // (len(equal) - 1))
            for n in (rows, fewer):  # a device that is nearly full may have room for slices that are equal, and smaller
                try:
                    bufs = [make_set(n) for _ in range(2)]
                    break
                except torch.OutOfMemoryError:
                    if n <= fewer:
                        raise
            st = {"bufs": bufs, "s_in": torch.cuda.Stream(device=dev), "s_out": torch.cuda.Stream(device=dev),
                  "computed": [None, None],   # per buffer set: kernel of the slice that last used it has finished
                  "drained": [None, None]}    # ... and its result has left the device
            if not capturing:
                _host_staging[key] = st
        if st["bufs"][0][0].shape[0] < rows:
            bounds = equal
        s_in, s_out = st["s_in"], st["s_out"]
        # Kept from call to call: a call on another stream finds the sets still in use by the one before it.
        computed, drained = st["computed"], st["drained"]
        cur = torch.cuda.current_stream(dev)
        start = torch.cuda.Event()
        start.record(cur)
        s_in.wait_event(start)
        s_out.wait_event(start)
        for c, (b0, b1) in enumerate(zip(bounds, bounds[1:])):
            bufs = [t[: b1 - b0] for t in st["bufs"][c & 1]]
            dq, dk, dv, do = bufs[:4]
            if computed[c & 1] is not None:
                s_in.wait_event(computed[c & 1])      # inputs of slice c-2 are no longer read
            with torch.cuda.stream(s_in):
                dq.copy_(Qu[b0:b1], non_blocking=True)
                dk.copy_(Ku[b0:b1], non_blocking=True)
                dv.copy_(Vu[b0:b1], non_blocking=True)
                arrived = torch.cuda.Event()
                arrived.record(s_in)
            cur.wait_event(arrived)
            if drained[c & 1] is not None:
                cur.wait_event(drained[c & 1])        # output buffers of slice c-2 have been copied out
            # a slice is itself an attention problem with batch = units in the slice, H = group, H_kv = 1
            flash_attn_cute(dq, dk, dv, do, causal=causal, scale=scale, lse=bufs[4] if lse is not None else None)
            computed[c & 1] = torch.cuda.Event()
            computed[c & 1].record(cur)
            s_out.wait_event(computed[c & 1])
            with torch.cuda.stream(s_out):
                Ou[b0:b1].copy_(do, non_blocking=True)
                if lse is not None:
                    Lu[b0:b1].copy_(bufs[4], non_blocking=True)
                drained[c & 1] = torch.cuda.Event()
                drained[c & 1].record(s_out)
        for ev in drained:
            if ev is not None:
                cur.wait_event(ev)

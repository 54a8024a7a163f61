"""Host-side glue shared by the op modules: pointers, streams, cached scratch, split policy."""
from __future__ import annotations

import ctypes
import os
from typing import Dict, Optional, Tuple

import torch

from . import _lib

CTAS_PER_PART = 2        # two CTAs (one per half of d_v) share a partition
FIXED_OVERHEAD = 5       # scheduler cost of starting a request, in 64-token blocks
BLOCK_N = 64

_scratch: Dict[Tuple, Dict[str, torch.Tensor]] = {}
_num_sms: Dict[int, int] = {}


def ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def stream_ptr(device: torch.device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def num_sms(device: torch.device) -> int:
    idx = device.index if device.index is not None else torch.cuda.current_device()
    if idx not in _num_sms:
        _num_sms[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _num_sms[idx]


def require_cuda(*tensors: Optional[torch.Tensor]) -> None:
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise ValueError("sparse_mla_sm120_b200 runs on CUDA tensors only (there is no CPU path)")


def kv_layout(kv_cache: torch.Tensor) -> int:
    """LAYOUT_V32 for 656-byte rows, LAYOUT_MODEL1 for 584-byte rows."""
    if kv_cache.dtype not in (torch.uint8, torch.int8, torch.float8_e4m3fn):
        raise ValueError(f"kv_cache must be a byte tensor, got {kv_cache.dtype}")
    row = kv_cache.shape[-1]
    if row == 656:
        return _lib.LAYOUT_V32
    if row == 584:
        return _lib.LAYOUT_MODEL1
    raise ValueError(f"kv_cache rows must be 656 bytes (V32) or 584 bytes (MODEL1), got {row}")


def kv_geometry(kv_cache: torch.Tensor) -> Tuple[int, int]:
    """(page_block_size, bytes between pages) of a packed cache tensor.

    V32 (656-byte rows): accepts [num_blocks, block, 1, 656], the legacy flat [pool, 1, 656] and
    [pool, 656].  MODEL1 (584 bytes per token, scales in a footer of the page): [num_blocks, block, 1, 584]
    only, since the position of the footer depends on the page size.  A page stride larger than
    block * row (a padded allocation) is honoured; flash_mla_sm120/ops.py:23-45 computes the same quantity."""
    layout = kv_layout(kv_cache)
    row = kv_cache.shape[-1]
    if kv_cache.stride(-1) != 1:
        raise ValueError("kv_cache rows must be contiguous")
    if kv_cache.dim() == 4:
        block = kv_cache.shape[1]
        if kv_cache.shape[2] != 1 or kv_cache.stride(1) != row:
            raise ValueError(f"kv_cache must be [num_blocks, block, 1, {row}] with {row}-byte rows")
        return block, kv_cache.stride(0)
    if layout != _lib.LAYOUT_V32:
        raise ValueError("a MODEL1 cache must be [num_blocks, block, 1, 584]")
    if kv_cache.dim() == 3:
        if kv_cache.shape[1] != 1 or kv_cache.stride(0) != 656:
            raise ValueError("kv_cache must be [pool, 1, 656] with 656-byte rows")
        pool = max(kv_cache.shape[0], 1)
        return pool, pool * 656
    if kv_cache.dim() == 2:
        if kv_cache.stride(0) != 656:
            raise ValueError("kv_cache must be [pool, 656] with 656-byte rows")
        pool = max(kv_cache.shape[0], 1)
        return pool, pool * 656
    raise ValueError(f"unsupported kv_cache rank {kv_cache.dim()}")


# What IMPL_AUTO means for a MODEL1 cache.  The FP8-class tensor-core kernel rounds V's RoPE columns to e4m3 (the reference
# keeps them in bf16), which costs up to about 2e-3 on rows with few entries and fails some of the reference's own V4
# tests by a small margin; the default is therefore exact numerics (IMPL_SCALAR: attn_exact_kernel, bf16 operands and fp32
# sums).  A deployment that accepts FP8-class error in those 64 columns sets SMLA_MODEL1_IMPL=tc in the environment (or
# assigns _lib.IMPL_TC here).
MODEL1_DEFAULT_IMPL = _lib.IMPL_TC if os.environ.get("SMLA_MODEL1_IMPL", "").lower() in ("tc", "2") else _lib.IMPL_SCALAR


def resolve_impl(impl: int, layout: int) -> int:
    """IMPL_AUTO for a MODEL1 cache -> MODEL1_DEFAULT_IMPL; everything else unchanged."""
    if impl == _lib.IMPL_AUTO and layout == _lib.LAYOUT_MODEL1:
        return MODEL1_DEFAULT_IMPL
    return impl


def tc_aligned(kv_cache: torch.Tensor, extra_kv: Optional[torch.Tensor] = None) -> bool:
    """What the tensor-core kernel's bulk copies need of the caches of an `_ext` call: base addresses and page
    strides that are multiples of 16 bytes (the library checks the same and falls back to the fp32 kernel)."""
    for t in (kv_cache, extra_kv):
        if t is not None and (t.data_ptr() % 16 != 0 or kv_geometry(t)[1] % 16 != 0):
            return False
    return True


def one_array(kv_cache: torch.Tensor) -> bool:
    """Whether the 656-byte rows of a cache are one linear, 16-byte aligned array (pages without padding between them):
    what attn_tile_kernel needs to name rows by their index (the library checks the same)."""
    block, stride = kv_geometry(kv_cache)
    return stride == block * 656 and kv_cache.data_ptr() % 16 == 0


def pick_num_sm_parts_fp32(num_tokens: int, num_heads: int, sms: int) -> int:
    """Partitions for the fp32 kernel, which runs ceil(heads / 8) CTAs per partition: requests stay
    whole when they already give two CTAs per SM, otherwise the work is cut so that they do."""
    tiles = -(-num_heads // 8)
    if num_tokens * tiles >= 2 * sms:
        return num_tokens
    return max(2 * sms // tiles, 1)


# attn_exact_kernel (exact numerics over MODEL1, aligned caches): microseconds of a partition's fixed part (q, epilogue),
# of a 128-token tile, and of what a split adds (scheduler and combine launches, partial records).  Estimates, not fitted, from before
# the launches ran under one another (a split adds less since): a tile takes about 11000 cycles (5.6 us) in the kernel; what the
# rule needs is their proportion.
_EXACT_US_FIXED, _EXACT_US_TILE, _EXACT_US_SPLIT = 6.0, 4.0, 9.0


def pick_num_sm_parts_exact(num_tokens: int, num_heads: int, sms: int, blocks_per_token: int) -> int:
    """Partitions for attn_exact_kernel, which runs one CTA per partition and 64 heads: whole requests when their tiles in
    full waves take no longer than cutting the work evenly over the machine and merging the pieces."""
    most = max(sms // -(-num_heads // 64), 1)
    tiles = max(-(-blocks_per_token // 2), 1)
    whole = -(-num_tokens // most) * (_EXACT_US_FIXED + tiles * _EXACT_US_TILE)
    parts = min(most, num_tokens * tiles)
    cut = _EXACT_US_FIXED + -(-num_tokens * tiles // parts) * _EXACT_US_TILE + _EXACT_US_SPLIT
    return num_tokens if whole <= cut else parts


BLOCKS_PER_PARTITION = 4  # a partition should be worth at least two 128-token tiles: below that the partials cost more than the split gains


def pick_num_sm_parts(num_tokens: int, sms: int, blocks_per_token: Optional[int] = None) -> int:
    """Partitions for the split-KV scheduler when nothing is known about the requests' lengths (or they differ).

    A partition is served by two CTAs, so at most sms // 2 partitions run at once.  When whole requests already
    fill half of the machine in full waves they are left unsplit (one partition per token: no partial outputs, no
    combine traffic; 40 requests of top-k 2048: 48 us unsplit, 64 us cut into 74 partitions that mostly straddle two
    requests).  Otherwise the work is cut into up to sms // 2 partitions, but not into partitions of fewer than
    BLOCKS_PER_PARTITION 64-token blocks (every extra partition is a partial output that the combine has to read
    back: one request of top-k 2048 is fastest in 8 partitions, 27 us, against 38 us in 74)."""
    max_parts = max(sms // CTAS_PER_PART, 1)
    ctas = num_tokens * CTAS_PER_PART
    waves = -(-ctas // sms)
    if ctas / (waves * sms) >= 0.5:
        return num_tokens
    if blocks_per_token is None:
        return max_parts
    want = -(-(num_tokens * max(blocks_per_token, 1)) // BLOCKS_PER_PARTITION)
    return max(num_tokens, min(max_parts, want))


# Cost model of a decode step at 128 heads on a B200, microseconds (fitted to measurements of 4 to 48 requests of
# top-k 2048 in 1, 2, 4 and 8 equal partitions each; it reproduces them to about 1 us): a partition pays a fixed part
# (set-up, Q quantisation, epilogue) and its 128-token tiles; a split step pays for every partial record, which is
# written and read back once, and at least the latency of the combine launch.
_US_FIXED, _US_TILE, _US_RECORD, _US_SPLIT_MIN = 11.3, 2.3, 0.15, 8.0


def pick_split(num_tokens: int, sms: int, blocks_per_token: Optional[int] = None, uniform: bool = False) -> Tuple[int, int]:
    """(partitions, fixed overhead) to give the scheduler.

    When every request has the same number of blocks (no ``topk_length``), the requests can be cut into k equal
    partitions each, k a divisor of the block count, by asking the scheduler for k * tokens partitions with a fixed
    overhead of 0: no partition then straddles two requests, i.e. none pays the fixed part of a partition twice.
    k is chosen by the cost model above (k = 1: nothing is split, the attention kernel runs alone).  Otherwise
    (lengths differ or are unknown) the choice is pick_num_sm_parts with the reference's fixed overhead."""
    if not uniform or blocks_per_token is None:
        return pick_num_sm_parts(num_tokens, sms, blocks_per_token), FIXED_OVERHEAD
    max_parts = max(sms // CTAS_PER_PART, 1)
    n = max(blocks_per_token, 1)
    waves = -(-num_tokens // max_parts)
    best = (waves * (_US_FIXED + -(-n // 2) * _US_TILE), num_tokens, FIXED_OVERHEAD)
    cuts = 0
    for k in range(2, n + 1):
        if n % k or k * num_tokens > max_parts or n // k < BLOCKS_PER_PARTITION:
            continue
        cuts += 1
        t = _US_FIXED + -(-(n // k) // 2) * _US_TILE + max(_US_SPLIT_MIN, _US_RECORD * k * num_tokens)
        if t < best[0]:
            best = (t, k * num_tokens, 0)
    if cuts == 0 and n >= 2 * BLOCKS_PER_PARTITION:
        # no equal cut exists although the requests are long enough to be worth cutting (a block count without a
        # suitable divisor, or too many requests for two partitions each): the general rule
        return pick_num_sm_parts(num_tokens, sms, blocks_per_token), FIXED_OVERHEAD
    return best[1], best[2]


# attn_tile_kernel (up to 64 heads over one linear array of rows): microseconds of a partition's fixed part, of a 128-token
# tile, and of what a split adds: a part that grows with the pieces of a request, and the records that are written and
# read back.  Fitted, before the kernel's last 15 %, to 1 to 64 requests of top-k 512, 1024 and 2048 in up to 16 equal partitions each, 16 and 64 heads (48
# requests of top-k 2048 at 16 heads: 40 us whole, 28.6 us in two partitions each; one: 38.5, 25.3, 18.5, 17.9 and 19.9 us in
# 1, 2, 4, 8 and 16); the cut that it names is the fastest measured one or within a microsecond of it.
def _tile_us(num_tokens: int, num_heads: int, blocks: int, k: int) -> float:
    t = 7.3 + 0.022 * num_heads + -(-(blocks // k) // 2) * (1.78 + 0.0077 * num_heads)
    return t if k == 1 else t + 1.9 + 0.45 * k + 0.03 * k * num_tokens


def pick_split_tile(num_tokens: int, num_heads: int, sms: int, blocks_per_token: int, uniform: bool) -> Tuple[int, int]:
    """(partitions, fixed overhead) for attn_tile_kernel, which runs one CTA per partition.  Requests of equal length are
    cut into as many equal partitions as pay off while all of them run at once.  Where no equal cut exists the rule is the
    general one: a partition that straddles two requests pays its fixed part twice, so that more of them, one per SM,
    are slower than half as many (ragged requests of top-k 2048, 16 heads: 16 of them 35 us in 148 partitions, 27 us in 74; 24: 35 and
    30).  That rule leaves 37 and more requests whole: 64 of them take 42.5 us so, 44.3 in 111 partitions and 46.7 in 148; 48: 41.9,
    41.2, 42.3; only near 37 is a cut better (39.7 whole, 35.2 in 74)."""
    n = max(blocks_per_token, 1)
    if not uniform:
        return pick_num_sm_parts(num_tokens, sms, blocks_per_token), FIXED_OVERHEAD
    cuts = [k for k in range(2, n // 2 + 1) if n % k == 0 and k * num_tokens <= sms]
    if not cuts and n >= 2 * BLOCKS_PER_PARTITION:
        return pick_num_sm_parts(num_tokens, sms, blocks_per_token), FIXED_OVERHEAD
    k = min([1] + cuts, key=lambda c: _tile_us(num_tokens, num_heads, n, c))
    return (num_tokens, FIXED_OVERHEAD) if k == 1 else (k * num_tokens, 0)


# attn_duo_kernel (65 to 128 heads over one linear array of rows): microseconds of a partition's fixed part, of a 128-token tile (more
# when many pairs of SMs share the memory), and of what a split adds per piece of a request and per record.  Fitted to 1 to 64
# requests of top-k 2048, 1024 and 512 in 1 to 16 equal partitions each, rows in HBM (one of 2048: 37.3, 28.2, 22.9, 22.8 and 24.9 us
# in 1, 2, 4, 8 and 16; 16: 39.3, 31.0, 27.8 in 1, 2, 4; 32: 39.9, 35.1; 64 whole 47.0); the cut that it names is the fastest measured
# one or within a microsecond of it.
def _duo_us(num_tokens: int, blocks: int, k: int, max_pairs: int) -> float:
    pairs = min(k * num_tokens, max_pairs)
    t = -(-num_tokens // max_pairs) * (12.3 + -(-(blocks // k) // 2) * (1.6 + 0.009 * max(pairs - 8, 0)))
    return t if k == 1 else t + 3.0 + 0.5 * k + 0.03 * k * num_tokens


def pick_split_duo(num_tokens: int, sms: int, blocks_per_token: int, uniform: bool) -> Tuple[int, int]:
    """(partitions, fixed overhead) where whole requests and equal partitions run on attn_duo_kernel and partitions of the
    scheduler on the pair kernel.

    Equal partitions leave fp16 records, so only calls that pick_split cuts equally are cut so here (lists of 8 blocks and more that
    have a suitable divisor, up to 37 requests), if into another number of pieces.  Others would be faster too (us whole / cut,
    rows in HBM: 4 requests of 640 entries 16.3 / 14.2, 10 of 896 19.1 / 17.1, 35 of 1024 23.0 / 22.5), but their results are whole
    requests' or go through fp32 records, without such a rounding.

    Ragged requests are left whole where the scheduler and combine launches and the partitions that straddle two requests cost
    more than the longest request: lists of up to 16 blocks (us before, with the scheduler and the pair kernel / whole, graph of steps:
    1 request of up to 512 entries 20.6 / 12.9, of up to 1024 22.2 / 15.0, 8: 25.0 / 19.9, 30: 34.0 / 20.2), and from half as
    many requests on as a list has blocks (us whole / cut, rows in HBM: 16 requests of up to 1024 entries 21.7 / 28.1; 8 of up to 1536 27.1 / 26.8, 13: 27.6 /
    29.7; 13 of up to 2048 33.6 / 30.7, 16: 33.5 / 34.1, 20: 34.1 / 39.6; 24 of up to 4096 59.4 / 54.6, 30: 60.1 / 60.4).  Otherwise the
    general rule cuts them into partitions of four blocks, as many as there are pairs of SMs at most; partitions of eight blocks
    take longer now that launches run under one another (4 requests of up to 2048 25.1 in 32, 27.2 in 16; 13: 30.7 in 74, 34.0 in
    52; 8: 29.3 and 29.6)."""
    n = max(blocks_per_token, 1)
    max_pairs = max(sms // CTAS_PER_PART, 1)
    whole = (num_tokens, FIXED_OVERHEAD)
    if uniform:
        parts, overhead = pick_split(num_tokens, sms, blocks_per_token, uniform=True)
        if parts == num_tokens:
            return whole
        if overhead == 0:
            cuts = [k for k in range(2, n // 2 + 1) if n % k == 0 and k * num_tokens <= max_pairs]
            k = min([1] + cuts, key=lambda c: _duo_us(num_tokens, n, c, max_pairs))
            return whole if k == 1 else (k * num_tokens, 0)
    if n <= 16 or 2 * num_tokens >= n:
        return whole
    return pick_num_sm_parts(num_tokens, sms, blocks_per_token), FIXED_OVERHEAD


def split_plan(device: int, num_tokens: int, num_heads: int, blocks: int, uniform: int, layout: int, ext: int, aligned: int,
               impl: int) -> Tuple[int, int, int]:
    """(partitions, the scheduler's fixed overhead, equal partitions per request) of a decode step: the one choice that
    the ops make.  A third value above 1 means that requests of equal length are cut into that many equal partitions each
    and the attention kernel derives the schedule itself (smla_decode_uniform).  ``ext``: MODEL1 or a second cache;
    ``aligned``: tc_aligned of the caches there, one_array of the cache otherwise."""
    if num_tokens == 0:
        return 0, FIXED_OVERHEAD, 0
    sms = num_sms(torch.device("cuda", device))
    if ext and aligned and layout == _lib.LAYOUT_MODEL1 and impl == _lib.IMPL_SCALAR:
        return pick_num_sm_parts_exact(num_tokens, num_heads, sms, blocks), FIXED_OVERHEAD, 0
    if ext and (impl == _lib.IMPL_SCALAR or not aligned):
        return pick_num_sm_parts_fp32(num_tokens, num_heads, sms), FIXED_OVERHEAD, 0
    if not ext and aligned and num_heads <= 64 and impl != _lib.IMPL_SCALAR:
        parts, overhead = pick_split_tile(num_tokens, num_heads, sms, blocks, bool(uniform))
    elif not ext and aligned and impl != _lib.IMPL_SCALAR:
        parts, overhead = pick_split_duo(num_tokens, sms, blocks, bool(uniform))
    else:
        parts, overhead = pick_split(num_tokens, sms, blocks, uniform=bool(uniform))
    k = parts // num_tokens
    equal = (uniform and not ext and impl != _lib.IMPL_SCALAR and overhead == 0 and k > 1 and k * num_tokens == parts
             and blocks % k == 0)
    return parts, overhead, k if equal else 0


_SCRATCH_LIMIT = 64      # cached call shapes per process before the least recently used one is dropped


def scratch(device: torch.device, total_splits: int, num_heads: int, num_tokens: int, num_parts: int):
    """Cached scratch for one call shape on the current stream (the reference allocates
    these on every call, flash_mla_sm120/ops.py:78-99).

    The key includes the stream: two calls of the same shape on different streams get different
    buffers, so they cannot race on ``o_accum``.  A capture gets buffers of its own, from the graph's
    memory, that never enter the cache: the graph may replay on any stream, beside eager calls on the
    stream that it was captured on.  Past _SCRATCH_LIMIT entries the least recently used one is dropped
    (it was allocated on, and only ever used on, its own stream, so the caching allocator may
    reuse it in stream order)."""
    def fresh():
        return {
            "o_accum": torch.empty((total_splits, 1, num_heads, 512), dtype=torch.float32, device=device),
            "lse_accum": torch.empty((total_splits, 1, num_heads), dtype=torch.float32, device=device),
            "sched_meta": torch.empty(num_parts * 8, dtype=torch.int32, device=device),
            "num_splits": torch.empty(num_tokens + 1, dtype=torch.int32, device=device),
        }
    if torch.cuda.is_current_stream_capturing():
        return fresh()
    key = (device.index, torch.cuda.current_stream(device).cuda_stream, total_splits, num_heads, num_tokens, num_parts)
    ws = _scratch.pop(key, None)
    _scratch[key] = fresh() if ws is None else ws                      # most recently used last
    if len(_scratch) > _SCRATCH_LIMIT:
        del _scratch[next(iter(_scratch))]
    return _scratch[key]


_status: Dict[int, torch.Tensor] = {}


def status_buffer(device: torch.device) -> torch.Tensor:
    idx = device.index if device.index is not None else torch.cuda.current_device()
    if idx not in _status:
        _status[idx] = torch.zeros(4, dtype=torch.int32, device=device)
    return _status[idx]


def status_pointer(index: int) -> int:
    return status_buffer(torch.device("cuda", index)).data_ptr()


def check_status(device: Optional[torch.device] = None) -> None:
    """Synchronises and raises if a kernel recorded a bounded wait that gave up.  Not called on
    the hot path (it reads device memory); tests and the benchmark call it."""
    if device is None:
        device = torch.device("cuda", torch.cuda.current_device())
    st = status_buffer(device)
    host = (ctypes.c_int32 * 4)()
    rc = _lib.load().smla_device_status(ptr(st), ctypes.addressof(host), stream_ptr(device))
    if rc != 0:
        raise _lib.SmlaError(_lib.load().smla_last_error().decode())

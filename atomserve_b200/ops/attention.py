"""Paged grouped-query attention over cache pages for a flat batch of requests."""

from __future__ import annotations

import ctypes
import functools
import os

import torch

from atomserve_b200.ops.library import KernelLibraryError, check, dtype_code, lib, ptr, require_cuda, stream

KEY_TILE = 32
TARGET_BLOCKS = 296  # two blocks for each of the 148 SMs before the key range is split
SHORT_ROWS = 8  # requests with at most this many new tokens run row by row in the decode kernel
MIXED_SCRATCH_BYTES = 128 << 20  # most that a step's partial results may take (see _paged_attention_parts)


# Which kernel serves prompt portions in bfloat16 with head size 128: "tcgen05" (scores and output
# in tensor memory; the default where its shape rules hold) or "mma" (the mma.sync kernel).
PREFILL_KERNEL = os.environ.get("ATOMSERVE_B200_PREFILL_ATTENTION", "tcgen05")


# In a step that holds prompt portions and single tokens, the two attention kernels touch disjoint
# rows and neither fills the device (a portion of a few hundred tokens is one block per SM or
# fewer; a few dozen single tokens are short chains of key tiles), so the single tokens' kernels
# run on a second stream beside the portions' kernel. "0" keeps them on one stream.
MIXED_OVERLAP = os.environ.get("ATOMSERVE_B200_MIXED_OVERLAP", "1") != "0"
_SIDE: dict[torch.device, tuple] = {}  # device -> (second stream, fork event, join event)


def _side_stream(device: torch.device):
    if device not in _SIDE:
        with torch.cuda.device(device):
            _SIDE[device] = (torch.cuda.Stream(), torch.cuda.Event(), torch.cuda.Event())
    return _SIDE[device]


def attention_tile_shape(group: int) -> tuple[int, int]:
    """(tokens per query tile, query heads per block) for `group` query heads per kv head."""
    qt, gc = ctypes.c_int(), ctypes.c_int()
    lib().asb_attention_tile_shape(group, ctypes.byref(qt), ctypes.byref(gc))
    return qt.value, gc.value


def plan_partitions(num_tokens: int, num_requests: int, num_kv_heads: int, group: int,
                    max_context: int, window: int) -> tuple[int, int]:  # fmt: skip
    """(partition size, partitions): split the keys only when the batch alone cannot fill the GPU.

    Partitions are aligned to absolute key positions, so the choice never changes which keys a
    row sees, only how its sum is grouped."""
    qt, gc = attention_tile_shape(group)
    blocks = (-(-num_tokens // qt) + num_requests) * num_kv_heads * -(-group // gc)
    span = max_context if window <= 0 else min(max_context, window + qt - 1)
    if blocks >= TARGET_BLOCKS or span <= 256:
        return 1 << 30, 1
    want = -(-TARGET_BLOCKS // blocks)
    size = max(256, -(-(-(-span // want)) // 256) * 256)
    if window <= 0:
        parts = (max_context - 1) // size + 1
    else:
        parts = min((max_context - 1) // size + 1, -(-span // size) + 1)
    return (size, parts) if parts > 1 else (1 << 30, 1)


@functools.lru_cache(maxsize=4096)
def plan_decode_partitions(rows: int, num_kv_heads: int, group: int, max_context: int, window: int,
                           head_dim: int = 128) -> tuple[int, int]:  # fmt: skip
    """(partition size, partitions) that even out the waves of blocks, one per (row, kv head, partition), if every row
    had the longest context: the fewest of waves x (64-key tiles per block + 3 tiles' worth of start-up) plus half a tile
    per partition for a merge. `plan_decode_ranges` asks it whether rows of several waves are worth cutting at all; how
    they are cut the decode kernel works out from the rows' own lengths."""
    blocks = rows * num_kv_heads * -(-group // 16)
    span = max_context if window <= 0 else min(max_context, window)
    resident = lib().asb_decode_attention_resident_blocks(head_dim) or 3 * 148
    best = None
    for want in range(1, max(1, span // 64) + 1):
        size = max(64, -(-(-(-span // want)) // 64) * 64)
        if window <= 0:
            parts = (max_context - 1) // size + 1
        else:
            parts = min((max_context - 1) // size + 1, -(-span // size) + 1)
        waves = -(-blocks * parts // resident)
        cost = waves * (size // 64 + 3) + 0.5 * parts
        if best is None or cost < best[0]:
            best = (cost, size, parts)
        if want > 64:
            break
    _, size, parts = best
    return (size, parts) if parts > 1 else (1 << 30, 1)


def plan_decode_ranges(rows: int, num_kv_heads: int, group: int, max_context: int, window: int, head_dim: int = 128,
                       partitions: tuple[int, int] | None = None) -> int:  # fmt: skip
    """Equal ranges into which the decode kernel cuts the keys of all rows, each for a block per kv head (and 16 of its
    heads); 0: each row is a range, and there is no merge. `partitions` (size, parts) asks for rows x parts of them.

    Nothing is cut where `plan_decode_partitions` would not split rows of the longest context (unless all rows run at once
    and walk more than 64 tiles, so that the longest row's end is worth a merge: 32 rows of 6,000 to 12,000 keys, 12 heads
    over 12 of size 64: 161 -> 136 us), nor where rows of up to 24 key tiles make blocks for half of what the device holds at once
    (64 rows of 100 to 300 keys, 8 kv heads: 25.6 -> 16.5 us). Otherwise as many ranges as the device holds blocks at
    once, if that leaves a block eight key tiles of the longest context; with less work three quarters of them, and no
    more than there are tiles: a merge of more shares then costs more than the shorter walk saves (one request of 12,288
    keys and 8 kv heads: 18.7 us in 16 ranges, 16.3 in 40, 19.3 in 55; of 2,048 keys: 10.8 us in 8, 9.4 in 32, 8.4 in 40;
    64 requests of 300 to 3,000 keys: 90.3 us in 24, 78.4 in 55).

    The merge costs about five tiles' time of a kernel with up to 8 heads a kv head (three with more, whose tiles take
    longer): rows that all run at once and walk no more than that further than a range would stay whole, and so do rows of
    up to eight tiles that would be cut in two (5 rows of 100 to 300 keys, 32 heads over 8: 7.7 -> 6.3 us; 16 of 500, 12 heads over 12 of size 64:
    12.6 -> 8.7; 128 of 500, 16 heads over one: 22.7 -> 16.7)."""
    if partitions:
        return rows * partitions[1] if partitions[1] > 1 else 0
    resident = lib().asb_decode_attention_resident(head_dim, group) or 3 * 148
    lanes = num_kv_heads * -(-group // 16)
    longest = -(-(min(max_context, window) if window > 0 else max_context) // 64)
    one_wave = rows * lanes <= resident
    if not (one_wave and longest > 64) and plan_decode_partitions(rows, num_kv_heads, group, max_context, window, head_dim)[1] <= 1:
        return 0
    if longest <= 24 and 2 * rows * lanes >= resident:
        return 0
    full, tiles = max(1, resident // lanes), rows * longest
    ranges = full if tiles >= 8 * full else max(1, min(3 * full // 4, tiles))
    walk = -(-tiles // ranges)
    if one_wave and longest <= max(walk + (5 if group <= 8 else 3), min(2 * walk, 8)):
        return 0
    return ranges


def decode_scratch_floats(rows: int, ranges: int, num_kv_heads: int, group: int, head_dim: int) -> int:
    """float32 elements of the decode kernel's scratch: four words a row, and per block (a range and a kv head, or 16 of its
    heads) two shares of up to 16 heads, each its output, maximum and sum."""
    return 4 * rows + 2 * ranges * num_kv_heads * -(-group // 16) * min(group, 16) * (head_dim + 2)


def plan_portion_parts(q_lens: list[int] | None, num_kv_heads: int, group: int, max_context: int, window: int) -> int:
    """Blocks (1, 2 or 4) that share the keys of each of the tcgen05 kernel's blocks (128 rows of one kv head's heads). By
    the estimate: waves of two blocks an SM, each of its share of the longest context's 64-key tiles (a tile's time 1, and
    1.3 where every SM has two blocks) and 4 tiles' time to start, 4 more to merge. (512 tokens, 32 heads over 8, one and
    two parts: at position 0 13.2 and 14.7 us, at 1,000 28.5 and 24.7, at 7,000 115 and 77; 100 tokens at 5,000: 99.7, and
    31.7 in four.) Divided only where that saves 15 % by the estimate: single tokens may run beside the portions."""
    tokens = 128 // group
    tiles = -(-(max_context if window <= 0 else min(max_context, window + tokens)) // 64)
    if q_lens is None or tiles < 8:
        return 1
    return _portion_parts(sum(-(-n // tokens) for n in q_lens if n > SHORT_ROWS) * num_kv_heads, tiles)


@functools.lru_cache(maxsize=4096)
def _portion_parts(blocks: int, tiles: int) -> int:
    def cost(parts):
        now = blocks * parts
        per_tile = 1 + 0.3 * min(1.0, max(0.0, 2 * now / TARGET_BLOCKS - 1))
        return -(-now // TARGET_BLOCKS) * (-(-tiles // parts) * per_tile + (8 if parts > 1 else 4))

    best = min((2, 4), key=cost)
    return best if cost(best) < 0.85 * cost(1) else 1


def paged_attention(
    q: torch.Tensor,
    k_cache: torch.Tensor,
    v_cache: torch.Tensor,
    block_tables: torch.Tensor,
    req_q_start: torch.Tensor,
    req_pos_start: torch.Tensor,
    *,
    num_requests: int,
    max_context: int,
    window: int | None,
    scale: float,
    partitions: tuple[int, int] | None = None,
    host_q_lens: list[int] | None = None,
    generic: bool = False,
    sink: torch.Tensor | None = None,
    chunk: int | None = None,
    softcap: float | None = None,
    keep_first: int = 0,
    earlier_keys_stored: bool = False,
    portions_context: int | None = None,
) -> torch.Tensor:
    """softmax(q k^T * scale) v for every new token, keys read in place from the pages.

    q: [T, H, hd]; k_cache, v_cache: [num_blocks, KV, block_size, hd]; block_tables: [R, W]
    int32; req_q_start: [R + 1] int32 (rows of each request in q); req_pos_start: [R] int32.
    max_context: the largest position + 1 any request reaches in this step (host int).
    A query at position p sees keys j <= p of its request, and j > p - window with a window.

    `sink` (float32 [H]): a logit per query head whose exponential joins the softmax's denominator
    once; it has no key and no value and is not scaled.

    `chunk`: the sequence is cut into runs of `chunk` positions, counted from position 0, and a
    query sees only the keys of its own run (still j <= p). `softcap`: every scaled score becomes
    softcap * tanh(score / softcap) before the softmax (the sink is not capped).

    `keep_first`: the first positions of a sequence, which stay visible behind the window and outside
    the chunk. q may be [T, H, KV, hd], a vector per key head: a head's score is then the sum of the
    products with all kv heads' keys (its values are still those of its own kv head): how scores that
    are mixed across heads run, the mix being part of the queries.

    `earlier_keys_stored`: the keys below every request's `req_pos_start` and the index tensors were written before the
    stream's previous kernel was launched (by earlier steps and by the step's upload, as in a model's step), so the kernels
    may read them while that kernel runs. Without it they read nothing before that kernel has completed.

    bfloat16 with head size 64 or 128 runs the tensor-core kernels (decode kernel for requests
    that bring at most 8 tokens, prefill kernel for longer portions; `host_q_lens`, the tokens
    each request brings, tells which are needed; `portions_context`, as max_context but of the
    requests that bring portions, is what these are planned for; heads with a vector per key head have kernels of
    their own); everything else, and `generic=True`, runs the
    general CUDA-core kernel.
    """
    require_cuda(q, k_cache, v_cache, block_tables, req_q_start, req_pos_start)
    KV, bs = k_cache.shape[1], k_cache.shape[2]
    parts, summed = 1, q.dim() == 4  # (with one kv head the sum has one term)
    if summed:
        parts = q.shape[2]
        if parts != KV:
            raise KernelLibraryError(f"paged_attention: queries of {parts} parts against {KV} key heads")
    T, H, hd = q.shape[0], q.shape[1], q.shape[-1]
    if not q.is_contiguous() or k_cache.shape != v_cache.shape or k_cache.shape[3] != hd:
        raise KernelLibraryError("paged_attention: q must be contiguous and the caches [blocks, KV, bs, hd]")
    if k_cache.dtype != q.dtype or v_cache.dtype != q.dtype:
        raise KernelLibraryError("paged_attention: cache and query dtypes differ")
    for t in (block_tables, req_q_start, req_pos_start):
        if t.dtype != torch.int32 or not t.is_contiguous():
            raise KernelLibraryError("paged_attention: index tensors must be contiguous int32")
    win = int(window) if window else 0
    chunk, softcap = int(chunk or 0), float(softcap or 0.0)
    out = torch.empty(T, H, hd, device=q.device, dtype=q.dtype)
    if sink is not None:
        require_cuda(sink)
        if sink.dtype != torch.float32 or sink.shape != (H,) or not sink.is_contiguous():
            raise KernelLibraryError(f"paged_attention: sink must be contiguous float32 [{H}]")
    span = min(win, chunk) if win and chunk else (win or chunk)  # a chunk bounds the keys of a row as a window does
    keep = int(keep_first) if span else 0
    if q.dtype == torch.bfloat16 and not generic and not summed and not keep and lib().asb_attention_mma_supported(hd, H // KV):
        return _paged_attention_mma(q, out, k_cache, v_cache, block_tables, req_q_start, req_pos_start,
                                    num_requests, max_context, win, scale, partitions, host_q_lens, sink, chunk, softcap, span,
                                    earlier_keys_stored, portions_context)  # fmt: skip
    if q.dtype == torch.bfloat16 and not generic and summed and not chunk and not softcap and sink is None and lib().asb_attention_parts_supported(hd, H, KV):
        return _paged_attention_parts(q, out, k_cache, v_cache, block_tables, req_q_start, req_pos_start, num_requests, max_context,
                                      win, keep, scale, partitions, host_q_lens, earlier_keys_stored)  # fmt: skip
    ps, np_ = partitions or plan_partitions(T, num_requests, KV, H // KV, max_context, span)
    part_m = part_l = part_acc = None
    if np_ > 1:
        part_m = torch.empty(T * H * np_, device=q.device, dtype=torch.float32)
        part_l = torch.empty_like(part_m)
        part_acc = torch.empty(T * H * np_ * hd, device=q.device, dtype=torch.float32)
    check(lib().asb_paged_attention_parts(
        ptr(out), ptr(q), ptr(k_cache), ptr(v_cache), ptr(block_tables), ptr(req_q_start),
        ptr(req_pos_start), ptr(part_m), ptr(part_l), ptr(part_acc), ptr(sink), T, num_requests, H, KV, hd, bs,
        block_tables.shape[1], win, chunk, keep, parts, ps, np_, float(scale), softcap, dtype_code(q), stream()))  # fmt: skip
    return out


def _paged_attention_mma(q, out, k_cache, v_cache, block_tables, req_q_start, req_pos_start, num_requests,
                         max_context, win, scale, partitions, host_q_lens, sink=None, chunk=0, softcap=0.0, span=None, earlier_keys_stored=False,
                         portions_context=None):  # fmt: skip
    span = win if span is None else span  # what bounds the keys of a row, for the planner
    T, H, hd = q.shape
    KV, bs = k_cache.shape[1], k_cache.shape[2]
    if host_q_lens is None:
        has_short = has_long = True
        all_single = False
        short_rows = T
    else:
        has_short = any(n <= SHORT_ROWS for n in host_q_lens)
        has_long = any(n > SHORT_ROWS for n in host_q_lens)
        all_single = all(n == 1 for n in host_q_lens)
        short_rows = sum(n for n in host_q_lens if n <= SHORT_ROWS)

    def decode(compact):
        """The launch for the rows of short requests: all T rows of the step, or the `compact` short ones of a step
        that holds longer portions too. Its scratch belongs to the stream that is current now."""
        group = H // KV
        ranges = plan_decode_ranges(short_rows, KV, group, max_context, span, hd, partitions)
        scratch = torch.empty(decode_scratch_floats(compact or T, ranges, KV, group, hd), device=q.device, dtype=torch.float32) if ranges else None

        def launch():
            check(lib().asb_decode_attention(
                ptr(out), ptr(q), ptr(k_cache), ptr(v_cache), ptr(block_tables), ptr(req_q_start), ptr(req_pos_start),
                ptr(scratch), ptr(sink), T, num_requests, H, KV, hd, bs, block_tables.shape[1], win, chunk, ranges,
                float(scale), softcap, int(all_single), compact, int(earlier_keys_stored), stream()))  # fmt: skip

        return launch

    if has_long and PREFILL_KERNEL == "tcgen05" and lib().asb_attention_tcgen05_supported(hd, H // KV, bs):
        from atomserve_b200.ops.linear import gemm_status

        parts = plan_portion_parts(host_q_lens, KV, H // KV, portions_context or max_context, span)

        def portions():
            check(lib().asb_prefill_attention_tcgen05_masked(
                ptr(out), ptr(q), ptr(k_cache), ptr(v_cache), ptr(block_tables), ptr(req_q_start), ptr(req_pos_start), ptr(sink),
                T, num_requests, H, KV, hd, bs, k_cache.shape[0], block_tables.shape[1], win, chunk, float(scale), softcap,
                parts, int(earlier_keys_stored), ptr(gemm_status(q.device)), stream()))  # fmt: skip

        if not has_short:
            portions()
            return out
        # What is left for the decode kernel: the short rows. When the caller says how many tokens
        # each request brings, the kernel's rows are the short ones only; otherwise it goes over
        # every row of the step and leaves the portions' alone.
        single_tokens = decode(short_rows if host_q_lens is not None else 0)
        if not MIXED_OVERLAP or torch.cuda.is_current_stream_capturing():
            portions()
            single_tokens()
            return out
        # Fork: the second stream starts from what this stream has done so far (q, the cache pages,
        # the scratch), runs the single tokens, and this stream goes on only when both are done.
        # The scratch is this stream's memory; it is given back after the join, so nothing that
        # reuses it can run before the second stream has finished with it.
        main = torch.cuda.current_stream(q.device)
        side, fork, join = _side_stream(q.device)
        fork.record(main)
        portions()
        with torch.cuda.stream(side):
            side.wait_event(fork)
            single_tokens()
            join.record(side)
        main.wait_event(join)
        return out
    if has_long:
        check(lib().asb_prefill_attention_mma(
            ptr(out), ptr(q), ptr(k_cache), ptr(v_cache), ptr(block_tables), ptr(req_q_start), ptr(req_pos_start), ptr(sink),
            T, num_requests, H, KV, hd, bs, block_tables.shape[1], win, chunk, float(scale), softcap, stream()))  # fmt: skip
    if has_short:
        decode(short_rows if has_long and host_q_lens is not None else 0)()
    return out


@functools.lru_cache(maxsize=4096)
def plan_parts_partitions(rows: int, heads: int, kv_heads: int, max_context: int, window: int, keep: int, head_dim: int) -> tuple[int, int]:
    """(key tiles of 64 per partition, partitions) for the decode kernel of heads with a vector per
    key head, one block per (row, up to 32 heads, partition): the same weighing as
    `plan_decode_partitions`, a tile's cost being the key and value heads that the block walks."""
    per_block = lib().asb_attention_parts_heads(heads, kv_heads)
    chunks = -(-heads // per_block)
    resident = lib().asb_attention_parts_resident(head_dim, heads, kv_heads) or 148
    tiles = -(-max_context // 64)
    if window:
        tiles = min(tiles, -(-min(keep, max_context) // 64) + -(-window // 64) + 1)
    items = (kv_heads + -(-kv_heads // chunks)) / 2  # a key head and a value head count as one tile of the plain kernel
    best = None
    for parts in range(1, min(tiles, 64) + 1):
        size = -(-tiles // parts)
        parts = -(-tiles // size)
        cost = -(-rows * chunks * parts // resident) * (size * items + 3) + 0.5 * parts
        if best is None or cost < best[0]:
            best = (cost, size, parts)
    return best[1], best[2]


def _paged_attention_parts(q, out, k_cache, v_cache, block_tables, req_q_start, req_pos_start, num_requests, max_context, win, keep,
                           scale, partitions, host_q_lens, earlier_keys_stored):  # fmt: skip
    T, H, KV, hd = q.shape
    bs = k_cache.shape[2]
    lens = host_q_lens
    has_short = lens is None or any(n <= SHORT_ROWS for n in lens)
    has_long = lens is None or any(n > SHORT_ROWS for n in lens)
    all_single = lens is not None and all(n == 1 for n in lens)
    short_rows = T if lens is None else sum(n for n in lens if n <= SHORT_ROWS)

    def launch(decode, long, pt, np_, m, l, acc, compact):
        check(lib().asb_attention_parts(
            ptr(out), ptr(q), ptr(k_cache), ptr(v_cache), ptr(block_tables), ptr(req_q_start), ptr(req_pos_start), ptr(m), ptr(l), ptr(acc),
            T, num_requests, H, KV, hd, bs, block_tables.shape[1], win, keep, pt, np_, float(scale), int(decode), int(long),
            int(all_single), compact, stream()))  # fmt: skip

    if has_long and PREFILL_KERNEL == "tcgen05" and scale > 0 and lib().asb_attention_parts_tcgen05_supported(hd, H // KV, bs):
        from atomserve_b200.ops.linear import gemm_status

        check(lib().asb_attention_parts_tcgen05(
            ptr(out), ptr(q), ptr(k_cache), ptr(v_cache), ptr(block_tables), ptr(req_q_start), ptr(req_pos_start), T, num_requests, H, KV, hd,
            bs, k_cache.shape[0], block_tables.shape[1], win, keep, float(scale), int(earlier_keys_stored), ptr(gemm_status(q.device)), stream()))  # fmt: skip
    elif has_long:
        launch(False, True, 1, 1, None, None, None, 0)
    if has_short:
        # a step that also holds long portions starts blocks, and holds partial results, for the short rows only
        compact = short_rows if has_long and lens is not None else 0
        rows = compact or T
        pt, np_ = partitions or plan_parts_partitions(short_rows, H, KV, max_context, win, keep, hd)
        if partitions is None and (lens is None or rows * H * np_ * (hd + 2) * 4 > MIXED_SCRATCH_BYTES):
            pt, np_ = 1 << 24, 1
        m = l = acc = None
        if np_ > 1:
            m = torch.empty(rows * H * np_, device=q.device, dtype=torch.float32)
            l = torch.empty_like(m)
            acc = torch.empty(rows * H * np_ * hd, device=q.device, dtype=torch.float32)
        launch(True, False, pt, np_, m, l, acc, compact)
        if np_ > 1 and compact:
            check(lib().asb_attention_reduce_short(ptr(out), ptr(m), ptr(l), ptr(acc), ptr(req_q_start), num_requests, SHORT_ROWS, compact,
                                                   H, np_, hd, dtype_code(q), stream()))  # fmt: skip
        elif np_ > 1:
            check(lib().asb_attention_reduce(ptr(out), ptr(m), ptr(l), ptr(acc), T * H, np_, hd, dtype_code(q), stream()))
    return out

"""Launch planning for the attention path, restated in Python.

These are mirrors of the planning rules compiled into ``libb200attn.so`` (csrc/decode.cu ``decode_pass_group`` /
``decode_ws_layout`` / ``decode_plan_kernel`` and the prefill grid in csrc/prefill.cu), which replace the
reference's split heuristics (kernels/attention.py:836-841, kernels/decode.py:271-278,
kernels/speculative_decode.py:301-309).  Nothing on the product path calls them: the library plans for itself.
They exist so that the rules can be unit-tested without a GPU, and ``decode_workspace_bytes`` is compared with the
library's own ``b200attn_decode_workspace_bytes`` in the GPU tests so that the two cannot drift apart unnoticed.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import List, Optional, Sequence, Tuple

DECODE_TILE_TOKENS = 64       # keys per cp.async stage
PREFILL_BLOCK_M = 128         # query rows per tensor-core tile
PREFILL_SLOTS = 2             # query tiles per CTA
PREFILL_BLOCK_N = 128         # keys per tile


@dataclass
class DecodePlan:
    target_items: int
    min_chunk: int
    max_items: int
    mma_tiles: int     # 16-row MMA tiles that hold group x q_len rows
    key_slices: int    # warps that split the keys of one stage
    threads: int
    wave_items: int = 0      # items of one KV head resident at once (one wave); 0: a single wave is never planned
    item_overhead: int = 0   # start-up + merge of an item in keys of streaming time (the planner's cost estimate)
    slots: int = 0           # CTAs per KV head of the persistent kernel that a batch may be dealt out to
    one_cta: bool = False    # that kernel has one CTA to an SM, not two


def decode_pass_group(group: int, q_len: int) -> int:
    """q heads of one KV head that one launch serves: at most 128 q rows (group x draft tokens) per CTA; a larger
    group is cut into the largest equal sub-groups that fit."""
    q_len = max(1, q_len)
    g = group
    while g > 1 and (g * q_len > 128 or group % g != 0):
        g -= 1
    return max(g, 1)


def decode_workspace_bytes(plan: "DecodePlan", batch: int, kv_heads: int, head_dim: int, rows: int,
                           cast_q_elems: int = 0, cast_kv_elems: int = 0) -> int:
    """Bytes of scratch a decode call needs: header, item prefix, merge tickets, item records, (m, l) and O partials,
    each rounded up to 256 bytes (csrc/decode.cu decode_ws_layout) - and, for fp32 inputs of a speculative-decode
    call, the fp16 copies of q, k and v (``cast_*_elems`` elements each)."""
    up = lambda x: (x + 255) & ~255
    off = 256
    off = up(off + 4 * (batch + 1))
    off = up(off + 4 * batch * kv_heads)
    off = up(off + 32 * plan.max_items)
    slots = plan.max_items * kv_heads
    off = up(off + 4 * slots * rows * 2)
    off = up(off + 4 * slots * rows * head_dim)
    if cast_kv_elems:
        off = up(off + 2 * cast_q_elems)
        off = up(off + 2 * cast_kv_elems)
        off = up(off + 2 * cast_kv_elems)
    return off


def tcgen05_plans_itself(sm_count: int, batch: int, kv_heads: int, keys: int) -> bool:
    """Whether a call of more than sixteen q rows per KV head in 16 bits goes without the planner's launch (csrc/decode.cu
    inline_plan_bits); ``keys``: of all sequences, as many as there can be (a packed tensor's rows, a table's width for each)."""
    return batch * kv_heads <= 96 and keys * kv_heads <= (1024 - 8 * batch) * 2 * sm_count


def keyrows_suit(sm_count: int, batch: int, kv_heads: int, rows: int, keys: int, head_dim: int, page_size: Optional[int] = None,
                 cache_keys: Optional[int] = None, equal: bool = True) -> bool:
    """Whether a call of 16-bit elements behind the planner goes to the kernel whose tiles have keys as their rows (csrc/decode.cu
    keyrows_suit); ``keys`` as in ``tcgen05_plans_itself``; for paged caches ``page_size`` and the rows of the cache (None: as many as
    it takes); ``equal``: a dense batch, whose sequences have one length."""
    if not 16 < rows <= 64 or (page_size is not None and page_size % 8):
        return False
    one_each = batch * kv_heads <= sm_count
    if one_each and head_dim == 64 and (not equal or page_size is not None or batch * kv_heads * 3 < sm_count * 2):
        return False

    def enough(n: int, quarters: int) -> bool:
        line = (512 << 7) // head_dim * (1 if one_each else 2) * quarters // 8
        return n >= line * batch and (one_each or n * kv_heads * head_dim >= (512 << 7) * quarters * sm_count)

    if page_size is None:
        return enough(keys, 4)
    return enough(keys, 8) and (cache_keys is None or enough(cache_keys, 3))


def decode_plan(sm_count: int, batch: int, q_heads: int, kv_heads: int, q_len: int, fp32: bool = False,
                keys: Optional[int] = None, head_dim: int = 64, page_size: Optional[int] = None, cache_keys: Optional[int] = None,
                equal: bool = True) -> DecodePlan:
    """``keys`` (see ``tcgen05_plans_itself``): with it, calls of the tcgen05 kernel that plan for themselves are planned as they do,
    without dealing the batch out, and up to three short sequences in items for one CTA an SM, and calls of the kernel with keys as rows
    (``keyrows_suit``, which ``head_dim`` and what follows it are for) as for that; without it all are the planner's, for the tcgen05 kernel
    with two CTAs an SM."""
    group = decode_pass_group(q_heads // kv_heads, q_len)
    rows = group * q_len
    # fp32 inputs of a speculative-decode call (several q rows per head) run the tensor-core kernels on fp16 copies
    # and are planned like 16-bit inputs (unless k and v would need more than 8 GiB of copies: csrc/decode.cu)
    fp32 = fp32 and rows <= 16 and q_len <= 1
    # six (item, kv head) CTAs per SM (a whole number of waves at 2 or 3 resident CTAs per SM)
    target = max(1, (sm_count * 6) // max(1, kv_heads))
    by_rows = -(-(rows * 8) // DECODE_TILE_TOKENS) * DECODE_TILE_TOKENS
    min_chunk = max(128, by_rows)
    tiles = -(-rows // 16)
    slices = 4 if tiles <= 2 else (2 if tiles <= 4 else 1)
    wide = rows > 16 and not fp32   # more than one 16-row tile: the tcgen05 kernel, two resident CTAs per SM (else three)
    wave = max(1, (sm_count * (2 if wide else 3)) // max(1, kv_heads))
    overhead = 448 if wide else 128
    slots, max_items = 2 * sm_count // max(1, kv_heads) if wide else 0, target + batch
    if wide and keys is not None and tcgen05_plans_itself(sm_count, batch, kv_heads, keys):
        slots = 0
        if batch <= 3 and keys * kv_heads <= 6 * min_chunk * sm_count:
            target, wave = max(1, sm_count // kv_heads), 0
    elif wide and keys is not None and keyrows_suit(sm_count, batch, kv_heads, rows, keys, head_dim, page_size, cache_keys, equal):
        slots, target, wave = sm_count // kv_heads, max(1, 3 * sm_count // kv_heads), max(1, sm_count // kv_heads)
        return DecodePlan(target, min_chunk, max_items, tiles, slices, 32 * (tiles * slices + 1), wave, overhead, slots, True)
    return DecodePlan(target, min_chunk, max_items, tiles, slices, 32 * (tiles * slices + 1), wave, overhead, slots)


def _round_up(x: int, m: int) -> int:
    return -(-x // m) * m


def _item_tokens(length: int, n: int) -> int:
    """Keys per item of a sequence cut into ``n`` items (csrc/decode.cu seq_chunk)."""
    return max(DECODE_TILE_TOKENS, _round_up(-(-length // n), DECODE_TILE_TOKENS))


def _pick_chunk(plan: DecodePlan, lens: Sequence[int], target: int):
    """First of 32 candidates between total / target and twice that with at most ``target`` items:
    (chunk, items, largest item, found)."""
    total = sum(lens)
    base = max(_round_up(-(-total // target), DECODE_TILE_TOKENS), plan.min_chunk)
    last = None
    for k in range(32):
        chunk = _round_up(base + (base * k) // 32, DECODE_TILE_TOKENS)
        counts = [max(1, -(-n // chunk)) for n in lens]
        biggest = max([min(n, _item_tokens(n, c)) for n, c in zip(lens, counts)], default=0)
        last = (chunk, sum(counts), biggest)
        if last[1] <= target:
            return last + (True,)
    return last + (False,)


def _plan_lengths(plan: DecodePlan, lens: Sequence[int]):
    """(chunk, dealt): the chunk size for several waves or a single one, and whether the batch is dealt out instead."""
    total = sum(lens)
    chunk, items, _, _ = _pick_chunk(plan, lens, plan.target_items)
    best = 0.0
    if plan.wave_items > 0:
        best = (total + items * plan.item_overhead) / plan.wave_items + 0.5 * (total / items + plan.item_overhead)
    if 0 < plan.wave_items < plan.target_items and items > plan.wave_items:
        w_chunk, _, w_biggest, found = _pick_chunk(plan, lens, plan.wave_items)
        if found and w_biggest + plan.item_overhead < best:
            best, chunk = w_biggest + plan.item_overhead, w_chunk
    if plan.one_cta:
        best = 0.89 * min(best, -(-items // plan.wave_items) * (chunk + plan.item_overhead)) - 500
    line = total + (len(lens) + plan.slots - 1) * plan.item_overhead
    dealt = (1 < plan.slots <= 512 and len(lens) <= 4096 and line < 1 << 30 and items > plan.wave_items
             and line / plan.slots + plan.min_chunk < best)
    return chunk, dealt


def decode_cuts(plan: DecodePlan, lengths: Sequence[int]) -> Optional[List[Tuple[int, int]]]:
    """First (sequence, key) of every slot when the batch is dealt out to the CTAs of the persistent kernel, one past the
    last sequence for slots that get nothing; None when it is planned in chunks."""
    lens = [max(0, int(n)) for n in lengths]
    if not _plan_lengths(plan, lens)[1]:
        return None
    ovh, starts = plan.item_overhead, [0]
    for n in lens:
        starts.append(starts[-1] + n + ovh)
    line = sum(lens) + (len(lens) + plan.slots - 1) * ovh
    stretch = max(_round_up(-(-line // plan.slots), DECODE_TILE_TOKENS), plan.min_chunk)
    cuts = []
    for i in range(plan.slots):
        x = i * stretch
        b, t = len(lens), 0
        if x < starts[-1]:
            b = max(j for j in range(len(lens)) if starts[j] <= x)
            off = x - starts[b] - ovh
            t = (off + DECODE_TILE_TOKENS // 2) // DECODE_TILE_TOKENS * DECODE_TILE_TOKENS if off > 0 else 0
            if t < plan.min_chunk:
                t = 0
            elif lens[b] - t < plan.min_chunk:
                b, t = b + 1, 0
        cuts.append((b, t))
    return cuts


def decode_chunk_tokens(plan: DecodePlan, lengths: Sequence[int]) -> int:
    """Chunk size the device planner picks for these lengths: the smallest of 32 candidates between
    total / target_items and twice that which splits the batch into at most target_items items - or, when the
    batch also fits a single wave of resident CTAs and the estimate favours it (largest item + per-item overhead
    against the average load of a resident CTA + half an item), the single-wave chunk.  A batch that is dealt out has no
    chunk size; its items have at least min_chunk keys (or are whole sequences)."""
    chunk, dealt = _plan_lengths(plan, [max(0, int(n)) for n in lengths])
    return plan.min_chunk if dealt else chunk


def decode_items(plan: DecodePlan, lengths: Sequence[int]) -> List[int]:
    """Work items (KV chunks) per sequence; their sum never exceeds plan.max_items."""
    cuts = decode_cuts(plan, lengths)
    if cuts is not None:
        return [1 + sum(1 for c, t in cuts if c == b and t > 0) for b in range(len(lengths))]
    chunk = decode_chunk_tokens(plan, lengths)
    return [max(1, -(-max(0, int(n)) // chunk)) for n in lengths]


def prefill_items(layout: str, batch: int, q_heads: int, kv_heads: int, max_q: int = 0, total_q: int = 0) -> int:
    """Work items of the persistent prefill kernel.  An item is two 128-row query tiles that share a KV head: two
    neighbouring q heads over the same rows when the GQA group is even, else two consecutive row tiles of one head."""
    head_pair = (q_heads // kv_heads) % 2 == 0
    rows = PREFILL_BLOCK_M if head_pair else PREFILL_BLOCK_M * PREFILL_SLOTS
    units = q_heads // 2 if head_pair else q_heads
    if layout == "ragged":
        return (total_q // rows + batch) * units
    return -(-max_q // rows) * units * batch


def paged_box_rows(page_size: int) -> int:
    """Tokens per TMA box for a paged cache: the largest power of two dividing the page size, at most one tile."""
    box = 1
    while box < PREFILL_BLOCK_N and page_size % (box * 2) == 0:
        box *= 2
    return box

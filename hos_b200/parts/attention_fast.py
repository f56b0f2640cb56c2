"""Python face of the tensor-core attention kernels (csrc/attention_decode.cu,
csrc/attention_prefill.cu).  They are compiled per head size (a multiple of 16, at most
256) as library `attn_hd<N>`; other head sizes are left to the plain kernel."""
from __future__ import annotations

import ctypes
import functools
import math
import os
from typing import Dict, NamedTuple, Optional

import numpy as np
import torch

from .. import ops

MAX_HEAD_DIM = 256
MAX_SPLITS = 64

_libs: Dict[int, ops.Library] = {}
enabled = {"decode": True, "prefill": True, "prefill_tc": True, "chunk": True, "chunk_tc": True,
           "prefill_pair": os.environ.get("HOS_ATTN_PAIR", "1") != "0",
           "decode_cluster": os.environ.get("HOS_ATTN_CLUSTER", "1") != "0",
           "decode_even": os.environ.get("HOS_ATTN_EVEN", "1") != "0"}
_pair_state: Dict[int, bool] = {}
_cluster_state: Dict[int, bool] = {}     # tests switch a kernel off to compare with the plain one


def supports(head_dim: int) -> bool:
    return head_dim % 16 == 0 and 16 <= head_dim <= MAX_HEAD_DIM


def lib_for(head_dim: int) -> ops.Library:
    lib = _libs.get(head_dim)
    if lib is None:
        lib = _libs[head_dim] = ops.Library(f"attn_hd{head_dim}")
    return lib


def decode_splits(n_tokens: int, n_kv_heads: int, group: int, max_len: int, window: Optional[int],
                  min_live: int = 0, clusters_fit=None, max_live: int = 0, fill: float = 1.0, head_dim: int = 256,
                  groups: int = 2) -> int:
    """How many shares the keys of one (token, kv head) are cut into; 0: even shares.  The kernel's CTAs (one per
    SM) take items one after another; the answer is the cut that makes the step shortest by the estimate below, for
    all `n_tokens` rows live and, if the step is
    a replayed one whose last rows may be padding, for `min_live` live rows and half-way as well
    (`max_live`: no more than that many of the rows are live; 0: all may be).  `fill`: the sequences' lengths add
    up to at most this fraction of live rows x what the longest holds (in this layer: of its window, if it has one):
    equal shares follow the longest sequence whatever the others hold, even shares follow the sum.
    `clusters_fit(s)`: how many clusters of s CTAs of the kernel run at once (None: no cluster merge); with
    all of a step's clusters on the GPU at once the shares merge through shared memory, which is cheaper.
    `groups`: the groups of consumers that even shares have with these heads (consumer_groups)."""
    return _decode_splits(_heads(n_kv_heads, group, head_dim), n_tokens, _pages(max_len, window), min_live, clusters_fit, max_live,
                          round(fill, 2), groups, enabled["decode_even"] and n_tokens <= EVEN_MAX_ROWS, ops.sm_count())


class _Heads(NamedTuple):
    per_token: int              # items of a row
    weight: float               # query heads of an item x head size / 512
    page: float                 # bytes of a page's keys and values / 64 KB
    alone: float                # us that a page takes a CTA by itself


def _heads(n_kv_heads: int, group: int, head_dim: int) -> _Heads:
    page = head_dim / 256
    return _Heads(max(1, n_kv_heads * ((group + 15) // 16)), min(group, 16) * head_dim / 512, page,
                  (0.41 + 0.26 * page) * (1.23 if group > 8 or group * head_dim > 1280 else 1.0))


def _pages(max_len: int, window: Optional[int]) -> int:
    span = min(max_len, window) if window else max_len
    return -(-span // ops.PAGE_TOKENS) + (1 if window else 0)


@functools.lru_cache(maxsize=1024)
def _decode_splits(h: _Heads, n_tokens, pages, min_live, clusters_fit, max_live, fill, groups, may_even, sms) -> int:
    hi = max(1, min(n_tokens, max_live) if max_live else n_tokens)
    lo = min(max(1, min_live), hi) if min_live else hi
    lives = (lo, (lo + hi) // 2, hi, hi) if lo < hi else (hi,)      # fewest, middle and most live rows (a full batch counts twice)

    def cluster(s: int) -> bool:
        return 1 < s <= CLUSTER_SHARES and hi * h.per_token * s <= sms and clusters_fit is not None and clusters_fit(s) >= hi * h.per_token

    best, best_cost = 1, None
    for s in range(1, min(MAX_SPLITS, max(1, (pages + 1) // 2)) + 1):
        if s > 1 and lo * h.per_token * (s - 1) > 2 * sms:          # more rounds than that never pay
            break
        merged = cluster(s)
        cost = sum(_equal_us(h, live, pages, fill, s, merged, sms) for live in lives)
        if s == 1:                                                  # (a round of whole items against even shares: see _whole)
            cost += sum(8.0 * ((live * h.per_token - 1) // sms) for live in lives)
        if best_cost is None or cost < 0.995 * best_cost:           # more shares only for a gain
            best, best_cost = s, cost
    if may_even and sum(_even_us(h, live, pages, fill, groups, sms) for live in lives) < best_cost:
        return 0
    return best


# The estimate, us a launch (weight, page, alone: see _Heads).
#   a page takes a CTA `alone`: 0.41 + 0.26 page, with more than eight heads to a kv head (the MMA's rows) or a ring of two stages (six
#   heads of 256) 1.23 times that; and the memory's speed is shared: 0.00964 page for every CTA that streams (6.8 TB/s);
#   an item 3.5 + 1.25 weight, a further round of items 3.45 less (its first pages come during the last one's merge);
#   a merge through a cluster 0.59 + weight (0.41 + 1.66 a CTA of it) and 0.45 + 0.25 weight more where the shares are no power of two, through
#   the workspace and a ticket 2.66 + weight (1.08 + 0.087 a share, 1.23 more likewise);
#   even shares 5.2 (one group of consumers: 6.5) + 6.3 weight, 0.21 weight for every CTA that the longest item lies in, and 1.2 for each of
#   the shortest rows' items, of which a CTA may have to do as many as a row has;
#   whole items by their length 6.3, 0.66 weight for every round after the first.
# Fitted to 1,017 batches of 1 to 128 rows of 200 to 8,184 keys, alike and not, with windows and without, head sizes 64, 128 and 256, 2 to 16
# query heads a kv head, each cut in up to 20 ways (B200, replayed launches on cold caches; deviation 7%).
# Examples of 8 heads of 256 over 4, us with even shares / one / two / four: 8 rows of 2,000 to
# 8,184 keys 39.6 / 89.6 / 50.0 / 33.9, 24 of 4,096 72.4 / 62.5 / 80.2 / 75.8, 40 of 8,184 205 / 246 / 221 / 223, 16 of 64 to 8,184 34.5 / 89.8 /
# 50.9 / 34.4, 36 of 1,024 30.3 / 27.9 / 35.1 / 45.8; of 32 heads of 256 over 2: 32 of 64 to 2,036 83 / 42 / 38 / 67.
def _page_us(h: _Heads, active: int) -> float:
    return max(h.alone, 0.00964 * h.page * active)


@functools.lru_cache(maxsize=256)
def _lengths(rows: int, fill: float) -> np.ndarray:
    """Lengths of `rows` rows, the longest (1) first, that fill `fill` of rows x the longest: evenly spread over their logarithm."""
    lo, hi = 1e-9, 1.0
    for _ in range(40):
        mid = math.sqrt(lo * hi)
        lo, hi = (mid, hi) if (mid - 1.0) / math.log(mid) < fill else (lo, mid)
    return hi ** (np.arange(rows) / max(1, rows - 1))


def _walks_us(h: _Heads, lengths: np.ndarray, per_row: int, sms: int, by_length: bool) -> float:
    """The time that CTAs take for the pages of items which are handed out in turn (by_length: every other round backwards), while the
    memory's speed is shared by those that are not done."""
    items = np.repeat(lengths, per_row)
    rounds = -(-items.size // sms)
    held = np.zeros((rounds, sms))
    held.reshape(-1)[:items.size] = items
    if by_length:
        held[1::2] = held[1::2, ::-1]
    held = np.sort(held.sum(axis=0))
    us = np.maximum(h.alone, 0.00964 * h.page * np.arange(sms, 0, -1))
    return float(np.dot(np.diff(held, prepend=0.0), us))


def _equal_us(h: _Heads, rows: int, pages: int, fill: float, s: int, cluster: bool, sms: int) -> float:
    full, rest = divmod(rows * h.per_token * s, sms)
    if fill > 0.99 or rows == 1:
        walks = -(-pages // s) * (full * _page_us(h, sms) + (_page_us(h, rest) if rest else 0.0))
    else:
        lengths = np.maximum(1.0, np.maximum(1.0, pages * _lengths(rows, fill)) / s)
        walks = _walks_us(h, lengths[np.argsort(np.arange(rows) * 0.6180339887 % 1.0)], h.per_token * s, sms, False)     # in no order
    rounds = full + (1 if rest else 0)
    odd = 1.0 if s & (s - 1) else 0.0
    if cluster:
        merge = 0.59 + h.weight * (0.41 + 1.66 / s) + (0.45 + 0.25 * h.weight) * odd
    else:
        merge = 2.66 + h.weight * (1.08 + 0.087 * s + 1.23 * odd) if s > 1 else 0.0
    return walks + rounds * (3.5 + 1.25 * h.weight + merge) - 3.45 * (rounds - 1)


def _even_us(h: _Heads, rows: int, pages: int, fill: float, groups: int, sms: int) -> float:
    share = max(1, -(-int(rows * h.per_token * max(1.0, pages * fill)) // sms), -(-pages // (EVEN_MOST_PARTS - 1)))
    short = max(1.0, pages * float(_lengths(rows, fill)[int(0.8 * (rows - 1))]))        # pages of a short row
    items = min(h.per_token, share / short) if rows > 1 else 0.0
    return ((5.2 if groups == 2 else 6.5) + 6.3 * h.weight + min(EVEN_MOST_PARTS, pages / share) * 0.21 * h.weight + 1.2 * items +
            share * _page_us(h, sms))


def _by_length_us(h: _Heads, rows: int, pages: int, fill: float, sms: int) -> float:
    rounds = -(-rows * h.per_token // sms)
    return _walks_us(h, np.maximum(1.0, pages * _lengths(rows, fill)), h.per_token, sms, True) + 6.3 + 0.66 * h.weight * (rounds - 1)


# Up to 16 shares of at most one wave of items merge as a cluster through shared memory: 2.3 to 2.8 us less
# than through the workspace (one sequence, 8,192 keys, 16 shares: 17.4 -> 14.6 us; a window of 4,096: 13.5 -> 10.7).
CLUSTER_SHARES = 16
EVEN_MAX_ROWS = 2048
EVEN_MOST_PARTS = 32        # CTAs that a (token, kv head) lies in, at most (csrc/attention_decode.cu: kEvenMaxParts)
SORTED_MAX_ROWS = 256


def whole_items_by_length(n_rows: int, per_token: int, pages: int, fill: float, weight: float = 1.0, page: float = 1.0) -> bool:
    """Whether whole (token, kv head), handed out by their length, finish before even shares do (both with two groups of consumers; see
    csrc/attention_decode.cu): `pages` of the longest row's keys, `fill` as for decode_splits.  64 rows of 16 heads of 128 over 4, 64 to
    2,036 keys, 25.6 / 32.5 us; 40 of 8,184 keys, whose 160 items are two rounds of 148 SMs, 166 / 114."""
    sms = ops.sm_count()
    if n_rows * per_token <= sms or n_rows > SORTED_MAX_ROWS:
        return False
    h = _Heads(per_token, weight, page, 0.41 + 0.26 * page)
    return _by_length_us(h, n_rows, pages, fill, sms) < _even_us(h, n_rows, pages, fill, 2, sms)


@functools.lru_cache(maxsize=1024)
def _whole(h: _Heads, splits: int, rows: int, pages: int, fill: float, even_groups: int, groups: int, sms: int) -> tuple:
    """(shares, by their length) where decode_splits chose even shares or whole items (`splits`: 0 or 1) and the items are more than the SMs:
    even shares (of `even_groups` groups of consumers), whole items as they come (one group, nothing sorted: rows all alike), or by
    their length (where `groups`, which that launch would have, are two).  64 rows of 8 heads of 256 over 4, us as they come / by length: 517
    keys each 28.8 / 30.1, 2,048 81.8 / 85.2; 16 heads of 128 over 4, 64 to 2,036 keys 31.9 / 25.6."""
    best = (splits, False)
    cost = _even_us(h, rows, pages, fill, even_groups, sms) if splits == 0 else None
    whole = _equal_us(h, rows, pages, fill, 1, False, sms)
    if cost is None or whole < 0.97 * cost:
        best, cost = (1, False), whole
    if groups == 2 and rows <= SORTED_MAX_ROWS and _by_length_us(h, rows, pages, fill, sms) < 0.97 * cost:
        best = (1, True)
    return best


def plan(head_dim: int, n_tokens: int, n_heads: int, n_kv_heads: int, max_len: int, window: Optional[int], min_live: int, clusters_fit,
         max_live: int, fill: float, groups_of) -> tuple:
    """(shares as decode_splits, whole items by their length) for a launch of n_tokens rows, of which as many are live as decode_splits is
    told; groups_of: consumer_groups.  Over the 1,017 batches beside the estimate the choice takes 1.01 times as long as the best of all cuts;
    one fitted at head size 256 with two query heads to a kv head took 1.05 times, up to 3.5 times."""
    group, heads = n_heads // n_kv_heads, _heads(n_kv_heads, n_heads // n_kv_heads, head_dim)
    even_groups = groups_of(head_dim, n_tokens, n_heads, n_kv_heads, True)
    splits = decode_splits(n_tokens, n_kv_heads, group, max_len, window, min_live, clusters_fit, max_live, fill, head_dim, even_groups)
    live = min(n_tokens, max_live) if max_live else n_tokens
    if splits > 1 or live * heads.per_token <= ops.sm_count():
        return splits, False
    return _whole(heads, splits, live, _pages(max_len, window), round(fill, 2), even_groups,
                  groups_of(head_dim, n_tokens, n_heads, n_kv_heads, False), ops.sm_count())


_groups_known: Dict[tuple, int] = {}
_fit_known: Dict[tuple, int] = {}


def consumer_groups(head_dim: int, n_tokens: int, n_heads: int, n_kv_heads: int, even: bool) -> int:
    """Groups of consumers of a launch with even shares, or with whole items by their length (asked once per shape)."""
    key = (head_dim, n_tokens, n_heads, n_kv_heads, even)
    n = _groups_known.get(key)
    if n is None:
        f = lib_for(head_dim).lib.hos_attn_decode_groups
        f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int] * 4
        n = _groups_known[key] = int(f(n_tokens, n_heads, n_kv_heads, int(even)))
    return n


@functools.lru_cache(maxsize=64)
def _fits(head_dim: int, n_heads: int, n_kv_heads: int):
    return functools.partial(clusters_fit, head_dim, n_heads, n_kv_heads)


def clusters_fit(head_dim: int, n_heads: int, n_kv_heads: int, n_splits: int) -> int:
    """Clusters of n_splits CTAs of the decode kernel that run on the GPU at once (asked once per shape)."""
    key = (head_dim, n_heads, n_kv_heads, n_splits)
    n = _fit_known.get(key)
    if n is None:
        f = lib_for(head_dim).lib.hos_attn_decode_clusters
        f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_int, ctypes.c_int]
        n = _fit_known[key] = int(f(n_heads, n_kv_heads, n_splits))
    return n


_ticket_store: Dict[object, list] = {}
_TICKETS_AT_LEAST = 1 << 16


def _tickets(device, n: int) -> torch.Tensor:
    """Zeroed counters that the kernel leaves zeroed, shared by all launches on a device.  Captured
    graphs keep the address they were given, so a buffer is never given up: if a launch needs more
    than the last one holds, another is made and the old ones stay."""
    held = _ticket_store.setdefault(device, [])
    if not held or held[-1].numel() < n:
        held.append(torch.zeros(max(n, _TICKETS_AT_LEAST), dtype=torch.int32, device=device))
    return held[-1]


def _clear_tickets() -> None:
    """After a kernel gave up: a share that left early took no ticket, so its counter is not at zero."""
    for held in _ticket_store.values():
        for t in held:
            t.zero_()


ops.on_give_up(_clear_tickets)


def decode(q: torch.Tensor, q_stride: int, out: torch.Tensor, token_pos, token_seq, seq_slot,
           cache: ops.PagedKVArgs, n_tokens: int, n_heads: int, scale: float, cap: float,
           window: Optional[int], max_len: int, n_splits: Optional[int] = None,
           max_new: Optional[int] = None, min_live: int = 0, token_slot=None, cluster: bool = True,
           max_live: int = 0, fill: float = 1.0, by_length: bool = True) -> None:
    """Attention of n_tokens single queries over the paged cache (each token at its own
    position in its own sequence).  `max_new`: the most tokens any sequence brings in this step;
    the kernel may fetch keys that lie below them while the kernel before it (which writes the
    step's new keys) still runs.  None: it fetches nothing ahead.  `token_slot`: each token's cache slot
    (seq_slot[token_seq]) if the step has it: the kernel then finds its first page one look-up sooner.
    `cluster`: up to 16 shares of at most one wave of work items may run as clusters that merge through
    shared memory (False: always through the workspace).  `by_length`, with n_splits 1: more items than SMs are handed out by
    their length."""
    hd, nkv = cache.head_dim, cache.n_kv_heads
    lib = lib_for(hd)
    want = bool(cluster and enabled["decode_cluster"])
    if _cluster_state.get(hd) != want:
        lib.call("hos_attn_decode_cluster", 1 if want else 0)
        _cluster_state[hd] = want
    if n_splits is None:
        n_splits, by_length = plan(hd, n_tokens, n_heads, nkv, max_len, window, min_live, _fits(hd, n_heads, nkv) if want else None,
                                   max_live, fill, consumer_groups)
    ws = tickets = None
    if n_splits == 0:            # even shares: every CTA the same number of pages, two places per CTA for what is cut
        f = lib.lib.hos_attn_decode_even_workspace
        f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_int, ctypes.c_int]
        ws = torch.empty(int(f(n_heads, nkv)), dtype=torch.float32, device=q.device)
    elif n_splits > 1:
        ws = torch.empty(n_tokens * n_heads * n_splits * (hd + 2), dtype=torch.float32, device=q.device)
    if n_splits != 1:
        tickets = _tickets(q.device, n_tokens * nkv * ((n_heads // nkv + 15) // 16))
    lib.call("hos_attn_decode", ops._ptr(q), q_stride, ops._ptr(out), out.shape[1], ops._ptr(ws),
             ops._ptr(tickets), ops._ptr(token_pos), ops._ptr(token_seq), ops._ptr(seq_slot), ops._ptr(token_slot),
             ops._ptr(cache.k_pages),
             ops._ptr(cache.v_pages), ops._ptr(cache.page_table), cache.table_stride, cache.ring_pages,
             n_tokens, n_heads, nkv, hd, float(scale), float(cap), int(window) if window else 0,
             int(n_splits), int(max_new) if max_new else 1 << 30, int(by_length), ops._stream())
    # one or two sequences' worth of CTAs leave most SMs free: the product after this kernel may be placed beside it
    ctas = ops.sm_count() if n_splits == 0 else n_tokens * nkv * ((n_heads // nkv + 15) // 16) * n_splits
    ops.note_room_left(2 * ctas <= ops.sm_count())


def decode_gave_up(head_dim: int) -> bool:
    """True if a launch since the last call left a bounded wait unfinished (synchronises)."""
    lib = lib_for(head_dim)
    f = lib.lib.hos_attn_decode_error
    f.restype = ctypes.c_int
    f.argtypes = []
    return bool(f())


def has_tc_prefill(head_dim: int) -> bool:
    f = lib_for(head_dim).lib.hos_attn_prefill_tc_available
    f.restype, f.argtypes = ctypes.c_int, []
    return bool(f())


def prompt_blocks(step, block: int):
    """(sequences, blocks of `block` queries) a prompt kernel's grid has to cover.  From the host's
    lists when the step has them; for a replayed step an upper bound (the kernels skip blocks
    beyond the sequences' real ends, which they read on the device)."""
    if step.replayed or not step.cu_host:
        return step.n_seqs, (step.n_tokens + block - 1) // block + step.n_seqs
    cu = step.cu_host
    return len(cu) - 1, sum((cu[i + 1] - cu[i] + block - 1) // block for i in range(len(cu) - 1))


PAIR_KEYS = 128             # keys of a tile of the pair kernel
MAX_SHARES = 8
SHARE_MIN_TILES = 2
# What a walk costs besides its tiles, and what cut walks cost besides theirs, in tiles of 2.2 us (head size 256): set-up and epilogue
# 5 to 8 us, partial sums written, read and merged 5.  Fits the times beside the kernel.
SHARE_TILES_FIXED, SHARE_TILES_MERGE = 3.0, 2.5


def cut_walks(tiles, pairs_per_block: int, pairs: int):
    """(shares, tiles of a share) for blocks of queries whose walks over the keys are `tiles` long (tiles of PAIR_KEYS keys), each
    walked by `pairs_per_block` pairs of SMs out of `pairs` at a time: (1, 0) where the walks stay whole.  A walk of n tiles is cut
    into min(shares, ceil(n / tiles of a share)) parts.  The estimate, in tiles: a part costs its tiles and a fixed part, cut
    walks a merge; parts that do not run at once share the pairs evenly, and end raggedly by half a part."""
    tiles = np.asarray(tiles, dtype=np.int64)
    longest = int(tiles.max()) if tiles.size else 0
    if longest < 2 * SHARE_MIN_TILES or tiles.size * pairs_per_block >= 2 * pairs:
        return 1, 0
    best, best_cost = (1, 0), None
    for shares in range(1, MAX_SHARES + 1):
        length = -(-longest // shares)
        if shares > 1 and length < SHARE_MIN_TILES:
            break
        parts = np.minimum(shares, -(-tiles // length))
        most = int((-(-tiles // parts)).max())
        n = int(parts.sum()) * pairs_per_block
        cost = most + SHARE_TILES_FIXED
        if n > pairs:
            cost = max(cost, (int(tiles.sum()) * pairs_per_block + SHARE_TILES_FIXED * n) / pairs + 0.5 * most)
        if shares > 1:
            cost += SHARE_TILES_MERGE
        if best_cost is None or cost < 0.95 * best_cost:
            best, best_cost = ((shares, length) if shares > 1 else (1, 0)), cost
    return best


def on_one_sm(pages, tiles, pairs_per_block: int, pairs: int, shares: int, share_tiles: int) -> bool:
    """Whether blocks of queries whose walks over the keys are `pages` tiles of 64 keys long, or `tiles` of PAIR_KEYS, are done sooner by the
    kernel on one SM a block and head than by pairs of SMs with cut_walks' answer.  The estimate, us: a walk on one SM 5.0 and 1.33 a tile
    of 64 keys, on a pair 7.0 and 2.12 a tile of 128, in shares 3.7 and 1.2 a share more; walks that do not run at once as in cut_walks.
    Measured (B200, us one SM / pairs as planned): 17 tokens on top of 40, 8 heads of 256, 6.2 / 9.1, of 500 16.8 / 18.7, of 1,500 36.8 / 22.2; 32
    heads of 128 over 16, 739 tokens on top of 40 22.9 / 27.0, of 500 40.3 / 38.9.  Over 504 such pieces the choice takes 1.00 times the best;
    always pairs 1.06 times, up to 1.54."""
    pages, tiles = np.asarray(pages, dtype=np.int64), np.asarray(tiles, dtype=np.int64)
    if pages.size == 0:
        return False
    alone = 5.0 + 1.33 * int(pages.max())
    walks = 2 * pairs_per_block * pages.size
    if walks > 2 * pairs:
        alone = max(alone, (1.33 * 2 * pairs_per_block * int(pages.sum()) + 5.0 * walks) / (2 * pairs) + 0.55 * int(pages.max()))
    parts = np.minimum(shares, -(-tiles // share_tiles)) if shares > 1 else np.ones_like(tiles)
    longest, n = int((-(-tiles // parts)).max()), int(parts.sum()) * pairs_per_block
    paired = 7.0 + 2.12 * longest
    if n > pairs:
        paired = max(paired, (2.12 * int(tiles.sum()) * pairs_per_block + 7.0 * n) / pairs + 1.08 * longest)
    if int(parts.max()) > 1:
        paired += 3.7 + 1.2 * int(parts.max())
    return alone < paired


def _walk_plan(part, n_heads: int, n_kv_heads: int, head_dim: int, window):
    """(pairs of SMs, shares, tiles of a share) for the sequences of `part`, once per step and kind of layer: see cut_walks and on_one_sm."""
    _set_pairs(head_dim, enabled["prefill_pair"])
    pairs = _pairs_at_once(head_dim, n_heads, n_kv_heads, enabled["prefill_pair"])
    if pairs == 0:
        return False, 1, 0
    key = ("attention walks", part.row_offset, part.n_tokens, n_heads, head_dim, window)
    got = part.shared.get(key)
    if got is None:
        w = int(window) if window else 0
        pages, tiles = [], []
        if part.replayed or not part.cu_host:         # what the launches are planned for: every block as long as the longest
            _, blocks = prompt_blocks(part, 128)
            span, n = min(part.max_len_after, w + 127) if w else part.max_len_after, max(1, blocks - part.n_seqs + 1)
            pages, tiles = [-(-span // ops.PAGE_TOKENS)] * n, [-(-span // PAIR_KEYS)] * n
        else:
            starts = part.starts_host or [0] * (len(part.cu_host) - 1)
            for i, start in enumerate(starts):
                n = part.cu_host[i + 1] - part.cu_host[i]
                for q0 in range(0, n, 128):
                    first, last = max(0, start + q0 + 1 - w) if w else 0, start + min(n, q0 + 128) - 1
                    pages.append(last // ops.PAGE_TOKENS - first // ops.PAGE_TOKENS + 1)
                    tiles.append(last // PAIR_KEYS - first // PAIR_KEYS + 1)
        shares, share_tiles = cut_walks(tiles, n_heads // 2, pairs)
        got = (False, 1, 0) if on_one_sm(pages, tiles, n_heads // 2, pairs, shares, share_tiles) else (True, shares, share_tiles)
        part.shared[key] = got
    return got


@functools.lru_cache(maxsize=64)
def _pairs_at_once(head_dim: int, n_heads: int, n_kv_heads: int, on: bool) -> int:
    """How many pairs of SMs the pieces of these heads run on at once; 0: they do not (asked once per shape and state of the switch)."""
    f = lib_for(head_dim).lib.hos_attn_prefill_pairs
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_int]
    return int(f(n_heads, n_kv_heads))


def _share_workspace(blocks: int, n_heads: int, head_dim: int, shares: int, device):
    """What the shares of cut walks leave: unnormalised sums, and (maximum, sum of weights) pairs."""
    if shares <= 1:
        return None, None
    places = blocks * n_heads * shares * 128
    return (torch.empty(places * head_dim, dtype=torch.float32, device=device),
            torch.empty(places * 2, dtype=torch.float32, device=device))


def _set_pairs(head_dim: int, want: bool) -> None:
    if _pair_state.get(head_dim) != want:
        lib_for(head_dim).call("hos_attn_prefill_pair", 1 if want else 0)
        _pair_state[head_dim] = want


def prefill_tc(rows: torch.Tensor, out, cu_seqlens, n_seqs: int, blocks: int, n_heads, n_kv_heads, head_dim, scale, cap,
               window, pairs: bool = True, wait_cycles: int = 0, stop_tile: int = -1) -> None:
    """Attention of whole prompts from position 0 on the tcgen05 tensor cores; `rows` is the
    fused projection output [N, (n_heads + 2 n_kv_heads) * head_dim] (head sizes 64, 128, 256).
    `blocks`: at least the sum over sequences of ceil(length / 128).  `pairs`: two query heads that
    share their keys may run as one pair of SMs (head sizes 128 and 256, an even group).
    wait_cycles, stop_tile: for tests of a wait that runs out (the limit of the waits; the tile at which one does)."""
    lib = lib_for(head_dim)
    _set_pairs(head_dim, bool(pairs and enabled["prefill_pair"]))
    lib.call("hos_attn_prefill_tc", ops._ptr(rows), rows.shape[0], rows.shape[1], ops._ptr(out), out.shape[1],
             ops._ptr(cu_seqlens), n_seqs, blocks, n_heads, n_kv_heads, head_dim, float(scale), float(cap),
             int(window) if window else 0, int(wait_cycles), int(stop_tile), ops._stream())


def prefill_tc_gave_up(head_dim: int) -> bool:
    f = lib_for(head_dim).lib.hos_attn_prefill_tc_error
    f.restype, f.argtypes = ctypes.c_int, []
    return bool(f())


def prefill(q, q_stride, k_rows, v_rows, kv_stride, out, cu_seqlens, n_seqs: int, blocks: int, n_heads, n_kv_heads,
            head_dim, scale, cap, window) -> None:
    """Attention of whole prompts from position 0 over their own packed rows (mma.sync kernel).
    `blocks`: at least the sum over sequences of ceil(length / 64)."""
    lib = lib_for(head_dim)
    lib.call("hos_attn_prefill", ops._ptr(q), q_stride, ops._ptr(k_rows), ops._ptr(v_rows), kv_stride,
             ops._ptr(out), out.shape[1], ops._ptr(cu_seqlens), n_seqs, blocks, n_heads, n_kv_heads, head_dim,
             float(scale), float(cap), int(window) if window else 0, ops._stream())


def chunk(q, q_stride, out, cu_seqlens, row_base: int, token_pos, seq_slot, n_seqs: int, blocks: int,
          cache: ops.PagedKVArgs, n_heads, scale, cap, window) -> None:
    """Attention of sequences that go on by many tokens over the paged cache (which holds the step's
    own keys already): sequence s has the rows cu_seqlens[s] - row_base .. of q and out, at consecutive
    positions from token_pos[its first row], and the page-table row seq_slot[s].  `blocks`: at least the
    sum over sequences of ceil(rows / 64)."""
    lib = lib_for(cache.head_dim)
    lib.call("hos_attn_chunk", ops._ptr(q), q_stride, ops._ptr(out), out.shape[1], ops._ptr(cu_seqlens), int(row_base),
             ops._ptr(token_pos), ops._ptr(seq_slot), n_seqs, blocks, ops._ptr(cache.k_pages), ops._ptr(cache.v_pages),
             ops._ptr(cache.page_table), cache.table_stride, cache.ring_pages, n_heads, cache.n_kv_heads,
             cache.head_dim, float(scale), float(cap), int(window) if window else 0, ops._stream())


def chunk_tc(q, out, cu_seqlens, row_base: int, token_pos, seq_slot, n_seqs: int, blocks: int,
             cache: ops.PagedKVArgs, n_heads, scale, cap, window, pairs: bool = True, shares: int = 1, share_tiles: int = 0) -> None:
    """As `chunk`, on the tcgen05 tensor cores (head sizes 64, 128, 256): q is [rows, stride] with the q heads
    first in a row; `blocks`: at least the sum over sequences of ceil(rows / 128); pairs: as prefill_tc's, False: one SM a block and head; shares,
    share_tiles: pairs of SMs walk over a block's keys in up to that many parts of about that many tiles (see cut_walks)."""
    lib = lib_for(cache.head_dim)
    _set_pairs(cache.head_dim, enabled["prefill_pair"])
    shares = max(1, int(shares)) if pairs else 0
    part_o, part_ml = _share_workspace(blocks, n_heads, cache.head_dim, shares, q.device)
    lib.call("hos_attn_chunk_tc", ops._ptr(q), q.shape[0], q.shape[1], ops._ptr(out), out.shape[1], ops._ptr(cu_seqlens),
             int(row_base), ops._ptr(token_pos), ops._ptr(seq_slot), n_seqs, blocks, ops._ptr(cache.k_pages),
             ops._ptr(cache.v_pages), cache.k_pages.shape[0], ops._ptr(cache.page_table), cache.table_stride,
             cache.ring_pages, n_heads, cache.n_kv_heads, cache.head_dim, float(scale), float(cap),
             int(window) if window else 0, int(shares), int(share_tiles), ops._ptr(part_o), ops._ptr(part_ml), ops._stream())


def attend_chunks(mixer, qkv, att, part, cache) -> bool:
    """The rows of `part` (sequences of a step that go on by many tokens; see StepInfo.rows) through
    a chunk kernel (the tcgen05 one where the head size has it); False if none takes the case."""
    if cache.k_pages.dtype != torch.bfloat16 or not supports(mixer.head_dim) or not enabled["chunk"]:
        return False
    if part.replayed:
        att.zero_()                          # which rows are padding is known on the device only: a defined output
    elif not part.cu_host:
        return False
    slots = part.seq_slot[part.seq_offset:]
    if enabled["chunk_tc"] and qkv.is_contiguous() and has_tc_prefill(mixer.head_dim):
        _, blocks = prompt_blocks(part, 128)
        pairs, shares, share_tiles = _walk_plan(part, mixer.n_heads, mixer.n_kv_heads, mixer.head_dim, mixer.window)
        chunk_tc(qkv, att, part.cu_seqlens, part.row_offset, part.token_pos, slots, part.n_seqs, blocks, cache,
                 mixer.n_heads, mixer.scale, mixer.softcap, mixer.window, pairs=pairs, shares=shares, share_tiles=share_tiles)
        return True
    _, blocks = prompt_blocks(part, 64)
    chunk(qkv, qkv.shape[1], att, part.cu_seqlens, part.row_offset, part.token_pos, slots, part.n_seqs, blocks, cache,
          mixer.n_heads, mixer.scale, mixer.softcap, mixer.window)
    return True


def attend(mixer, qkv, att, step, cache, packed: bool) -> bool:
    """Runs the tensor-core kernel if it takes the case; False hands it to the plain kernel."""
    if cache.k_pages.dtype != torch.bfloat16 or not supports(mixer.head_dim):
        return False
    if packed:
        if not enabled["prefill"]:
            return False
        if step.replayed or not step.cu_host:
            att.zero_()                          # which rows are padding is known on the device only
        elif step.n_tokens > step.cu_host[-1]:
            att[step.cu_host[-1]:].zero_()       # padding rows: a defined output
        if enabled["prefill_tc"] and qkv.is_contiguous() and has_tc_prefill(mixer.head_dim):
            n_seqs, blocks = prompt_blocks(step, 128)
            prefill_tc(qkv, att, step.cu_seqlens, n_seqs, blocks, mixer.n_heads, mixer.n_kv_heads, mixer.head_dim,
                       mixer.scale, mixer.softcap, mixer.window)
            return True
        n_seqs, blocks = prompt_blocks(step, 64)
        prefill(qkv, qkv.shape[1], qkv[:, mixer.q_dim:], qkv[:, mixer.q_dim + mixer.kv_dim:], qkv.shape[1],
                att, step.cu_seqlens, n_seqs, blocks, mixer.n_heads, mixer.n_kv_heads, mixer.head_dim,
                mixer.scale, mixer.softcap, mixer.window)
        return True
    if not enabled["decode"]:
        return False
    decode(qkv, qkv.shape[1], att, step.token_pos, step.token_seq, step.seq_slot, cache, step.n_tokens,
           mixer.n_heads, mixer.scale, mixer.softcap, mixer.window, step.max_len_after, max_new=step.max_new,
           min_live=getattr(step, "min_live", 0), token_slot=getattr(step, "token_slot", None),
           max_live=getattr(step, "max_live", 0),
           fill=step.fill_for(mixer.window) if hasattr(step, "fill_for") else 1.0)
    return True

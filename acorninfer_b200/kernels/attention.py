"""Choice of the attention kernel for a step, behind one call.

The float32 engine runs its own prefill and decode kernels (head sizes 64 and 128, causal masks with or without a
window) and the plain kernel for everything else.  The bfloat16 engine runs the split-K
decode kernel when every row of the step is a single token, the tensor-core prefill kernel
otherwise (a single-token row is then a tile of one query), and the plain kernel for head
sizes and group sizes the fast kernels do not take.
"""

from __future__ import annotations

from functools import lru_cache

import numpy as np
import torch

from . import ops

B200_SMS = 148          # what planning functions assume when no device is given (CPU-side tests)
_CHUNK = 64

Q_TILE = 64             # query tokens per tile of the mma.sync prefill kernel
TILE_LARGE = 128        # query tokens per tile of the tcgen05 prefill kernel
LARGE_MIN = 32          # rows shorter than this stay with the small-tile kernel


def _tiles(plan, lo: int, hi: int | None, tile: int) -> np.ndarray:
    """(row, first token within the row) of every ``tile``-token query tile of the rows that bring
    lo <= n (< hi) tokens."""
    t = [(r, q0) for r, n in enumerate(plan.row_lens) if n >= lo and (hi is None or n < hi)
         for q0 in range(0, n, tile)]
    return np.asarray(t, np.int32).reshape(-1, 2)


def _single_tokens(plan) -> np.ndarray:
    return np.asarray([int(plan.row_start[r]) for r, n in enumerate(plan.row_lens) if n == 1], np.int32)


def _large_tiles(plan) -> np.ndarray:
    """Tiles of the tcgen05 kernel, longest first: a tile's work grows with the keys before its
    last query (the row's cached length plus the tile's end), and CTAs are handed out in list
    order, so the long ones start first and the short ones fill the tail of the last wave."""
    t = _tiles(plan, LARGE_MIN, None, TILE_LARGE)
    if t.shape[0] > 1:
        keys = plan.row_pos[t[:, 0]] + np.minimum(t[:, 1] + TILE_LARGE, np.asarray(plan.row_lens, np.int32)[t[:, 0]])
        t = t[np.argsort(-keys, kind="stable")]
    return np.ascontiguousarray(t)


# The per-step arrays the attention kernels read (``Part.step_arrays``): rows of one token go to the
# decode kernel by token list, longer rows to a prefill kernel in query tiles.
STEP_ARRAYS = {
    "attention.single_tokens": _single_tokens,
    "attention.q_tiles": lambda plan: _tiles(plan, 2, None, Q_TILE),
    "attention.q_tiles_large": _large_tiles,
    "attention.q_tiles_small": lambda plan: _tiles(plan, 2, LARGE_MIN, Q_TILE),
}

sm_count = ops.device_sms


# What the split choice assumes of the decode kernel on this GPU (measured: 10 to 128 rows of 8 kv
# heads at contexts 1,024 to 16,384, 1 to 8 splits each): one CTA streams its keys and values at
# about 35 GB/s at most (three stages of 32 KB in flight), all CTAs together at the memory's 6.5
# TB/s, a wave of CTAs costs about 2 us beyond its streaming, the merge pass about 3 us.
_CTA_GBS, _HBM_GBS, _WAVE_US, _MERGE_US = 35.0, 6500.0, 2.0, 3.0


def merged_in_kernel(splits: int, limit: int) -> bool:
    """Whether a decode kernel that merges up to ``limit`` splits inside itself (a cluster) does so for
    this many: clusters of up to 8 CTAs, and of 16; sizes between (9 splits took 24 us where the
    separate merge pass took 17) are left to the merge pass."""
    return splits <= min(limit, 8) or (splits == 16 and limit >= 16)


@lru_cache(maxsize=4096)        # asked by every layer of a step, with the same sizes
def decode_splits(rows: int, num_kv_heads: int, key_bound: int, head_dim: int, num_sms: int = B200_SMS) -> int:
    """Splits of the key range for the decode kernels that end in a merge pass (``decode_plan`` has the TMA kernel's).
    ``key_bound`` bounds the keys any row reads; it changes only with the table stride, so a captured step keeps its grid.

    Two CTAs of the decode kernel fit on an SM: ``2 * num_sms`` (296 on a B200) run at a time, in waves.  A CTA is bound by
    its own streaming rate, a full wave by the memory.  So few (row, kv head) pairs want many
    splits (more CTAs in flight); a count just above a multiple of 296 wants splits too (a last
    wave of few long CTAs takes as long as one CTA takes alone); a count that fills its last wave well wants
    none.  The splits with the least estimated time are taken."""
    _TARGET_CTAS = 2 * num_sms
    pairs = max(1, rows * num_kv_heads)
    most = max(1, min(-(-key_bound // _CHUNK), 32))
    pair_kb = key_bound * head_dim * 4 / 1e3                         # K and V of one pair, bfloat16, in KB
    best, best_us = 1, None
    for s in range(1, most + 1):
        kb = pair_kb / s
        alone_us = kb / _CTA_GBS                                     # KB / (GB/s) = us
        full, rest = divmod(pairs * s, _TARGET_CTAS)
        us = full * (max(alone_us, _TARGET_CTAS * kb / _HBM_GBS) + _WAVE_US)
        if rest:
            us += max(alone_us, rest * kb / _HBM_GBS) + _WAVE_US
        if s > 1:
            us += _MERGE_US
        if best_us is None or us <= best_us + 1e-9:                  # equal estimates: more CTAs in flight
            best, best_us = s, us
    return best


# How the TMA decode kernel's launches share the work (measured: 1 to 90 rows of 8 kv heads and 40 to 90 of 4 at contexts of 300 to
# 16,384, equal and of 35 to 100 %, every number of splits).  Clusters run in one wave only as long as they fill no more than seven
# eighths of the CTAs that single ones would (5 rows of 900 keys: 6 splits, 240 CTAs, 9.1 us; 7 splits, 280 CTAs, 15.4; 12 rows: 2
# splits 13.9, 3 splits, 288 CTAs, 21.6), pairs of CTAs fill all of them, clusters of sixteen half.  At short contexts a second
# wave of clusters costs more than its splits bring (41 rows of 900: unsplit 43.7, 3 splits 50.7; of 1,700: 69 and 67; a step of 41
# rows of 600 to 1,700 keys at Qwen3-4B: 3,866 and 4,280 us).
_START_US, _CLUSTER_US = 3.5, 1.5
# From here on the keys of a row that is left whole take longer than another wave's start: ``_waves_us`` has the choice for more
# rows than two splits of each fit one wave.  40 rows of 8 kv heads, equal / ragged, us, whole and in the splits it takes: 4,096 keys
# 149 / 93 and 131 / 86 (2), 8,192 289 / 176 and 222 / 154 (3), 16,384 569 / 342 and 406 / 281 (4); 20 rows of 16,384 250 / 226 and
# 204 / 158 (3); 48 of 8,192 294 / 208 and 247 / 180 (2); 80 of 16,384 902 / 586 and 800 / 548 (2); 64 rows, which fill two waves
# well, stay whole (16,384 keys: 610 / 507, in 4 splits 650 / 441).  The table is a power of two of pages wide, so a bound of 4,096
# stands for contexts from 2,049 on: those of 2,500 gain less (40 rows 95 / 60 and 89 / 60) and lose at 76 rows (147 / 96 and 150 / 103).
_LONG_KEYS = 2048


def _wave(splits: int, num_sms: int) -> int:
    """CTAs that run at once where a (row, kv head) has so many."""
    return 2 * num_sms if splits <= 2 or splits > 16 else 2 * num_sms * 7 // 8 if splits <= 8 else num_sms


def _waves_us(pairs: int, keys: float, splits: int, num_sms: int) -> float:
    """Estimated time of the TMA decode kernel over several waves, fitted to the measurements above (2.3 % above the best choice on
    average): a lone CTA streams 40 GB/s and two on an SM 33 each, all together 6.8 TB/s; a wave's start takes 2 us, of clusters of
    three and more 6."""
    kb, wave, start = keys * 128 * 4 / 1e3 / splits, _wave(splits, num_sms), 2.0 if splits <= 2 else 6.0
    full, rest = divmod(pairs * splits, wave)
    us = full * (max(kb / 33.0, wave * kb / 6800.0) + start)
    return us + (max(kb / (40.0 if rest <= num_sms else 33.0), rest * kb / 6800.0) + start if rest else 0.0)


@lru_cache(maxsize=4096)
def decode_plan(rows: int, num_kv_heads: int, key_bound: int, num_sms: int = B200_SMS, merge_limit: int = 16) -> int:
    """Splits of the key range for the TMA decode kernel (head size 128, ``merge_limit`` splits merged inside it)."""
    pairs, wave = rows * num_kv_heads, 2 * num_sms
    most = max(1, -(-key_bound // _CHUNK))
    if key_bound > _LONG_KEYS and 2 * pairs > wave:
        # contexts are anywhere between half of the bound and all of it: the sum of two estimates
        return min(range(1, min(merge_limit, 8) + 1),
                   key=lambda s: (_waves_us(pairs, key_bound, s, num_sms) + _waves_us(pairs, 0.75 * key_bound, s, num_sms), s))
    if pairs > wave:
        return 1
    pair_kb = key_bound * 128 * 4 / 1e3                             # K and V of one pair, bfloat16, in KB
    best, best_us = 1, None
    for s in (1, 2, 3, 4, 5, 6, 7, 8, 16, 24, 32):
        if s > most or (s > 1 and pairs * s > _wave(s, num_sms)):
            continue
        us = _START_US + pair_kb / s / min(_CTA_GBS, _HBM_GBS / (pairs * s))
        if s > 1:
            us += _CLUSTER_US if merged_in_kernel(s, merge_limit) else _WAVE_US + _MERGE_US
        if best_us is None or us <= best_us + 1e-9:                  # equal estimates: more CTAs in flight
            best, best_us = s, us
    return best


_MERGE_FREE: dict = {}


def _merge_free(nq: int, nkv: int, d: int, P: int) -> int:
    """Splits that the decode kernel for these sizes merges itself (1: none)."""
    key = (nq, nkv, d, P)
    if key not in _MERGE_FREE:
        _MERGE_FREE[key] = (ops.lib().acorn_attention_decode_tma_merges(nq, nkv)
                            if ops.lib().acorn_attention_decode_tma_supported(nq, nkv, d, P) else 1)
    return _MERGE_FREE[key]


def choose_splits(rows: int, nq: int, nkv: int, d: int, P: int, key_bound: int, windowed_only: bool, num_sms: int) -> int:
    """Splits for the decode kernel that takes these sizes."""
    limit = _merge_free(nq, nkv, d, P) if windowed_only else 1
    # (a limit above 1: the TMA kernel takes them)
    return decode_plan(rows, nkv, key_bound, num_sms, limit) if limit > 1 else decode_splits(rows, nkv, key_bound, d, num_sms)


def _decode(qkv, inputs, group, cache, nq, nkv, d, P, scale, window, bound, n, windowed_only, mask, token_list=None, out=None):
    """The step's ``n`` single-token rows (``token_list``, or all tokens) on a decode kernel."""
    splits = choose_splits(n, nq, nkv, d, P, bound, windowed_only, sm_count(qkv.device))
    return ops.attention_decode(qkv, qkv.stride(0), cache.k_pages, cache.v_pages, group.block_table, group.page_base, inputs.token_row,
                                inputs.positions, inputs.num_tokens, nq, nkv, d, scale, window, splits, token_list=token_list, out=out,
                                **mask)


def _key_bound(table_keys: int, window: int | None, chunk: int | None, keep_first: int) -> int:
    """A bound on the keys any query of the step reads, from the table's width and the mask."""
    spans = [s for s in (window, chunk) if s]
    return min(table_keys, min(spans) + keep_first) if spans else table_keys


def paged_attention(qkv: torch.Tensor, inputs, group, cache, nq: int, nkv: int, d: int, scale: float,
                    window: int | None, chunk: int | None = None, keep_first: int = 0,
                    value_dim: int | None = None, slopes32: torch.Tensor | None = None,
                    q: torch.Tensor | None = None, sink32: torch.Tensor | None = None, softcap: float | None = None,
                    maps: int = 1) -> torch.Tensor:
    """Attention of all tokens of the step; q is the head of ``qkv`` ([T, >= nq d]).  ``window``, ``chunk``,
    ``keep_first``: which earlier keys a query reads (see ``parts/attention.py``); ``value_dim``: width of the
    value rows where it is not ``d``; ``slopes32`` (float32 [nq]): a penalty ``slope_h * distance to the key`` on
    the scores; ``q``: the queries where they are not the head of ``qkv`` ([T, >= nq d]).  The tensor-core kernels
    take values as wide as keys; the TMA decode kernel knows windows only.  ``sink32`` (float32 [nq]): a term
    ``exp(sink_h)`` in the softmax denominator; ``softcap`` c: the scaled score becomes ``c tanh(score / c)``; ``maps``
    n > 1: every head holds n score maps side by side and ``nq`` counts (head, map) pairs (see
    ``ops.attention_plain``).  The tcgen05 prefill kernel knows the sink and the cap and the TMA decode kernel none
    of the three: score maps run the mma.sync prefill kernel (unless the caller lays the pairs' queries out with
    zeros itself and passes ``maps`` 1), all three the cp.async split-K decode kernel."""
    if q is not None:
        qkv = q
    P = cache.k_pages.shape[2]
    scored = sink32 is not None or bool(softcap) or maps != 1           # what only some of the kernels know
    windowed_only = not chunk and not keep_first and slopes32 is None and not scored
    mask = {"chunk": chunk, "keep_first": keep_first, "slopes32": slopes32}
    if scored:
        mask.update(sink32=sink32, softcap=softcap, maps=maps)
    tc_mask = {"chunk": chunk, "keep_first": keep_first, "slopes32": slopes32, "sink32": sink32, "softcap": softcap}
    tc_knows = maps == 1 and not (softcap and slopes32 is not None) and scale > 0
    if qkv.dtype == torch.bfloat16 and (value_dim is None or value_dim == d):
        if inputs.plan.all_decode and ops.attention_decode_supported(nq, nkv, d) and inputs.num_tokens <= 65535:
            bound = _key_bound(group.block_table.shape[1] * P, window, chunk, keep_first)
            return _decode(qkv, inputs, group, cache, nq, nkv, d, P, scale, window, bound, inputs.num_rows, windowed_only, mask)
        x, hx = inputs.extra, inputs.plan.extra
        n_single = int(hx["attention.single_tokens"].size)
        if ops.attention_prefill_supported(nq, nkv, d) and (n_single == 0 or (
                ops.attention_decode_supported(nq, nkv, d) and n_single <= 65535)):
            # a mixed step: prompt portions through the prefill kernel, decoded tokens through the
            # decode kernel, both writing their rows of one output
            out = torch.empty((inputs.num_tokens, nq * d), dtype=qkv.dtype, device=qkv.device)
            if ops.attention_prefill_tc_supported(nq, nkv, d, P) and qkv.stride(0) % 8 == 0 and tc_knows:
                # long rows on the tcgen05 kernel (tiles of 128 queries), short ones on the mma.sync kernel
                if hx["attention.q_tiles_large"].shape[0]:
                    ops.attention_prefill_tc(qkv, qkv.stride(0), cache.k_pages, cache.v_pages, group.block_table,
                                             group.page_base, inputs.row_start, inputs.row_pos, x["attention.q_tiles_large"],
                                             inputs.num_tokens, nq, nkv, d, scale, window, out=out, **tc_mask)
                if hx["attention.q_tiles_small"].shape[0]:
                    ops.attention_prefill(qkv, qkv.stride(0), cache.k_pages, cache.v_pages, group.block_table,
                                          group.page_base, inputs.row_start, inputs.row_pos, x["attention.q_tiles_small"],
                                          inputs.num_tokens, nq, nkv, d, scale, window, out=out, **mask)
            elif hx["attention.q_tiles"].shape[0]:
                ops.attention_prefill(qkv, qkv.stride(0), cache.k_pages, cache.v_pages, group.block_table,
                                      group.page_base, inputs.row_start, inputs.row_pos, x["attention.q_tiles"],
                                      inputs.num_tokens, nq, nkv, d, scale, window, out=out, **mask)
            if n_single:
                bound = _key_bound(group.block_table.shape[1] * P, window, chunk, keep_first)
                _decode(qkv, inputs, group, cache, nq, nkv, d, P, scale, window, bound, n_single, windowed_only, mask,
                        token_list=x["attention.single_tokens"], out=out)
            return out
    if qkv.dtype == torch.float32 and (value_dim is None or value_dim == d) and windowed_only and cache.k_pages.shape == cache.v_pages.shape:
        # a row of one token goes to the decode kernel whatever else is in the step, so that its bits stay the same
        n_single = inputs.num_tokens if inputs.plan.all_decode else int(inputs.plan.extra["attention.single_tokens"].size)
        chunks = ops.f32_decode_chunks(_key_bound(group.block_table.shape[1] * P, window, None, 0), window)
        runs = ops.f32_prefill_chunks(group.block_table.shape[1] * P, window) if n_single < inputs.num_tokens else 0
        if n_single <= 65535 and ops.attention_f32_supported(nq, nkv, d, n_single, chunks, runs):
            out = torch.empty((inputs.num_tokens, nq * d), dtype=qkv.dtype, device=qkv.device)
            if n_single < inputs.num_tokens:
                ops.attention_f32_prefill(qkv, qkv.stride(0), cache.k_pages, cache.v_pages, group.block_table, group.page_base,
                                          inputs.row_start, inputs.row_pos, inputs.extra["attention.q_tiles"], nq, nkv, d, scale,
                                          window, runs, out)
            if n_single:
                ops.attention_f32_decode(qkv, qkv.stride(0), cache.k_pages, cache.v_pages, group.block_table, group.page_base,
                                         inputs.token_row, inputs.positions,
                                         None if inputs.plan.all_decode else inputs.extra["attention.single_tokens"], n_single, nq,
                                         nkv, d, scale, window, chunks, out)
            return out
    return ops.attention_plain(qkv, qkv.stride(0), cache.k_pages, cache.v_pages, group.block_table,
                               group.page_base, inputs.token_row, inputs.positions, inputs.num_tokens,
                               nq, nkv, d, scale, window, value_dim=value_dim, **mask)

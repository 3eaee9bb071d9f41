"""Chooses the attention kernels of a step.

float32: the CUDA-core kernel for every token (true 32-bit).  bfloat16: tensor-core kernels
where the sizes of keys and values are multiples of 16 — one launch for the sequences that bring one token
(keys split across CTAs when there are few sequences and long contexts) and one for the longer
portions, which takes the tcgen05 + TMA kernel when head and page size allow it and the
mma.sync kernel otherwise — and the CUDA-core kernel for any other head size.
"""

from __future__ import annotations

import torch

from . import ops

import functools


@functools.lru_cache(maxsize=None)
def sm_count() -> int:
    """SMs of the current CUDA device; without one (host-side tests) the B200's 148."""
    if torch.cuda.is_available():
        return int(torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count)
    return 148


def one_wave(ctas_per_sm: int) -> int:
    """CTAs resident at once: the mma.sync decode kernel holds two per SM in its few-sequences shape, the
    TMA-fed decode kernel four at head size 64 and two at head size 128."""
    return sm_count() * ctas_per_sm


MIN_TILES_PER_SPLIT = 2  # key tiles (of 64) a split should at least cover


CLUSTER_SPLITS_MAX = ops.DECODE_TMA_CLUSTER_SPLITS  # splits that the TMA decode kernel merges inside one thread-block cluster
# Splits of the TMA-fed kernel, measured on a B200 with the keys and values not in L2 (head size 64, 8 KV heads;
# us at 1 / 2 / 4 sequences):  8 K keys: 16 splits 15 / 21 / 35, 8 splits 23 / 25 / 27, 64 splits 30 / 36 / 48;
# 32 K keys: 16 splits 27 / 39 / 89, 8 splits 60 / 66 / 68, 32 splits 32 / 48 / 79;  one sequence of 128 K keys: 16
# splits 68, 32 splits 70.  A cluster's merge on the chip beats more splits with a merge kernel at every length a
# model here reaches; a cluster of 16 is worth its narrower placement only while the grid is small (one or two
# sequences' head groups).  (More than 16 splits, merged by a second kernel, remain for callers that ask for them.)
CLUSTER_16_MAX_CTAS_PER_SPLIT = 16


def choose_splits(num_seqs: int, ctas_per_seq: int, max_kv_len: int, wave: int | None = None, fill_last_wave: bool = True,
                  min_tiles: int | None = None) -> int:
    """Key splits for single-token sequences: as many as still fit the GPU in one wave (a second,
    partly filled wave costs more than the extra parallelism brings), none shorter than
    MIN_TILES_PER_SPLIT key tiles (the role of src/dli/model/paged_attention.py:63-74)."""
    wave = one_wave(2) if wave is None else wave
    pairs = max(1, num_seqs * ctas_per_seq)
    tiles = -(-max_kv_len // 64)
    most = max(1, tiles // (min_tiles or MIN_TILES_PER_SPLIT))
    if pairs <= wave:
        return max(1, min(wave // pairs, most))
    if not fill_last_wave:
        return 1
    # More CTAs than one wave holds even without splits: a few splits can still fill the last wave
    # (512 CTAs on 296 places leave the second wave 27 % empty; 2,048 fill seven waves to 99 %).  Each
    # split costs merging, so it has to buy three points of occupancy.  (Measured: the mma.sync
    # kernel at head size 128 gains a fifth at 64 sequences; the TMA-fed kernel loses, so it opts out.)
    def score(s: int) -> float:
        ctas = pairs * s
        return ctas / (-(-ctas // wave) * wave) - 0.03 * (s - 1)

    return max(range(1, min(4, most) + 1), key=score)


def _slab_kernels(head_dim: int, one_pool: bool) -> bool:
    """Whether the TMA-fed kernels may serve these rows (``ops.decode_tma_supported`` and its sister also look at the page size).
    They copy keys and values separately: where the values lie in the keys' rows (``one_pool``) they are only taken at the sizes
    that fill their slabs, and the mma.sync kernels, which then copy a row once, serve the rest."""
    return not one_pool or head_dim in (64, 128)


def decode_splits(num_seqs: int, num_heads: int, nkv: int, head_dim: int, page_size: int, max_kv_len: int, value_dim: int | None = None,
                  one_pool: bool = False) -> int:
    """Key splits of the decode kernel that will serve these sizes (``value_dim`` None: values as long as keys)."""
    ctas_per_seq = nkv * -(-(num_heads // nkv) // 16)
    value_dim = value_dim or head_dim
    tma = ops.decode_tma_supported(head_dim, page_size, value_dim) and _slab_kernels(head_dim, one_pool)
    wave = one_wave(4 if max(head_dim, value_dim) <= 64 else 2) if tma else one_wave(2)
    splits = choose_splits(num_seqs, ctas_per_seq, max_kv_len, wave, fill_last_wave=not tma)
    if tma and splits > 8:  # a cluster merges its splits on the chip: 16 of them for one or two sequences' head groups, else 8
        pairs = num_seqs * ctas_per_seq
        splits = CLUSTER_SPLITS_MAX if splits >= CLUSTER_SPLITS_MAX and pairs <= CLUSTER_16_MAX_CTAS_PER_SPLIT else 8
    elif tma:
        # The splits of a sequence are a cluster, and clusters of 3 or 6 CTAs run slower than the power of two below
        # them.  Measured in replayed graphs (us a launch, splits 2 / 3 / 4): 24 sequences at head size 64 and 2 K keys
        # 21.8 / 31.4 / 28.7, at 16 K keys 139 / 161 / 136; 12 sequences at head size 128 and 2 K keys 21.9 / 34.5 /
        # 29.5; 12 sequences at head size 64 with 4 / 6 splits 13.5 / 20.1.
        splits = 1 << (splits.bit_length() - 1)
    return splits


ONE_KEY_TILE = 64  # keys that one tile of the mma.sync kernels holds


def _portion_keys(batch) -> int:
    """The most keys that a portion of the step sees; where the step does not say, its longest sequence bounds it."""
    return getattr(batch, "max_kv_len_portion", 0) or batch.max_kv_len


def portions_pay_for_tiles_of_rows(batch) -> bool:
    """Whether portions over one pool of rows go to the tcgen05 kernel: from the second key tile of the mma.sync kernel on.  Measured (us, mma.sync /
    tcgen05, 16 heads, rows of 256): 2 tokens alone 9.3 / 9.9, 64 tokens 11.8 / 13.4, 16 portions of 16 tokens 11.9 / 14.0, 2 tokens behind 64 12.6 / 9.9,
    80 tokens 15.2 / 13.6, 128 tokens 16.0 / 13.9; 8 heads, rows of 192: 2 tokens 7.1 / 9.2, 2 behind 64 10.5 / 9.2."""
    return not 0 < _portion_keys(batch) <= ONE_KEY_TILE


def paged_attention(out: torch.Tensor, qkv: torch.Tensor, cache, batch, num_heads: int, scale: float, window: int | None,
                    splits: int | None = None, sink: float | torch.Tensor | None = None, softcap: float | None = None,
                    slopes: torch.Tensor | None = None, value_dim: int | None = None) -> None:
    """Attention of every token of the step over its sequence's pages.  ``splits``: key runs per single-token
    sequence, if the caller fixed them (a recorded graph); otherwise chosen from this step's shape.  ``sink``: the
    score of a term that is added to every softmax denominator and carries no value (None: no such term); a float32 tensor
    gives a score per query head.  ``softcap`` c: a score s (after the scale) becomes c tanh(s / c); ``slopes`` (float32, one per
    query head): then slopes[h] * (position - key position) is taken off (None: neither).  ``value_dim``: where keys and values are one pool, how many
    leading numbers of each head's output the caller reads (a kernel may leave the others as they are)."""
    group = batch.group(cache.group)
    _, nkv, _, d = cache.k.shape
    dv = cache.v.shape[3]  # a value's size may differ from a key's
    one_pool = cache.v.data_ptr() == cache.k.data_ptr()
    bend = {"softcap": softcap, "slopes": slopes} if softcap or slopes is not None else {}
    if out.dtype != torch.bfloat16 or not (ops.mma_head_dim_supported(d) and ops.mma_head_dim_supported(dv)):
        ops.paged_attention_simt(out, qkv, cache.k, cache.v, group.block_tables, batch.seq_of_token, batch.positions,
                                 num_heads, scale, window, sink, **bend)
        return
    singles, total = batch.num_single, batch.num_seqs
    if singles:
        tma = ops.decode_tma_supported(d, cache.page_size, dv) and _slab_kernels(d, one_pool)
        splits = splits or decode_splits(singles, num_heads, nkv, d, cache.page_size, batch.max_kv_len_single, dv, one_pool)
        scratch = None
        if splits > 1:
            rows = singles * num_heads
            scratch = (torch.empty(rows * splits * dv, dtype=torch.float32, device=out.device),
                       torch.empty(rows * splits * 2, dtype=torch.float32, device=out.device))
        kernel = ops.paged_decode_tma if tma else ops.paged_attention_mma
        args = (out, qkv, cache.k, cache.v, group.block_tables, batch.q_start, batch.kv_len, 0, singles) + (() if tma else (1,))
        kernel(*args, 0, num_heads, scale, window, splits, scratch, *((batch.max_kv_len_single,) if tma else ()), sink=sink, **bend)
    if total > singles and ops.prefill_tc_supported(d, cache.page_size, dv) and _slab_kernels(d, one_pool):
        ops.paged_prefill_tc(out, qkv, cache.k, cache.v, group.block_tables, batch.q_start, batch.kv_len, singles, total - singles,
                             batch.max_q_len, num_heads, scale, window, sink=sink, **bend)
    elif (total > singles and one_pool and not bend and ops.prefill_rows_supported(d, cache.page_size) and portions_pay_for_tiles_of_rows(batch)
          and (out.data_ptr() | qkv.data_ptr() | cache.k.data_ptr()) % 16 == 0):
        ops.paged_prefill_rows(out, qkv, cache.k, group.block_tables, batch.q_start, batch.kv_len, singles, total - singles, batch.max_q_len, num_heads, scale,
                               window, sink=sink, value_dim=value_dim if value_dim and value_dim % 8 == 0 else None)
    elif total > singles:
        ops.paged_attention_mma(out, qkv, cache.k, cache.v, group.block_tables, batch.q_start, batch.kv_len, singles,
                                total - singles, batch.max_q_len, singles, num_heads, scale, window, sink=sink, **bend)


def diff_portions_apart(batch, tokens: int, num_heads: int, nkv: int, window: int | None, keep_first: int) -> bool:
    """Whether the portions of a step of ``tokens`` rows of differential attention go to the tcgen05 kernel, single tokens following in a launch of their own, or everything to
    one launch of the mma.sync kernel.

    Estimates of both, us, fitted to 800 steps (16 and 32 heads on 4 and 8, 8 on 2, 16 on 16; with and without a window of 1,024; 0 to 64 single tokens
    at 200 to 3,000 keys; portions of 2 to 1,024 tokens behind 0 to 3,000).  One launch takes as long as its slowest part: 23 us for 1,000 keys of a
    single token, 13 to 53 of a portion (the more of its 64 rows are queries), more where CTAs queue.  Two launches add up: 12 us and 17 for
    1,000 keys, and behind them 11 us and some 5 for 1,000 keys.  The new kernel is taken where it promises 15 % or more: then 5 of the 800 steps took over 5 %
    longer than in one launch (29 % at most), with two launches throughout 359 did.  Measured, us, one / two launches: 2 tokens 6.1 / 12.1,
    64 tokens 16 / 14, 1,024 76 / 29; 24 single tokens at 200 keys beside 16 tokens 16 / 30, beside 512 behind 512 80 / 44; at 3,000 keys 82 / 65, 106 / 80."""
    singles, portions = batch.num_single, batch.num_seqs - batch.num_single
    tokens -= singles

    def seen(keys: int) -> float:  # thousands of keys that a query reads
        return (min(keys, window + keep_first + 64) if window else keys) / 1000

    group, sms = num_heads // nkv, sm_count()
    keys, single_keys = seen(_portion_keys(batch)), seen(batch.max_kv_len_single) if singles else 0.0
    rows = min(1.0, batch.max_q_len * group / 64)
    portion = 9 * rows + keys * (13 + 40 * rows) * max(1.0, nkv * max(portions, tokens * group / 64) / (1.3 * sms))
    one = 6 + max(portion, single_keys * 23 * max(1.0, singles * nkv / sms))
    two = 12 + keys * 17 * max(1.0, nkv * max(portions, tokens * group / 128) / sms) + (11 + single_keys * 20 * max(0.26, singles * nkv / sms) if singles else 0)
    return two <= 0.85 * one


def diff_singles_beside(batch, num_heads: int, nkv: int, window: int | None, keep_first: int) -> bool:
    """Whether the single tokens of a step go to the launch of its portions (``ops.paged_prefill_diff``), whose last CTAs they are, or to their own.

    Where the portions' last wave of CTAs leaves places for all of them they start when the last portion CTAs have started, and what they see beyond those takes the
    launch longer, 17 us for 1,000 keys.  A launch of their own and the merge of its partial results behind it take 11 us and 5 to 20 for 1,000 keys (both slopes as in
    ``diff_portions_apart``).  Measured, us, apart / beside, 16 heads on 4: 9 tokens at 1,500 keys (a window of 1,024) beside 1,535 behind 1,024 93 / 78, 24 at 3,000 beside 1,200 behind
    1,024 126 / 120, 1 at 1,000 beside 1,200 49 / 40, 2 at 1,500 beside 500 behind 512 48 / 38; 8 heads on 2: 1 at 8,000 beside 200 64 / 123, 40 at 8,000 beside 200 behind 1,024 166 / 181; 32 on
    8: 2 at 3,000 beside 200 behind 1,024 55 / 66.  Of 120 steps (1 to 64 tokens at 100 to 8,000 keys, 1 to 4 portions, windows of 512 and 1,024) none takes over 3 % longer for this rule than
    apart, and six that it keeps apart could save 3 to 20 %.  A recorded step (its portions have no lengths yet) keeps them apart."""
    singles, lens, starts = batch.num_single, getattr(batch, "q_lens", [])[batch.num_single :], getattr(batch, "starts", [])[batch.num_single :]
    if not lens or min(lens) < 1 or len(starts) != len(lens):
        return False

    def seen(keys: int) -> float:  # thousands of keys that a query reads
        return (min(keys, window + keep_first + 64) if window else keys) / 1000

    group, sms = num_heads // nkv, sm_count()
    heads = min(group, 128)  # of a CTA's rows
    wide = nkv * -(-group // heads)
    ctas = wide * sum(-(-q // (128 // heads)) for q in lens)
    if wide * singles > -ctas % sms:
        return False
    last = seen(max(q + before for q, before in zip(lens, starts))) if ctas <= sms else seen(min(starts))
    alone = seen(batch.max_kv_len_single)
    return 17 * (alone - last) <= 0.6 * (11 + alone * 20 * max(0.26, singles * nkv / sms))


def diff_attention(out: torch.Tensor, q: torch.Tensor, cache, batch, gate: torch.Tensor | None, num_heads: int, scale: float,
                   window: int | None, keep_first: int, lam: float, post: float, eps: float) -> None:
    """Differential attention of every token of the step over its sequence's pages (``ops.diff_attention_simt`` says what is
    computed).  bfloat16 with sizes that are multiples of 16: portions of maps of 64 go to a tcgen05 kernel where that pays (``diff_portions_apart``),
    everything else to the mma.sync kernel (portions and single tokens in one launch); float32 and any other size: the CUDA-core kernel."""
    group = batch.group(cache.group)
    if out.dtype == torch.bfloat16 and ops.diff_attention_tc_supported(cache.k.shape[3] // 2, cache.v.shape[3]):
        _, nkv, _, d2 = cache.k.shape
        vdim, singles, seqs, longest, seen = cache.v.shape[3], batch.num_single, batch.num_seqs, batch.max_q_len, batch.max_kv_len
        if (seqs > singles and ops.prefill_diff_supported(d2 // 2, vdim, cache.page_size) and diff_portions_apart(batch, q.shape[0], num_heads, nkv, window, keep_first)
                and (out.data_ptr() | q.data_ptr() | cache.k.data_ptr() | cache.v.data_ptr()) % 16 == 0):
            beside = singles if singles and diff_singles_beside(batch, num_heads, nkv, window, keep_first) else 0
            ops.paged_prefill_diff(out, q, cache.k, cache.v, group.block_tables, batch.q_start, batch.kv_len, singles, seqs - singles, longest, gate, num_heads,
                                   scale, window, keep_first, lam, post, eps, beside)
            if beside == singles:
                return
            seqs, longest, seen = singles, 1, batch.max_kv_len_single
        splits, scratch = 1, None
        if longest == 1 and out.is_cuda:  # few single tokens: their key tiles are divided between CTAs to fill the GPU
            seen = min(seen, window + keep_first + 64) if window else seen
            wave = one_wave(ops.diff_attention_tc_ctas_per_sm(d2 // 2, vdim))
            splits = choose_splits(seqs, nkv * -(-(num_heads // nkv) // 64), seen, wave, fill_last_wave=False, min_tiles=1)
            if splits > 1:
                scratch = torch.empty(ops.diff_attention_scratch(seqs, num_heads, vdim, splits), dtype=torch.float32, device=out.device)
        ops.diff_attention_tc(out, q, cache.k, cache.v, group.block_tables, batch.q_start, batch.kv_len, seqs, longest, gate, num_heads, scale, window,
                              keep_first, lam, post, eps, splits, scratch)
        return
    ops.diff_attention_simt(out, q, cache.k, cache.v, group.block_tables, batch.seq_of_token, batch.positions, gate, num_heads, scale,
                            window, keep_first, lam, post, eps)

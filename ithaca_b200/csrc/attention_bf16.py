"""Attention kernels of the bfloat16 path: one compiled module per head size.

``attention_bf16.cu`` is specialised at compile time for a head size; the module for the
size a model has is compiled the first time that model runs a step (a few seconds) and kept
beside the core library.
"""
from __future__ import annotations

import ctypes
from typing import Dict, Optional, Tuple

import torch

from . import build
from . import ops
from .ops import KernelError, _check, _ptr, _stream, sm_count

_vp, _i, _f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
_modules: Dict[tuple, ctypes.CDLL] = {}

# Modules with options, measured on B200 (head sizes 64 and 128, contexts 2k-8k, batches 8-64): a ring of 60 KB a block leaves room for
# enough blocks per SM; where heads stop early the blocks of a sequence are unequal, and chunks of at most 8 pages even them out.
OPTION_RING_KB, REACH_CHUNK_PAGES = 60, 8
DECODE_CHUNK_PAGES = 4        # default: a decode block covers 4 pages = 256 keys; chunks start at multiples of that


def decode_chunk_pages(n_seqs: int, n_heads: int, n_kv_heads: int, max_kv_len: int, page_size: int = 64,
                       n_sm: Optional[int] = None) -> int:
    """Pages per decode block.  Measured on B200 (head size 128, 8 kv heads, contexts 1k-16k, batches 1-64,
    chunks of 2-32 pages): the kernel is fastest with about two blocks per SM in ONE wave, so the pages of a
    sequence are cut into as many chunks as that allows, but into chunks of at least 4 pages (2 when even
    that leaves most SMs idle: set-up and merging per block cost about as much as reading two pages).  With
    more (sequence, kv head) groups than two per SM, or a count that would load the SMs unevenly, there
    are several waves anyway; a long chunk and a short rest then pack best (the short blocks of the last chunk
    start last and fill the tail).  Over 72 measured (batch, context) pairs the chunk picked here is within 1 % of
    the best one's time on average, 13 % at worst."""
    N_SM = n_sm if n_sm is not None else sm_count()
    groups = n_seqs * n_kv_heads * -(-(n_heads // n_kv_heads) // 16)
    pages = max(1, -(-max_kv_len // page_size))
    if groups <= N_SM or groups > 1.5 * N_SM and groups <= 2 * N_SM:
        # (between one and one and a half groups per SM a single wave would give some SMs two blocks and others one)
        n_chunks = max(1, (2 * N_SM) // groups)
        least = 4 if groups * -(-pages // 4) >= 128 else 2
        return min(pages, max(-(-pages // n_chunks), least))
    return -(-pages * 3 // 4) if pages <= 24 else 20


def decode_chunk_pages_uneven(pages, n_heads: int, n_kv_heads: int, chunk: int, n_sm: int) -> int:
    """Pages per decode block for sequences of so many ``pages`` each, ``chunk`` being what would suit them all as long as the longest.  Where they come
    to less than 85 % of that, blocks are fewer and longer than the SMs want.  Then the shortest chunk of up to 12 pages that makes at most three
    blocks per SM and 18 pieces of a sequence (more cost more to merge than they gain); where there are more blocks whatever the chunk, 12 pages if the
    sequences differ by more, and nothing shorter where there are so many sequences and kv heads that they fill the SMs anyway.
    us on B200, lengths between a quarter and all of the longest, ``chunk`` / this, 32 heads of 128 on 8 kv heads: 8 sequences up to 4,000 30.4 / 21.0, 16 of 3,000
    41.5 / 28.0, 10 of 6,000 53.7 / 34.3, 20 of 600 18.4 / 15.0, 3 of 8,000 24.2 / 23; 40 heads on 40: 3 of 8,000 97 / 65, 8 of 4,000 79 / 70; one of 8,000 beside 15 of
    500 74 / 26."""
    n, most, total = len(pages), max(pages), sum(pages)
    if n < 2 or total >= 0.85 * n * most:
        return chunk
    groups = n_kv_heads * -(-(n_heads // n_kv_heads) // 16)
    if n * groups > 2.4 * n_sm:
        return min(12, chunk) if total < 0.35 * n * most else chunk
    least = max(2, -(-most // 18))
    for c in range(least, max(13, least + 1)):
        if sum(-(-p // c) for p in pages) * groups <= 3 * n_sm:
            return c if c <= 0.8 * chunk else chunk
    return min(12, chunk) if total < 0.75 * n * most else chunk


def seen_pages(kv_len_bound: int, window: int, keep: int, page_size: int = 64) -> int:
    """The most pages a query of a sequence of up to ``kv_len_bound`` positions sees: all, or under a window (> 0) those of
    the first ``keep`` keys and those a window of that many keys can reach into."""
    pages = max(1, -(-kv_len_bound // page_size))
    if window <= 0:
        return pages
    return min(pages, -(-keep // page_size) + (window + page_size - 2) // page_size + 1)


def supported(head_dim: int) -> bool:
    return head_dim % 16 == 0 and 16 <= head_dim <= 256


def module(head_dim: int, slopes: bool = False, one_row: bool = False) -> ctypes.CDLL:
    """The module of a head size; ``slopes``: with a distance bias, ``one_row``: for pages whose rows are keys and values."""
    key = (head_dim, slopes, one_row)
    m = _modules.get(key)
    if m is None:
        m = build.load_library(*build.attention_module(head_dim, slopes, one_row))
        m.ik_attn_prefill.argtypes = [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _f, _f, _i, _i, _i, _vp, _vp, _vp, _f, _f, _i, _i, _i, _vp, _vp]
        m.ik_attn_prefill.restype = _i
        m.ik_attn_prefill_tc.argtypes = [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _f, _f, _i, _i, _i, _vp, _vp, _vp, _f, _f, _i, _i, _i, _vp, _vp]
        m.ik_attn_prefill_tc.restype = _i
        m.ik_attn_prefill_two_heads.argtypes = m.ik_attn_prefill_tc.argtypes
        m.ik_attn_prefill_two_heads.restype = _i
        m.ik_attn_decode.argtypes = [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _f, _f, _i, _i, _i, _vp, _vp, _vp, _f, _f, _i, _i, _i, _i, _i, _i,
                                     _vp, _vp]
        m.ik_attn_decode.restype = _i
        m.ik_attn_take_wait_record.argtypes = [_vp]
        m.ik_attn_take_wait_record.restype = _i
        if m.ik_attn_head_dim() != head_dim:
            raise KernelError("the attention module was compiled for another head size")
        _modules[key] = m
    return ops.timed(m)


def prefill(q: torch.Tensor, k_pages: torch.Tensor, v_pages: torch.Tensor, cu_seqlens: torch.Tensor,
            kv_lens: torch.Tensor, table: torch.Tensor, n_seqs: int, max_new: int, n_heads: int, scale: float,
            window: int, status: Optional[torch.Tensor], out: Optional[torch.Tensor] = None,
            kind: str = "auto", work: Optional[Tuple[int, int]] = None, softcap: float = 0.0, sink=False, keep: int = 0,
            key_scales: Optional[torch.Tensor] = None, slopes: Optional[torch.Tensor] = None, reach=None,
            two_heads: bool = False) -> torch.Tensor:
    """``kind``: "tc" = the tcgen05 kernel (head sizes 64 and 128), "two_heads" = the one with two heads a block, "mma" = the
    warp-level kernel, "auto" = tcgen05 where it applies (``two_heads``: with two heads a block where that kernel takes the call).  ``softcap``: scores become cap * tanh(score / cap) (0 = no cap).  ``sink``: the
    softmax's denominator counts one more key of score 0 that carries no value (True), or of a score per head (a float32
    tensor [n_heads], not scaled).  ``key_scales``: the pages' rows are keys and values (``v_pages`` None), and every score is
    multiplied by its key's number.  ``slopes`` [n_heads]: a score loses slope * distance, behind the cap.  ``reach`` = (norm, coef, every): no
    score in front of cap and bias is larger than norm * |1 + coef ln(floor((pos + 1) / every) + 1)| (every 0: than norm), so that keys
    the bias makes negligible need not be visited (None: nothing is known).  ``keep``: under a window the first ``keep`` keys stay visible."""
    n_pages, nkv, page_size, hd = k_pages.shape
    ops.check_score_extras(key_scales, slopes, k_pages, n_heads)
    m = module(hd, slopes is not None, key_scales is not None)
    if out is None:
        out = torch.empty_like(q)
    ways = [kind] if kind in ("tc", "two_heads") else []
    if kind == "auto" and hd in (64, 128):
        ways = ["two_heads", "tc"] if two_heads else ["tc"]
    for way in ways:
        ops._work(f"attention prefill tcgen05 {q.shape[0]}x{n_heads}", *(work or (0, 0)))
        st = (m.ik_attn_prefill_two_heads if way == "two_heads" else m.ik_attn_prefill_tc)(_ptr(q), _ptr(k_pages), _ptr(v_pages), _ptr(out), _ptr(cu_seqlens), _ptr(kv_lens),
                                  _ptr(table), table.stride(0), q.shape[0], n_seqs, max_new, n_heads, nkv, scale, softcap, window, keep,
                                  ops.sink_flag(sink), _ptr(ops.sink_values(sink, n_heads)), _ptr(key_scales), _ptr(slopes), *(reach or (0.0, 0.0, 0)), page_size, n_pages, _ptr(status), _stream())
        if st != -2:
            _check(st, "attention prefill (tcgen05)")
            return out
    if kind in ("tc", "two_heads"):
        raise KernelError("attention prefill (tcgen05): head size or alignment not supported")
    ops._work(f"attention prefill mma {q.shape[0]}x{n_heads}", *(work or (0, 0)))
    _check(m.ik_attn_prefill(_ptr(q), _ptr(k_pages), _ptr(v_pages), _ptr(out), _ptr(cu_seqlens), _ptr(kv_lens),
                             _ptr(table), table.stride(0), n_seqs, max_new, n_heads, nkv, scale, softcap, window, keep, ops.sink_flag(sink),
                             _ptr(ops.sink_values(sink, n_heads)), _ptr(key_scales), _ptr(slopes), *(reach or (0.0, 0.0, 0)), page_size, n_pages, _ptr(status), _stream()), "attention prefill")
    return out


# Per head size and kernel (one head a block, two): us of a block besides its keys (with a window: more), per step of 64 or 128 keys
# beside other blocks and alone, of a block whose tile a shorter sequence does not have, the share of a whole round that a last round
# of equal blocks costs, of a launch, and the share of the longest block that unequal sequences add.
_Ways = Tuple[float, float, float, float, float, float, float, float]
PREFILL_COSTS: Dict[int, Tuple[_Ways, _Ways]] = {
    64: ((4.75, 1.37, 1.028, 0.743, 1.64, 0.80, 4.31, 0.27), (7.04, 2.39, 1.722, 1.594, 0.90, 1.06, 3.65, 0.05)),
    128: ((6.04, 1.96, 1.086, 0.757, 1.56, 0.70, 4.58, 0.30), (8.51, 2.67, 2.051, 1.907, 0.74, 1.03, 2.63, 0.09))}


def two_heads_pay(n_new, kv_lens, n_heads: int, hd: int, window: int, n_sm: int) -> bool:
    """Whether the prompts of a step run two heads a block (prompts without options, an even number of heads per kv head).

    Such a block has an SM to itself; of those with one head an SM holds two, and there are twice as many.  So two heads pay where
    tiles of 128 queries see many keys, and lose where they see few (short prompts, windows) or where the last round of the SMs is nearly
    empty.  The times of both are estimated from the tiles that exist; the estimates' figures are fitted to measurements, 5 to 7 % off.
    Measured on B200 (us, one head / two; 32 heads on 8), heads of 128 and of 64: one prompt of 1,024 23 / 27 and 21 / 23, of 2,048 52 / 49 and
    49 / 42, of 4,096 148 / 143 and 134 / 121; 24 of 100 28 / 33 and 25 / 29, 64 of 130 124 / 168 and 104 / 139, eight of 1,000 114 / 128 and
    98 / 105, six of 50 to 2,000 134 / 118 and 112 / 92; 4,096 under a window of 128 52 / 63 and 45 / 56, of 1,024 94 / 97 and 84 / 85;
    512 behind 3,000 54 / 66 and 51 / 57."""
    counts = {}                                                     # tiles by the pages they see
    n_tiles = most = 0
    for n, e in zip(n_new, kv_lens):
        most = max(most, -(-n // 128))
        for lo in range(e - n, e, 128):
            pages = (min(lo + 128, e) - 1) // 64 - (max(0, lo + 1 - window) // 64 if window else 0) + 1
            counts[pages] = counts.get(pages, 0) + 1
            n_tiles += 1
    if not n_tiles:
        return False
    missing = most * len(n_new) - n_tiles

    def time(heads, slots, step_pages, costs):
        base, windowed, step, alone, none, last, launch, uneven = costs
        base += windowed if window else 0.0
        mean = base + step * sum(-(-p // step_pages) * c for p, c in counts.items()) / n_tiles
        top = -(-max(counts) // step_pages)
        longest = base + alone * top
        rounds = n_tiles * heads / slots
        us = longest
        if n_tiles * heads > n_sm:
            us = max(longest, mean * (rounds + last * (mean / (base + step * top)) ** 3 * (-(-n_tiles * heads // slots) - rounds)))
        return us + none * heads * missing / slots + uneven * longest * min(1.0, 2.5 * missing / n_tiles) + launch

    # near a tie two heads of 64 come out 2 % too cheap, and two of 128 4 % too dear for a prompt alone
    one, two = PREFILL_COSTS[hd]
    return time(n_heads // 2, n_sm, 2, two) < (0.98 if hd == 64 else 1.04 if len(n_new) == 1 else 1.0) * time(n_heads, 2 * n_sm, 1, one)


def _two_heads_of(ctx, n_heads: int, hd: int, window: int) -> bool:
    """``two_heads_pay`` of a step, once for all its layers of one kind."""
    key = ("two_heads_pay", n_heads, hd, window)
    if key not in ctx.shared:
        ctx.shared[key] = two_heads_pay(ctx.host_n_new, ctx.host_kv_lens, n_heads, hd, window, ops.sm_count())
    return ctx.shared[key]


def decode(q: torch.Tensor, k_pages: torch.Tensor, v_pages: torch.Tensor, kv_lens: torch.Tensor, table: torch.Tensor,
           n_seqs: int, kv_len_bound: int, n_heads: int, scale: float, window: int, status: Optional[torch.Tensor],
           out: Optional[torch.Tensor] = None, chunk_pages: int = DECODE_CHUNK_PAGES, ring_kb: int = 0,
           work: Optional[Tuple[int, int]] = None, softcap: float = 0.0, sink=False, keep: int = 0,
            key_scales: Optional[torch.Tensor] = None, slopes: Optional[torch.Tensor] = None, reach=None) -> torch.Tensor:
    """``kv_len_bound``: no sequence of the step is longer than this (it sizes the grid and the
    scratch for the partial results; blocks beyond a sequence's length return at once).  ``keep``: under a window the
    first ``keep`` keys stay visible."""
    n_pages, nkv, page_size, hd = k_pages.shape
    ops.check_score_extras(key_scales, slopes, k_pages, n_heads)
    m = module(hd, slopes is not None, key_scales is not None)
    n_splits = max(1, -(-seen_pages(kv_len_bound, window, keep, page_size) // chunk_pages))
    part_o = torch.empty((n_seqs, n_heads, n_splits, hd), dtype=torch.float32, device=q.device)
    part_ml = torch.empty((n_seqs, n_heads, n_splits, 2), dtype=torch.float32, device=q.device)
    if out is None:
        out = torch.empty_like(q)
    ops._work(f"attention decode {n_seqs}x{n_heads}", *(work or (0, 0)))
    _check(m.ik_attn_decode(_ptr(q), _ptr(k_pages), _ptr(v_pages), _ptr(out), _ptr(part_o), _ptr(part_ml),
                            _ptr(kv_lens), _ptr(table), table.stride(0), n_seqs, n_heads, nkv, scale, softcap, window, keep,
                            ops.sink_flag(sink), _ptr(ops.sink_values(sink, n_heads)), _ptr(key_scales), _ptr(slopes), *(reach or (0.0, 0.0, 0)), page_size, n_pages, chunk_pages, n_splits, ring_kb,
                            _ptr(status), _stream()), "attention decode", kernels=2)
    return out


def attend(q, k_pages, v_pages, ctx, table, n_heads: int, scale: float, window: int,
           status, softcap: float = 0.0, sink=False, keep: int = 0,
            key_scales: Optional[torch.Tensor] = None, slopes: Optional[torch.Tensor] = None, reach=None) -> Optional[torch.Tensor]:
    """Returns None when no specialised kernel takes these sizes or options (the caller then uses the
    CUDA-core kernel)."""
    n_pages, nkv, page_size, hd = k_pages.shape
    if k_pages.dtype != torch.bfloat16 or q.dtype != torch.bfloat16 or page_size != 64 or not supported(hd):
        return None
    work = None
    if ops.profiling():
        # (query, key) pairs under the causal mask (and the window), from the host's copy of the lengths
        pairs = 0
        for n, end in zip(ctx.host_n_new, ctx.host_kv_lens):
            for p in range(end - n, end):
                pairs += min(p + 1, window + keep) if window else p + 1
        keys = sum(min(e, window + keep + n) if window else e for n, e in zip(ctx.host_n_new, ctx.host_kv_lens))
        rows = hd * 2 + 4 if key_scales is not None else 2 * hd * 2             # bytes of a key (and value) per kv head
        work = (2 * q.numel() * 2 + keys * nkv * rows, 4 * hd * n_heads * pairs)
    if ctx.is_decode:
        # from the bound; the single lengths have a say only where the step is not captured: a graph is replayed for other lengths
        chunk = decode_chunk_pages(ctx.n_seqs, n_heads, nkv, seen_pages(ctx.kv_len_bound, window, keep, page_size) * page_size, page_size)
        if len(ctx.host_kv_lens) == ctx.n_seqs > 1 and not getattr(ctx, "replayed", False):
            key = ("decode_chunk", n_heads, nkv, window, keep, page_size)              # once for all layers of a kind
            if key not in ctx.shared:
                ctx.shared[key] = decode_chunk_pages_uneven([seen_pages(e, window, keep, page_size) for e in ctx.host_kv_lens], n_heads, nkv, chunk, sm_count())
            chunk = ctx.shared[key]
        options = {}
        if key_scales is not None or slopes is not None:
            options["ring_kb"] = OPTION_RING_KB
        if reach is not None:
            chunk = min(chunk, REACH_CHUNK_PAGES)
        return decode(q, k_pages, v_pages, ctx.kv_lens, table, ctx.n_seqs, ctx.kv_len_bound, n_heads, scale, window,
                      status, chunk_pages=chunk, work=work, **options, softcap=softcap, sink=sink, keep=keep, key_scales=key_scales, slopes=slopes, reach=reach)
    plain = hd in (64, 128) and key_scales is None and slopes is None and not softcap and not ops.sink_flag(sink) and not keep and n_heads // nkv % 2 == 0
    return prefill(q, k_pages, v_pages, ctx.cu_seqlens, ctx.kv_lens, table, ctx.n_seqs, ctx.max_new, n_heads, scale,
                   window, status, work=work, softcap=softcap, sink=sink, keep=keep, key_scales=key_scales, slopes=slopes, reach=reach,
                   two_heads=plain and _two_heads_of(ctx, n_heads, hd, int(window or 0)))

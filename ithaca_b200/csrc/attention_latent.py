"""Attention over bfloat16 key rows that carry their own values (a latent that is key and value at once): one compiled
module per (row size, value size).

``attention_latent.cu`` makes the query heads of a key/value group the rows of its tensor-core tile, so a cached row is
read once for all of them.  The module for the sizes a model has is compiled the first time that model runs a step.
"""
from __future__ import annotations

import ctypes
from typing import Dict, Optional, Tuple

import torch

from . import build
from . import ops
from .ops import KernelError, _check, _ptr, _stream, sm_count

_vp, _i, _f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
_modules: Dict[Tuple[int, int], ctypes.CDLL] = {}

ROWS = 32                     # (token, head) rows of a block
SMEM_LIMIT = 227 * 1024


def supported(row_size: int, value_size: int) -> bool:
    """Rows in multiples of 16, values in multiples of 64 (four column groups of whole 16-wide tiles), and two pages,
    the queries and the weights must fit into a block's shared memory."""
    if row_size % 16 or value_size % 64 or not 64 <= value_size <= row_size:
        return False
    ld = row_size + 8
    return (ROWS * ld + 2 * 64 * ld + ROWS * 72) * 2 + 512 <= SMEM_LIMIT


def module(row_size: int, value_size: int) -> ctypes.CDLL:
    key = (row_size, value_size)
    m = _modules.get(key)
    if m is None:
        m = build.load_library(f"ithaca_attn_latent_{row_size}_{value_size}", ["attention_latent.cu"],
                               defines=[f"IK_HD={row_size}", f"IK_HDV={value_size}"])
        m.ik_attn_latent.argtypes = [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _f, _i, _i, _i, _i, _i, _i, _vp, _vp]
        m.ik_attn_latent.restype = _i
        if m.ik_attn_latent_rows() != ROWS:
            raise KernelError("the latent attention module was compiled for another tile")
        _modules[key] = m
    return ops.timed(m)


def splits_for(n_blocks: int, pages: int, n_sm: Optional[int] = None) -> Tuple[int, int]:
    """(pages per split, splits) for blocks that would each walk ``pages`` pages: about two blocks per SM when the
    step has fewer, in runs of at least two pages."""
    n_sm = n_sm if n_sm is not None else sm_count()
    want = max(1, (2 * n_sm) // max(n_blocks, 1))
    chunk = max(2, -(-pages // want))
    if chunk >= pages:
        return pages, 1
    return chunk, -(-pages // chunk)


def attend(q: torch.Tensor, k_pages: torch.Tensor, ctx, table: torch.Tensor, n_heads: int, scale: float, window: int,
           status: Optional[torch.Tensor], value_size: int, sink: bool = False) -> Optional[torch.Tensor]:
    """q [T, n_heads * row size] against the rows of ``k_pages`` [pages, kv heads, 64, row size]; a row's leading
    ``value_size`` columns are its value.  Returns [T, n_heads * value_size], or None when the kernel does not take
    these sizes or types (the caller then uses the CUDA-core kernel)."""
    n_pages, nkv, page_size, hd = k_pages.shape
    if k_pages.dtype != torch.bfloat16 or q.dtype != torch.bfloat16 or page_size != 64 or not supported(hd, value_size):
        return None
    if n_heads % nkv or q.shape[1] != n_heads * hd:
        raise KernelError("latent attention: q has the wrong shape")
    T, B = q.shape[0], ctx.n_seqs
    group = n_heads // nkv
    hpb = min(group, ROWS)
    tpb = ROWS // hpb
    # pages a block's rows can see, from the bound (a captured graph is replayed for other lengths)
    bound = max(ctx.kv_len_bound, ctx.max_kv_len, 1)
    reach = min(bound, window + tpb) if window else bound
    pages = -(-reach // page_size) + (1 if window else 0)
    chunk, n_splits = pages, 1
    if ctx.max_new == 1:
        chunk, n_splits = splits_for(B * nkv * -(-group // hpb), pages)
    out = torch.empty((T, n_heads * value_size), dtype=torch.bfloat16, device=q.device)
    part_o = part_ml = None
    if n_splits > 1:
        part_o = torch.empty((T * n_heads, n_splits, value_size), dtype=torch.float32, device=q.device)
        part_ml = torch.empty((T * n_heads, n_splits, 2), dtype=torch.float32, device=q.device)
    if ops.profiling():
        pairs = 0
        for n, end in zip(ctx.host_n_new, ctx.host_kv_lens):
            for p in range(end - n, end):
                pairs += min(p + 1, window) if window else p + 1
        keys = sum(min(e, window + n) if window else e for n, e in zip(ctx.host_n_new, ctx.host_kv_lens))
        ops._work(f"attention latent {T}x{n_heads}", ops._nbytes(q, out) + keys * nkv * hd * 2, 2 * pairs * n_heads * (hd + value_size))
    m = module(hd, value_size)
    _check(m.ik_attn_latent(_ptr(q), _ptr(k_pages), _ptr(out), _ptr(part_o), _ptr(part_ml), _ptr(ctx.cu_seqlens),
                            _ptr(ctx.kv_lens), _ptr(table), table.stride(0), T, B, ctx.max_new, n_heads, nkv, scale,
                            int(window or 0), 1 if sink else 0, page_size, n_pages, chunk, n_splits, _ptr(status), _stream()),
           "attention latent", kernels=2 if n_splits > 1 else 1)
    return out


PROMPT_BYTES_MOST = 1 << 30       # of formed keys, values and gathered latents at a time: sequences take turns where a step's are more
FORM_KEYS_QUERIES = 64


def formed_bytes(keys: int, n_heads: int, rank: int) -> int:
    """What ``prompt`` allocates for a sequence of so many keys: a latent, and every head's key and value of 128, in whole pages."""
    return -(-keys // 64) * 64 * 2 * (rank + 256 * n_heads)


def forms_keys(ctx, k_pages: torch.Tensor, dtype: torch.dtype, dk: int, dr: int, dv: int, rank: int, window: int = 0, n_heads: int = 32,
               scale: float = 1.0) -> bool:
    """Whether a step's attention goes over keys and values formed per head (``prompt``) rather than over the cached rows.  Forming
    them costs heads x rank x (dk + dv) products a key; a query that sees the key then saves 2 rank - dk - dv of the 2 rank + dr
    products per head (768 of 1,088), and runs on tcgen05.  Measured on B200 (rank 512, one sequence; us for the layer, over the rows /
    formed): 16 heads, 64 new tokens behind 2,000 190 / 155, 512 behind 2,000 371 / 168, 4,096 from the start 2,056 / 348; 32 heads,
    64 behind 2,000 228 / 183, 512 behind 2,000 674 / 245; below 64 not measured.  With a rank of 64 a query saves no products, only the kernel's
    rate: 32 heads, 16 sequences of 64 behind 500 203 / 217, one of 512 behind 2,000 245 / 188, so twice as many queries are asked for.  Under a window a query sees that many keys at
    most, while every key is formed.  A sequence whose formed keys and values alone exceed ``PROMPT_BYTES_MOST`` (1 GB: 61,680 keys with 32
    heads, 16,131 with 128) goes over the rows, with the others of its step."""
    if dtype != torch.bfloat16 or k_pages.dtype != torch.bfloat16 or ctx.is_decode or k_pages.shape[1:3] != (1, 64):
        return False
    if dk != 128 or dv != 128 or dr not in (0, 64) or rank % 64 or k_pages.shape[3] != rank + dr or not scale > 0:
        return False
    lens, new = ctx.host_kv_lens, ctx.host_n_new
    keys = sum(lens)
    return len(lens) == ctx.n_seqs and all(formed_bytes(e, n_heads, rank) <= PROMPT_BYTES_MOST for e in lens) and sum(n * min(e, window or e) for n, e in zip(new, lens)) >= \
        FORM_KEYS_QUERIES * (2 if rank < 128 else 1) * keys


def prompt(q_plain: torch.Tensor, q_full: torch.Tensor, k_pages: torch.Tensor, w_kv: torch.Tensor, ctx, table: torch.Tensor, n_heads: int,
           rank: int, scale: float, window: int, status: Optional[torch.Tensor]) -> torch.Tensor:
    """q_plain [T, heads * 128] and the turning parts in q_full [T, heads * (rank + dr)]; ``w_kv`` [2 * heads * 128, rank]: all heads'
    key matrices, then their value matrices.  Returns the heads' results [T, heads * 128]."""
    from . import gemm_bf16
    n_pages, _, _, hd = k_pages.shape
    T, lens = q_plain.shape[0], ctx.host_kv_lens
    lib = ops.lib()
    out = torch.empty((T, n_heads * 128), dtype=torch.bfloat16, device=q_plain.device)
    first = 0
    while first < ctx.n_seqs:                             # as many sequences at a time as ``PROMPT_BYTES_MOST`` has room for
        end, used = first, 0
        while end < ctx.n_seqs and (end == first or used + formed_bytes(lens[end], n_heads, rank) <= PROMPT_BYTES_MOST):
            used += formed_bytes(lens[end], n_heads, rank)
            end += 1
        B, n_keys, longest = end - first, sum(-(-e // 64) * 64 for e in lens[first:end]), max(lens[first:end])
        cu_seqlens, kv_lens, rows = ctx.cu_seqlens[first:], ctx.kv_lens[first:], table[first:]
        latents = torch.empty((n_keys, rank), dtype=torch.bfloat16, device=q_plain.device)
        ops._work(f"latent_gather {n_keys}x{rank}", 2 * ops._nbytes(latents))
        _check(lib.ik_latent_gather(_ptr(k_pages), _ptr(cu_seqlens), _ptr(kv_lens), _ptr(rows), rows.stride(0), _ptr(latents), B, longest,
                                    hd, rank, int(window or 0), n_pages, _ptr(status), _stream()), "latent_gather")
        kv = gemm_bf16.gemm(latents, w_kv, out_dtype=torch.bfloat16)
        if ops.profiling():
            pairs = sum(min(p + 1, window) if window else p + 1
                        for n, e in zip(ctx.host_n_new[first:end], lens[first:end]) for p in range(e - n, e))
            ops._work(f"attention latent prompt {T}x{n_heads}", ops._nbytes(q_plain, out, kv), 2 * pairs * n_heads * (256 + hd - rank))
        _check(lib.ik_latent_prompt(_ptr(q_plain), _ptr(q_full), _ptr(kv), _ptr(k_pages), _ptr(out), _ptr(cu_seqlens), _ptr(kv_lens), _ptr(rows),
                                    rows.stride(0), T, B, ctx.max_new, n_keys, n_heads, hd, rank, scale, int(window or 0), n_pages, _ptr(status),
                                    _stream()), "attention latent prompt")
        del latents, kv                                   # the next sequences' are made where these were
        first = end
    return out

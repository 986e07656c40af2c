"""Paged-KV ops: cache write and page gather (csrc/kv_cache.cu) and attention over the paged
cache.  Attention runs on the tcgen05 kernel (csrc/attention_sm100.cu) whose TMA producer walks
the block table: decode maps the query heads that share a KV head onto the rows of one MMA
tile, chunked prefill is the causal kernel with a query offset.  A CUDA-core decode kernel
(csrc/kv_cache.cu) remains for page sizes the TMA path does not take.  CPU paths restate the
same semantics in PyTorch for the engine's CPU tests."""
from __future__ import annotations

import ctypes
import math

import torch

from . import _native as nv

c_int, c_long, c_float = ctypes.c_int, ctypes.c_long, ctypes.c_float


def _set_bounds(k_cache) -> None:
    """Checked build only: tell the library how many slots / pages the cache holds."""
    if nv.bounds_check_enabled():
        nb, bs = k_cache.shape[0], k_cache.shape[1]
        nv.lib("kv_cache").omni_kv_set_bounds(c_long(nb * bs), c_int(nb), nv.ptr(nv.status_word(k_cache.device)))


def kv_write(k, v, k_cache, v_cache, slots):
    """k, v: [T, Hkv, D]; caches: [num_blocks, block_size, Hkv, D]; slots int32 [T] (<0 = skip)."""
    T = k.shape[0]
    row = k_cache.shape[2] * k_cache.shape[3]
    if not k.is_cuda:
        kf, vf = k_cache.view(-1, row), v_cache.view(-1, row)
        ok = slots >= 0
        kf[slots[ok].long()] = k.reshape(T, row)[ok]
        vf[slots[ok].long()] = v.reshape(T, row)[ok]
        return
    assert k.stride(-1) == 1 and k.stride(1) == k.shape[2] and slots.dtype == torch.int32
    _set_bounds(k_cache)
    rc = nv.lib("kv_cache").omni_kv_write(nv.ptr(k), nv.ptr(v), c_long(k.stride(0)), c_long(v.stride(0)),
                                          nv.ptr(k_cache), nv.ptr(v_cache), nv.ptr(slots), c_int(T), c_int(row),
                                          nv.stream_ptr())
    nv.check_rc(rc, "omni_kv_write")


def kv_gather(k_cache, v_cache, block_table, T, out_k=None, out_v=None):
    """Pages of one sequence -> contiguous [T, Hkv, D] tensors (or the given buffers, which may
    live in another GPU's peer-mapped memory)."""
    nb, bs, Hkv, D = k_cache.shape
    if out_k is None:
        out_k, out_v = (torch.empty(T, *c.shape[2:], dtype=c.dtype, device=c.device) for c in (k_cache, v_cache))
    if not k_cache.is_cuda or k_cache.shape != v_cache.shape or k_cache.dtype != torch.bfloat16:
        out_k.copy_(rows_gather(k_cache, block_table, T))
        out_v.copy_(rows_gather(v_cache, block_table, T))
        return out_k, out_v
    _set_bounds(k_cache)
    rc = nv.lib("kv_cache").omni_kv_gather(nv.ptr(k_cache), nv.ptr(v_cache), nv.ptr(block_table), c_int(bs), c_int(T),
                                           c_int(Hkv * D), nv.ptr(out_k), nv.ptr(out_v), nv.stream_ptr())
    nv.check_rc(rc, "omni_kv_gather")
    return out_k, out_v


def rows_gather(k_cache, block_table, T):
    """Pages of one sequence that hold one tensor (or none) -> contiguous [T, Hkv, D]."""
    if not k_cache.numel():
        return k_cache.new_empty(T, *k_cache.shape[2:])
    bs = k_cache.shape[1]
    j = torch.arange(T, device=k_cache.device)
    return k_cache.view(-1, *k_cache.shape[2:])[block_table.long()[j // bs] * bs + j % bs]


def _scratch_for(device, n_part: int, D: int):
    """Partial sums and their maxima and weights of a split call, its own: other threads and streams run calls of the same size."""
    return (torch.empty(n_part * D, dtype=torch.float32, device=device), torch.empty(n_part * 2, dtype=torch.float32, device=device))


def tma_pages_ok(block_size: int, D: int) -> bool:
    """Page shapes the tensor-core path takes: head_dim 128, pages of 8..128 tokens that tile 128."""
    return D == 128 and block_size >= 8 and block_size % 8 == 0 and 128 % block_size == 0


def _attn_paged(q, q_rs, q_hs, q_bs, k_cache, v_cache, block_tables, kv_lens, out, o_rs, o_hs, o_bs, B, H, Hkv, Sq,
                max_kv, scale, causal, q_offset, kv_splits, lse=None):
    nb, bs = k_cache.shape[0], k_cache.shape[1]
    part_o = part_ml = None
    if kv_splits > 1:
        part_o, part_ml = _scratch_for(q.device, B * H * Sq * kv_splits, 128)
    st = nv.status_word(q.device)
    rc = nv.lib("attention_sm100").omni_attn_fwd_paged(
        nv.ptr(q), c_long(q_rs), c_long(q_hs), c_long(q_bs), nv.ptr(k_cache), nv.ptr(v_cache), c_int(nb), c_int(bs),
        nv.ptr(block_tables), c_int(block_tables.stride(0)), nv.ptr(out), c_long(o_rs), c_long(o_hs), c_long(o_bs),
        nv.ptr(lse), c_int(B), c_int(H), c_int(Hkv), c_int(Sq), c_int(max_kv), nv.ptr(kv_lens), c_float(scale),
        c_int(1 if causal else 0), c_int(q_offset), c_int(kv_splits), nv.ptr(part_o), nv.ptr(part_ml), nv.ptr(st),
        nv.stream_ptr())
    nv.check_rc(rc, "omni_attn_fwd_paged")


def decode_impl(n: int, H: int, Hkv: int, D: int, block_size: int, num_splits, q_stride: int, out_stride: int) -> str:
    """The kernel that decodes ``n`` sequences.  Pages that the tensor-core kernel does not take: "simt", which keeps the weights in fp32
    where the others round them to bf16 ("stream" for group sizes it does not have).  Else "tc" where a number of splits is asked for or
    more than 16 heads share a KV head, and "stream" for up to 8 of them.  Groups of 9 to 16 heads fill both halves of its products and
    leave room for fewer loads in flight: it wins where the tensor-core kernel, a block per sequence and KV head, has very few blocks or
    a last round that is less than nine tenths full, and loses where it has nearly one or two rounds of them.  Of "tc"'s time, 64 / 4 and
    32 / 2 heads at 64 to 32768 keys: 16 groups 0.57 to 0.84, 32 groups 0.77 to 1.12, 128 groups 0.95 to 1.34, 160 groups 0.36 to 0.95,
    256 groups 0.45 to 1.06, 288 groups 0.88 to 1.17, 320 groups 0.33 to 0.86."""
    G, groups, sms = H // Hkv, n * Hkv, 148
    if not tma_pages_ok(block_size, D) or G > 128:
        return "stream" if D == 128 and block_size % 8 == 0 and G <= 16 and G not in (1, 2, 4, 8) and num_splits is None else "simt"
    if G > 16 or num_splits is not None or q_stride % 8 or out_stride % 8:
        return "tc"
    if G <= 8:
        return "stream"
    whole = Hkv % 4 == 0 or Hkv <= 2                   # all four warps of a block have heads: 36 / 3 heads, 576 groups, 1.10 of "tc"'s time
    return "stream" if whole and (groups <= 16 or (groups > sms and not 1.8 * sms <= groups <= 2 * sms)) else "tc"


def paged_decode(q, k_cache, v_cache, block_tables, seq_lens, scale=None, num_splits=None, out=None, impl=None, rows=None):
    """q: [num_seqs, H, D] (one new token per sequence) -> [num_seqs, H, D].

    ``rows`` (int64 [num_seqs]): sequence i is row rows[i] of q and of ``out``, which is then needed; other rows of it stay.

    ``impl``: "stream" (csrc/decode_attn.cu), "tc" (tcgen05 kernel) or "simt"; by default as ``decode_impl`` says."""
    n, H, D = q.shape if rows is None else (rows.numel(), *q.shape[1:])
    nb, bs, Hkv, _ = k_cache.shape
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if rows is not None:
        asked = impl
        if impl is None and q.is_cuda:
            impl = decode_impl(n, H, Hkv, D, bs, num_splits, q.stride(0), out.stride(0))
        if impl != "stream" or rows.dtype != torch.int64 or not rows.is_contiguous() or rows.device != q.device:
            out[rows] = paged_decode(q[rows].contiguous(), k_cache, v_cache, block_tables, seq_lens, scale, num_splits, impl=asked)
            return out
    if out is None:
        out = torch.empty_like(q)
    if not q.is_cuda:
        from .attention import attention_reference
        for i in range(n):
            L = int(seq_lens[i])
            gk, gv = kv_gather(k_cache, v_cache, block_tables[i], L)
            out[i] = attention_reference(q[i:i + 1, None].reshape(1, 1, H, D), gk[None], gv[None], scale)[0, 0]
        return out
    assert q.stride(-1) == 1 and q.stride(1) == D and block_tables.dtype == torch.int32 and seq_lens.dtype == torch.int32
    G = H // Hkv
    if impl is None:
        impl = decode_impl(n, H, Hkv, D, bs, num_splits, q.stride(0), out.stride(0))
    if impl == "stream":
        assert out.stride(-1) == 1 and out.stride(1) == D and q.dtype == torch.bfloat16
        lib, max_kv = nv.lib("decode_attn"), block_tables.shape[1] * bs
        shares = lib.omni_paged_decode_shares(c_int(n), c_int(Hkv), c_int(max_kv))
        part = torch.empty(n * H * shares * (D + 2), dtype=torch.float32, device=q.device) if shares > 1 else None
        rc = lib.omni_paged_decode_attn(
            nv.ptr(q), c_long(q.stride(0)), nv.ptr(k_cache), nv.ptr(v_cache), nv.ptr(block_tables), c_int(block_tables.stride(0)), c_int(bs),
            nv.ptr(seq_lens), c_int(n), c_int(H), c_int(Hkv), c_int(max_kv), c_float(scale), nv.ptr(part),
            nv.ptr(None if part is None else part[n * H * shares * D:]), nv.ptr(out), c_long(out.stride(0)), nv.ptr(rows), c_int(q.shape[0]),
            nv.ptr(nv.status_word(q.device)), nv.stream_ptr())
        nv.check_rc(rc, "omni_paged_decode_attn")
        return out
    if impl == "tc":
        # the G heads of a group are the rows of the query tile: row pitch = one head (D),
        # "head" pitch = one group (G * D), batch pitch = one token
        max_kv = block_tables.shape[1] * bs
        tiles = (max_kv + 127) // 128
        if num_splits is None:
            # one CTA per SM: pick the split count with the fewest (fractional) waves of 148 CTAs
            ctas = n * Hkv
            num_splits = min(range(1, min(tiles, 16) + 1),
                             key=lambda sp: -(-ctas * sp // 148) / sp + 0.02 * sp)
        assert out.stride(-1) == 1 and out.stride(1) == D
        _attn_paged(q, D, G * D, q.stride(0), k_cache, v_cache, block_tables, seq_lens, out, D, G * D, out.stride(0),
                    n, Hkv, Hkv, G, max_kv, scale, False, 0, num_splits)
        return out
    if num_splits is None:
        # enough CTAs to fill the GPU: seqs x kv heads x splits >= ~2 waves of 148 SMs
        num_splits = max(1, min(32, (148 * 8 + n * Hkv - 1) // (n * Hkv)))
    sc = _scratch_for(q.device, n * H * num_splits, D)
    rc = nv.lib("kv_cache").omni_paged_decode(
        nv.ptr(q), c_long(q.stride(0)), nv.ptr(k_cache), nv.ptr(v_cache), nv.ptr(block_tables),
        c_int(block_tables.shape[1]), nv.ptr(seq_lens), c_int(n), c_int(bs), c_int(H), c_int(Hkv), c_int(D),
        c_float(scale), c_int(num_splits), nv.ptr(sc[0]), nv.ptr(sc[1]), nv.ptr(out), c_long(out.stride(0)),
        nv.stream_ptr())
    nv.check_rc(rc, "omni_paged_decode")
    return out


def prefill_segments_ok(q, k_cache, contexts) -> bool:
    """Whether ``prefill_segments`` takes these operands: bf16, head size 64 or 128, at most 4096 query blocks of 256 rows, and pages of its kind where a
    segment has a context."""
    T, _, D = q.shape
    return q.is_cuda and q.dtype == torch.bfloat16 and D in (64, 128) and T <= 4096 * 256 and (not any(contexts) or tma_pages_ok(k_cache.shape[1], D))


def prefill_segments(q, k, v, k_cache, v_cache, segs, scale=None, out=None):
    """Causal attention of all prompt segments of one step in one launch (csrc/attention_sm100.cu, eight segments at a time).

    q [T, H, D], k, v [T, Hkv, D]: rows of the step; ``segs``: (first row, rows, context, block table) each.  A segment without context reads its keys from
    k and v, another all of its keys from the pages, where this step's were written before.  Rows of no segment stay as they are in ``out``."""
    T, H, D = q.shape
    Hkv = k.shape[1]
    assert q.stride(2) == 1 and k.stride(2) == 1 and v.stride(2) == 1 and out.stride(2) == 1
    n = len(segs)
    ints = lambda i: (c_int * n)(*(s[i] for s in segs))
    tables = [s[3] if s[2] else None for s in segs]
    assert all(t is None or (t.dtype == torch.int32 and t.stride(-1) == 1) for t in tables)
    nb, bs = (k_cache.shape[0], k_cache.shape[1]) if k_cache is not None else (0, 0)
    rc = nv.lib("attention_sm100").omni_attn_prefill_segs(
        nv.ptr(q), c_long(q.stride(0)), c_long(q.stride(1)), nv.ptr(k), c_long(k.stride(0)), c_long(k.stride(1)), nv.ptr(v), c_long(v.stride(0)),
        c_long(v.stride(1)), nv.ptr(k_cache), nv.ptr(v_cache), c_int(nb), c_int(bs), nv.ptr(out), c_long(out.stride(0)), c_long(out.stride(1)), c_int(T),
        c_int(H), c_int(Hkv), c_int(D), c_int(n), ints(0), ints(1), ints(2), (ctypes.c_void_p * n)(*(0 if t is None else t.data_ptr() for t in tables)),
        c_float(scale if scale is not None else 1.0 / math.sqrt(D)), nv.ptr(nv.status_word(q.device)), nv.stream_ptr())
    nv.check_rc(rc, "omni_attn_prefill_segs")
    if n > 8 or T > 248 * 256:                               # more than eight segments or 256 blocks of 256 rows
        blocks = [sum(-(-s[1] // 256) for s in segs[i:i + 8]) for i in range(0, n, 8)]
        nv.count_launches(sum(-(-b // 256) for b in blocks) - 1)
    return out


def paged_prefill(q, k_cache, v_cache, block_table, kv_len: int, scale=None, out=None):
    """Causal attention of the LAST ``T`` tokens of one sequence against its whole paged context (a decoder's step takes all of its portions through
    ``prefill_segments``).

    q: [T, H, D]; block_table: int32 [max_blocks]; kv_len: tokens in the cache including these T
    (their K/V already written).  Query row i sees keys [0, kv_len - T + i]."""
    T, H, D = q.shape
    nb, bs, Hkv, _ = k_cache.shape
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if out is None:
        out = torch.empty_like(q)
    if not q.is_cuda or not tma_pages_ok(bs, D):
        from .attention import attention, attention_reference
        gk, gv = kv_gather(k_cache, v_cache, block_table, kv_len)
        if q.is_cuda:
            attention(q[None], gk[None], gv[None], scale=scale, causal=True, q_offset=kv_len - T, out=out[None])
        else:
            out.copy_(attention_reference(q[None], gk[None], gv[None], scale, causal=True, q_offset=kv_len - T)[0])
        return out
    assert q.stride(-1) == 1 and out.stride(-1) == 1 and block_table.dtype == torch.int32
    lens = torch.full((1,), kv_len, dtype=torch.int32, device=q.device)
    bt = block_table.view(1, -1)
    _attn_paged(q, q.stride(0), q.stride(1), T * q.stride(0), k_cache, v_cache, bt, lens, out, out.stride(0),
                out.stride(1), T * out.stride(0), 1, H, Hkv, T, kv_len, scale, True, kv_len - T, 1)
    return out

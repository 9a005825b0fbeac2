"""DeepSeek MLA on the GPU.  The absorbed form is used for prefill and decode alike: grouped tcgen05 GEMMs (one group per head) around the
latent-cache attention kernel (csrc/kernels/mla.cu), which works per token.  With XFT_MLA_EXPAND=1 longer portions of prompts take the
expanded form (csrc/kernels/latent_prefill_sm100.cu, see native_latent): the latents that they see times W_uk and W_uv once, then
attention in tiles of 128 queries.  It is faster, but rounds keys and values of each head to bf16 where the absorbed form rounds its query
and its latent result, so a model's logits differ by as much as either differs from 64 bits."""
from __future__ import annotations

import ctypes as C
from typing import Dict

import torch

from . import native as N

_ready = False
_tables: Dict[tuple, tuple] = {}


def _lib():
    global _ready
    lib = N.lib()
    if not _ready:
        lib.xft_mla_attention_ext.restype = C.c_int
        lib.xft_gemm_bf16_grouped.restype = lib.xft_gemm_bf16_grouped_tm.restype = C.c_int
        _ready = True
    return lib


def _head_tiles(H: int, T: int, dev):
    """Static tile table of a per-head grouped GEMM: rows of head h are [h*T, (h+1)*T)."""
    bn = 16 if T <= 16 else 32 if T <= 32 else 64 if T <= 64 else 128 if T < 512 else 256
    key = (H, T, bn, dev.index)
    if key not in _tables:
        rows = []
        for h in range(H):
            for j in range(0, T, bn):
                rows.append([h, h * T + j, min(bn, T - j), 0])
        tiles = torch.tensor(rows, dtype=torch.int32, device=dev)
        meta = torch.tensor([len(rows), H * T], dtype=torch.int32, device=dev)
        _tables[key] = (tiles, meta, len(rows), bn)
    return _tables[key]


def _per_head_gemm(x_ht, w_stacked, H, T, n_out, k_in):
    """x_ht [H*T, k_in] bf16 (rows grouped by head) x per-head weights [H*n_out, k_in] -> [H*T, n_out] bf16."""
    tiles, meta, nt, bn = _head_tiles(H, T, x_ht.device)
    out = torch.empty(H * T, n_out, dtype=torch.bfloat16, device=x_ht.device)
    ws = N.Workspace.get(x_ht.device)
    if bn >= 128:
        # prompts: the token-major kernel (3000 tokens, 128 heads of 512 x 128: 1980 us with the kernel of the decode steps)
        N._check(_lib().xft_gemm_bf16_grouped_tm(N._p(x_ht), k_in, H * T, N._p(w_stacked), H * n_out, k_in, N._p(out), n_out, n_out, k_in,
                                                 0, 0, n_out, N._p(tiles), N._p(meta), nt, bn, 0, N._p(ws.status), N._stream()),
                 "per-head grouped gemm")
        ws.launches += 1
        return out
    rc = _lib().xft_gemm_bf16_grouped(N._p(x_ht), k_in, H * T, N._p(w_stacked), H * n_out, k_in, N._p(out), n_out, 0,
                                      n_out, k_in, 0, 0, n_out, N._p(tiles), N._p(meta), nt, bn, N._p(None), 0,
                                      N._p(ws.status), N._stream())
    N._check(rc, "per-head grouped gemm")
    ws.launches += 1
    return out


def expands(cu_q, nope, rope, kvl, vd, kv_lens=None) -> bool:
    """Whether a batch's portions of at least XFT_LATENT_EXPAND_MIN_Q new tokens pay for the expanded form: sizes that attn_flat_tc_kernel
    has, 64 tokens that take it, or 256 where shorter portions beside them need a launch of the other form, and, as it works per visible key
    and the absorbed form per key and token, 40 tokens per visible key or 256 keys per portion.  us of a layer's attention with its
    per-head products, 128 heads, absorbed / expanded (error against 64 bits): 32 prompts of about 97 tokens 2087 / 339 (2.682e-3 and
    2.680e-3 of the result), 32 of 16 351 / 212, one of 200 169 / 78, of 2000 3866 / 344 (2.84e-3, 2.76e-3); 4 x 16 tokens behind 300 keys
    141 / 116, 4000 511 / 840, 32000 3345 / 6757; 32 x 16 behind 300 529 / 648; 8 x 32 behind 1000 574 / 509, 16000 5690 / 6534; 4 x 64
    behind 4000 1566 / 853, 32000 11339 / 6909; one of 16 tokens 58 / 78; 140 tokens in two portions beside two short ones 128 / 174."""
    if nope % 64 or rope % 64 or nope + rope > 256 or kvl % 8 or vd % 64 or vd > 128:
        return False
    least = N._ENV().latent_expand_min_q
    n = [cu_q[i + 1] - cu_q[i] for i in range(len(cu_q) - 1)]
    long = [i for i, q in enumerate(n) if q >= least]
    if sum(n[i] for i in long) < (64 if min(n) >= least else 256):
        return False
    if kv_lens is None:
        return True
    keys = sum(kv_lens[i] for i in long)
    return keys <= 256 * len(long) or sum(n[i] * kv_lens[i] for i in long) >= 40 * keys


class _Heads:
    """What native_latent.flat_attention asks of packed rows."""

    def __init__(self, heads, nope, rope, vd, rank):
        self.heads, self.dim, self.rot, self.vdim, self.rank = heads, nope, rope, vd, rank
        self.q_width, self.gate, self.head_gate = heads * (nope + rope), False, False


def _expanded(q_nope, q_rope, cache, block_table, sp, w_uk, w_uv, scale, out) -> bool:
    """Portions `sp.long` into `out`; False where keys and values have no room."""
    from . import native_latent as NL
    T, Hl, nope = q_nope.shape
    rope, L, vd = q_rope.shape[2], w_uk.shape[2], w_uv.shape[1]
    step = (Hl * (nope + rope), nope + rope, 1)
    if q_nope.stride() == step and q_rope.stride() == step and q_rope.data_ptr() == q_nope.data_ptr() + 2 * nope:
        q = q_nope.as_strided((T, step[0]), (step[0], 1))                # the packed heads of mla_prep
    else:
        q = torch.cat([q_nope, q_rope], -1).view(T, -1)
    nb, _, bs, W = cache.shape
    per = max(1, min(Hl, NL.EXPAND_BYTES // (2 * sp.rows * (nope + vd))))
    try:
        flat = torch.empty(sp.rows, W, dtype=q.dtype, device=q.device)
        kv = torch.empty(sp.rows * per * (nope + vd), dtype=q.dtype, device=q.device)
    except torch.OutOfMemoryError:
        return False
    ws, d = N.Workspace.get(q.device), _Heads(Hl, nope, rope, vd, L)
    N._check(NL._fn("xft_latent_gather")(N._p(cache), W, bs, nb, N._p(block_table), block_table.stride(0), N._p(sp.seq), N._p(sp.lo),
                                         N._p(sp.row), len(sp.long), sp.rows, N._p(flat), N._p(ws.status), N._stream()), "latent_gather")
    ws.launches += 1
    wk, wv = w_uk.reshape(Hl * nope, L), w_uv.reshape(Hl * vd, L)
    for h0 in range(0, Hl, per):
        n = min(per, Hl - h0)
        part = kv[:sp.rows * n * (nope + vd)].view(sp.rows, n * (nope + vd))
        N.gemm_bf16(flat[:, :L], wk[h0 * nope:(h0 + n) * nope], n * nope, out=part[:, :n * nope])
        N.gemm_bf16(flat[:, :L], wv[h0 * vd:(h0 + n) * vd], n * vd, out=part[:, n * nope:])
        NL.flat_attention(q, d, part, flat, sp, h0, n, scale, 0, out)
    return True


def mla_attention(q_nope, q_rope, latent_cache, block_table, cu_q, kv_lens, w_uk, w_uv, scale, absorbed=True, meta=None):
    T, Hl, nope = q_nope.shape
    L = w_uk.shape[2]
    vd = w_uv.shape[1]
    rope = q_rope.shape[2]
    assert L == 512 and rope == 64, "MLA kernel is specialised for kv_lora_rank 512 + rope 64"
    dev = q_nope.device
    cu_dev, kv_dev, B, decode, max_kv = N.batch_arrays(cu_q, kv_lens, meta, dev)
    if N._ENV().mla_expand and not decode and scale > 0 and expands(cu_q, nope, rope, L, vd, kv_lens):
        from .native_latent import _Spans
        kept = meta.meta if meta is not None else {}
        key = ("latent spans", 0, N._ENV().latent_expand_min_q)
        sp = kept.get(key)
        if sp is None:
            sp = kept[key] = _Spans(cu_q, kv_lens, 0, key[2], dev)
        out = torch.empty(T, Hl * vd, dtype=torch.bfloat16, device=dev)
        if _expanded(q_nope, q_rope, latent_cache, block_table, sp, w_uk, w_uv, scale, out):
            if sp.part is not None:
                rows, seqs, cu, kv, n, most = sp.part
                out.index_copy_(0, rows.long(), _absorbed(q_nope.index_select(0, rows), q_rope.index_select(0, rows), latent_cache,
                                                          block_table.index_select(0, seqs), cu, kv, n, most, w_uk, w_uv, scale,
                                                          None).view(rows.shape[0], Hl * vd))
            return out.view(T, Hl, vd)
    return _absorbed(q_nope, q_rope, latent_cache, block_table, cu_dev, kv_dev, B, max_kv, w_uk, w_uv, scale,
                     meta.meta.get("nsplit") if meta is not None else None)


def _absorbed(q_nope, q_rope, latent_cache, block_table, cu_dev, kv_dev, B, max_kv, w_uk, w_uv, scale, splits):
    T, Hl, nope = q_nope.shape
    L, vd, rope = w_uk.shape[2], w_uv.shape[1], q_rope.shape[2]
    dev = q_nope.device
    ws = N.Workspace.get(dev)
    # W_uk^T stacked per head: [Hl*L, nope] (linear weight [out=L, in=nope])
    # cached on the tensor itself (an id()-keyed table would hand a dead tensor's copy to a new tensor that reuses
    # its address)
    wk = getattr(w_uk, "_xft_wk_t", None)
    if wk is None or wk.shape != (Hl * L, nope):
        wk = w_uk.transpose(1, 2).contiguous().view(Hl * L, nope)
        w_uk._xft_wk_t = wk
    wv = w_uv.reshape(Hl * vd, L)
    q_ht = q_nope.transpose(0, 1).contiguous().view(Hl * T, nope)
    q_abs = _per_head_gemm(q_ht, wk, Hl, T, L, nope)                 # [Hl*T, L]
    o_lat = torch.empty(Hl * T, L, dtype=torch.bfloat16, device=dev)
    nb, _, bs, W = latent_cache.shape
    chunks = (Hl + 15) // 16
    from .native_latent import mla_scratch, mla_splits
    nsplit, groups = splits or mla_splits(T * chunks, max_kv)
    po, pm, cnt = mla_scratch(ws, T * chunks, nsplit, groups, L)
    q_rope = q_rope.contiguous()
    LL = C.c_longlong
    rc = _lib().xft_mla_attention_ext(N._p(q_abs), LL(T * L), LL(L), N._p(q_rope), LL(rope), LL(Hl * rope), N._p(o_lat), LL(T * L),
                                      LL(L), N._p(latent_cache), N._p(block_table), block_table.stride(0), N._p(cu_dev),
                                      N._p(kv_dev), B, T, Hl, L, bs, nb, C.c_float(scale), N._p(None), 0, nsplit, groups, N._p(po), N._p(pm),
                                      N._p(cnt), N._p(ws.status), N._stream())
    N._check(rc, "mla_attention")
    ws.launches += 1
    o = _per_head_gemm(o_lat, wv, Hl, T, vd, L)                      # [Hl*T, vd]
    return o.view(Hl, T, vd).transpose(0, 1).contiguous()

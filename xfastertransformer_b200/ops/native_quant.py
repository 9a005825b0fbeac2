"""Bindings of the quantised GEMM kernels: weight-only int8 / nf4 dequant-GEMM and W8A8 (dynamic int8 activations x int8 weights
on the int8 tensor path) in csrc/kernels/quant_gemm_sm100.cu, fp8-e4m3 and uint4 weights on the fp8 tensor path in
csrc/kernels/gemm_e4m3_sm100.cu, prompts over int8 weights in csrc/kernels/gemm_prefill_sm100.cu (CODES_ROWS)."""
from __future__ import annotations

import ctypes as C

import torch

from . import native as N

_QT = {"int8": 0, "nf4": 2}
_E4M3 = {"fp8": 0, "int4": 1}             # weights that e4m3 holds: csrc/kernels/gemm_e4m3_sm100.cu
_ready = False


def _lib():
    global _ready
    lib = N.lib()
    if not _ready:
        for fn in ("xft_qgemm", "xft_quant_act", "xft_row_sum", "xft_w8a8_gemm", "xft_split_e4m3", "xft_split_e4m3_cols",
                   "xft_gemm_e4m3", "xft_w8a8_gemm_gated", "xft_rms_quant_act", "xft_rms_split_e4m3"):
            getattr(lib, fn).restype = C.c_int
        _ready = True
    return lib


def _row_sums(x2, ldx):
    T, K = x2.shape
    out = torch.empty(T, dtype=torch.float32, device=x2.device)
    N._check(_lib().xft_row_sum(N._p(x2), ldx, N._p(out), T, K, N._stream()), "row_sum")
    N.Workspace.get(x2.device).launches += 1
    return out


def split_e4m3(x2, ldx, nibbles=False, want_sum=False, src=None, rows_used=None, rows=None, norm=None):
    """Rows of x2 (or rows `src` of it) as sums of two e4m3 numbers -> (uint8 [rows, 2 * cols], scale [rows], sum [rows] or
    None).  `nibbles`: in the order in which 4-bit codes expand.  `rows_used`: device count; later rows stay unwritten.  `norm`:
    (gain, eps) of an RMSNorm in front (norm_fits)."""
    T, K = x2.shape
    rows = T if rows is None else rows
    xs = torch.empty(rows, 2 * _lib().xft_split_e4m3_cols(K), dtype=torch.uint8, device=x2.device)
    st = torch.empty(2, rows, dtype=torch.float32, device=x2.device)
    if norm is not None:
        N._check(_lib().xft_rms_split_e4m3(N._p(x2), ldx, N._p(norm[0]), C.c_float(norm[1]), rows, K, int(nibbles), N._p(xs), N._p(st[0]),
                                           N._p(st[1] if want_sum else None), N._stream()), "rms_split_e4m3")
    else:
        N._check(_lib().xft_split_e4m3(N._p(x2), ldx, N._p(src), N._p(rows_used), rows, K, int(nibbles), N._p(xs), N._p(st[0]),
                                       N._p(st[1] if want_sum else None), N._stream()), "split_e4m3")
    N.Workspace.get(x2.device).launches += 1
    return xs, st[0], st[1] if want_sum else None


def gemm_e4m3(split, w, pitch, src, out, T, n_out, K, gated, dual_off, scale, zero, scale_ld, bias=None, r2=None, ldr=0, res_scale=1.0,
              act=None, tiles=None, n_tiles=None, group_rows=0, max_tiles=0, bn=0, col_scale=None):
    xs, xscale, xsum = split
    ws = N.Workspace.get(xs.device)
    rc = _lib().xft_gemm_e4m3(N._p(xs), xs.shape[0], N._p(xscale), N._p(xsum), N._p(w), w.shape[0], pitch, src, N._p(out), out.stride(0),
                              int(out.dtype == torch.float32), T, n_out, K, int(gated), dual_off, N._p(scale), N._p(zero), scale_ld,
                              N._p(bias), N._p(r2), ldr, C.c_float(res_scale), N._ACT[act], N._p(tiles), N._p(n_tiles), group_rows,
                              max_tiles, bn, N._p(col_scale), N._p(ws.status), N._stream())
    N._check(rc, "gemm_e4m3")
    ws.launches += 1


# Prompts over int8 weights: above so many rows a product's codes are written out as bf16, which holds them exactly, for the kernel of
# bf16 prompts (gemm_prefill_sm100.cu), as long as that copy stays below a bound.  qgemm_kernel, which expands them once for every 128
# rows, keeps what it cuts into parts of k: those sums have another order.  B200, us there / here: 2 x 11008 x 4096 128 rows 112 / 119, 192
# rows 199 / 118, 1210 rows 592 / 225; 12288 x 4096 128 rows 74 / 71, 192 rows 128 / 71.  uint4 weights stay with the halves in e4m3
# (gemm_e4m3_sm100.cu) at any size: their sums are others too, 0.9 % of the logits after eight layers.
CODES_ROWS = 128
CODES_MAX_COPY = 1 << 30


def _codes_copy(W, n_out, rows, K, T, gated, ws, dev):
    """Room for a product's codes in bf16, or None where it does not pay, would change sums or has no room."""
    if W.kind != "int8" or T <= CODES_ROWS or rows * K * 2 > CODES_MAX_COPY or not N._ENV().gemm_prefill_tm:
        return None
    parts, per = C.c_int(), C.c_int()
    _lib().xft_plan_splits((n_out + 127) // 128 * ((T + 127) // 128), (K + 63) // 64, 128, 1 + gated, C.c_size_t(ws.ws_bytes), ws.n_counters,
                           C.byref(parts), C.byref(per))
    if parts.value > 1:
        return None
    try:
        return torch.empty(rows, K, dtype=torch.bfloat16, device=dev)
    except torch.OutOfMemoryError:
        return None


def norm_fits(W, T, K, gated, gain) -> bool:
    """Whether a product of W takes (gain, eps) of an RMSNorm of its rows (csrc/kernels/quant_rows.cu): kinds that rewrite the rows in any
    case, at the sizes at which that adds a row's squares as xft_rmsnorm does."""
    return (W.kind == "w8a8" or W.kind in _E4M3) and 2048 <= K <= 8192 and K % 8 == 0 and gain.dtype == torch.float32 \
        and gain.data_ptr() % 16 == 0 and not (gated and W.kind == "fp8" and W.out_features % 256)


def _qgemm(x, W, n_out, gated, bias, act, residual, res_scale, out_dtype, norm=None):
    x2, ldx = N._rows2d(x)
    T, K = x2.shape
    if K % 8:
        raise N.KernelError(f"quantised GEMM needs K % 8 == 0 (got {K})")
    fp32 = out_dtype == torch.float32
    out = torch.empty(T, n_out, dtype=torch.float32 if fp32 else torch.bfloat16, device=x.device)
    ws = N.Workspace.get(x.device)
    r2, ldr = (None, 0)
    if residual is not None:
        r2 = residual.reshape(-1, residual.shape[-1])
        ldr = r2.stride(0)
    w = W.w if W.w.dtype != torch.float8_e4m3fn else W.w.view(torch.uint8)
    if (w.stride(0) * w.element_size()) % 16:
        # TMA rows must start on 16-byte boundaries: keep a copy whose row pitch is padded (zero codes past K
        # multiply zero-filled activations, so they add nothing)
        wp = W.cache.get("w_pitch16")
        if wp is None:
            cols = w.shape[1]
            pad = (-cols * w.element_size()) % 16 // w.element_size()
            wp = torch.nn.functional.pad(w, (0, pad)).contiguous()[:, :cols]
            W.cache["w_pitch16"] = wp
        w = wp
    zero = W.zero
    copy = _codes_copy(W, n_out, w.shape[0], K, T, gated, ws, x.device)
    if copy is not None:
        fn = _lib().xft_gemm_codes_tm
        fn.restype = C.c_int
        N._check(fn(N._p(x2), ldx, N._p(w), w.shape[0], w.stride(0) * w.element_size(), N._p(copy), N._p(out),
                    out.stride(0), int(fp32), T, n_out, K, int(gated), n_out if gated else 0, N._p(W.scale), N._p(zero),
                    N._p(_row_sums(x2, ldx) if zero is not None else None), N._p(bias), N._p(r2), ldr, C.c_float(res_scale), N._ACT[act],
                    N._p(ws.status), N._stream()), "gemm_codes_tm")
        ws.launches += 2
        return out
    if W.kind in _E4M3:
        codes = W.kind == "int4"
        if codes and zero is None:
            zero = W.cache.get("zero0")
            if zero is None:
                zero = W.cache["zero0"] = torch.zeros_like(W.scale)
        gemm_e4m3(split_e4m3(x2, ldx, codes, codes, norm=norm), w, w.stride(0), _E4M3[W.kind], out, T, n_out, K, gated, n_out if gated else 0,
                  W.scale, zero if codes else None, 0 if codes else W.scale.shape[1], bias, r2, ldr, res_scale, act)
        return out
    if W.kind == "nf4":
        zero = None
    xsum = _row_sums(x2, ldx) if zero is not None else None
    rc = _lib().xft_qgemm(N._p(x2), ldx, N._p(w), w.shape[0], w.stride(0) * w.element_size(), _QT[W.kind], N._p(out),
                          out.stride(0), int(fp32), T, n_out, K, int(gated), n_out if gated else 0, N._p(W.scale),
                          N._p(zero), N._p(xsum), 0, N._p(bias), N._p(r2), ldr, C.c_float(res_scale),
                          N._ACT[act], N._p(ws.ws), C.c_size_t(ws.ws_bytes), N._p(ws.counters), ws.n_counters,
                          N._p(ws.status), N._stream())
    N._check(rc, f"qgemm[{W.kind}]")
    ws.launches += 1
    return out


_QMODE = {"int8": 0, "w8a8": 0, "int4": 1, "nf4": 2}
_SRC_DT = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}


def quantize_rows(w, kind):
    """Quantise-at-load on the device: dense w [out, in] (fp32 / fp16 / bf16, on the GPU) -> (codes, scale[out],
    zero[out], wsum[out] or None) in the layouts of `ops.reference.quantize_{int8,uint4,nf4}_per_channel`: int8 codes
    [out, in], or two 4-bit codes per byte [out, in / 2].  `wsum` (sum of the codes per row) only for kind "w8a8"."""
    if w.dim() != 2 or w.stride(1) != 1 or w.dtype not in _SRC_DT:
        w = w.contiguous() if w.dtype in _SRC_DT else w.float().contiguous()
    rows, K = w.shape
    mode = _QMODE[kind]
    if mode and K % 2:
        raise ValueError("4-bit weights need an even input dimension")
    q = torch.empty(rows, K if mode == 0 else K // 2, dtype=torch.int8 if mode == 0 else torch.uint8, device=w.device)
    sz = torch.empty(3, rows, dtype=torch.float32, device=w.device)
    wsum = sz[2] if kind == "w8a8" else None
    fn = _lib().xft_quantize_rows
    fn.restype = C.c_int
    N._check(fn(N._p(w), _SRC_DT[w.dtype], C.c_longlong(w.stride(0)), rows, K, mode, N._p(q), C.c_longlong(q.stride(0)),
                N._p(sz[0]), N._p(sz[1]), N._p(wsum), N._stream()), "quantize_rows")
    N.Workspace.get(w.device).launches += 1
    return q, sz[0], sz[1], wsum


def quant_act(x2, ldx, norm=None):
    """bf16 [T,K] -> (int8 [T,K], scale[T], zero[T], qsum[T]) per-row dynamic asymmetric.  `norm`: as in split_e4m3."""
    T, K = x2.shape
    q = torch.empty(T, K, dtype=torch.int8, device=x2.device)
    s = torch.empty(3, T, dtype=torch.float32, device=x2.device)
    if norm is not None:
        N._check(_lib().xft_rms_quant_act(N._p(x2), ldx, N._p(norm[0]), C.c_float(norm[1]), N._p(q), K, N._p(s[0]), N._p(s[1]), N._p(s[2]), T, K,
                                          N._stream()), "rms_quant_act")
    else:
        N._check(_lib().xft_quant_act(N._p(x2), ldx, N._p(q), K, N._p(s[0]), N._p(s[1]), N._p(s[2]), T, K, N._stream()),
                 "quant_act")
    N.Workspace.get(x2.device).launches += 1
    return q, s[0], s[1], s[2]


def _w8a8(x, W, rows, bias, act, residual, res_scale, out_dtype, row0=0, norm=None):
    x2, ldx = N._rows2d(x)
    T, K = x2.shape
    q, sa, za, qs = quant_act(x2, ldx, norm)
    fp32 = out_dtype == torch.float32
    out = torch.empty(T, rows, dtype=torch.float32 if fp32 else torch.bfloat16, device=x.device)
    ws = N.Workspace.get(x.device)
    r2, ldr = (None, 0)
    if residual is not None:
        r2 = residual.reshape(-1, residual.shape[-1])
        ldr = r2.stride(0)
    w = W.w[row0:row0 + rows]
    sl = slice(row0, row0 + rows)
    rc = _lib().xft_w8a8_gemm(N._p(q), K, N._p(w), W.w.stride(0), N._p(out), out.stride(0), int(fp32), T, rows, K,
                              N._p(sa), N._p(za), N._p(qs), N._p(W.scale[sl]), N._p(W.zero[sl]), N._p(W.wsum[sl]),
                              N._p(bias), N._p(r2), ldr, C.c_float(res_scale), N._ACT[act], N._p(ws.ws),
                              C.c_size_t(ws.ws_bytes), N._p(ws.counters), ws.n_counters, N._p(ws.status), N._stream())
    N._check(rc, "w8a8_gemm")
    ws.launches += 1
    return out


def linear(x, W, bias=None, act=None, residual=None, res_scale=1.0, out_dtype=None, norm=None):
    if W.kind == "w8a8":
        return _w8a8(x, W, W.out_features, bias, act, residual, res_scale, out_dtype, norm=norm)
    if W.kind in _QT or W.kind in _E4M3:
        return _qgemm(x, W, W.out_features, False, bias, act, residual, res_scale, out_dtype, norm)
    raise N.KernelError(f"no sm_100a GEMM for weight kind {W.kind}")


def linear_gated(x, W, act="silu", bias=None, norm=None):
    I = W.out_features // 2
    if W.kind == "w8a8":
        x2, ldx = N._rows2d(x)
        T, K = x2.shape
        q, sa, za, qs = quant_act(x2, ldx, norm)
        out = torch.empty(T, I, dtype=torch.bfloat16, device=x.device)
        ws = N.Workspace.get(x.device)
        N._check(_lib().xft_w8a8_gemm_gated(N._p(q), K, N._p(W.w), W.w.stride(0), N._p(out), I, T, I, K, I, N._p(sa), N._p(za), N._p(qs),
                                            N._p(W.scale), N._p(W.zero), N._p(W.wsum), N._p(bias), N._ACT[act], N._p(ws.status),
                                            N._stream()), "w8a8_gemm_gated")
        ws.launches += 1
        return out
    if W.kind == "fp8" and I % 128:
        gu = _qgemm(x, W, 2 * I, False, bias, None, None, 1.0, None)
        return N.gated_act(gu, act)
    return _qgemm(x, W, I, True, bias, act, None, 1.0, None, norm)

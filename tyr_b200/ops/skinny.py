"""Decode-sized linear layers (1..32 rows) on the weight-streaming kernel (csrc/skinny_gemm.cu)."""
from __future__ import annotations

import ctypes
import os
from typing import List, Optional, Sequence

import torch

from .._native import register_signatures
from ._common import check, cur_stream, lib, ptr

MAX_ROWS = 32
MAX_MATRICES = 4         # of one launch (skinny_many)


@register_signatures
def _sigs(lib_):
    P, I, L = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    fn = getattr(lib_, "tyr_skinny_gemm_bf16", None)
    if fn is not None:
        fn.argtypes = [P, P, P, P, L, L, L, I, I, I, P]
        fn.restype = I
    F = ctypes.c_float
    for name, args in (("tyr_skinny_gemm_act_bf16", [P, P, P, P, L, L, L, I, I, I, I, F, F, P]),
                       ("tyr_skinny_heads_bf16", [P, P, P, L, L, L, L, L, L, I, I, I, I, P]),
                       ("tyr_skinny_gelu_mul_bf16", [P, P, P, P, L, L, L, L, I, I, I, P]),
                       ("tyr_skinny_many_bf16", [P, L, I, P, P, P, P, P, I, I, I, P]),
                       ("tyr_skinny_norm_many_bf16", [P, P, P, P, L, L, I, P, P, P, P, P, I, I, F, I, P]),
                       ("tyr_skinny_norm_swiglu_bf16", [P, P, P, P, L, L, P, P, P, L, I, I, I, F, I, P])):
        fn = getattr(lib_, name, None)
        if fn is not None:
            fn.argtypes, fn.restype = args, I
    fn = getattr(lib_, "tyr_skinny_swiglu_bf16", None)
    if fn is not None:
        fn.argtypes = [P, P, P, P, L, L, L, I, I, I, P]
        fn.restype = I


LINEAR_MAX_ROWS = 16     # plain products above this many rows go to the library GEMM (measured 2.5x faster at 32 rows)


def supported(x2: torch.Tensor, w: torch.Tensor, max_rows: int = LINEAR_MAX_ROWS) -> bool:
    M, K = x2.shape
    # 9..16 rows with a long contraction leave too few loads in flight per warp; the library GEMM is faster there
    return (x2.is_cuda and x2.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and 1 <= M <= min(max_rows, MAX_ROWS) and (M <= 8 or K <= 8192) and K >= 32 and K % 32 == 0
            and x2.stride(1) == 1 and w.stride(1) == 1 and x2.stride(0) % 8 == 0 and w.stride(0) % 8 == 0
            and x2.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


def skinny_linear(x2: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """x2: [M <= 32, K] bf16, w: [N, K] bf16 (rows may be strided) -> [M, N] bf16 with fp32 accumulation; ``out`` (rows may be
    strided, e.g. a window of a symmetric-heap buffer) receives the result when given."""
    M, K = x2.shape
    N = w.shape[0]
    if not x2.is_cuda:
        y = x2.float() @ w.float().T
        y = (y if bias is None else y + bias.float()).to(x2.dtype)
        if out is not None:
            out.copy_(y)
            return out
        return y
    y = torch.empty((M, N), dtype=torch.bfloat16, device=x2.device) if out is None else out
    assert y.shape == (M, N) and y.dtype == torch.bfloat16 and y.stride(1) == 1
    b = None if bias is None else bias.to(torch.bfloat16).contiguous()
    check(lib().tyr_skinny_gemm_bf16(ptr(x2), ptr(w), ptr(b), ptr(y), x2.stride(0), w.stride(0), y.stride(0), M, N, K, cur_stream(x2.device)), "skinny_gemm_bf16")
    return y


def shared_launch(M: int, K: int, widths: Sequence[int]) -> List[int]:
    """Which of the matrices [N_i, K] are best read by one launch over M rows; the others are left to the products of their own.

    Up to 8 rows a launch holds 888 tiles of 16 columns at once, and a few tiles more are a wave of their own: 12288, 1024 and 1024 columns of 5120 take 35.2 us in
    one launch, and 23.1 and 6.9 with the widest by itself.  Above 16 rows the tensor-core kernel does not take narrow matrices and the library stands against the
    shared launch, at about 2.5 us and 1.5 a 1024 channels a matrix whatever its width, where the launch takes 4.5 us and one more a million numbers.
    20 rows, library / shared: two of 1024 x 4096 17.2 / 10.7, two of 2048 x 4096 15.7 / 19.1, 4096 x 5120 10.6 / 24.2, two of 48 x 5120 16.1 / 6.1."""
    idx = sorted(range(len(widths)), key=widths.__getitem__)
    if M > LINEAR_MAX_ROWS:
        while idx and 4.5 + 1e-6 * K * sum(widths[i] for i in idx) >= len(idx) * (2.5 + 1.5e-3 * K):
            idx.pop()
    elif M <= 8 and len(idx) > 1:
        tiles = [-(-widths[i] // 16) for i in idx]
        if tiles[-1] <= 888 < sum(tiles) <= 976:
            idx.pop()
    return sorted(idx)


def skinny_many(x2: torch.Tensor, ws: Sequence[torch.Tensor], splits: int = 0) -> List[torch.Tensor]:
    """``[x2 w^T for w in ws]`` in one launch: x2 [M <= 32, K] bf16, up to four matrices [N_i, K] bf16 (rows may be strided).  ``splits``: CTAs
    of a cluster that share a contraction (0: by size)."""
    M, K = x2.shape
    if not x2.is_cuda:
        return [(x2.float() @ w.float().T).to(x2.dtype) for w in ws]
    if not (all(w.shape[1] == K and w.dtype == torch.bfloat16 and w.stride(1) == 1 and w.device == x2.device for w in ws) and x2.dtype == torch.bfloat16 and x2.stride(1) == 1):
        raise ValueError("skinny_many takes bf16 rows and matrices over one contraction")
    n = len(ws)
    ys = [torch.empty((M, w.shape[0]), dtype=torch.bfloat16, device=x2.device) for w in ws]
    P, L, I = ctypes.c_void_p * n, ctypes.c_longlong * n, ctypes.c_int * n
    check(lib().tyr_skinny_many_bf16(ptr(x2), x2.stride(0), n, P(*[w.data_ptr() for w in ws]), P(*[y.data_ptr() for y in ys]), L(*[w.stride(0) for w in ws]),
                                     L(*[y.stride(0) for y in ys]), I(*[w.shape[0] for w in ws]), M, K, splits, cur_stream(x2.device)), "skinny_many")
    return ys


NORM_NUMBERS = 16384       # of the normalised rows that a CTA of the forms below keeps


def norm_supported(x2: torch.Tensor, norm_w: torch.Tensor, ws: Sequence[torch.Tensor]) -> bool:
    """Up to 8 rows whose norm every CTA of the products takes again."""
    M, K = x2.shape
    return (len(ws) <= MAX_MATRICES and M <= 8 and M * (K + 8) <= NORM_NUMBERS and all(supported(x2, w) and w.shape[1] == K for w in ws)
            and norm_w.dtype == torch.bfloat16 and norm_w.is_contiguous() and norm_w.data_ptr() % 16 == 0 and norm_w.numel() == K)


def norm_fit(x2: torch.Tensor, resid: Optional[torch.Tensor], norm_w: torch.Tensor, ws: Sequence[torch.Tensor]) -> bool:
    """Types, shapes and devices of the norm's operands and of the matrices behind it go together."""
    M, K = x2.shape
    return (all(t.dtype == torch.bfloat16 and t.device == x2.device for t in (x2, norm_w, *ws, *(() if resid is None else (resid,))))
            and (resid is None or resid.shape == x2.shape) and norm_w.shape == (K,) and norm_w.is_contiguous()
            and all(w.dim() == 2 and w.shape[1] == K and w.stride(1) == 1 for w in ws))


def _norm_operands(x2, resid, norm_w, ws):
    if not norm_fit(x2, resid, norm_w, ws):
        raise ValueError(f"norm and products of rows {tuple(x2.shape)} ({x2.dtype}) take bf16 operands over the same channels, on one device")
    M, K = x2.shape
    r = None if resid is None else resid if resid.stride(1) == 1 and resid.stride(0) % 8 == 0 and resid.data_ptr() % 16 == 0 else resid.contiguous()
    return r, None if r is None else torch.empty((M, K), dtype=x2.dtype, device=x2.device), 0 if r is None else r.stride(0)


def skinny_norm_many(x2: torch.Tensor, resid: Optional[torch.Tensor], norm_w: torch.Tensor, eps: float, ws: Sequence[torch.Tensor], one_plus_w: bool = False):
    """``([h w^T for w in ws], s)`` with ``s = x2 + resid`` (bf16; x2 itself without ``resid``) and h its RMS norm times the gain, in one launch."""
    M, K = x2.shape
    r, out, ldr = _norm_operands(x2, resid, norm_w, ws)
    n = len(ws)
    ys = [torch.empty((M, w.shape[0]), dtype=torch.bfloat16, device=x2.device) for w in ws]
    P, L, I = ctypes.c_void_p * n, ctypes.c_longlong * n, ctypes.c_int * n
    check(lib().tyr_skinny_norm_many_bf16(ptr(x2), ptr(r), ptr(norm_w), ptr(out), x2.stride(0), ldr, n, P(*[w.data_ptr() for w in ws]),
                                          P(*[y.data_ptr() for y in ys]), L(*[w.stride(0) for w in ws]), L(*[y.stride(0) for y in ys]),
                                          I(*[w.shape[0] for w in ws]), M, K, eps, 1 if one_plus_w else 0, cur_stream(x2.device)), "skinny_norm_many")
    return ys, x2 if out is None else out


def skinny_norm_swiglu(x2: torch.Tensor, resid: Optional[torch.Tensor], norm_w: torch.Tensor, eps: float, gate_w: torch.Tensor, up_w: torch.Tensor,
                       one_plus_w: bool = False):
    """``(silu(h gate_w^T) * (h up_w^T), s)`` with h and s as in :func:`skinny_norm_many`."""
    M, K = x2.shape
    N = gate_w.shape[0]
    if up_w.shape != gate_w.shape or up_w.stride() != gate_w.stride():
        raise ValueError(f"gate and up matrices {tuple(gate_w.shape)} and {tuple(up_w.shape)} differ in shape or strides")
    r, out, ldr = _norm_operands(x2, resid, norm_w, (gate_w, up_w))
    y = torch.empty((M, N), dtype=torch.bfloat16, device=x2.device)
    check(lib().tyr_skinny_norm_swiglu_bf16(ptr(x2), ptr(r), ptr(norm_w), ptr(out), x2.stride(0), ldr, ptr(gate_w), ptr(up_w), ptr(y), gate_w.stride(0), M, N, K,
                                            eps, 1 if one_plus_w else 0, cur_stream(x2.device)), "skinny_norm_swiglu")
    return y, x2 if out is None else out


_SWIGLU = os.environ.get("TYR_SKINNY_SWIGLU", "1") != "0"


def swiglu_supported(x2: torch.Tensor, gate_w: torch.Tensor, up_w: torch.Tensor) -> bool:
    # the gated form replaces a library product plus two element-wise launches and stays ahead of them up to 32 rows
    return (_SWIGLU and supported(x2, gate_w, MAX_ROWS) and supported(x2, up_w, MAX_ROWS) and gate_w.shape == up_w.shape and gate_w.stride(0) == up_w.stride(0)
            and hasattr(lib(), "tyr_skinny_swiglu_bf16"))


def skinny_swiglu(x2: torch.Tensor, gate_w: torch.Tensor, up_w: torch.Tensor) -> torch.Tensor:
    """x2: [M <= 32, K] bf16 -> silu(x2 gate_w^T) * (x2 up_w^T) as [M, N] bf16: both matrices streamed once, one launch."""
    M, K = x2.shape
    N = gate_w.shape[0]
    if not x2.is_cuda:
        return (torch.nn.functional.silu(x2.float() @ gate_w.float().T) * (x2.float() @ up_w.float().T)).to(x2.dtype)
    y = torch.empty((M, N), dtype=torch.bfloat16, device=x2.device)
    check(lib().tyr_skinny_swiglu_bf16(ptr(x2), ptr(gate_w), ptr(up_w), ptr(y), x2.stride(0), gate_w.stride(0), N, M, N, K, cur_stream(x2.device)),
          "skinny_swiglu")
    return y


def skinny_xielu(x2: torch.Tensor, w: torch.Tensor, a: float, b: float) -> torch.Tensor:
    """x2: [M <= 32, K] bf16 -> xIELU of ``x2 w^T`` (factors ``a`` above zero, ``b`` below) as [M, N] bf16, in the product's epilogue."""
    M, K = x2.shape
    N = w.shape[0]
    y = torch.empty((M, N), dtype=torch.bfloat16, device=x2.device)
    check(lib().tyr_skinny_gemm_act_bf16(ptr(x2), ptr(w), None, ptr(y), x2.stride(0), w.stride(0), N, M, N, K, 6, a, b, cur_stream(x2.device)),
          "skinny_xielu")
    return y


def skinny_gelu_mul(x2: torch.Tensor, w: torch.Tensor, e: torch.Tensor) -> torch.Tensor:
    """x2: [M <= 32, K] bf16 -> tanh-GELU of ``x2 w^T`` times ``e`` [M, N] (rows may be strided) as [M, N] bf16, in the product's epilogue."""
    M, K = x2.shape
    N = w.shape[0]
    assert e.shape == (M, N) and e.dtype == torch.bfloat16 and e.stride(1) == 1
    y = torch.empty((M, N), dtype=torch.bfloat16, device=x2.device)
    check(lib().tyr_skinny_gelu_mul_bf16(ptr(x2), ptr(w), ptr(e), ptr(y), x2.stride(0), w.stride(0), e.stride(0), N, M, N, K, cur_stream(x2.device)),
          "skinny_gelu_mul")
    return y


def head_products_supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype == w.dtype == torch.bfloat16 and w.shape[2] % 32 == 0 and x.stride(2) == w.stride(2) == 1
            and all(s % 8 == 0 for s in (*x.stride()[:2], *w.stride()[:2])) and x.data_ptr() % 16 == w.data_ptr() % 16 == 0)


def head_products(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """A matrix of its own for each head: out[m, h, :N] = x[m, h, :K] w[h]^T.  x: [M, H, >= K] and out: [M, H, >= N] (views with contiguous
    channels), w: [H, N, K].  Channels of x past K and of out past N are left alone."""
    M, H = x.shape[:2]
    _, N, K = w.shape
    if not head_products_supported(x, w):
        out[..., :N] = torch.einsum("mhk,hnk->mhn", x[..., :K], w) if x.is_cuda else torch.einsum("mhk,hnk->mhn", x[..., :K].float(), w.float()).to(out.dtype)
        return out
    assert x.shape[2] >= K and out.shape[:2] == (M, H) and out.shape[2] >= N and out.stride(2) == 1 and out.dtype == x.dtype
    for m in range(0, M, MAX_ROWS):
        n = min(MAX_ROWS, M - m)
        check(lib().tyr_skinny_heads_bf16(ptr(x[m:]), ptr(w), ptr(out[m:]), x.stride(0), x.stride(1), w.stride(0), w.stride(1), out.stride(0), out.stride(1),
                                          H, n, N, K, cur_stream(x.device)), "skinny_heads")
    return out

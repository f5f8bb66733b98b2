"""Element-wise passes of a gated full-attention layer over prompts (csrc/prompt_mix.cu): normalised and rotated queries, keys and values
in the store, and the gated output.  Off the GPU and for what the kernels do not take, callers keep the plain operations."""
from __future__ import annotations

import ctypes

import torch

from .._native import register_signatures
from ._common import check, cur_stream, lib, ptr


@register_signatures
def _sigs(lib_):
    P, I, L, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    for name, args in (("tyr_attention_operands", [P, P, P, ctypes.POINTER(L), P, P, P, P, P, P, P, ctypes.POINTER(I), F, P]),
                       ("tyr_attention_gate", [P, P, ctypes.POINTER(L), P, L, I, I, I, P])):
        fn = getattr(lib_, name, None)
        if fn is not None:
            fn.argtypes, fn.restype = args, I


def _rows(t: torch.Tensor) -> bool:
    """[B, S, C] whose rows are evenly spaced over the batch, 16-byte aligned."""
    return (t.stride(2) == 1 and t.stride(0) % 8 == 0 and t.stride(1) % 8 == 0 and t.data_ptr() % 16 == 0
            and (t.shape[0] == 1 or t.shape[1] == 1 or t.stride(0) == t.shape[1] * t.stride(1)))


def operands_fit(q, k, v, store, q_norm, k_norm, cos, D: int, sin=None) -> bool:
    """The part of :func:`operands_supported` that does not ask where the tensors lie.  The kernel reads one row of the tables for each token, so tables
    that broadcast over the tokens are not for it."""
    bf16, f32 = torch.bfloat16, torch.float32
    B, S, C = q.shape
    sin = cos if sin is None else sin
    if not (q.dtype == k.dtype == v.dtype == q_norm.dtype == k_norm.dtype == bf16 and cos.dtype == sin.dtype == f32 and D % 8 == 0 and D <= 256
            and cos.dim() == 2 and store is not None and not store.ring):
        return False
    half, sk, sv = cos.shape[1], store.k, store.v
    return (cos.shape == sin.shape == (S, half) and half % 8 == 0 and 0 < 2 * half <= D and cos.is_contiguous() and sin.is_contiguous()
            and C % (2 * D) == 0 and k.shape == v.shape == (B, S, sk.shape[1] * D) and _rows(q) and _rows(k) and _rows(v)
            and sk.dtype == sv.dtype == bf16 and sk.shape == sv.shape and sk.shape[0] == B and sk.shape[3] == D and sk.is_contiguous() and sv.is_contiguous()
            and q_norm.shape == k_norm.shape == (D,) and q_norm.is_contiguous() and k_norm.is_contiguous()
            and (cos.data_ptr() | sin.data_ptr() | sk.data_ptr() | sv.data_ptr() | q_norm.data_ptr() | k_norm.data_ptr()) % 16 == 0)


def operands_supported(q, k, v, store, q_norm, k_norm, cos, D: int, sin=None) -> bool:
    """q, k, v: projections [B, S, C]; ``store``: a plain ``KVCache`` of bf16 rows of D; cos, sin: [S, half] fp32."""
    return q.is_cuda and operands_fit(q, k, v, store, q_norm, k_norm, cos, D, sin)


def attention_operands(q: torch.Tensor, q_head: int, k: torch.Tensor, v: torch.Tensor, q_norm: torch.Tensor, k_norm: torch.Tensor, cos: torch.Tensor,
                       sin: torch.Tensor, eps: float, H: int, G: int, D: int, store) -> torch.Tensor:
    """Queries [B, S, H, D] (head h of ``q`` starts at column ``h * q_head``) after norm and rotation; keys and values go to the slots of
    ``store`` behind its length, which is advanced."""
    B, S = q.shape[:2]
    if q.shape[2] != H * q_head or k.shape[2] != G * D or store.k.shape[1] != G or cos.shape[0] != S:
        raise ValueError(f"{H} and {G} heads of {D} over {S} tokens do not fit projections {tuple(q.shape)}, {tuple(k.shape)}, a store "
                         f"{tuple(store.k.shape)} and tables {tuple(cos.shape)}")
    if store.length + S > store.cap:
        raise ValueError(f"KV cache overflow: {store.length}+{S} > {store.cap}")
    out = torch.empty((B, S, H, D), dtype=q.dtype, device=q.device)
    row = lambda t: t.stride(1) if t.shape[1] > 1 else t.stride(0)
    strides = (ctypes.c_longlong * 4)(row(q), row(k), row(v), q_head)
    dims = (ctypes.c_int * 8)(B, S, H, G, D, cos.shape[1], store.cap, store.length)
    check(lib().tyr_attention_operands(ptr(q), ptr(k), ptr(v), strides, ptr(q_norm), ptr(k_norm), ptr(cos), ptr(sin), ptr(out), ptr(store.k), ptr(store.v), dims,
                                       eps, cur_stream(q.device)), "attention_operands")
    store.length += S
    return out


def attention_gate(o: torch.Tensor, gate: torch.Tensor, gate_head: int) -> torch.Tensor:
    """o [B, S, H, D] (a view) times sigmoid(gate) -> [B, S, H * D]; ``gate`` [B, S, C]: head h's gates start at column ``h * gate_head``."""
    B, S, H, D = o.shape
    y = torch.empty((B, S, H * D), dtype=o.dtype, device=o.device)
    strides = (ctypes.c_longlong * 5)(o.stride(0), o.stride(1), o.stride(2), gate.stride(1) if S > 1 else gate.stride(0), gate_head)
    check(lib().tyr_attention_gate(ptr(o), ptr(gate), strides, ptr(y), B * S, S, H, D, cur_stream(o.device)), "attention_gate")
    return y

"""Bindings of the fused token-generation projections (``csrc/decode_fused.cu``): RMSNorm + fused QKV GEMV + RoPE + KV-cache
write in one launch, RMSNorm + gate/up GEMV + SwiGLU in one launch.  With the two row-parallel GEMVs that take the
residual in their epilogue (``fused_comm.skinny_gemm``) and the decode attention (split + merge) a decoder layer of the
token-generation graph is six launches (reference graph: ``examples/inference/modules/model_base.py:459-518``).  One sequence of the
compiled layer sizes takes all layers in one launch instead (``token_stack``).

Batches of 1 to 128 sequences on one process take the tensor-core counterparts (``csrc/gemm_smallm.cu``: weight rows as the
UMMA M dimension, cluster split-K) unless the weights are small (``gemm.streams_on_tensor_cores``): fused QKV GEMM + RoPE + cache
write, gate/up GEMM + SwiGLU (<= 64 rows), and the plain GEMM with the residual in its epilogue.  Few sequences of a narrow model
(``norm_fits``) have the two RMSNorms inside the projections behind them, six launches per layer; else they are launches of their own,
eight.  Their weights are fetched before the kernel in front has ended, so no kernel that may still run may write them."""
from __future__ import annotations

import ctypes as _c
from typing import Optional, Sequence, Tuple

import torch

from . import _lib

MAX_ROWS = 8
BATCHED_MAX_ROWS = 128          # gemm_smallm kernels
BATCHED_SWIGLU_MAX_ROWS = 64


def qualifies(x: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and 1 <= x.shape[0] <= MAX_ROWS
            and x.shape[1] % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and _lib.available())


def qkv_rope_cache(x: torch.Tensor, norm_w: Optional[torch.Tensor], eps: float, w_qkv: torch.Tensor, cos: torch.Tensor,
                   sin: torch.Tensor, positions: torch.Tensor, cache_k: torch.Tensor, cache_v: torch.Tensor, n_q: int,
                   n_kv: int, D: int, seq_ids: Optional[torch.Tensor] = None, block_table: Optional[torch.Tensor] = None,
                   page_size: int = 0) -> torch.Tensor:
    """``x [B, H]`` -> ``q [B, n_q, D]`` (rotated); the rotated K row and the V row of every sequence are written into
    the cache at ``positions[b]``.  ``positions`` / ``seq_ids`` / ``block_table`` must be int32."""
    B, K = x.shape
    assert w_qkv.shape == ((n_q + 2 * n_kv) * D, K) and w_qkv.stride(1) == 1
    assert positions.dtype == torch.int32 and cos.dtype == torch.float32 and cos.shape[1] == D // 2
    q = torch.empty((B, n_q, D), dtype=torch.bfloat16, device=x.device)
    rc = _lib.lib().nxd_decode_qkv_rope_cache(
        _lib.ptr(x), _c.c_longlong(x.stride(0)), _lib.ptr(norm_w), _c.c_float(eps), _lib.ptr(w_qkv),
        _c.c_longlong(w_qkv.stride(0)), _lib.ptr(cos), _lib.ptr(sin), _lib.ptr(positions), _lib.ptr(q), _lib.ptr(cache_k),
        _lib.ptr(cache_v), _lib.ptr(seq_ids), _lib.ptr(block_table), _c.c_longlong(cache_k.stride(0)),
        _c.c_longlong(cache_k.stride(1)), _c.c_int(page_size), _c.c_int(block_table.shape[1] if block_table is not None else 0),
        _c.c_int(B), _c.c_int(K), _c.c_int(n_q), _c.c_int(n_kv), _c.c_int(D), _lib.stream_ptr())
    _lib.check(rc, "nxd_decode_qkv_rope_cache")
    return q


def gate_up_swiglu(x: torch.Tensor, norm_w: Optional[torch.Tensor], eps: float, w_gate_up: torch.Tensor) -> torch.Tensor:
    """``silu(W_gate n(x)) * (W_up n(x))`` for ``x [B, H]``; ``w_gate_up [2 I, H]`` holds the gate rows first."""
    B, K = x.shape
    I = w_gate_up.shape[0] // 2
    assert w_gate_up.shape[1] == K and w_gate_up.stride(1) == 1
    out = torch.empty((B, I), dtype=torch.bfloat16, device=x.device)
    rc = _lib.lib().nxd_decode_gate_up_swiglu(
        _lib.ptr(x), _c.c_longlong(x.stride(0)), _lib.ptr(norm_w), _c.c_float(eps), _lib.ptr(w_gate_up),
        _c.c_longlong(w_gate_up.stride(0)), _lib.ptr(out), _c.c_longlong(out.stride(0)), _c.c_int(B), _c.c_int(K),
        _c.c_int(I), _lib.stream_ptr())
    _lib.check(rc, "nxd_decode_gate_up_swiglu")
    return out


def qualifies_batched(x: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and 1 <= x.shape[0] <= BATCHED_MAX_ROWS
            and x.shape[1] % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and _lib.available())


def qkv_rope_cache_batched(xn: torch.Tensor, w_qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor,
                           positions: torch.Tensor, cache_k: torch.Tensor, cache_v: torch.Tensor, n_q: int, n_kv: int,
                           D: int, seq_ids: Optional[torch.Tensor] = None, block_table: Optional[torch.Tensor] = None,
                           page_size: int = 0, splits: int = 0) -> torch.Tensor:
    """``xn [B, H]`` (already normalised, ``1 <= B <= 128``) -> ``q [B, n_q, D]`` rotated; rotated K rows and V rows go into
    the cache at ``positions[b]`` -- ONE tensor-core launch (``nxd_smallm_qkv_rope_cache``)."""
    B, K = xn.shape
    assert w_qkv.shape == ((n_q + 2 * n_kv) * D, K) and w_qkv.stride(1) == 1
    assert positions.dtype == torch.int32 and cos.dtype == torch.float32 and cos.shape[1] == D // 2
    q = torch.empty((B, n_q, D), dtype=torch.bfloat16, device=xn.device)
    rc = _lib.lib().nxd_smallm_qkv_rope_cache(
        _lib.ptr(xn), _c.c_longlong(xn.stride(0)), _lib.ptr(w_qkv), _c.c_longlong(w_qkv.stride(0)), _lib.ptr(cos),
        _lib.ptr(sin), _lib.ptr(positions), _lib.ptr(q), _lib.ptr(cache_k), _lib.ptr(cache_v), _lib.ptr(seq_ids),
        _lib.ptr(block_table), _c.c_longlong(cache_k.stride(0)), _c.c_longlong(cache_k.stride(1)), _c.c_int(page_size),
        _c.c_int(block_table.shape[1] if block_table is not None else 0), _c.c_int(B), _c.c_int(K), _c.c_int(n_q),
        _c.c_int(n_kv), _c.c_int(D), _c.c_int(splits), _lib.stream_ptr())
    _lib.check(rc, "nxd_smallm_qkv_rope_cache")
    return q


def norm_fits(x: torch.Tensor, w: torch.Tensor, gate_up: bool) -> bool:
    """Whether ``norm_qkv_rope_cache`` / ``norm_gate_up_swiglu`` take these rows (few and narrow: ``csrc/gemm_smallm.cu`` has the
    measurements)."""
    B, K = x.shape
    return (1 <= B <= MAX_ROWS and K % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and bool(
        _lib.lib().nxd_smallm_norm_applies(_c.c_int(int(gate_up)), _c.c_int(B), _c.c_int(K),
                                           _c.c_int(w.shape[0] // 2 if gate_up else w.shape[0]))))


def norm_qkv_rope_cache(x: torch.Tensor, norm_w: torch.Tensor, eps: float, w_qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor,
                        positions: torch.Tensor, cache_k: torch.Tensor, cache_v: torch.Tensor, n_q: int, n_kv: int, D: int,
                        seq_ids: Optional[torch.Tensor] = None, block_table: Optional[torch.Tensor] = None,
                        page_size: int = 0) -> torch.Tensor:
    """``qkv_rope_cache_batched`` of ``rmsnorm(x) * norm_w``: the projection's kernel normalises its rows itself
    (``nxd_smallm_norm_qkv_rope_cache``)."""
    B, K = x.shape
    assert w_qkv.shape == ((n_q + 2 * n_kv) * D, K) and w_qkv.stride(1) == 1 and norm_w.is_contiguous()
    assert positions.dtype == torch.int32 and cos.dtype == torch.float32 and cos.shape[1] == D // 2
    q = torch.empty((B, n_q, D), dtype=torch.bfloat16, device=x.device)
    rc = _lib.lib().nxd_smallm_norm_qkv_rope_cache(
        _lib.ptr(x), _c.c_longlong(x.stride(0)), _lib.ptr(norm_w), _c.c_float(eps), _lib.ptr(w_qkv),
        _c.c_longlong(w_qkv.stride(0)), _lib.ptr(cos), _lib.ptr(sin), _lib.ptr(positions), _lib.ptr(q), _lib.ptr(cache_k),
        _lib.ptr(cache_v), _lib.ptr(seq_ids), _lib.ptr(block_table), _c.c_longlong(cache_k.stride(0)),
        _c.c_longlong(cache_k.stride(1)), _c.c_int(page_size), _c.c_int(block_table.shape[1] if block_table is not None else 0),
        _c.c_int(B), _c.c_int(K), _c.c_int(n_q), _c.c_int(n_kv), _c.c_int(D), _lib.stream_ptr())
    _lib.check(rc, "nxd_smallm_norm_qkv_rope_cache")
    return q


def norm_gate_up_swiglu(x: torch.Tensor, norm_w: torch.Tensor, eps: float, w_gate_up: torch.Tensor) -> torch.Tensor:
    """``gate_up_swiglu_batched`` of ``rmsnorm(x) * norm_w`` (``nxd_smallm_norm_gate_up_swiglu``)."""
    B, K = x.shape
    I = w_gate_up.shape[0] // 2
    assert w_gate_up.shape[1] == K and w_gate_up.stride(1) == 1 and I % 8 == 0 and norm_w.is_contiguous()
    out = torch.empty((B, I), dtype=torch.bfloat16, device=x.device)
    rc = _lib.lib().nxd_smallm_norm_gate_up_swiglu(
        _lib.ptr(x), _c.c_longlong(x.stride(0)), _lib.ptr(norm_w), _c.c_float(eps), _lib.ptr(w_gate_up),
        _c.c_longlong(w_gate_up.stride(0)), _lib.ptr(out), _c.c_longlong(out.stride(0)), _c.c_int(B), _c.c_int(K), _c.c_int(I),
        _lib.stream_ptr())
    _lib.check(rc, "nxd_smallm_norm_gate_up_swiglu")
    return out


def gate_up_swiglu_batched(xn: torch.Tensor, w_gate_up: torch.Tensor, splits: int = 0) -> torch.Tensor:
    """``silu(xn W_gate^T) * (xn W_up^T)`` for ``xn [B, H]``, ``B <= 64``; ``w_gate_up [2 I, H]`` gate rows first: one
    launch with two accumulators per CTA (``nxd_smallm_gate_up_swiglu``)."""
    B, K = xn.shape
    I = w_gate_up.shape[0] // 2
    assert B <= BATCHED_SWIGLU_MAX_ROWS and w_gate_up.shape[1] == K and w_gate_up.stride(1) == 1 and I % 8 == 0
    out = torch.empty((B, I), dtype=torch.bfloat16, device=xn.device)
    rc = _lib.lib().nxd_smallm_gate_up_swiglu(
        _lib.ptr(xn), _c.c_longlong(xn.stride(0)), _lib.ptr(w_gate_up), _c.c_longlong(w_gate_up.stride(0)), _lib.ptr(out),
        _c.c_longlong(out.stride(0)), _c.c_int(B), _c.c_int(K), _c.c_int(I), _c.c_int(splits), _lib.stream_ptr())
    _lib.check(rc, "nxd_smallm_gate_up_swiglu")
    return out


def token_stack_scratch(layers: int, B: int, H: int, I: int, n_q: int, n_kv: int, D: int) -> int:
    """Bytes of scratch with which ``token_stack`` takes such layers, 0 where it does not (``csrc/token_stack.cu``)."""
    fn = _lib.lib().nxd_token_stack_scratch
    fn.restype = _c.c_longlong
    return int(fn(*(_c.c_int(v) for v in (layers, B, H, I, n_q, n_kv, D))))


def token_stack_runs_here() -> bool:
    """Whether the current stream has all SMs of the device, as ``token_stack`` needs (one of a green context has not)."""
    return bool(_lib.lib().nxd_token_stack_runs_on(_lib.stream_ptr()))


def token_stack(x: torch.Tensor, layers: Sequence[Tuple[Sequence[torch.Tensor], float, float]], cos: torch.Tensor, sin: torch.Tensor,
                positions: torch.Tensor, lengths: torch.Tensor, n_q: int, n_kv: int, D: int, scratch: int,
                seq_ids: Optional[torch.Tensor] = None, block_table: Optional[torch.Tensor] = None, page_size: int = 0,
                wait_clocks: int = -1, gave_up: Optional["GaveUp"] = None) -> torch.Tensor:
    """A token-generation step ``x [1, H]`` through whole decoder layers in one launch -> ``[1, H]`` (``nxd_token_stack``).  A layer is
    ``((input norm, q|k|v, o, norm behind the attention, gate|up, down, cache of keys, of values), eps, eps)``; the caches are written
    at ``positions``.  ``scratch``: bytes, of ``token_stack_scratch``.  ``wait_clocks``: clocks after which a wait inside gives up, -1:
    two seconds (``gave_up`` and ``token_stack_gave_up`` say so then)."""
    H = x.shape[1]
    tensors = [t for layer in layers for t in layer[0]]
    ck = layers[0][0][6]
    assert x.shape[0] == 1 and x.is_contiguous() and cos.is_contiguous() and sin.is_contiguous() and cos.shape[1] == D // 2
    assert all(t.dtype == torch.bfloat16 for t in tensors) and all(t.stride() == ck.stride() for s, _, _ in layers for t in s[6:])
    assert all(t.is_contiguous() for s, _, _ in layers for t in s[:6]) and positions.dtype == lengths.dtype == torch.int32
    out = torch.empty_like(x)
    work = torch.empty(scratch, dtype=torch.uint8, device=x.device)
    pointers = (_c.c_void_p * len(tensors))(*(t.data_ptr() for t in tensors))
    eps = (_c.c_float * (2 * len(layers)))(*(e for layer in layers for e in layer[1:]))
    rc = _lib.lib().nxd_token_stack_telling(
        _lib.ptr(x), _lib.ptr(out), pointers, eps, _c.c_int(len(layers)), _lib.ptr(cos), _lib.ptr(sin), _lib.ptr(positions),
        _lib.ptr(lengths), _lib.ptr(seq_ids), _lib.ptr(block_table), _c.c_longlong(ck.stride(0)), _c.c_longlong(ck.stride(1)),
        _c.c_int(page_size), _c.c_int(block_table.shape[1] if block_table is not None else 0), _lib.ptr(work), _c.c_int(H),
        _c.c_int(layers[0][0][5].shape[1]), _c.c_int(n_q), _c.c_int(n_kv), _c.c_int(D), _c.c_float(D ** -0.5),
        _c.c_longlong(wait_clocks), _lib.ptr(gave_up.word) if gave_up is not None else None, _lib.stream_ptr())
    _lib.check(rc, "nxd_token_stack_telling")
    return out


class GaveUp:
    """A word of pinned host memory that a ``token_stack`` whose waits gave up sets: read without a copy, of use once the step has ended."""

    def __init__(self):
        self.word = torch.zeros(1, dtype=torch.int32, device="cpu", pin_memory=torch.cuda.is_available())
        self._view = self.word.numpy()

    def take(self) -> bool:
        """Whether it was set since the last call."""
        told = bool(self._view[0])
        if told:
            self._view[0] = 0
        return told

    def __deepcopy__(self, memo):
        return GaveUp()

    def __reduce__(self):
        return GaveUp, ()


def token_stack_gave_up() -> bool:
    """Whether a ``token_stack`` on this device has given up a wait since the last call (its results are NaN).  Waits for the stream."""
    flag = _c.c_int(0)
    _lib.check(_lib.lib().nxd_token_stack_status(_c.byref(flag), _lib.stream_ptr()), "nxd_token_stack_status")
    return bool(flag.value)

"""Python face of the tcgen05 GEMM (csrc/src/gemm_sm100.cu).

``gemm(a, w)`` computes ``a @ w.T`` for bf16 ``a [M, K]`` and ``w [N, K]`` (the nn.Linear weight layout) with
fp32 accumulation in tensor memory.  ``gemm_swiglu(a, w_interleaved)`` fuses ``silu(gate) * up`` into the
epilogue; ``interleave_gate_up`` prepares the weight for it once at load time.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from .. import _native, _stream

EPI_STORE, EPI_SWIGLU = 0, 1
_declared = False


def _lib():
    global _declared
    lib = _native.cuda()
    if not _declared:
        vp, i = C.c_void_p, C.c_int
        lib.purlin_gemm_bf16.argtypes = [vp, vp, vp, i, i, i, i, i, vp, vp]
        lib.purlin_gemm_grouped_bf16.argtypes = [vp, vp, vp, i, i, i, i, vp, i, i, vp, C.c_uint64, vp]
        _declared = True
    return lib


def _check(a: torch.Tensor, w: torch.Tensor):
    if a.dtype != torch.bfloat16 or w.dtype != torch.bfloat16:
        raise TypeError("the tcgen05 GEMM takes bf16 operands")
    if not (a.is_cuda and w.is_cuda and a.is_contiguous() and w.is_contiguous()):
        raise ValueError("operands must be contiguous CUDA tensors")
    if a.shape[1] != w.shape[1]:
        raise ValueError("a is [M, K] and w is [N, K]")


def gemm(a: torch.Tensor, w: torch.Tensor, out: Optional[torch.Tensor] = None, bn: int = 0) -> torch.Tensor:
    _check(a, w)
    m, k = a.shape
    n = w.shape[0]
    if out is None:
        out = torch.empty(m, n, dtype=torch.bfloat16, device=a.device)
    lib = _lib()
    rc = lib.purlin_gemm_bf16(a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, EPI_STORE, bn, None,
                              _stream(None))
    _native.check(lib, rc)
    return out


def interleave_gate_up(w_gate: torch.Tensor, w_up: torch.Tensor) -> torch.Tensor:
    """[I, K] gate and up weights -> [2I, K] with rows alternating 16 of gate and 16 of up, so that one 32-column
    slice of an accumulator tile holds both factors of 16 output columns."""
    i, k = w_gate.shape
    if i % 16:
        raise ValueError("the intermediate size must be a multiple of 16")
    g = w_gate.reshape(i // 16, 16, k)
    u = w_up.reshape(i // 16, 16, k)
    return torch.stack([g, u], dim=1).reshape(2 * i, k).contiguous()


def gemm_swiglu(a: torch.Tensor, w_gu: torch.Tensor, out: Optional[torch.Tensor] = None, bn: int = 0) -> torch.Tensor:
    """out[M, I] = silu(a @ w_gate.T) * (a @ w_up.T) with ``w_gu = interleave_gate_up(w_gate, w_up)``."""
    _check(a, w_gu)
    m, k = a.shape
    n = w_gu.shape[0]
    if out is None:
        out = torch.empty(m, n // 2, dtype=torch.bfloat16, device=a.device)
    lib = _lib()
    rc = lib.purlin_gemm_bf16(a.data_ptr(), w_gu.data_ptr(), out.data_ptr(), m, n, k, EPI_SWIGLU, bn, None,
                              _stream(None))
    _native.check(lib, rc)
    return out


def grouped_gemm(a: torch.Tensor, w: torch.Tensor, counts: torch.Tensor, likely_rows: int, out: torch.Tensor, swiglu: bool = False,
                 status_ptr: int = 0, timeout_ns: int = 0) -> torch.Tensor:
    """``out[rows of e] = a[rows of e] @ w[e].T`` (or the SwiGLU form) for every expert e, in one launch: expert e owns
    ``counts[e]`` consecutive rows of ``a [rows, K]`` and ``w[e] [N, K]``; ``w`` is one contiguous tensor. ``counts`` (int32)
    stays on the device; rows beyond the sum of the counts are left alone. ``likely_rows`` says how many rows an expert is
    expected to have. ``status_ptr``: four device words for the first wait inside the kernel that took longer than
    ``timeout_ns`` (0: two seconds); rows that were not finished by then are left alone too."""
    if a.dtype != torch.bfloat16 or w.dtype != torch.bfloat16 or out.dtype != torch.bfloat16 or counts.dtype != torch.int32:
        raise TypeError("the grouped GEMM takes bf16 operands and int32 counts")
    if not (a.is_cuda and w.is_cuda and out.is_cuda and counts.is_cuda):
        raise ValueError("operands must be CUDA tensors")
    if not (a.is_contiguous() and w.is_contiguous() and out.is_contiguous() and counts.is_contiguous()):
        raise ValueError("operands must be contiguous")
    experts, n, k = w.shape
    if a.shape[1] != k or out.shape != (a.shape[0], n // 2 if swiglu else n) or counts.numel() < experts:
        raise ValueError("a is [rows, K], w is [experts, N, K], out is [rows, N or N / 2] and counts has an entry per expert")
    if swiglu and n % 32:
        raise ValueError("the SwiGLU epilogue needs N to be a multiple of 32 (16 rows of gate and 16 of up in turn)")
    lib = _lib()
    rc = lib.purlin_gemm_grouped_bf16(a.data_ptr(), w.data_ptr(), out.data_ptr(), a.shape[0], experts, n, k, counts.data_ptr(), likely_rows,
                                      EPI_SWIGLU if swiglu else EPI_STORE, status_ptr or None, timeout_ns, _stream(None))
    _native.check(lib, rc)
    return out

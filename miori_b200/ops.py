"""The tensor-level operators over the C ABI.  torch is used for device memory and streams only; every
computation happens in libmiori_b200.so.

The operators themselves are C functions (csrc/binding.cpp, built as _native.so): each checks its
tensors, allocates the output when none is given and enqueues on the current stream.  An operator's
device work is a few microseconds, so the call path is native as well.  As with the library there is
no fallback: without _native.so this module does not import.
"""
from __future__ import annotations

import torch

from ._lib import MioriError, check, lib
from . import _native

_native.bind(lib._handle, MioriError)

from ._native import (argmax, dequant4_cache, dequant4_rowmajor, dequant8_rowmajor, embed8,  # noqa: E402,F401
                      gemm_bf16_cache, gemm_bf16_strided, gemv4, gemv4_post_norm_add, gemv4_rmsnorm,
                      gemv4_rmsnorm_silu, gemv4_silu, gemv8, gemv8_rmsnorm, gemv_bf16_cache, linear4,
                      post_norm_add, rmsnorm, silu_mul)


def cache_to_rowmajor(cache, N, K):
    """The row-major [N][K] tensor behind a cache of dequant4_cache."""
    if not cache.is_cuda:
        raise ValueError("miori_b200 ops need CUDA tensors (there is no CPU path)")
    if not cache.is_contiguous():
        raise ValueError("miori_b200 ops need contiguous tensors")
    o = torch.empty((N, K), dtype=torch.bfloat16, device=cache.device)
    check(lib.miori_cache_to_rowmajor(cache.data_ptr(), o.data_ptr(), N, K, torch.cuda.current_stream().cuda_stream))
    return o


def gemm_workspace(M, N, K, device):
    """Scratch tensor of the size miori_gemm_workspace_bytes recommends, or None."""
    nbytes = lib.miori_gemm_workspace_bytes(M, N, K)
    return torch.empty(nbytes // 4, dtype=torch.float32, device=device) if nbytes else None

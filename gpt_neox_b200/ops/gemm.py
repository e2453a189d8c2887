"""16-bit (bf16 / fp16) GEMM front-end for the tcgen05 kernels in ``csrc/gemm_sm100.cu`` and ``csrc/gemm_2cta_sm100.cu``.

``gemm(a, b, ...)`` computes ``epilogue(alpha * op(a) @ op(b))`` where each operand is given as a
2-D tensor and a flag telling whether it is stored "K-major" (contraction index contiguous) or
"MN-major".  The three GEMMs of a linear layer map onto it without any transposition copy:

=========  =======================  ==================  ==================
pass       math                     A (stored)          B (stored)
=========  =======================  ==================  ==================
forward    Y[M,N] = X W^T           X[M,K]  K-major     W[N,K]  K-major
dgrad      dX[M,K] = dY W           dY[M,N] K-major     W[N,K]  MN-major
wgrad      dW[N,K] = dY^T X         dY[M,N] MN-major    X[M,K]  MN-major
=========  =======================  ==================  ==================

On CPU (no device) the same function evaluates the identical math with torch ops in fp32, which is
the oracle the GPU tests compare against.
"""
from __future__ import annotations

import ctypes

import torch
import torch.nn.functional as F

from . import flop_count, native

ACT_NONE, ACT_GELU, ACT_DGELU = 0, 1, 2


def gelu_tanh_ref(x):
    return F.gelu(x, approximate="tanh")


def dgelu_tanh_ref(x):
    k0, k1 = 0.7978845608028654, 0.044715
    t = torch.tanh(k0 * x * (1 + k1 * x * x))
    return 0.5 * x * ((1 - t * t) * (k0 + 3 * k0 * k1 * x * x)) + 0.5 * (1 + t)


def gemm_ref(a, b, a_mn=False, b_mn=False, out_dtype=torch.bfloat16, bias=None, add=None, act=ACT_NONE, aux=None,
             alpha=1.0, want_preact=False):
    """fp32 eager statement of the kernel's math (oracle and CPU path)."""
    A = a.float().t() if a_mn else a.float()          # [M, K]
    B = b.float() if b_mn else b.float().t()          # [K, N]
    v = alpha * (A @ B)
    if bias is not None:
        v = v + bias.float()
    pre = v.to(a.dtype if a.dtype in (torch.bfloat16, torch.float16) else torch.bfloat16) if want_preact else None
    if act == ACT_GELU:
        v = gelu_tanh_ref(v)
    elif act == ACT_DGELU:
        v = v * dgelu_tanh_ref(aux.float())
    if add is not None:
        v = v + add.float()
    v = v.to(out_dtype)
    return (v, pre) if want_preact else v


_PAIR = None


def use_pair_kernel(M, N, K):
    """The CTA-pair kernel (``csrc/gemm_2cta_sm100.cu``, 256 x 256 tiles on two SMs) pays off once the problem
    fills the machine with such tiles; small problems keep the one-CTA kernel.  ``NEOX_GEMM_2CTA=0/1`` forces it."""
    global _PAIR
    if _PAIR is None:
        import os
        _PAIR = os.environ.get("NEOX_GEMM_2CTA", "auto")
    if _PAIR == "0":
        return False
    if _PAIR == "1":
        return True
    return PAIR_DEFAULT and ((M + 255) // 256) * ((N + 255) // 256) >= 74 and K >= 256


PAIR_DEFAULT = True
SKINNY_MAX_M = 32       # csrc/gemm_skinny.cu
SKINNY_MAX_MNK = 1.75e9


def use_skinny_kernel(M, N, K, a_mn, b_mn):
    """The weight-streaming kernel (``csrc/gemm_skinny.cu``) takes the products of few rows with a K-major weight matrix:
    the linear layers of a decoding step.  It reads the rows of ``a`` again for every 16 rows of ``b``, so with more than 8 rows
    it only pays where the tile kernels do not fill the machine (N <= 8192), with 9 to 16 also while the product is small.
    Measured, us, this kernel and the tile kernel that would run: 16 rows 12288 x 4096 31.9 / 34.2, 50304 x 2048 51.6 / 53.2,
    18432 x 6144 52.2 / 50.1, 32000 x 4096 65.7 / 55.5; 12 rows 32000 x 4096 61.9 / 62.4, 24576 x 6144 71.8 / 63.4; 9 rows
    50432 x 6144 129 / 128; 32 rows 2048 x 8192 14.6 / 53.2, 8192 x 2048 15.6 / 18.9, 12288 x 4096 39.1 / 34.3, 50304 x 1024
    46.0 / 29.5; up to 8 rows it was faster everywhere (8 rows 50432 x 6144 109 / 147).
    ``NEOX_GEMM_2CTA=0/1`` forces one of the two tile kernels instead."""
    if M > SKINNY_MAX_M or a_mn or b_mn or K % 8 or (M > 8 and N > 8192 and (M > 16 or M * N * K > SKINNY_MAX_MNK)):
        return False
    use_pair_kernel(M, 1, 1)                # reads the switch
    return _PAIR not in ("0", "1")


def gemm_rowmap(a, b, row_ptrs, b_mn=False, bias=None):
    """``a @ op(b) + bias`` whose output row r is stored (bf16) at device address ``row_ptrs[r]`` (int64 tensor of
    M addresses, 16-byte aligned, possibly in other GPUs' peer-mapped memory) instead of into one matrix."""
    assert a.is_cuda and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and row_ptrs.dtype == torch.int64
    M, K = a.shape
    N = b.shape[1] if b_mn else b.shape[0]
    assert row_ptrs.numel() == M and N % 8 == 0
    if M == 0:
        return
    rc = native.lib().neox_gemm_bf16_rowmap(
        native.ptr(a), native.ptr(b), None, M, N, K, ctypes.c_longlong(a.stride(0)), ctypes.c_longlong(b.stride(0)),
        ctypes.c_longlong(N), 0, int(b_mn), 0, native.ptr(bias), None, ctypes.c_longlong(0), 0, None,
        ctypes.c_longlong(0), None, ctypes.c_longlong(0), ACT_NONE, ctypes.c_float(1.0), native.ptr(row_ptrs),
        ctypes.c_void_p(native.stream_ptr()))
    native.check(rc, "neox_gemm_bf16_rowmap")


def _accumulates(out, bias, add, act, pre):
    """``out += alpha * op(a) @ op(b)`` in fp32 and nothing else: the form that may split its contraction."""
    return (add is not None and out.dtype == torch.float32 and add.dtype == torch.float32 and bias is None
            and act == ACT_NONE and pre is None and add.data_ptr() == out.data_ptr() and add.stride(0) == out.stride(0))


def gemm(a, b, a_mn=False, b_mn=False, out=None, out_dtype=torch.bfloat16, bias=None, add=None, act=ACT_NONE,
         aux=None, alpha=1.0, want_preact=False):
    """See module docstring.  ``add`` may alias ``out`` (in-place accumulate, e.g. wgrad into main_grad)."""
    if flop_count.ACTIVE[0] is not None:
        flop_count.gemm(a.shape[0], b.shape[1] if b_mn else b.shape[0], a.shape[1]) if not a_mn else \
            flop_count.gemm(a.shape[1], b.shape[1] if b_mn else b.shape[0], a.shape[0])
    if not a.is_cuda:
        r = gemm_ref(a, b, a_mn, b_mn, out_dtype if out is None else out.dtype, bias, add, act, aux, alpha, want_preact)
        if out is not None:
            if want_preact:
                out.copy_(r[0]); return out, r[1]
            out.copy_(r); return out
        return r
    dt = a.dtype
    assert dt in (torch.bfloat16, torch.float16) and b.dtype == dt, "tcgen05 GEMM takes two bf16 or two fp16 operands"
    if out is None and out_dtype == torch.bfloat16:
        out_dtype = dt                      # the default output type is the operand type
    assert a.dim() == 2 and b.dim() == 2 and a.stride(1) == 1 and b.stride(1) == 1
    if a_mn:
        K, M = a.shape
    else:
        M, K = a.shape
    if b_mn:
        Kb, N = b.shape
    else:
        N, Kb = b.shape
    assert K == Kb, f"contraction mismatch {K} vs {Kb}"
    if out is None:
        out = torch.empty(M, N, device=a.device, dtype=out_dtype)
    assert out.shape == (M, N) and out.stride(1) == 1 and out.dtype in (dt, torch.float32)
    pre = torch.empty(M, N, device=a.device, dtype=dt) if want_preact else None
    if add is not None:
        assert add.shape == (M, N) and add.stride(1) == 1 and add.dtype in (dt, torch.float32)
    if bias is not None:
        assert bias.dtype == dt and bias.numel() == N and bias.is_contiguous()
    if act == ACT_DGELU:
        assert aux is not None and aux.shape == (M, N) and aux.dtype == dt and aux.stride(1) == 1
    L = native.lib()
    h16 = 1 if dt == torch.float16 else 0
    head = (a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0))
    epilogue = (1 if out.dtype == torch.float32 else 0, None if bias is None else bias.data_ptr(),
                *((None, 0, 0) if add is None else (add.data_ptr(), add.stride(0), 1 if add.dtype == torch.float32 else 0)),
                *((None, 0) if pre is None else (pre.data_ptr(), pre.stride(0))),
                *((None, 0) if aux is None else (aux.data_ptr(), aux.stride(0))), act, alpha)
    if use_skinny_kernel(M, N, K, a_mn, b_mn):
        rc = L.neox_gemm_skinny_16(*head, *epilogue, h16, native.stream_ptr())
    elif use_pair_kernel(M, N, K):
        rc = L.neox_gemm_16_2cta(*head, int(a_mn), int(b_mn), *epilogue, h16, native.stream_ptr())
    else:
        splits = L.neox_gemm_splits(M, N, K) if _accumulates(out, bias, add, act, pre) else 1
        if splits > 1:
            parts = torch.empty(splits * M * ((N + 3) // 4 * 4), dtype=torch.float32, device=a.device)
            rc = L.neox_gemm_accumulate_16(*head, int(a_mn), int(b_mn), alpha, splits, parts.data_ptr(), h16,
                                           native.stream_ptr())
        else:
            rc = L.neox_gemm_16(*head, int(a_mn), int(b_mn), *epilogue, None, h16, native.stream_ptr())
    if rc:
        native.check(rc, "neox_gemm_16")
    return (out, pre) if want_preact else out

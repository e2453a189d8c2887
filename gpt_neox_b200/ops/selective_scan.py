"""Mamba selective scan (S6) and causal depth-wise conv1d.

    delta = softplus(dt + dt_bias);  h_t = exp(delta_t A) * h_{t-1} + delta_t B_t u_t;  y_t = C_t . h_t + D u_t
    out = y * silu(z)

Layouts are channel-last -- u, dt, z ``[b, l, d]``, B, C ``[b, l, n]``, with any batch and time strides -- so consecutive
threads of the CUDA kernels (``csrc/selective_scan.cu``: chunks of 32 steps side by side, combined in a short pass; their
start states are the checkpoints of the backward recomputation) touch consecutive addresses and no ``b d l`` transposes
are needed.
``selective_scan_ref`` states the same recurrence in PyTorch (CPU path and oracle).
Reference: mamba_ssm ``selective_scan_fn`` / ``causal_conv1d_fn`` as called from ``megatron/model/mamba/mamba.py:207-300``.
"""
from __future__ import annotations

import ctypes

import torch
import torch.nn.functional as F

from . import native


def selective_scan_ref(u, dt, A, B, C, D=None, z=None, dt_bias=None, dt_softplus=True):
    b, l, d = u.shape
    n = A.shape[1]
    uf, dtf = u.float(), dt.float()
    if dt_bias is not None:
        dtf = dtf + dt_bias.float()
    if dt_softplus:
        dtf = F.softplus(dtf)
    Af, Bf, Cf = A.float(), B.float(), C.float()
    h = torch.zeros(b, d, n, dtype=torch.float32, device=u.device)
    ys = []
    for t in range(l):
        dA = torch.exp(dtf[:, t, :, None] * Af[None])                    # [b, d, n]
        dBu = dtf[:, t, :, None] * Bf[:, t, None, :] * uf[:, t, :, None]
        h = dA * h + dBu
        ys.append(torch.einsum("bdn,bn->bd", h, Cf[:, t]))
    y = torch.stack(ys, dim=1)
    if D is not None:
        y = y + uf * D.float()
    if z is not None:
        y = y * F.silu(z.float())
    return y.to(u.dtype)


def _rows(t, dtype=None):
    """``t`` ([b, l, x], any batch and time strides) with a contiguous last dimension, as the kernels read it."""
    t = t if dtype is None else t.to(dtype)
    return t if t.stride(2) == 1 else t.contiguous()


def _like_rows(t):
    """A new tensor of the shape of ``t``, in its order of batch and time where that leaves the last dimension contiguous, as the
    kernels write it.  (The dense copy of overlapping windows, strides (s, 1, 1), may put time innermost.)"""
    new = torch.empty_like(t)
    return new if new.stride(2) == 1 else torch.empty(t.shape, dtype=t.dtype, device=t.device)


def _strides(*ts):
    return (ctypes.c_longlong * (2 * len(ts)))(*[s for t in ts for s in t.stride()[:2]])


class _Scan(torch.autograd.Function):
    @staticmethod
    def forward(ctx, u, dt, A, B, C, D, z, dt_bias):
        b, l, d = u.shape
        n = A.shape[1]
        u, dt, z = _rows(u), _rows(dt), _rows(z)
        Bc, Cc = _rows(B, torch.float32), _rows(C, torch.float32)
        Af, Df, bias = A.float().contiguous(), D.float().contiguous(), dt_bias.float().contiguous()
        nchk = (l + 31) // 32
        y = _like_rows(u)
        ckpt = torch.empty(b, nchk, n, d, dtype=torch.float32, device=u.device)
        sumd = torch.empty(b, nchk, d, dtype=torch.float32, device=u.device)
        rc = native.lib().neox_selective_scan_fwd(native.ptr(u), native.ptr(dt), native.ptr(Af), native.ptr(Bc),
                                                  native.ptr(Cc), native.ptr(Df), native.ptr(z), native.ptr(bias),
                                                  native.ptr(y), native.ptr(ckpt), native.ptr(sumd),
                                                  _strides(u, dt, z, y, Bc, Cc), b, l, d, n,
                                                  ctypes.c_void_p(native.stream_ptr()))
        native.check(rc, "neox_selective_scan_fwd")
        ctx.save_for_backward(u, dt, Af, Bc, Cc, Df, z, bias, ckpt)
        ctx.dtypes = (A.dtype, B.dtype, C.dtype, D.dtype, dt_bias.dtype)
        return y

    @staticmethod
    def backward(ctx, gy):
        u, dt, Af, Bc, Cc, Df, z, bias, ckpt = ctx.saved_tensors
        b, l, d = u.shape
        n = Af.shape[1]
        gy = _rows(gy)
        du, ddt, dz = _like_rows(u), _like_rows(dt), _like_rows(z)
        sums = torch.zeros(d * n + 2 * b * l * n + 2 * d, dtype=torch.float32, device=u.device)
        dA, dB, dC, dD, dbias = sums.split([d * n, b * l * n, b * l * n, d, d])
        dA, dB, dC = dA.view(d, n), dB.view(b, l, n), dC.view(b, l, n)
        gst, sumd = torch.empty_like(ckpt), torch.empty(b, ckpt.shape[1], d, dtype=torch.float32, device=u.device)
        rc = native.lib().neox_selective_scan_bwd(native.ptr(u), native.ptr(dt), native.ptr(Af), native.ptr(Bc),
                                                  native.ptr(Cc), native.ptr(Df), native.ptr(z), native.ptr(bias),
                                                  native.ptr(ckpt), native.ptr(gy), native.ptr(du), native.ptr(ddt),
                                                  native.ptr(dz), native.ptr(dA), native.ptr(dB), native.ptr(dC),
                                                  native.ptr(dD), native.ptr(dbias), native.ptr(gst), native.ptr(sumd),
                                                  _strides(u, dt, z, gy, Bc, Cc, du, ddt, dz, dB), b, l, d, n,
                                                  ctypes.c_void_p(native.stream_ptr()))
        native.check(rc, "neox_selective_scan_bwd")
        ta, tb, tc, td, tbias = ctx.dtypes
        return du, ddt, dA.to(ta), dB.to(tb), dC.to(tc), dD.to(td), dz, dbias.to(tbias)


def have_scan_kernel():
    return native.available() and native.lib().has("neox_selective_scan_fwd")


def selective_scan(u, dt, A, B, C, D, z, dt_bias):
    """All of D, z, dt_bias are required on the kernel path (the Mamba block always has them)."""
    if u.is_cuda and u.dtype == torch.bfloat16 and A.shape[1] == 16 and have_scan_kernel():
        return _Scan.apply(u, dt, A, B, C, D, z, dt_bias)
    return selective_scan_ref(u, dt, A, B, C, D, z, dt_bias, True)


class _CausalConv(torch.autograd.Function):
    """``xz`` ``[b, l, d or 2 d]`` -> (activation(conv(first d channels)), the other d channels or None).  The second half is
    a view: with it, the gradient of a projection that feeds both halves is born packed."""

    @staticmethod
    def forward(ctx, xz, weight, bias, silu):
        b, l, _ = xz.shape
        d = weight.shape[0]
        w = weight.contiguous()
        out = torch.empty(l, b, d, dtype=xz.dtype, device=xz.device).transpose(0, 1) if xz.stride(0) < xz.stride(1) \
            else torch.empty(b, l, d, dtype=xz.dtype, device=xz.device)
        rc = native.lib().neox_causal_conv_fwd(native.ptr(xz), native.ptr(w), native.ptr(bias), native.ptr(out),
                                               _strides(xz, out), b, l, d, int(silu), int(xz.dtype == torch.float16),
                                               ctypes.c_void_p(native.stream_ptr()))
        native.check(rc, "neox_causal_conv_fwd")
        ctx.save_for_backward(xz, weight, bias)
        ctx.silu = silu
        return out, xz[..., d:]

    @staticmethod
    def backward(ctx, g, gz):
        xz, weight, bias = ctx.saved_tensors
        b, l, width = xz.shape
        d = weight.shape[0]
        if torch.is_grad_enabled():
            # create_graph: the gradients are to be differentiated once more, which the kernel's are not
            leaves = [t for t, wanted in zip((xz, weight, bias), ctx.needs_input_grad) if wanted]
            out = _library_conv(xz[..., :d], weight, bias, ctx.silu)
            found = iter(torch.autograd.grad(out, leaves, g, create_graph=True))
            gxz, gw, gb = (next(found) if wanted else None for wanted in ctx.needs_input_grad[:3])
            if gxz is not None and width > d:
                gxz = gxz + torch.cat([torch.zeros_like(g), gz], dim=-1)
            return gxz, gw, gb, None
        w = weight.contiguous()
        g = _aligned_rows(g)
        gxz = torch.empty(l, b, width, dtype=xz.dtype, device=xz.device).transpose(0, 1) if xz.stride(0) < xz.stride(1) \
            else torch.empty(b, l, width, dtype=xz.dtype, device=xz.device)
        if width > d:
            gxz[..., d:].copy_(gz)
        part = torch.empty(native.lib().neox_causal_conv_blocks(b, l, d), d, w.shape[1] + 1, dtype=torch.float32, device=xz.device)
        rc = native.lib().neox_causal_conv_bwd(native.ptr(xz), native.ptr(w), native.ptr(bias), native.ptr(g),
                                               native.ptr(gxz), native.ptr(part), _strides(xz, g, gxz), b, l, d,
                                               int(ctx.silu), int(xz.dtype == torch.float16),
                                               ctypes.c_void_p(native.stream_ptr()))
        native.check(rc, "neox_causal_conv_bwd")
        sums = part.sum(0).to(w.dtype)
        return gxz, sums[:, :-1], sums[:, -1] if bias is not None else None, None


def _aligned_rows(t):
    """``t`` with unit channel stride and every row on a 16-byte boundary (the channels are a multiple of 8)."""
    ok = t.stride(2) == 1 and t.stride(0) % 8 == 0 and t.stride(1) % 8 == 0 and t.data_ptr() % 16 == 0
    return t if ok else t.clone(memory_format=torch.contiguous_format)      # contiguous() keeps one that starts off a boundary


def _conv_kernel_ok(x, weight, bias):
    """Do ``x`` ([b, l, d] or [b, l, 2 d]), ``weight`` ([d, 4]) and ``bias`` fit the kernels, which read ``d`` channels of every
    row of ``x`` and ``d`` contiguous bias elements without asking again?  Whatever does not goes to the library
    convolution, which takes it or refuses it with a message; so do calls under a transform (vmap, forward mode, tracing)
    that an autograd function would not follow."""
    if not (x.is_cuda and native.available() and x.dim() == 3 and weight.dim() == 2 and native.untransformed(x, weight, bias)):
        return False
    b, _, width = x.shape
    d, taps = weight.shape
    if bias is not None and not (bias.shape == (d,) and bias.is_contiguous() and bias.dtype == x.dtype
                                 and bias.device == x.device):
        return False
    return (x.dtype in (torch.bfloat16, torch.float16) and weight.dtype == x.dtype and weight.device == x.device
            and taps == 4 and d % 8 == 0 and width in (d, 2 * d) and b <= 65535 and x.numel() > 0 and x.stride(2) == 1
            and x.stride(0) % 8 == 0 and x.stride(1) % 8 == 0 and x.data_ptr() % 16 == 0)


def causal_conv1d(x, weight, bias, activation="silu"):
    """Depth-wise causal conv over time for channel-last ``x`` ``[b, l, d]`` (any batch and time strides); ``weight``
    ``[d, w]``.  Width 4 in 16 bits on a GPU: one kernel with bias and SiLU (``csrc/causal_conv.cu``)."""
    if _conv_kernel_ok(x, weight, bias) and x.shape[-1] == weight.shape[0]:
        return _CausalConv.apply(x, weight, bias, activation == "silu")[0]
    return _library_conv(x, weight, bias, activation == "silu")


def _library_conv(x, weight, bias, silu):
    w = weight.shape[1]
    y = F.conv1d(x.transpose(1, 2), weight.unsqueeze(1), bias, padding=w - 1, groups=weight.shape[0])[..., : x.shape[1]]
    y = y.transpose(1, 2)
    return F.silu(y) if silu else y


def causal_conv1d_split(xz, weight, bias):
    """``xz`` ``[b, l, 2 d]`` -> (``silu(conv(first half))``, second half)."""
    if _conv_kernel_ok(xz, weight, bias) and xz.shape[-1] == 2 * weight.shape[0]:
        return _CausalConv.apply(xz, weight, bias, True)
    x, z = xz.chunk(2, dim=-1)
    return causal_conv1d(x, weight, bias), z

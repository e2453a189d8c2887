"""Numerics of every CUDA kernel against the plain PyTorch fp32 statement of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from gpt_neox_b200.ops import functional as OF
from gpt_neox_b200.ops import gemm as G
from gpt_neox_b200.ops import native

DEV = "cuda"


def _close(a, b, atol, rtol=1e-2):
    a, b = a.float(), b.float()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    assert bool((err <= tol).all()), f"max err {err.max().item():.4g} (tol {atol}, {rtol})"


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(128, 256, 64, 0, 0), (256, 512, 256, 0, 1), (256, 512, 256, 1, 0),
                                             (384, 264, 136, 1, 1), (1000, 840, 328, 0, 0), (77, 96, 200, 0, 1)])
def test_gemm_layouts(M, N, K, a_mn, b_mn):
    torch.manual_seed(0)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV, dtype=torch.bfloat16)
    out = G.gemm(a, b, a_mn, b_mn)
    ref = G.gemm_ref(a, b, a_mn, b_mn, out_dtype=torch.float32)
    assert native.read_status() == 0
    _close(out, ref, atol=0.02 * ref.abs().max().item(), rtol=1e-2)


def test_gemm_epilogues():
    torch.manual_seed(1)
    M, N, K = 512, 1024, 512
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16) * 0.05
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
    out, pre = G.gemm(a, b, bias=bias, act=G.ACT_GELU, add=res, want_preact=True)
    ro, rp = G.gemm_ref(a, b, bias=bias, act=G.ACT_GELU, add=res, want_preact=True, out_dtype=torch.float32)
    _close(out, ro, atol=0.05)
    _close(pre, rp, atol=0.05)
    aux = torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
    out = G.gemm(a, b, act=G.ACT_DGELU, aux=aux)
    _close(out, G.gemm_ref(a, b, act=G.ACT_DGELU, aux=aux, out_dtype=torch.float32), atol=0.05)
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    want = G.gemm_ref(a, b, add=acc, out_dtype=torch.float32)
    G.gemm(a, b, out=acc, add=acc)
    _close(acc, want, atol=0.02)
    assert native.read_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("rows,cols", [(33, 64), (128, 2048), (17, 6144), (5, 16384)])
def test_layernorm(dtype, rows, cols):
    torch.manual_seed(0)
    x = torch.randn(rows, cols, device=DEV, dtype=dtype, requires_grad=True)
    w = (1 + 0.1 * torch.randn(cols, device=DEV)).to(dtype).requires_grad_()
    b = (0.1 * torch.randn(cols, device=DEV)).to(dtype).requires_grad_()
    y = OF.layer_norm(x, w, b, 1e-5)
    g = torch.randn_like(y)
    y.backward(g)
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = torch.nn.functional.layer_norm(xr, (cols,), wr, br, 1e-5)
    yr.backward(g.float())
    tol = 1e-4 if dtype == torch.float32 else 3e-2
    _close(y, yr, tol)
    _close(x.grad, xr.grad, tol)
    _close(w.grad, wr.grad, tol * math.sqrt(rows), rtol=2e-2)
    _close(b.grad, br.grad, tol * math.sqrt(rows), rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(33, 64), (64, 4096)])
def test_rmsnorm(dtype, rows, cols):
    torch.manual_seed(0)
    x = torch.randn(rows, cols, device=DEV, dtype=dtype, requires_grad=True)
    w = (1 + 0.1 * torch.randn(cols, device=DEV)).to(dtype).requires_grad_()
    y = OF.rms_norm(x, w, None, 1e-5)
    g = torch.randn_like(y)
    y.backward(g)
    xr, wr = (t.detach().float().requires_grad_() for t in (x, w))
    yr = OF.rms_norm_ref(xr, wr, None, 1e-5)
    yr.backward(g.float())
    tol = 1e-4 if dtype == torch.float32 else 3e-2
    _close(y, yr, tol)
    _close(x.grad, xr.grad, tol)
    _close(w.grad, wr.grad, tol * math.sqrt(rows), rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_bias_gelu_and_gated(dtype):
    torch.manual_seed(0)
    x = torch.randn(37, 512, device=DEV, dtype=dtype, requires_grad=True)
    bias = torch.randn(512, device=DEV, dtype=dtype, requires_grad=True)
    y = OF.bias_gelu(x, bias)
    g = torch.randn_like(y)
    y.backward(g)
    xr, br = x.detach().float().requires_grad_(), bias.detach().float().requires_grad_()
    yr = torch.nn.functional.gelu(xr + br, approximate="tanh")
    yr.backward(g.float())
    tol = 2e-3 if dtype == torch.float32 else 3e-2
    _close(y, yr, tol)
    _close(x.grad, xr.grad, tol)
    for kind in ("geglu", "swiglu", "reglu", "bilinear", "glu"):
        x2 = torch.randn(19, 256, device=DEV, dtype=dtype, requires_grad=True)
        y2 = OF.gated_act(x2, kind)
        g2 = torch.randn_like(y2)
        y2.backward(g2)
        x2r = x2.detach().float().requires_grad_()
        y2r = OF.gated_act_ref(x2r, kind)
        y2r.backward(g2.float())
        _close(y2, y2r, tol)
        _close(x2.grad, x2r.grad, tol)


@pytest.mark.parametrize("sk", [17, 128, 1000, 2048, 5000])
def test_softmax(sk):
    torch.manual_seed(0)
    b, h, sq = 2, 3, 8
    x = torch.randn(b, h, sq, sk, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    mask = torch.rand(b, 1, sq, sk, device=DEV) < 0.3
    y = OF.scaled_masked_softmax(x, mask, 0.7)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    yr = OF.scaled_masked_softmax_ref(xr, mask, 0.7)
    yr.backward(g.float())
    # the reference bar for this kernel is a mean absolute difference <= 1e-3
    assert (y.float() - yr).abs().mean().item() <= 1e-3
    _close(y, yr, 1e-2)
    _close(x.grad, xr.grad, 2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("s", [16, 129, 2048])
def test_causal_softmax(s, dtype):
    torch.manual_seed(0)
    x = torch.randn(4, s, s, device=DEV, dtype=dtype, requires_grad=True)
    y = OF.scaled_upper_triang_masked_softmax(x, 0.5)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    yr = OF.scaled_causal_softmax_ref(xr, 0.5)
    yr.backward(g.float())
    assert (y.float() - yr).abs().mean().item() <= 1e-3
    assert bool((y.float().triu(1) == 0).all())
    _close(x.grad, xr.grad, 2e-2)


@pytest.mark.parametrize("d,rot", [(64, 16), (96, 24), (128, 128)])
def test_rope_strided(d, rot):
    torch.manual_seed(0)
    s, b, h = 33, 2, 4
    qkv = torch.randn(s, b, h, 3 * d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    q = qkv[..., d:2 * d]                    # a strided view, as sliced from the fused projection
    t = torch.arange(s, device=DEV).float()
    inv = 1.0 / (10000 ** (torch.arange(0, rot, 2, device=DEV).float() / rot))
    emb = torch.cat([torch.outer(t, inv)] * 2, dim=-1)
    cos, sin = emb.cos()[:, None, None, :], emb.sin()[:, None, None, :]
    y = OF.rope(q, cos, sin)
    g = torch.randn_like(y)
    y.backward(g)
    qr = qkv.detach().float().requires_grad_()
    yr = OF.rope_ref(qr[..., d:2 * d], cos, sin)
    yr.backward(g.float())
    _close(y, yr, 3e-2)
    _close(qkv.grad, qr.grad, 3e-2)


@pytest.mark.parametrize("dtype,d,rot", [(torch.float32, 64, 64), (torch.float32, 80, 20), (torch.float32, 66, 6),
                                         (torch.float16, 96, 24), (torch.float16, 128, 64), (torch.float16, 80, 20)])
def test_rope_every_vector_width(dtype, d, rot):
    """16-byte, 8-byte and scalar accesses (chosen from rot / 2, d - rot and the strides) give the same rotation."""
    torch.manual_seed(0)
    s, b, h = 17, 3, 5
    x = torch.randn(s, b, h, d, device=DEV, dtype=dtype, requires_grad=True)
    t = torch.arange(s, device=DEV).float()
    inv = 1.0 / (10000 ** (torch.arange(0, rot, 2, device=DEV).float() / rot))
    emb = torch.cat([torch.outer(t, inv)] * 2, dim=-1)
    cos, sin = emb.cos()[:, None, None, :], emb.sin()[:, None, None, :]
    y = OF.rope(x, cos, sin)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    yr = OF.rope_ref(xr, cos, sin)
    yr.backward(g.float())
    tol = 1e-5 if dtype == torch.float32 else 4e-3
    _close(y, yr, tol)
    _close(x.grad, xr.grad, tol)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_cross_entropy(dtype):
    from gpt_neox_b200.parallel.cross_entropy import vocab_parallel_cross_entropy
    torch.manual_seed(0)
    logits = (torch.randn(4, 9, 1000, device=DEV) * 3).to(dtype).requires_grad_()
    tgt = torch.randint(0, 1000, (4, 9), device=DEV)
    loss = vocab_parallel_cross_entropy(logits, tgt)
    w = torch.rand_like(loss)
    (loss * w).sum().backward()
    lr = logits.detach().float().requires_grad_()
    ref = OF.cross_entropy_ref(lr, tgt)
    (ref * w).sum().backward()
    _close(loss, ref, 2e-3 if dtype == torch.float32 else 2e-2)
    _close(logits.grad, lr.grad, 1e-4 if dtype == torch.float32 else 1e-2)


def test_fused_adam_matches_torch():
    from gpt_neox_b200.optim.fused_adam import FusedAdam
    torch.manual_seed(0)
    p0 = torch.randn(10007, device=DEV)
    p1 = torch.nn.Parameter(p0.clone())
    p2 = torch.nn.Parameter(p0.clone())
    out = torch.empty(10007, device=DEV, dtype=torch.bfloat16)
    p1.model_out = out
    o1 = FusedAdam([p1], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    o2 = torch.optim.AdamW([p2], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for _ in range(5):
        g = torch.randn(10007, device=DEV)
        p1.grad, p2.grad = g.clone(), g.clone()
        o1.step()
        o2.step()
    _close(p1, p2, 1e-5, rtol=1e-5)
    _close(out, p2, 1e-2)


def test_bounded_wait_reports_instead_of_hanging():
    """A device-side wait that nobody satisfies gives up after its cycle limit, records a status code the host can
    read, and leaves the context usable: a flag-wait kernel is pointed at a flag word that stays 0 (it waits for
    epoch 7 of a second rank that does not exist), on one GPU.  A clean launch before and after reads status 0."""
    import ctypes
    a = torch.randn(128, 64, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(256, 64, device=DEV, dtype=torch.bfloat16)
    G.gemm(a, b)
    assert native.read_status() == 0
    flags = torch.zeros(64, dtype=torch.int32, device=DEV)
    rc = native.lib().neox_wait_flags(native.ptr(flags), ctypes.c_uint(7), 2, 0,
                                      ctypes.c_void_p(native.stream_ptr()))
    assert rc == 0
    assert native.read_status() == 561            # 560 + the rank whose flag never arrived
    out = G.gemm(a, b)                            # the context is intact: kernels still run and are correct
    _close(out, G.gemm_ref(a, b, out_dtype=torch.float32), atol=0.5)
    assert native.read_status() == 0


@pytest.mark.parametrize("sq,sk,b,hq,hkv,d,causal,window,alibi,fused", [
    (128, 128, 1, 1, 1, 64, True, None, False, False),
    (256, 256, 2, 4, 4, 96, True, None, False, True),
    (300, 300, 2, 4, 2, 64, True, None, False, False),      # GQA + ragged tiles
    (200, 200, 1, 2, 2, 128, False, None, False, False),
    (77, 500, 1, 2, 1, 96, True, None, False, False),       # sq < sk: bottom-right aligned causal mask
    (512, 512, 1, 2, 2, 64, True, 100, False, False),       # sliding window
    (512, 512, 1, 2, 2, 64, True, None, True, False),       # ALiBi
    (1024, 1024, 1, 4, 4, 96, True, None, False, True),
])
def test_flash_attention_fwd_bwd(sq, sk, b, hq, hkv, d, causal, window, alibi, fused):
    from gpt_neox_b200.ops import attention as A
    torch.manual_seed(0)
    if fused and hq == hkv:
        qkv = torch.randn(sq, b, hq, 3 * d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
        q, k, v = qkv[..., :d], qkv[..., d:2 * d], qkv[..., 2 * d:]
        leaves = [qkv]
    else:
        q = torch.randn(sq, b, hq, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
        k = torch.randn(sk, b, hkv, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
        v = torch.randn(sk, b, hkv, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
        leaves = [q, k, v]
    slopes = (torch.rand(hq, device=DEV) * 0.1) if alibi else None
    assert A.have_flash_kernel()
    out = A.flash_attention(q, k, v, causal=causal, window=window, alibi_slopes=slopes)
    g = torch.randn_like(out)
    out.backward(g)
    assert native.read_status() == 0
    refl = [l.detach().float().requires_grad_() for l in leaves]
    if len(refl) == 1:
        rq, rk, rv = refl[0][..., :d], refl[0][..., d:2 * d], refl[0][..., 2 * d:]
    else:
        rq, rk, rv = refl
    ref = A.attention_ref(rq, rk, rv, causal, None, window, slopes)
    ref.backward(g.float())
    _close(out, ref, 3e-2)
    for got, want in zip(leaves, refl):
        _close(got.grad, want.grad, 0.02 + 0.02 * want.grad.abs().max().item(), rtol=3e-2)


@pytest.mark.parametrize("s,b,h,d,rot", [(256, 2, 4, 96, 24), (300, 1, 2, 64, 64), (512, 1, 2, 128, 0)])
def test_packed_qkv_attention_with_inplace_rotary(s, b, h, d, rot):
    """rotary + attention on the packed projection, in place, against fp32 rotary + fp32 attention."""
    from gpt_neox_b200.models.positional import RotaryEmbedding
    from gpt_neox_b200.ops import attention as A
    from gpt_neox_b200.ops import functional as OF
    torch.manual_seed(0)
    mixed = torch.randn(s, b, h, 3 * d, device=DEV, dtype=torch.bfloat16)
    leaf = mixed.clone().requires_grad_(True)
    cos = sin = None
    if rot:
        cos, sin = RotaryEmbedding(rot, s, precision=torch.bfloat16).to(DEV)(mixed, seq_len=s)
    work = leaf * 1.0                                   # non-leaf copy: the op overwrites its input
    out = A.packed_qkv_attention(work, cos, sin)
    g = torch.randn_like(out)
    out.backward(g)
    assert native.read_status() == 0
    ref_leaf = mixed.detach().float().requires_grad_(True)
    q, k, v = ref_leaf[..., :d], ref_leaf[..., d:2 * d], ref_leaf[..., 2 * d:]
    if rot:
        q, k = OF.rope_ref(q, cos, sin), OF.rope_ref(k, cos, sin)
    ref = A.attention_ref(q, k, v, True, None, None, None)
    ref.backward(g.float())
    _close(out, ref, 3e-2)
    _close(leaf.grad, ref_leaf.grad, 0.02 + 0.02 * ref_leaf.grad.abs().max().item(), rtol=3e-2)


def test_flash_attention_is_deterministic():
    from gpt_neox_b200.ops import attention as A
    torch.manual_seed(0)
    q, k, v = (torch.randn(512, 2, 4, 96, device=DEV, dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
    outs, grads = [], []
    for _ in range(2):
        for t in (q, k, v):
            t.grad = None
        o = A.flash_attention(q, k, v)
        o.backward(torch.ones_like(o))
        outs.append(o.detach().clone())
        grads.append([t.grad.clone() for t in (q, k, v)])
    assert torch.equal(outs[0], outs[1])
    for a, b_ in zip(grads[0], grads[1]):
        assert torch.equal(a, b_)      # no atomics anywhere: bitwise repeatable


@pytest.mark.parametrize("b,l,d", [(2, 70, 192), (1, 256, 100)])
def test_selective_scan_fwd_bwd(b, l, d):
    """Mamba S6 scan kernel (state in registers, 32-step checkpoints) against the step-by-step fp32 recurrence."""
    from gpt_neox_b200.ops import selective_scan as SS
    torch.manual_seed(0)
    n = 16
    mk = lambda *s, scale=1.0: (torch.randn(*s, device=DEV) * scale)
    u = mk(b, l, d).to(torch.bfloat16).requires_grad_(True)
    dt = mk(b, l, d, scale=0.5).to(torch.bfloat16).requires_grad_(True)
    z = mk(b, l, d).to(torch.bfloat16).requires_grad_(True)
    A = (-torch.rand(d, n, device=DEV) * 2 - 0.1).requires_grad_(True)
    B = mk(b, l, n, scale=0.5).requires_grad_(True)
    C = mk(b, l, n, scale=0.5).requires_grad_(True)
    D = mk(d).requires_grad_(True)
    bias = mk(d, scale=0.3).requires_grad_(True)
    leaves = [u, dt, A, B, C, D, z, bias]
    assert SS.have_scan_kernel()
    out = SS.selective_scan(u, dt, A, B, C, D, z, bias)
    g = torch.randn_like(out)
    out.backward(g)
    got = [t.grad.clone() for t in leaves]
    for t in leaves:
        t.grad = None
    ref = SS.selective_scan_ref(u.float(), dt.float(), A, B, C, D, z.float(), bias, True)
    ref.backward(g.float())
    _close(out, ref, 3e-2)
    for have, t in zip(got, leaves):
        _close(have, t.grad, 0.03 + 0.03 * t.grad.abs().max().item(), rtol=5e-2)


def test_embedding_kernels_vocab_parallel_slice():
    from gpt_neox_b200.ops import embedding as E
    torch.manual_seed(0)
    V, h, v0 = 1000, 256, 300
    w = torch.randn(400, h, device=DEV, dtype=torch.bfloat16, requires_grad=True)        # owns rows [300, 700)
    ids = torch.randint(0, V, (4, 33), device=DEV)
    ids[0, :5] = 345                                                                      # duplicates: atomics must add
    out = E.embedding(ids, w, v0)
    ref_w = w.detach().float().requires_grad_(True)
    ref = E.embedding_ref(ids, ref_w, v0)
    assert torch.equal(out.float(), ref)
    g = torch.randn_like(out)
    out.backward(g)
    ref.backward(g.float())
    _close(w.grad, ref_w.grad, 2e-2, rtol=2e-2)
    # with an fp32 main-gradient view the kernel accumulates there and autograd sees no .grad
    w2 = w.detach().clone().requires_grad_(True)
    w2.main_grad = torch.ones(400, h, device=DEV, dtype=torch.float32)
    E.embedding(ids, w2, v0).backward(g)
    assert w2.grad is None
    _close(w2.main_grad, 1.0 + ref_w.grad, 1e-3, rtol=1e-4)


@pytest.mark.parametrize("top_k,top_p", [(5, 0.0), (0, 0.9), (50, 0.5), (1, 0.0), (0, 0.999)])
def test_sampling_filter_matches_sort_based_filter(top_k, top_p):
    from gpt_neox_b200 import text_generation as TG
    torch.manual_seed(0)
    logits = torch.randn(7, 50304, device=DEV) * 3
    got = TG.filter_logits(logits, top_k=top_k, top_p=top_p)
    want = TG.filter_logits(logits.cpu(), top_k=top_k, top_p=top_p).to(DEV)
    kept_g, kept_w = torch.isfinite(got), torch.isfinite(want)
    # the sorted reference accumulates 50k fp32 probabilities in another order, so deep in the tail the boundary may
    # move by a few tokens: the sets must agree up to a negligible probability mass
    probs = torch.softmax(logits.float(), dim=-1)
    assert (probs * (kept_g != kept_w)).sum(dim=-1).max().item() < 1e-3
    if top_p < 0.99:
        assert (kept_g != kept_w).sum(dim=-1).max().item() <= 1
    assert torch.equal(got[kept_g & kept_w], logits[kept_g & kept_w])


@pytest.mark.parametrize("along_rows,e5m2", [(False, False), (True, False), (False, True), (True, True)])
def test_mxfp8_quantise_round_trip_matches_torch_float8(along_rows, e5m2):
    from gpt_neox_b200.ops import mxfp8 as MX
    torch.manual_seed(0)
    x = (torch.randn(200, 176, device=DEV) * torch.logspace(-3, 2, 176, device=DEV)).to(torch.bfloat16)
    x[3, :40] = 0
    got = MX.qdq(x, along_rows, e5m2)
    want = MX.qdq_ref(x, along_rows, e5m2)
    assert torch.equal(got, want)
    q, s = MX.quantize(x, along_rows, e5m2)
    assert torch.equal(MX.dequantize(q, s, along_rows, e5m2), got)
    # error of every element is at most 1/8 of its block's maximum: half an ulp of the top binade, or the
    # saturation of scaled values in (max_fp8, 2 * 2^emax) that the power-of-two scale allows
    blk, _, _ = MX._blocks((got.float() - x.float()).abs(), along_rows)
    ref_blk, _, _ = MX._blocks(x.float().abs(), along_rows)
    assert bool((blk.amax(-1) <= ref_blk.amax(-1) * 0.125 + 1e-30).all())


def test_mxfp8_linear_fwd_bwd_against_fp32_on_quantised_operands():
    from gpt_neox_b200.ops import mxfp8 as MX
    torch.manual_seed(0)
    x = torch.randn(256, 192, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(320, 192, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_(True)
    b = torch.randn(320, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    y = MX.mx_linear(x, w, b, hybrid=True, fp8_wgrad=True)
    g = torch.randn_like(y)
    y.backward(g)
    xq, wq = MX.qdq_ref(x.detach(), False), MX.qdq_ref(w.detach(), False)
    _close(y, xq.float() @ wq.float().t() + b.float(), 2e-2, rtol=2e-2)
    gq, wq2 = MX.qdq_ref(g, False, True), MX.qdq_ref(w.detach(), True)
    _close(x.grad, gq.float() @ wq2.float(), 2e-2, rtol=2e-2)
    gq2, xq2 = MX.qdq_ref(g, True, True), MX.qdq_ref(x.detach(), True)
    _close(w.grad, gq2.float().t() @ xq2.float(), 5e-2, rtol=2e-2)
    # and the block-scaled result stays close to the unquantised layer
    ref = x.detach().float() @ w.detach().float().t() + b.detach().float()
    assert ((y.float() - ref).abs().mean() / ref.abs().mean()).item() < 0.05


# ------------------------------------------------------------------ per-tensor fp8 (fp8 tensor cores)
@pytest.mark.parametrize("e5m2", [False, True])
def test_fp8_cast_matches_torch_float8(e5m2):
    from gpt_neox_b200.ops import fp8 as F8
    torch.manual_seed(0)
    x = (torch.randn(203, 176, device=DEV) * torch.logspace(-2, 1, 176, device=DEV)).to(torch.bfloat16)
    got = F8.cast(x, e5m2, margin=1)
    want = F8._cast_ref(x, e5m2, 1, None)
    assert torch.allclose(got.inv, want.inv, rtol=1e-6)
    assert torch.equal(got.q, want.q)
    # delayed scaling: the first cast runs at scale 1 and records the amax, the second uses it
    meta = F8.DelayedMeta(x.device, length=4, e5m2=e5m2)
    meta.update()
    first = F8.cast(x, e5m2, meta=meta)
    assert float(first.inv) == 1.0
    meta.update()
    second = F8.cast(x, e5m2, meta=meta)
    lim = F8.E5M2_MAX if e5m2 else F8.E4M3_MAX
    assert abs(float(second.inv) - float(x.float().abs().max()) / lim) < 1e-6 * float(second.inv) + 1e-12
    assert torch.equal(second.q, F8._cast_ref(x, e5m2, 0, None).q)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("a_e5,b_e5", [(False, False), (True, False)])
def test_fp8_gemm_matches_fp32_on_the_same_fp8_operands(a_mn, b_mn, a_e5, b_e5):
    from gpt_neox_b200.ops import fp8 as F8
    from gpt_neox_b200.ops import gemm as G
    torch.manual_seed(1)
    M, N, K = 304, 528, 400               # ragged against the 128 x 256 x 128 tile in every dimension
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.bfloat16)
    b = (torch.randn((K, N) if b_mn else (N, K), device=DEV) * 0.1).to(torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    aq, bq = F8.cast(a, a_e5), F8.cast(b, b_e5)
    got = F8.gemm_fp8(aq, bq, a_mn, b_mn, bias=bias, out_dtype=torch.float32)
    want = F8.gemm_fp8_ref(aq, bq, a_mn, b_mn, bias=bias, out_dtype=torch.float32)
    _close(got, want, 2e-3, rtol=1e-3)
    acc = torch.randn(M, N, device=DEV)
    got2 = F8.gemm_fp8(aq, bq, a_mn, b_mn, out=acc.clone(), add=acc)
    _close(got2, F8.gemm_fp8_ref(aq, bq, a_mn, b_mn, out_dtype=torch.float32) + acc, 2e-3, rtol=1e-3)


@pytest.mark.parametrize("recipe", ["current", "delayed"])
def test_fp8_linear_fwd_bwd_tracks_the_bf16_layer(recipe):
    from gpt_neox_b200.ops import fp8 as F8
    torch.manual_seed(2)
    x = torch.randn(512, 384, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = torch.nn.Parameter((torch.randn(640, 384, device=DEV) * 0.05).to(torch.bfloat16))
    b = torch.nn.Parameter(torch.randn(640, device=DEV, dtype=torch.bfloat16))
    g = torch.randn(512, 640, device=DEV, dtype=torch.bfloat16)
    rec = F8.Fp8Recipe(recipe=recipe, history_len=4)
    for _ in range(3 if recipe == "delayed" else 1):     # delayed scaling needs a step to learn its scales
        x.grad = w.grad = b.grad = None
        F8.invalidate_weight_cache()                      # what the engine does after an optimizer step
        y = F8.fp8_linear(x, w, b, rec)
        y.backward(g)
    xr, wr = x.detach().float(), w.detach().float()
    rel = lambda got, want: ((got.float() - want).norm() / want.norm()).item()
    assert rel(y, xr @ wr.t() + b.detach().float()) < 0.05
    assert rel(x.grad, g.float() @ wr) < 0.08
    assert rel(w.grad, g.float().t() @ xr) < 0.08
    _close(b.grad, g.float().sum(0), 0.5, rtol=2e-2)
    # exactness against the quantised operands (forward)
    xq, wq = F8._cast_ref(x.detach(), False, 0, None), F8._cast_ref(w.detach(), False, 0, None)
    if recipe == "current":
        _close(y, xq.dequant() @ wq.dequant().t() + b.detach().float(), 3e-2, rtol=1e-2)


# ------------------------------------------------------------------ CTA-pair GEMM (tcgen05 cta_group::2)
@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(256, 256, 64, 0, 0), (512, 512, 256, 0, 1), (512, 512, 256, 1, 0),
                                             (640, 264, 136, 1, 1), (1000, 840, 328, 0, 0), (77, 96, 200, 0, 1),
                                             (2304, 1536, 512, 0, 0)])
def test_gemm_cta_pair_kernel_matches_fp32(M, N, K, a_mn, b_mn, monkeypatch):
    from gpt_neox_b200.ops import gemm as G
    monkeypatch.setattr(G, "_PAIR", "1")
    torch.manual_seed(0)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV, dtype=torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    add = torch.randn(M, N, device=DEV, dtype=torch.float32)
    got = G.gemm(a, b, a_mn, b_mn, bias=bias, add=add, out_dtype=torch.float32)
    want = G.gemm_ref(a, b, a_mn, b_mn, out_dtype=torch.float32, bias=bias, add=add)
    _close(got, want, 2e-2 * (K ** 0.5) / 8, rtol=1e-3)
    got2, pre = G.gemm(a, b, a_mn, b_mn, bias=bias, act=G.ACT_GELU, want_preact=True)
    want2, wpre = G.gemm_ref(a, b, a_mn, b_mn, bias=bias, act=G.ACT_GELU, want_preact=True)
    _close(pre, wpre, 0.25, rtol=1e-2)
    _close(got2, want2, 0.25, rtol=1e-2)
    from gpt_neox_b200.ops import native
    assert native.read_status() == 0


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_fp8_gemm_cta_pair_kernel_matches_fp32_on_the_same_fp8_operands(a_mn, b_mn, monkeypatch):
    from gpt_neox_b200.ops import fp8 as F8
    from gpt_neox_b200.ops import gemm as G
    from gpt_neox_b200.ops import native
    monkeypatch.setattr(G, "_PAIR", "1")
    torch.manual_seed(1)
    M, N, K = 560, 528, 400
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.bfloat16)
    b = (torch.randn((K, N) if b_mn else (N, K), device=DEV) * 0.1).to(torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    aq, bq = F8.cast(a, True), F8.cast(b, False)
    got = F8.gemm_fp8(aq, bq, a_mn, b_mn, bias=bias, out_dtype=torch.float32)
    want = F8.gemm_fp8_ref(aq, bq, a_mn, b_mn, bias=bias, out_dtype=torch.float32)
    _close(got, want, 2e-3, rtol=1e-3)
    assert native.read_status() == 0


# ------------------------------------------------------------------ MXFP8 on the block-scaled tensor cores
@pytest.mark.parametrize("a_rows,b_rows", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("mode", ["unit_scales", "row_scales", "k_scales", "random"])
def test_mxfp8_block_scaled_gemm_matches_dequantised_product(a_rows, b_rows, mode):
    """forward (K-major, K-major), dgrad (K-major, MN-major) and wgrad (MN-major, MN-major) layouts; the scale
    patterns isolate the scale plumbing: all scales equal / varying along mn only / along K blocks only / both."""
    from gpt_neox_b200.ops import mxfp8 as MX
    from gpt_neox_b200.ops import gemm as G
    torch.manual_seed(3)
    M, N, K = 272, 464, 416          # N: three 192-wide tiles (even, odd, ragged); K: ragged against 128
    def make(mn, k, rows_are_k):
        base = torch.empty(mn, k, device=DEV).uniform_(1.0, 1.9)
        sign = torch.where(torch.rand(mn, k, device=DEV) < 0.5, -1.0, 1.0)
        mn_e = torch.randint(-3, 4, (mn, 1), device=DEV).float()
        k_e = torch.randint(-3, 4, (1, (k + 31) // 32), device=DEV).float().repeat_interleave(32, dim=1)[:, :k]
        e = {"unit_scales": 0 * mn_e + 0 * k_e, "row_scales": mn_e + 0 * k_e, "k_scales": 0 * mn_e + k_e,
             "random": mn_e + k_e}[mode]
        t = (base * sign * torch.exp2(e)).to(torch.bfloat16)          # [mn, k]
        return t.t().contiguous() if rows_are_k else t
    a = make(M, K, a_rows)           # [M, K] or [K, M]
    b = make(N, K, b_rows)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    got = MX.gemm_mx(MX.quantize_tiled(a, a_rows, False), MX.quantize_tiled(b, b_rows, True), bias=bias,
                     out_dtype=torch.float32)
    want = G.gemm_ref(MX.qdq_ref(a, a_rows, False), MX.qdq_ref(b, b_rows, True), a_rows, b_rows,
                      out_dtype=torch.float32, bias=bias)
    assert native.read_status() == 0
    _close(got, want, 1e-2, rtol=2e-3)


def test_mxfp8_hardware_linear_matches_the_emulated_layer():
    from gpt_neox_b200.ops import mxfp8 as MX
    torch.manual_seed(0)
    x = torch.randn(256, 192, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(320, 192, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_(True)
    b = torch.randn(320, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn(256, 320, device=DEV, dtype=torch.bfloat16)
    outs = []
    for hw in (False, True):
        x.grad = w.grad = b.grad = None
        y = MX.mx_linear(x, w, b, hybrid=True, fp8_wgrad=True, hardware=hw)
        y.backward(g)
        outs.append((y.detach().float(), x.grad.float().clone(), w.grad.float().clone()))
    for e, h in zip(*outs):
        _close(h, e, 3e-2, rtol=2e-2)


@pytest.mark.parametrize("e5m2", [False, True])
def test_mxfp8_dual_quantise_equals_the_two_single_direction_passes(e5m2):
    from gpt_neox_b200.ops import mxfp8 as MX
    torch.manual_seed(5)
    x = (torch.randn(203, 2184, device=DEV) * torch.logspace(-3, 2, 2184, device=DEV)).to(torch.bfloat16)
    x[40:80, 64:96] = 0
    tc, tr = MX.quantize_dual(x, e5m2)
    sc, sr = MX.quantize_tiled(x, False, e5m2), MX.quantize_tiled(x, True, e5m2)
    assert torch.equal(tc.q, sc.q) and torch.equal(tc.sf, sc.sf) and tc.mnb == sc.mnb
    assert torch.equal(tr.q, sr.q) and torch.equal(tr.sf, sr.sf) and tr.mnb == sr.mnb


# ------------------------------------------------------------------ fp16 operands, long persistent loops, small kernels
@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_gemm_fp16_operands(a_mn, b_mn, pair, monkeypatch):
    """fp16 A / B / bias / output through both tcgen05 kernels (instruction-descriptor format bit + fp16 epilogue)."""
    monkeypatch.setattr(G, "_PAIR", pair)
    torch.manual_seed(0)
    M, N, K = 520, 776, 392
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.float16)
    b = (torch.randn((K, N) if b_mn else (N, K), device=DEV) * 0.1).to(torch.float16)
    bias = torch.randn(N, device=DEV, dtype=torch.float16)
    res = torch.randn(M, N, device=DEV, dtype=torch.float16)
    got, pre = G.gemm(a, b, a_mn, b_mn, bias=bias, act=G.ACT_GELU, add=res, want_preact=True)
    assert got.dtype == torch.float16 and pre.dtype == torch.float16
    want, wpre = G.gemm_ref(a, b, a_mn, b_mn, bias=bias, act=G.ACT_GELU, add=res, want_preact=True, out_dtype=torch.float32)
    _close(pre, wpre, 0.02, rtol=4e-3)           # fp16 keeps 11 bits: tighter than the bf16 cases above
    _close(got, want, 0.02, rtol=4e-3)
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    want = G.gemm_ref(a, b, a_mn, b_mn, add=acc, out_dtype=torch.float32)
    G.gemm(a, b, a_mn, b_mn, out=acc, add=acc)
    _close(acc, want, 0.02, rtol=2e-3)
    assert native.read_status() == 0


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("M,N,K", [(4096, 4096, 512), (8192, 6144, 1024)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_gemm_many_tiles_per_cta(M, N, K, a_mn, b_mn, pair, monkeypatch):
    """Problems with several tiles per persistent CTA (accumulator double-buffering, barrier phase flips over many
    tiles, L2 tile order) against the fp32 product."""
    monkeypatch.setattr(G, "_PAIR", pair)
    torch.manual_seed(2)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.bfloat16)
    b = (torch.randn((K, N) if b_mn else (N, K), device=DEV) * 0.05).to(torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    got = G.gemm(a, b, a_mn, b_mn, bias=bias, out_dtype=torch.float32)
    want = G.gemm_ref(a, b, a_mn, b_mn, bias=bias, out_dtype=torch.float32)
    _close(got, want, 0.03, rtol=2e-3)
    assert native.read_status() == 0


@pytest.mark.parametrize("sq,sk,b,hq,hkv,d,causal", [(256, 256, 2, 4, 4, 96, True), (300, 300, 1, 4, 2, 64, True),
                                                     (200, 328, 1, 2, 2, 128, False)])
def test_flash_attention_fp16(sq, sk, b, hq, hkv, d, causal):
    from gpt_neox_b200.ops import attention as A
    torch.manual_seed(0)
    q = torch.randn(sq, b, hq, d, device=DEV, dtype=torch.float16, requires_grad=True)
    k = torch.randn(sk, b, hkv, d, device=DEV, dtype=torch.float16, requires_grad=True)
    v = torch.randn(sk, b, hkv, d, device=DEV, dtype=torch.float16, requires_grad=True)
    out = A.flash_attention(q, k, v, causal=causal)
    assert out.dtype == torch.float16
    g = torch.randn_like(out)
    out.backward(g)
    assert native.read_status() == 0
    refl = [t.detach().float().requires_grad_() for t in (q, k, v)]
    ref = A.attention_ref(*refl, causal, None, None, None)
    ref.backward(g.float())
    _close(out, ref, 1e-2)
    for got, want in zip((q, k, v), refl):
        _close(got.grad, want.grad, 0.01 + 0.01 * want.grad.abs().max().item(), rtol=1e-2)


@pytest.mark.parametrize("B,T,H,N", [(2, 64, 4, 64), (1, 100, 2, 64)])
def test_wkv6_kernel_matches_reference_scan(B, T, H, N):
    """RWKV-6 wkv forward and backward (CUDA) against the sequential fp32 recurrence."""
    from gpt_neox_b200.ops import wkv6 as W
    torch.manual_seed(0)
    C = H * N
    mk = lambda scale=1.0: (torch.randn(B, T, C, device=DEV) * scale).to(torch.bfloat16).requires_grad_()
    r, k, v = mk(), mk(0.5), mk()
    w = (-torch.rand(B, T, C, device=DEV) * 2 - 0.1).to(torch.bfloat16).requires_grad_()      # log-decay, negative
    u = (torch.randn(H, N, device=DEV) * 0.3).to(torch.bfloat16).requires_grad_()
    y = W.wkv6(r, k, v, w, u)
    g = torch.randn_like(y)
    y.backward(g)
    got = [t.grad.clone() for t in (r, k, v, w, u)]
    ref_in = [t.detach().float().requires_grad_() for t in (r, k, v, w, u)]
    yr = W.wkv6_ref(*ref_in)
    yr.backward(g.float())
    _close(y, yr, 0.05 + 0.02 * yr.abs().max().item(), rtol=2e-2)
    for a, b_ in zip(got, ref_in):
        _close(a, b_.grad, 0.05 + 0.03 * b_.grad.abs().max().item(), rtol=3e-2)


def test_lion_kernel_matches_eager_update():
    from gpt_neox_b200.optim.lion import Lion
    torch.manual_seed(0)
    n = 100_003
    p0 = torch.randn(n, device=DEV)
    grads = [torch.randn(n, device=DEV) for _ in range(3)]
    p_gpu = torch.nn.Parameter(p0.clone())
    out = torch.empty(n, device=DEV, dtype=torch.bfloat16)
    p_gpu.model_out = out
    p_cpu = torch.nn.Parameter(p0.cpu().clone())
    o_gpu = Lion([p_gpu], lr=1e-2, betas=(0.9, 0.98), weight_decay=0.1)
    o_cpu = Lion([p_cpu], lr=1e-2, betas=(0.9, 0.98), weight_decay=0.1)
    for g in grads:
        p_gpu.grad, p_cpu.grad = g.clone(), g.cpu().clone()
        o_gpu.step()
        o_cpu.step()
    # a sign flip needs |m*b1 + g*(1-b1)| at rounding level: allow a handful of elements to differ by 2*lr
    diff = (p_gpu.detach().cpu() - p_cpu.detach()).abs()
    assert (diff > 1e-5).sum().item() <= 3, diff.max()
    _close(out, p_gpu.detach(), 1e-2, rtol=1e-2)
    _close(o_gpu.state[p_gpu]["exp_avg"].cpu(), o_cpu.state[p_cpu]["exp_avg"], 1e-5, rtol=1e-4)


def test_adam8bit_tracks_fp32_adam():
    """Block-wise 8-bit optimizer states: after 20 steps on a quadratic the parameters stay close to fp32 Adam."""
    from gpt_neox_b200.optim.adam8bit import Adam8bit
    torch.manual_seed(0)
    n = 4096 + 77
    target = torch.randn(n, device=DEV)
    p8 = torch.nn.Parameter(torch.zeros(n, device=DEV))
    p32 = torch.nn.Parameter(torch.zeros(n, device=DEV))
    o8 = Adam8bit([p8], lr=5e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.0)
    o32 = torch.optim.Adam([p32], lr=5e-2, betas=(0.9, 0.95), eps=1e-8)
    for _ in range(20):
        for p, o in ((p8, o8), (p32, o32)):
            p.grad = (p.detach() - target) * (1 + 0.1 * torch.randn(n, device=DEV, generator=None))
            o.step()
    assert (p8 - p32).abs().max().item() < 0.15 and (p8 - target).norm() < 0.8 * target.norm()
    st = o8.state[p8]
    assert any(t.dtype in (torch.int8, torch.uint8) for t in st.values() if torch.is_tensor(t))
    # the CUDA kernel and the chunked torch statement of the same update agree (same quantised states, same result)
    pc = torch.nn.Parameter(torch.zeros(n))
    oc = Adam8bit([pc], lr=5e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.01)
    pg = torch.nn.Parameter(torch.zeros(n, device=DEV))
    og = Adam8bit([pg], lr=5e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.01)
    gen = torch.Generator().manual_seed(5)
    for _ in range(5):
        gr = torch.randn(n, generator=gen)
        pc.grad, pg.grad = gr.clone(), gr.to(DEV)
        oc.step()
        og.step()
    _close(pg.detach().cpu(), pc.detach(), 2e-3, rtol=1e-3)
    assert (og.state[pg]["qm"].cpu().int() - oc.state[pc]["qm"].int()).abs().max().item() <= 1
    # the 16-bit model copy written by the same kernel is the rounded fp32 parameter, tail block included
    pm = torch.nn.Parameter(torch.zeros(n, device=DEV))
    pm.model_out = torch.full((n,), 7.0, device=DEV, dtype=torch.bfloat16)
    om = Adam8bit([pm], lr=5e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.01)
    for _ in range(3):
        pm.grad = torch.randn(n, device=DEV)
        om.step()
    assert torch.equal(pm.model_out, pm.detach().bfloat16())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_bias_dropout_add_kernel_matches_the_philox_mask(dtype):
    """Training-mode bias + dropout + residual add in one kernel: forward and backward against the same Philox
    mask generated in plain torch; the keep rate is 1 - p; a replayed generator state reproduces the mask."""
    torch.manual_seed(123)
    rows, cols, p = 300, 1024, 0.1
    x = torch.randn(rows, cols, device=DEV, dtype=dtype, requires_grad=True)
    bias = torch.randn(cols, device=DEV, dtype=dtype, requires_grad=True)
    res = torch.randn(rows, cols, device=DEV, dtype=dtype, requires_grad=True)
    gen = torch.cuda.default_generators[torch.cuda.current_device()]
    state = torch.cuda.get_rng_state()
    seed, offset = gen.initial_seed(), gen.get_offset()
    out = OF.bias_dropout_add(x, bias, res, p, True)
    assert gen.get_offset() > offset                       # the stream was advanced: the next call draws a new mask
    keep = OF.philox_mask_ref(rows * cols, p, seed, offset, device=DEV).view(rows, cols)
    assert abs(keep.float().mean().item() - (1 - p)) < 5e-3
    want = res.float() + torch.where(keep, (x.float() + bias.float()) / (1 - p), torch.zeros((), device=DEV))
    _close(out, want, 2e-2 if dtype != torch.float32 else 1e-5)
    g = torch.randn_like(out)
    out.backward(g)
    gx = torch.where(keep, g.float() / (1 - p), torch.zeros((), device=DEV))
    _close(x.grad, gx, 2e-2 if dtype != torch.float32 else 1e-5)
    _close(res.grad, g, 0.0, rtol=0.0)
    _close(bias.grad, gx.sum(0), 0.5 if dtype != torch.float32 else 1e-3, rtol=2e-2)
    torch.cuda.set_rng_state(state)                        # what activation checkpointing does before recomputing
    again = OF.bias_dropout_add(x.detach(), bias.detach(), res.detach(), p, True)
    assert torch.equal(again, out.detach())
    other = OF.bias_dropout_add(x.detach(), bias.detach(), res.detach(), p, True)
    assert not torch.equal(other, out.detach())


# ------------------------------------------------------------------ mixture-of-experts kernels
@pytest.mark.parametrize("T,E,k,dtype", [(1000, 8, 2, torch.bfloat16), (513, 64, 1, torch.float32),
                                         (300, 200, 4, torch.float16)])
def test_moe_router_kernel_matches_eager(T, E, k, dtype):
    from gpt_neox_b200.ops import moe_ops as MO
    torch.manual_seed(0)
    logits = (torch.randn(T, E, device=DEV) * 2).to(dtype)
    a = logits.clone().requires_grad_(True)
    b = logits.clone().requires_grad_(True)
    probs, w, idx, counts = MO.router(a, k)
    probs_r, w_r, idx_r, counts_r = MO.router_ref(b, k)
    _close(probs, probs_r, 1e-6, rtol=1e-4)
    _close(w, w_r, 1e-6, rtol=1e-4)
    # ties between equal probabilities (frequent with 16-bit logits) may be broken differently: the selected
    # probabilities always agree; indices, histogram and gradients are compared on the rows without a tie
    assert torch.equal(probs_r.gather(1, idx).sort(1).values, probs_r.gather(1, idx_r).sort(1).values)
    rows = (idx == idx_r).all(1)
    assert rows.float().mean().item() > 0.9
    if bool(rows.all()):
        assert torch.equal(counts, counts_r)
    assert int(counts.sum()) == T * k
    gw = torch.randn(T, k, device=DEV)
    gp = torch.randn(T, E, device=DEV) * 0.1
    (w * gw).sum().add((probs * gp).sum()).backward()
    (w_r * gw).sum().add((probs_r * gp).sum()).backward()
    lo = dtype != torch.float32
    _close(a.grad[rows], b.grad[rows], 4e-3 if lo else 1e-5, rtol=2e-2 if lo else 1e-3)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_moe_dispatch_and_combine_kernels(dtype):
    from gpt_neox_b200.ops import moe_ops as MO
    torch.manual_seed(1)
    T, E, k, h = 700, 8, 2, 264
    idx = torch.stack([torch.randperm(E, device=DEV)[:k] for _ in range(T)])
    counts = torch.bincount(idx.reshape(-1), minlength=E)
    for cap in (None, 100):
        row_of, kept = MO.plan_rows(idx, counts, cap)
        rows = MO.padded_rows(T * k, E)
        # every kept assignment has its own row inside its expert's segment
        flat = row_of.reshape(-1)
        ok = flat >= 0
        assert flat[ok].unique().numel() == int(ok.sum()) == int(kept.sum())
        starts = torch.cumsum((kept + 63) // 64 * 64, 0) - (kept + 63) // 64 * 64
        e_of = idx.reshape(-1)[ok]
        assert bool(((flat[ok] >= starts[e_of]) & (flat[ok] < starts[e_of] + kept[e_of])).all())
        x = torch.randn(T, h, device=DEV).to(dtype)
        gate = torch.rand(T, k, device=DEV)
        xa = x.clone().requires_grad_(True)
        xb = x.clone().requires_grad_(True)
        ga = gate.clone().requires_grad_(True)
        gb = gate.clone().requires_grad_(True)
        pa = MO.dispatch(xa, row_of, rows)
        pb = MO.dispatch_ref(xb, row_of, rows)
        assert torch.equal(pa, pb)
        ya = MO.combine(pa * 1.0, row_of, ga)
        yb = MO.combine_ref(pb * 1.0, row_of, gb)
        _close(ya, yb, 1e-2)
        gy = torch.randn_like(ya)
        ya.backward(gy)
        yb.backward(gy)
        _close(xa.grad, xb.grad, 2e-2)
        _close(ga.grad, gb.grad, 5e-2, rtol=2e-2)


@pytest.mark.parametrize("counts,N,K,act", [([300, 0, 129, 64, 1, 700, 5, 90], 512, 256, None),
                                            ([37, 1000], 384, 192, "gelu"),
                                            ([0, 0, 0, 256], 256, 64, "gelu")])
def test_grouped_gemm_matches_per_expert_eager(counts, N, K, act):
    from gpt_neox_b200.ops import moe_ops as MO
    torch.manual_seed(2)
    E = len(counts)
    cnt = torch.tensor(counts, device=DEV)
    rows = MO.padded_rows(sum(counts), E)
    x = torch.zeros(rows, K, device=DEV, dtype=torch.bfloat16)
    g = torch.zeros(rows, N, device=DEV, dtype=torch.bfloat16)
    row = 0
    for c in counts:
        x[row:row + c] = torch.randn(c, K, device=DEV).to(torch.bfloat16)
        g[row:row + c] = torch.randn(c, N, device=DEV).to(torch.bfloat16)
        row += (c + 63) // 64 * 64
    w = (torch.randn(E, N, K, device=DEV) / math.sqrt(K)).to(torch.bfloat16)
    assert MO.grouped_kernel_ok(x, w)
    xa, wa = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    xb, wb = x.float().requires_grad_(True), w.float().requires_grad_(True)
    ya = MO.grouped_linear(xa, wa, cnt, act)
    yb = MO.grouped_linear_ref(xb, wb, cnt, act)
    assert native.read_status() == 0
    _close(ya, yb, 3e-2, rtol=2e-2)
    ya.backward(g)
    yb.backward(g.float())
    assert native.read_status() == 0
    _close(xa.grad, xb.grad, 5e-2, rtol=3e-2)
    _close(wa.grad, wb.grad, 0.25, rtol=3e-2)
    # weight gradients accumulate into the optimizer's fp32 buffer when it is attached
    wa2 = w.clone().requires_grad_(True)
    wa2.main_grad = torch.ones(E, N, K, device=DEV)
    MO.grouped_linear(x.clone().requires_grad_(True), wa2, cnt, act).backward(g)
    _close(wa2.main_grad - 1.0, wb.grad, 0.25, rtol=3e-2)


@pytest.mark.parametrize("rows,cols,dtype", [(4096, 6144, torch.bfloat16), (1000, 264, torch.float16), (7, 8, torch.bfloat16)])
def test_bias_grad_column_sum_kernel(rows, cols, dtype):
    torch.manual_seed(3)
    g = torch.randn(rows, cols, device=DEV).to(dtype)
    ref = g.float().sum(0)
    out = OF.bias_grad(g)
    assert out.dtype == dtype
    _close(out, ref, 0.05 * math.sqrt(rows) / 8, rtol=1e-2)
    # with the optimizer's fp32 buffer attached the sum is accumulated there and the parameter is reported ready
    bias = torch.nn.Parameter(torch.zeros(cols, device=DEV, dtype=dtype))
    bias.main_grad = torch.full((cols,), 2.0, device=DEV)
    seen = []
    bias._grad_ready = lambda: seen.append(1)
    assert OF.bias_grad(g, bias) is None and seen == [1] and bias.grad_in_main
    _close(bias.main_grad - 2.0, ref, 1e-3 * math.sqrt(rows), rtol=1e-5)
    # a strided view (the rows of a wider matrix)
    wide = torch.randn(rows, cols * 2, device=DEV).to(dtype)
    _close(OF.bias_grad(wide[:, :cols]), wide[:, :cols].float().sum(0), 0.05 * math.sqrt(rows) / 8, rtol=1e-2)


@pytest.mark.parametrize("kinds", [("ln", "ln"), ("ln",), ("rms",), ("rms", "ln")])
def test_norm_fan_out_adds_all_gradient_contributions_in_the_kernels(kinds):
    """Block head ``x -> (norms(x)..., x)``: outputs equal the separate norm kernels bit for bit; the input gradient is
    the sum of the residual gradient and every norm's gradient (fp32 oracle); parameter gradients as usual."""
    from gpt_neox_b200.models.norms import LayerNorm, RMSNorm
    torch.manual_seed(4)
    rows, b, h = 192, 3, 1024
    mods = [LayerNorm(h, eps=1e-5, device=DEV, dtype=torch.bfloat16) if k == "ln"
            else RMSNorm(h, eps=1e-6, device=DEV, dtype=torch.bfloat16) for k in kinds]
    for m in mods:
        for p in m.parameters():
            p.data.add_(torch.randn_like(p) * 0.2)
    x = torch.randn(rows, b, h, device=DEV).to(torch.bfloat16)
    gs = [torch.randn(rows, b, h, device=DEV).to(torch.bfloat16) for _ in range(len(mods) + 1)]
    xa = x.clone().requires_grad_(True)
    outs = OF.norm_fan_out(xa, mods)
    assert len(outs) == len(mods) + 1 and outs[-1].data_ptr() == xa.data_ptr()
    sep = [m(x) for m in mods]
    for o, s in zip(outs, sep):
        assert torch.equal(o, s)
    torch.autograd.backward(list(outs), gs)
    got = {id(p): p.grad.clone() for m in mods for p in m.parameters()}
    for m in mods:
        m.zero_grad()
    # fp32 oracle through the modules' eager math
    xb = x.float().requires_grad_(True)
    ws = [p for m in mods for p in m.parameters()]
    wf = [p.detach().float().requires_grad_(True) for p in ws]
    ref_outs = []
    it = iter(wf)
    for m, k in zip(mods, kinds):
        if k == "ln":
            w_, b_ = next(it), next(it)
            ref_outs.append(torch.nn.functional.layer_norm(xb, (h,), w_, b_, m.eps))
        else:
            s_ = next(it)
            ref_outs.append(xb / (xb.norm(2, dim=-1, keepdim=True) * h ** -0.5 + m.eps) * s_)
    torch.autograd.backward(ref_outs + [xb * 1.0], [g.float() for g in gs])
    _close(xa.grad, xb.grad, 0.06, rtol=2e-2)
    for p, f in zip(ws, wf):
        _close(got[id(p)], f.grad, 0.02 * math.sqrt(rows * b), rtol=3e-2)
    # only some outputs used: the others contribute nothing (no zero tensors are materialised for them)
    xc = x.clone().requires_grad_(True)
    outs = OF.norm_fan_out(xc, mods)
    outs[0].backward(gs[0])
    xd = x.clone().requires_grad_(True)
    mods[0](xd).backward(gs[0])
    _close(xc.grad, xd.grad, 1e-6, rtol=0)


def test_block_sparse_attention_on_device_bf16():
    from gpt_neox_b200.models.transformer import sparse_layout_mask
    from gpt_neox_b200.ops.sparse_attention import block_sparse_attention
    torch.manual_seed(0)
    s, b, h, d = 1000, 2, 8, 64
    cfg = {"block": 16, "num_sliding_window_blocks": 5, "num_global_blocks": 2, "num_random_blocks": 2}
    q, k, v = [torch.randn(s, b, h, d, device=DEV).to(torch.bfloat16).requires_grad_(True) for _ in range(3)]
    out = block_sparse_attention(q, k, v, "bigbird", cfg, d ** -0.5)
    g = torch.randn_like(out)
    out.backward(g)
    mask = sparse_layout_mask("bigbird", s, s, cfg, q.device) | \
        (torch.arange(s, device=DEV)[None, :] > torch.arange(s, device=DEV)[:, None])
    qf, kf, vf = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    probs = torch.softmax((torch.einsum("sbhd,tbhd->bhst", qf, kf) * d ** -0.5).masked_fill(mask[None, None],
                                                                                           float("-inf")), dim=-1)
    ref = torch.einsum("bhst,tbhd->sbhd", probs, vf)
    ref.backward(g.float())
    _close(out, ref, 2e-2, rtol=2e-2)
    for a, r in ((q.grad, qf.grad), (k.grad, kf.grad), (v.grad, vf.grad)):
        _close(a, r, 6e-2, rtol=5e-2)


@pytest.mark.parametrize("n,offset", [(1, 0), (7, 1), (1000003, 0), (1000003, 3), (4096, 2)])
def test_squared_norm_kernel_any_alignment(n, offset):
    import ctypes
    torch.manual_seed(6)
    base = torch.randn(n + offset + 8, device=DEV)
    x = base[offset:offset + n]
    out = torch.zeros((), device=DEV)
    rc = native.lib().neox_sumsq_f32(native.ptr(x), ctypes.c_longlong(n), native.ptr(out),
                                     ctypes.c_void_p(native.stream_ptr()))
    native.check(rc, "neox_sumsq_f32")
    ref = (x.double() ** 2).sum().item()
    assert abs(out.item() - ref) <= 2e-5 * max(ref, 1.0), (out.item(), ref)


@pytest.mark.parametrize("b,l,d,time_major", [(1, 1, 64, False), (2, 33, 65, True), (3, 96, 136, True), (1, 300, 40, False),
                                              (2, 40, 75776, False)])
def test_selective_scan_chunks_and_strides(b, l, d, time_major):
    """Edges of the chunked scan -- one step, a chunk and one step, whole chunks, many chunks, channels that leave a block
    part full, channels that fill the machine (no split of time) -- on operands that are slices of wider [l, b, ...]
    tensors, against the recurrence in fp32.  bf16 outputs: half an ulp (2^-9) of the value plus the summation error."""
    from gpt_neox_b200.ops import selective_scan as SS
    torch.manual_seed(l)
    n = 16

    def mk(w, dtype, scale=1.0):
        t = (torch.randn(l, b, w + 8, device=DEV) * scale).to(dtype)[..., 8:].transpose(0, 1) if time_major \
            else (torch.randn(b, l, w, device=DEV) * scale).to(dtype)
        return t.detach().requires_grad_(True)
    u, dt, z = mk(d, torch.bfloat16), mk(d, torch.bfloat16, 0.5), mk(d, torch.bfloat16)
    B, C = mk(n, torch.float32, 0.5), mk(n, torch.float32, 0.5)
    A = (-torch.rand(d, n, device=DEV) * 2 - 0.1).requires_grad_(True)
    D, bias = torch.randn(d, device=DEV).requires_grad_(True), (torch.randn(d, device=DEV) * 0.3).requires_grad_(True)
    leaves = [u, dt, A, B, C, D, z, bias]
    out = SS.selective_scan(u, dt, A, B, C, D, z, bias)
    g = torch.randn(l, b, d, device=DEV).to(torch.bfloat16).transpose(0, 1) if time_major else torch.randn_like(out)
    got = torch.autograd.grad(out, leaves, g)
    ref_leaves = [t.detach().float().requires_grad_(True) for t in leaves]
    ru, rdt, rA, rB, rC, rD, rz, rbias = ref_leaves
    ref = SS.selective_scan_ref(ru, rdt, rA, rB, rC, rD, rz, rbias, True)
    want = torch.autograd.grad(ref, ref_leaves, g.float())
    for have, exact in zip([out, *got], [ref, *want]):
        _close(have, exact, 4e-3 + 2e-3 * exact.abs().max().item(), rtol=4e-3)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("b,l,d,time_major,bias", [(1, 1, 8, False, True), (2, 3, 264, True, True), (3, 17, 136, True, False),
                                                   (1, 256, 128, False, True), (2, 300, 1032, True, True)])
def test_causal_conv_matches_fp32(b, l, d, time_major, bias, dtype):
    """Width-4 causal convolution + SiLU of the first half of a projection, sequences shorter than the window, runs and
    blocks part full, both orders of batch and time; forward, input, weight and bias gradients.  Outputs round once, so
    they are within half an ulp; the weight gradient rounds once after a sum of b * l fp32 products."""
    from gpt_neox_b200.ops import selective_scan as SS
    torch.manual_seed(l + d)
    xz = torch.randn(l, b, 2 * d, device=DEV).to(dtype).transpose(0, 1) if time_major else \
        torch.randn(b, l, 2 * d, device=DEV).to(dtype)
    xz.requires_grad_()
    w = (torch.randn(d, 4, device=DEV) * 0.5).to(dtype).requires_grad_()
    bs = (torch.randn(d, device=DEV) * 0.5).to(dtype).requires_grad_() if bias else None
    assert SS._conv_kernel_ok(xz, w, bs)
    leaves = [xz, w] + ([bs] if bias else [])
    x, z = SS.causal_conv1d_split(xz, w, bs)
    gx, gz = torch.randn(b, l, d, device=DEV).to(dtype), torch.randn(b, l, d, device=DEV).to(dtype)
    got = torch.autograd.grad([x, z], leaves, [gx, gz])
    ref = [t.detach().cpu().float().requires_grad_() for t in leaves]
    rx, rz = SS.causal_conv1d_split(ref[0], ref[1], ref[2] if bias else None)
    want = torch.autograd.grad([rx, rz], ref, [gx.cpu().float(), gz.cpu().float()])
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b_ in zip([x, z, *got], [rx, rz, *want]):
        _close(a.cpu(), b_, 2e-4 + ulp / 2 * b_.abs().mean().item(), rtol=ulp)
    plain = SS.causal_conv1d(xz.detach()[..., :d], w, bs, activation=None)
    _close(plain.cpu(), SS.causal_conv1d(xz.detach().cpu().float()[..., :d], ref[1], ref[2] if bias else None, activation=None),
           2e-4 + ulp / 2, rtol=ulp)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 2048, 4096), (3, 24, 72), (8, 1000, 1032), (9, 16, 64), (16, 4104, 520),
                                   (17, 40, 2056), (32, 264, 136), (33, 64, 128)])
def test_few_row_gemm_matches_fp32(M, N, K, dtype):
    """The weight-streaming kernel (up to 32 rows; 33 takes the tile kernel): part-filled row groups, weight tiles and
    k-blocks, one k-block and K split over a cluster, all epilogues.  The 16-bit result is within half an ulp of the fp32
    value, whose own summation error is below K * 2^-24 of the sum of magnitudes."""
    from gpt_neox_b200.ops import gemm as G
    torch.manual_seed(M * N + K)
    x = torch.randn(M, K + 8, device=DEV).to(dtype)[:, :K]
    w, bias, add = torch.randn(N, K, device=DEV).to(dtype), torch.randn(N, device=DEV).to(dtype), torch.randn(M, N, device=DEV)
    aux, scale = torch.randn(M, N, device=DEV).to(dtype), K ** -0.5
    assert G.use_skinny_kernel(M, N, K, False, False) == (M <= 32)
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11

    def check(**kw):
        got, want = G.gemm(x, w, alpha=scale, **kw), G.gemm_ref(x, w, alpha=scale, **{"out_dtype": dtype, **kw})
        for a, b in zip(got, want) if kw.get("want_preact") else [(got, want)]:
            _close(a, b, 1e-4 if kw.get("out_dtype") == torch.float32 else half_ulp / 8,
                   rtol=1e-4 if kw.get("out_dtype") == torch.float32 else 2 * half_ulp)
    check()
    check(bias=bias, add=add.to(dtype))
    check(bias=bias, act=G.ACT_GELU, want_preact=True)
    check(act=G.ACT_DGELU, aux=aux)
    check(out_dtype=torch.float32, add=add)
    assert torch.equal(G.gemm(x, w, bias=bias), G.gemm(x, w, bias=bias))       # fixed summation order


@pytest.mark.parametrize("n,b,hq,hkv,d,rot,window,alibi,dtype", [
    (1, 1, 4, 4, 64, 16, None, False, torch.float16), (31, 2, 4, 1, 128, 128, None, False, torch.bfloat16),
    (129, 1, 4, 2, 96, 24, None, True, torch.bfloat16), (700, 2, 8, 8, 64, 64, None, False, torch.bfloat16),
    (700, 1, 4, 4, 128, 32, 37, False, torch.float16), (2047, 1, 2, 2, 128, 0, 1500, True, torch.bfloat16),
    (300, 20, 16, 16, 64, 16, 0, False, torch.bfloat16)])
def test_decode_attention_matches_rotary_append_and_attention(n, b, hq, hkv, d, rot, window, alibi, dtype):
    """One launch against the separate steps in fp32: rotary embedding, append, softmax over the cache (split over one
    to eight CTAs), grouped queries, window, ALiBi, packed strided projections, position on the host and on the device.
    The output is a convex combination of values, so its error is that of 16-bit weights' fp32 sums plus half an ulp."""
    from gpt_neox_b200.models.positional import RotaryEmbedding
    from gpt_neox_b200.ops import attention as A
    from gpt_neox_b200.ops import functional as OF
    torch.manual_seed(n + d)
    packed = torch.randn(1, b, hq + 2 * hkv, d, device=DEV).to(dtype)
    q, k, v = packed.split([hq, hkv, hkv], dim=2)
    cap = n + 1 if n == 2047 else n + 9
    cache = torch.randn(2, cap, b, hkv, d, device=DEV).to(dtype)
    cos = sin = None
    kr, qr = k, q
    if rot:
        cos, sin = RotaryEmbedding(rot, cap).to(DEV)(q, seq_len=cap)
        qr, kr = OF.rope_ref(q, cos[n:n + 1], sin[n:n + 1]), OF.rope_ref(k, cos[n:n + 1], sin[n:n + 1])
    slopes = torch.rand(hq, device=DEV) if alibi else None
    keys = torch.cat([cache[0, :n], kr]).float()
    vals = torch.cat([cache[1, :n], v]).float()
    want = A.attention_ref(qr.float(), keys, vals, True, 0.1, window, slopes)
    assert A.decode_attention_ok(q, k, v)
    for pos in (None, torch.tensor([n], device=DEV)):
        c = cache.clone()
        got = A.decode_attention(q, k, v, c, n if pos is None else cap - 1, pos, cos, sin, 0.1, window, slopes)
        _close(got, want, 1e-3, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10)
        _close(c[0, n], kr[0], 1e-3, rtol=2.0 ** -8)                   # the rotated key, to the rounding of its 16 bits
        assert torch.equal(c[1, n], v[0])
        keep = torch.arange(cap, device=DEV) != n
        assert torch.equal(c[:, keep], cache[:, keep])


@pytest.mark.parametrize("kind", ["ln", "rms"])
@pytest.mark.parametrize("rows,cols,dtype", [
    (1, 8, torch.bfloat16), (700, 256, torch.float16), (5, 264, torch.bfloat16), (3001, 520, torch.bfloat16),
    (900, 776, torch.float32), (1300, 1024, torch.float16), (700, 1032, torch.bfloat16), (9, 3080, torch.bfloat16),
    (650, 6152, torch.float16), (3, 9224, torch.bfloat16)])
def test_norm_row_splits_match_fp64(kind, rows, cols, dtype):
    """Every split of a row (one to four warps, one to three vectors of a CTA's threads, re-read rows), part-filled warps, row
    counts that leave CTAs or row groups without a row; addend aliasing the result, parameter gradients stored and
    accumulated.  Row results round once (half an ulp) after fp32 sums; column sums are fp32 over ``rows`` terms."""
    torch.manual_seed(rows + cols)
    x, g, res = (torch.randn(rows, cols, device=DEV).to(dtype) for _ in range(3))
    w, b = (1 + 0.1 * torch.randn(cols, device=DEV)).to(dtype), (0.1 * torch.randn(cols, device=DEV)).to(dtype)
    xr, wr, br = (t.double().requires_grad_() for t in (x, w, b))
    if kind == "ln":
        yr, y = torch.nn.functional.layer_norm(xr, (cols,), wr, br, 1e-5), OF.layer_norm(x, w, b, 1e-5)
        mean, sc = xr.mean(-1), (xr.var(-1, unbiased=False) + 1e-5).rsqrt()
    else:
        rms = xr.pow(2).mean(-1, keepdim=True).sqrt()
        yr, y = xr / (rms + 1e-5) * wr + br, OF.rms_norm(x, w, b, 1e-5)
        mean, sc = None, 1 / (rms[:, 0] + 1e-5)
    yr.backward(g.double())
    ulp = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -18}[dtype]
    _close(y, yr, ulp, rtol=ulp)
    w.main_grad = torch.full((cols,), 2.0, device=DEV)
    dx = res.clone()
    mean, sc = (None if t is None else t.detach().float().contiguous() for t in (mean, sc))
    gw, gb = OF._norm_backward(kind, g, x, w, b, mean, sc, dx, dx, 1e-5, True, True)
    _close(dx, xr.grad + res.double(), ulp, rtol=ulp)
    assert gw is None and w.grad_in_main
    sums = 1e-5 * math.sqrt(rows) + 1e-5
    _close(w.main_grad - 2.0, wr.grad, sums, rtol=1e-5)
    _close(gb, br.grad, sums, rtol=1e-5 + (0 if dtype == torch.float32 else ulp))


@pytest.mark.parametrize("M,N,K", [(128, 256, 8192), (136, 40, 4104), (768, 768, 1000), (72, 1032, 3000), (2048, 2048, 1024)])
def test_accumulating_gemm_splits_the_contraction(M, N, K):
    """``acc += a^T b`` where few output tiles make the kernel split K (up to 8 parts, uneven, ragged edges of the output in
    element-wise additions) and where it does not.  fp32 accumulation: error below sqrt(K) * 2^-22 of the terms' size."""
    from gpt_neox_b200.ops import gemm as G
    torch.manual_seed(K)
    a, b = torch.randn(K, M, device=DEV).to(torch.bfloat16), torch.randn(K, N, device=DEV).to(torch.bfloat16)
    acc = torch.randn(M, N, device=DEV)
    want = acc.double() + a.double().t() @ b.double()
    G.gemm(a, b, a_mn=True, b_mn=True, out=acc, add=acc)
    _close(acc, want, 1e-5 * math.sqrt(K), rtol=1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("s,b,hq,hk,d,rot", [(7, 3, 5, 5, 64, 64), (33, 1, 3, 1, 96, 24), (5, 2, 4, 4, 128, 32), (9, 1, 2, 2, 64, 20),
                                             (4, 1, 1, 1, 96, 6)])
def test_rope_in_place_every_access_width(s, b, hq, hk, d, rot, dtype):
    """In-place rotation of q and k inside a packed projection: vectors of 8 and 4 and single elements, head counts that leave
    a thread's group of four part full, and the inverse.  One rounding, half an ulp, after two products in fp32 that may cancel:
    2^-24 of each product's size, with and without a fused multiply-add."""
    import ctypes
    torch.manual_seed(rot)
    packed = torch.randn(s, b, hq + 2 * hk, d, device=DEV).to(dtype)
    before = packed.clone()
    q, k = packed[:, :, :hq], packed[:, :, hq:hq + hk]
    cos, sin = torch.randn(s, rot, device=DEV), torch.randn(s, rot, device=DEV)
    ll = ctypes.c_longlong
    ulp = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}[dtype]
    for inverse in (0, 1):
        want = OF.rope_ref(packed[:, :, :hq + hk], cos.view(s, 1, 1, rot), (-sin if inverse else sin).view(s, 1, 1, rot))
        native.check(native.lib().neox_rope_qk_inplace(
            native.ptr(q), native.ptr(k), native.ptr(cos), native.ptr(sin), s, b, hq, hk, rot, ll(q.stride(0)),
            ll(q.stride(1)), ll(q.stride(2)), ll(k.stride(0)), ll(k.stride(1)), ll(k.stride(2)), inverse, OF._DT[dtype],
            OF._s()), "rope")
        products = 2.0 ** -22 * before.float().abs().max().item() * max(cos.abs().max().item(), sin.abs().max().item()) ** 2
        _close(packed[:, :, :hq + hk], want, ulp / 8 + products, rtol=ulp)
        assert torch.equal(packed[:, :, hq + hk:], before[:, :, hq + hk:])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n,offset", [(1, 0), (4, 0), (1027, 0), (1027, 4), (1027, 1), (300000, 0), (300000, 2)])
def test_adam_shards_of_any_alignment(n, offset, dtype):
    """A shard that starts anywhere in a flat buffer: four elements at a time where all tensors allow it, one otherwise, the
    remainder, and nothing outside the shard.  The update in fp64, fp32 rounding of a few operations."""
    import ctypes
    torch.manual_seed(n)
    full = n + offset + 8
    p, m, g = (torch.randn(full, device=DEV) for _ in range(3))
    v, out = torch.rand(full, device=DEV), torch.zeros(full, device=DEV, dtype=dtype)
    keep = [t.clone() for t in (p, m, v, out)]
    sl = slice(offset, offset + n)
    f = ctypes.c_float
    native.check(native.lib().neox_adam_step(
        native.ptr(p[sl]), native.ptr(m[sl]), native.ptr(v[sl]), native.ptr(g[sl]), native.ptr(out[sl]), OF._DT[dtype],
        ctypes.c_longlong(n), f(1e-2), f(0.9), f(0.95), f(1e-8), f(0.1), f(0.1), f(0.05), f(0.5), 1, OF._s()), "adam")
    P, M, V, G = (t[sl].double() for t in (*keep[:3], g))
    G = G * 0.5
    M, V = 0.9 * M + 0.1 * G, 0.95 * V + 0.05 * G * G
    P = P - (1e-2 / 0.1 * M / (V.sqrt() / 0.05 ** 0.5 + 1e-8) + 1e-2 * 0.1 * P)
    for have, want in ((p, P), (m, M), (v, V)):
        _close(have[sl], want, 1e-6, rtol=2e-6)
    assert torch.equal(out[sl], p[sl].to(dtype))
    for have, was in zip((p, m, v, out), keep):
        assert torch.equal(have[:offset], was[:offset]) and torch.equal(have[offset + n:], was[offset + n:])


@pytest.mark.parametrize("B,T,H,N", [(1, 1, 1, 32), (2, 16, 2, 64), (1, 65, 3, 64), (2, 200, 2, 128), (1, 700, 2, 32),
                                     (300, 130, 4, 32)])
def test_wkv6_groups_match_reference_scan(B, T, H, N):
    """Edges of the staged groups of eight steps (one step, whole groups, a group and one step, fewer groups than pieces of a
    state row, more heads than the machine holds) against the sequential recurrence in fp32.  bf16 results: half an ulp (2^-9) of the value plus the
    fp32 sums' error, which scales with the largest result."""
    from gpt_neox_b200.ops import wkv6 as W
    torch.manual_seed(T)
    C = H * N
    mk = lambda scale=1.0: (torch.randn(B, T, C, device=DEV) * scale).to(torch.bfloat16).requires_grad_()
    r, k, v, w = mk(), mk(0.5), mk(), mk(1.5)
    u = (torch.randn(H, N, device=DEV) * 0.3).to(torch.bfloat16).requires_grad_()
    y = W.wkv6(r, k, v, w, u)
    g = torch.randn_like(y)
    got = torch.autograd.grad(y, (r, k, v, w, u), g)
    ref_in = [t.detach().float().requires_grad_() for t in (r, k, v, w, u)]
    yr = W.wkv6_ref(*ref_in)
    want = torch.autograd.grad(yr, ref_in, g.float(), allow_unused=True)       # one step uses no decay
    want = [torch.zeros_like(t) if w_ is None else w_ for t, w_ in zip(ref_in, want)]
    # The decay gradient is ew times the difference of two sums over all later steps: T additions, each rounded to 2^-24 of a
    # running sum that is far larger than the difference, so its error is of the size sqrt(T) 2^-24 |ew| |running sum|
    # (twice, for the two sums; twice again for the largest of all elements).
    rr, kr, vr, wr, ur = (t.detach() for t in ref_in)
    vg = (vr * g.float()).view(B, T, H, N).sum(-1, keepdim=True).expand(B, T, H, N).reshape(B, T, C)
    running = (rr * (want[0] - ur.reshape(1, 1, C) * kr * vg)).flip(1).cumsum(1).abs().max().item()
    decay = 4 * math.sqrt(T) * 2.0 ** -24 * running * wr.exp().max().item()
    for n_, (a, b_) in enumerate(zip([y, *got], [yr, *want])):
        _close(a, b_, 1e-3 + 2e-3 * b_.abs().max().item() + (decay if n_ == 4 else 0.0), rtol=4e-3)


@pytest.mark.parametrize("kind", ["gemm", "pair", "few_rows", "attention"])
def test_first_cuda_work_of_a_thread(kind):
    """A backward pass may begin with one of these kernels on an autograd thread that has done no CUDA work yet: a fresh
    thread without a current context computes what this one does."""
    import threading
    from gpt_neox_b200.ops import attention as A
    from gpt_neox_b200.ops import gemm as G
    torch.manual_seed(0)
    M, N = {"gemm": (200, 264), "pair": (2560, 2304), "few_rows": (3, 264), "attention": (8, 8)}[kind]
    a, b = torch.randn(M, 320, device=DEV).to(torch.bfloat16), torch.randn(N, 320, device=DEV).to(torch.bfloat16)
    q = torch.randn(130, 2, 3, 64, device=DEV).to(torch.bfloat16)
    run = (lambda: A.flash_attention(q, q, q)) if kind == "attention" else (lambda: G.gemm(a, b))
    want, got = run(), []
    torch.cuda.synchronize()
    a, b, q = a.clone(), b.clone(), q.clone()              # other addresses: no tensor map of the call above is found again

    def work():
        try:
            got.append(run())
        except Exception as e:
            got.append(e)
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert torch.is_tensor(got[0]), got[0]
    torch.cuda.synchronize()
    assert torch.equal(got[0], want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,narrow", [(2331, 2048, 328, True), (5781, 1024, 520, True), (8192, 768, 264, True),
                                          (4000, 1160, 1000, True), (2331, 6144, 264, False)])
def test_pair_gemm_tile_widths(M, N, K, narrow, dtype):
    """Products that fill a round of 256 x 256 tiles poorly take tiles of 192 columns: column counts that are and are not
    multiples of 192, a last tile whose second half lies outside, ragged rows and contraction, every epilogue.  16-bit
    results within half an ulp of the fp32 value (sums of K products, error below K 2^-24 of their size)."""
    torch.manual_seed(M + N)
    rows = -(-M // 256)
    assert (-(-rows * -(-N // 192) // 74) * 92 < -(-rows * -(-N // 256) // 74) * 100) == narrow and G.use_pair_kernel(M, N, K)
    x, w = torch.randn(M, K, device=DEV).to(dtype), torch.randn(N, K, device=DEV).to(dtype)
    bias, add, s = torch.randn(N, device=DEV).to(dtype), torch.randn(M, N, device=DEV).to(dtype), K ** -0.5
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for kw in ({}, {"bias": bias, "add": add}, {"bias": bias, "act": G.ACT_GELU, "want_preact": True}, {"out_dtype": torch.float32}):
        got, want = G.gemm(x, w, alpha=s, **kw), G.gemm_ref(x, w, alpha=s, **{"out_dtype": dtype, **kw})
        for a, b in zip(got, want) if kw.get("want_preact") else [(got, want)]:
            _close(a, b, 2e-4 if kw.get("out_dtype") == torch.float32 else half_ulp / 4, rtol=2 * half_ulp)
    assert native.read_status() == 0


def test_causal_conv_second_derivatives_and_transforms():
    """What the library convolution offered beside first gradients: second derivatives, vmap and forward mode, in bf16 against
    the same in fp32 (a few roundings of 2^-8 each)."""
    from torch.autograd import forward_ad
    from gpt_neox_b200.ops import selective_scan as SS
    torch.manual_seed(0)
    x, w, bs = torch.randn(2, 3, 12, 16, device=DEV), torch.randn(16, 4, device=DEV) * 0.5, torch.randn(16, device=DEV)

    def second(x, w, bs):
        x, w, bs = (t.detach().requires_grad_() for t in (x, w, bs))
        y = SS.causal_conv1d(x, w, bs)
        gx, gw = torch.autograd.grad(y.float().square().sum(), (x, w), create_graph=True)
        return torch.autograd.grad(gx.float().sum() + gw.float().sum(), (x, w, bs))
    b16 = lambda *ts: [t.to(torch.bfloat16) for t in ts]
    for a, b in zip(second(*b16(x[0], w, bs)), second(*(t.float() for t in b16(x[0], w, bs)))):
        _close(a, b, 0.02 * b.abs().max().item(), rtol=0.02)
    xb, wb, bb = b16(x, w, bs)
    plain = torch.stack([SS.causal_conv1d(t, wb, bb) for t in xb])
    _close(torch.func.vmap(lambda t: SS.causal_conv1d(t, wb, bb))(xb), plain, 2.0 ** -7, rtol=2.0 ** -6)
    with forward_ad.dual_level():
        out = SS.causal_conv1d(forward_ad.make_dual(xb[0], torch.ones_like(xb[0])), wb, bb)
        assert forward_ad.unpack_dual(out).tangent is not None


def test_selective_scan_on_overlapping_windows():
    """Windows of one signal (strides (s, 1, 1)) as the input: results and gradients equal those on its copy, bit for bit in
    the outputs."""
    from gpt_neox_b200.ops import selective_scan as SS
    torch.manual_seed(0)
    b, l, d, n = 2, 40, 64, 16
    u = torch.randn(b, 256, device=DEV).to(torch.bfloat16).as_strided((b, l, d), (256, 1, 1))
    dt, z, g = (torch.randn(b, l, d, device=DEV).to(torch.bfloat16) for _ in range(3))
    B, C, A = torch.randn(b, l, n, device=DEV), torch.randn(b, l, n, device=DEV), -torch.rand(d, n, device=DEV) - 0.1
    D, bias = torch.randn(d, device=DEV), torch.randn(d, device=DEV)
    got = []
    for t in (u, u.contiguous()):
        zz = z.clone().requires_grad_()
        y = SS.selective_scan(t, dt, A, B, C, D, zz, bias)
        got.append((y, *torch.autograd.grad(y, zz, g)))
    for a, c in zip(*got):
        assert torch.equal(a, c)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(128, 256, 8192), (136, 40, 4104), (768, 768, 1000), (72, 1030, 3000), (200, 264, 700),
                                   (768, 2304, 8192)])
def test_accumulating_gemm_is_repeatable(M, N, K, dtype):
    """``acc += a^T b`` gives the same bits every time, whatever order the parts of a split contraction finish in, and touches
    nothing beside the product's columns when the output is a slice of a wider buffer.  Values: the tensor cores truncate the
    running sum (about 5 sqrt(K) at most for products of unit normals) to 24 bits after each of K / 16 steps."""
    torch.manual_seed(K)
    a, b = torch.randn(K, M, device=DEV).to(dtype), torch.randn(K, (N + 7) // 8 * 8, device=DEV).to(dtype)[:, :N]
    wide = torch.randn(M, N + 3, device=DEV)
    results = []
    for view in (lambda t: t[:, :N], lambda t: t[:, 3:]):
        for _ in range(6):
            acc = wide.clone()
            G.gemm(a, b, a_mn=True, b_mn=True, out=view(acc), add=view(acc))
            keep = acc.clone()
            view(keep).copy_(view(wide))
            assert torch.equal(keep, wide)
            results.append(view(acc).clone())
        want = view(wide).double() + a.double().t() @ b.double()
        _close(results[-1], want, K / 16 * 2.0 ** -23 * 5 * math.sqrt(K), rtol=1e-5)
        assert all(torch.equal(r, results[-1]) for r in results[-6:])
    dense = [wide[:, :N].clone() for _ in range(6)]
    for t in dense:
        G.gemm(a, b, a_mn=True, b_mn=True, out=t, add=t)
    assert all(torch.equal(t, results[0]) for t in dense)


@pytest.mark.parametrize("B,H", [(1, 2), (3, 4)])
def test_wkv6_without_steps_has_zero_gradients(B, H):
    """No steps: empty results, and a gradient of zero for the bonus, whatever was in memory before."""
    from gpt_neox_b200.ops import wkv6 as W
    N = 64
    r, k, v, w = (torch.zeros(B, 0, H * N, device=DEV, dtype=torch.bfloat16, requires_grad=True) for _ in range(4))
    u = torch.randn(H, N, device=DEV).to(torch.bfloat16).requires_grad_()
    y = W.wkv6(r, k, v, w, u)
    assert y.shape == (B, 0, H * N)
    for _ in range(4):
        torch.full((B, H, N), float("nan"), device=DEV)                       # what a fresh allocation may hold
        grads = torch.autograd.grad(y, (r, k, v, w, u), torch.empty_like(y), retain_graph=True)
        assert all(g.numel() == 0 for g in grads[:4]) and torch.equal(grads[4], torch.zeros_like(u))


@pytest.mark.parametrize("first", [1e30, float("inf"), -float("inf")])
def test_selective_scan_carries_extreme_states_between_chunks(first):
    """A state that is huge, or has overflowed, and decays by more than fp32's range over a chunk of 32 steps, though by a normal
    number in each: it is handed on as in the step-by-step recurrence.  (Outputs in bf16, 2^-8 each; 96 factors of a relative
    error of 2^-22 and an exponent of up to 400 in each product of factors.)"""
    from gpt_neox_b200.ops import selective_scan as SS
    b, l, d, n = 1, 100, 64, 16
    u = torch.zeros(b, l, d, device=DEV).to(torch.bfloat16)
    u[:, 0] = first
    dt = torch.full((b, l, d), 0.5413, device=DEV).to(torch.bfloat16)          # softplus: 1
    A = -torch.linspace(0.5, 4.0, d, device=DEV)[:, None].expand(d, n).contiguous()
    B, C, z = torch.ones(b, l, n, device=DEV), torch.ones(b, l, n, device=DEV), torch.ones(b, l, d, device=DEV).to(torch.bfloat16)
    D, bias = torch.zeros(d, device=DEV), torch.zeros(d, device=DEV)
    got = SS.selective_scan(u, dt, A, B, C, D, z, bias).float()
    want = SS.selective_scan_ref(u.double(), dt.double(), A.double(), B.double(), C.double(), D.double(), z.double(), bias.double(),
                                 True) if math.isfinite(first) else None
    if want is not None:
        normal = want.abs() > 2.0 ** -120
        assert int(normal[:, 64:].sum()) > 0
        assert bool(((got.double() - want).abs() <= 0.01 * want.abs())[normal].all())
    else:
        assert bool((got[:, 1:] == first).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols,shift,rank", [(8, 0, 0), (1000, 0, 1), (50304, 0, 0), (1001, 0, 1), (1000, 1, 0)])
def test_cross_entropy_of_extreme_16_bit_logits(cols, shift, rank, dtype, monkeypatch):
    """Loss and gradient over one rank's share of the vocabulary: targets owned and not owned, the largest 16-bit values, rows with
    -inf (also at the target), with nothing but -inf and with inf, where fp64 gives inf or NaN and so must the kernels.  Both
    forms (vector loads; odd widths and unaligned rows).  Statistics in fp32 with fast exponentials (an error of some 2^-21 of
    the exponent, at most 2^4 where it counts), gradients rounded to 16 bits."""
    from gpt_neox_b200.parallel import cross_entropy as CE
    torch.manual_seed(cols)
    rows, top = 12, torch.finfo(dtype).max if dtype == torch.float16 else 1e4
    v0 = rank * cols
    monkeypatch.setattr(CE.mpu, "get_model_parallel_rank", lambda: rank)
    x = (torch.randn(rows, cols, device=DEV) * 4).to(dtype)
    tgt = torch.randint(0, cols, (rows,), device=DEV) + v0
    tgt[0], tgt[1], tgt[2] = v0, v0 + cols - 1, v0 + cols // 2
    tgt[3], tgt[4] = v0 + cols, v0 - 1                                        # another rank's
    x[5, ::2] = -float("inf")
    tgt[5] = v0 + 1
    x[6, tgt[6] - v0] = -float("inf")
    x[7] = -float("inf")
    x[8, cols // 2] = float("inf")
    x[9, 1], x[9, 2] = top, -top
    x[10] = top
    x[11, 3] = float("nan")
    buf = torch.empty(rows * cols + 8, device=DEV, dtype=dtype)
    logits = buf[shift:shift + rows * cols].view(rows, cols).copy_(x)
    logits = logits.detach().requires_grad_()
    g = torch.rand(rows, device=DEV) + 0.5
    loss = CE.vocab_parallel_cross_entropy(logits, tgt)
    grad, = torch.autograd.grad(loss, logits, g)
    xd, owned = x.double(), (tgt >= v0) & (tgt < v0 + cols)
    m = xd.max(1).values
    e = (xd - m[:, None]).exp()
    at = (tgt - v0).clamp(0, cols - 1)
    want = e.sum(1).log() - torch.where(owned, xd.gather(1, at[:, None])[:, 0] - m, torch.zeros_like(m))
    p = e / e.sum(1, keepdim=True)
    p[torch.arange(rows, device=DEV), at] -= owned.double()
    want_grad = p * g.double()[:, None]
    nan_rows = torch.zeros(rows, dtype=torch.bool, device=DEV)
    nan_rows[[7, 8, 11]] = True
    assert torch.equal(want.isnan(), nan_rows) and float(want[6]) == float("inf")
    torch.testing.assert_close(loss.double(), want, atol=2e-5, rtol=2e-5, equal_nan=True)
    rounding = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11           # 8 and 11 bits of significand
    bound = (rounding + 2.0 ** -15) * want_grad.abs() + 2.0 ** -24
    bound[torch.arange(rows, device=DEV), at] += 2.0 ** -16                  # p - 1 carries the whole error of p
    bad = ~((grad.double() - want_grad).abs() <= bound) & ~(grad.isnan() & want_grad.isnan())
    assert not bad.any(), (bad.nonzero()[:5].tolist(), grad[bad][:5], want_grad[bad][:5])


@pytest.mark.parametrize("s,b,hq,hkv,d,window,dtype", [(16384, 2, 4, 4, 128, None, torch.bfloat16), (16000, 3, 3, 3, 96, None, torch.float16),
                                                       (16384, 4, 8, 2, 128, 1000, torch.bfloat16)])
def test_attention_in_several_head_groups_equals_head_by_head(s, b, hq, hkv, d, window, dtype):
    """Operands that exceed the share of L2 a group of heads may take, so that the tiles of several groups (the last one part
    full; one key head a group with grouped queries) follow each other: the same bits as one key head at a time, forward and
    all gradients, and some rows against fp64 (a weighted mean of values, weights of 16 bits)."""
    from gpt_neox_b200.ops import attention as A
    torch.manual_seed(d)
    rep = hq // hkv
    fwd, dkv = (48 << 20) // (4 * s * d // rep), (48 << 20) // (4 * s * d * rep)
    assert fwd < b * hq and (b * hq) % fwd and dkv < b * hkv
    q = torch.randn(s, b, hq, d, device=DEV).to(dtype).requires_grad_()
    k, v = (torch.randn(s, b, hkv, d, device=DEV).to(dtype).requires_grad_() for _ in range(2))
    g = torch.randn(s, b, hq, d, device=DEV).to(dtype)
    out = A.flash_attention(q, k, v, True, None, window)
    grads = torch.autograd.grad(out, (q, k, v), g)
    for i in range(b):
        for h in range(hkv):
            hs = slice(h * rep, (h + 1) * rep)
            one = [t.detach()[:, i:i + 1, sl].contiguous().requires_grad_() for t, sl in ((q, hs), (k, slice(h, h + 1)), (v, slice(h, h + 1)))]
            o1 = A.flash_attention(*one, True, None, window)
            g1 = torch.autograd.grad(o1, one, g[:, i:i + 1, hs].contiguous())
            assert torch.equal(out[:, i:i + 1, hs], o1)
            for have, want, sl in zip(grads, g1, (hs, slice(h, h + 1), slice(h, h + 1))):
                assert torch.equal(have[:, i:i + 1, sl], want)
    rows = torch.tensor([0, 1, 127, 128, 4095, s // 2 + 3, s - 1], device=DEV)
    keys = torch.arange(s, device=DEV)
    banned = keys[None] > rows[:, None]
    if window is not None:
        banned |= keys[None] < rows[:, None] - window
    for i, h in ((0, 0), (b - 1, hq - 1)):
        sc = q[rows, i, h].double() @ k[:, i, h // rep].double().t() / math.sqrt(d)
        want = sc.masked_fill(banned, -float("inf")).softmax(-1) @ v[:, i, h // rep].double()
        _close(out[rows, i, h], want, 2e-2 if dtype == torch.bfloat16 else 4e-3, rtol=1e-2)
    assert native.read_status() == 0


def test_overlapped_kernels_read_what_the_launch_before_wrote():
    """A product whose second operand, and norms whose scale and bias, are results of the overlapped launch right before, many
    times over in recycled memory: the values of the same calls with a wait in between."""
    torch.manual_seed(0)
    cols, n = 1024, 256
    src = [torch.randn(n, cols, device=DEV).to(torch.bfloat16) for _ in range(40)]
    x, ones, zeros = (t.to(torch.bfloat16) for t in (torch.randn(3, cols, device=DEV), torch.ones(cols, device=DEV), torch.zeros(cols, device=DEV)))

    def step(s, wait):
        sync = torch.cuda.synchronize if wait else (lambda: None)
        w = OF.layer_norm(s, ones, zeros, 1e-5)
        sync()
        y = G.gemm(x, w)                                       # [3, n]
        sync()
        scale, bias = (G.gemm(s[i:i + 1, :], s) for i in (0, 1))         # [1, n] each
        sync()
        a = OF.layer_norm(y, scale.view(-1), bias.view(-1), 1e-5)
        b = OF.rms_norm(y, G.gemm(s[2:3, :], s).view(-1), None, 1e-5)
        return y, a, b
    with torch.no_grad():
        want = [step(s, True) for s in src]
        torch.cuda.synchronize()
        for _ in range(5):
            got = [step(s, False) for s in src]
            for p, q in zip(want, got):
                assert all(torch.equal(s, t) for s, t in zip(p, q))


@pytest.mark.parametrize("kind", ["ln", "rms"])
@pytest.mark.parametrize("rows,cols,dtype", [(9, 520, torch.bfloat16), (700, 1032, torch.bfloat16), (9, 3080, torch.float32),
                                             (650, 6152, torch.float16), (310, 8200, torch.bfloat16), (3, 9224, torch.bfloat16)])
def test_norm_backward_without_addend_matches_fp64(kind, rows, cols, dtype):
    """The backward forms without another gradient to add, through autograd: row results round once after fp32 sums, column sums are
    fp32 over ``rows`` terms and round to the parameter's type."""
    torch.manual_seed(rows + cols)
    x, g = (torch.randn(rows, cols, device=DEV).to(dtype) for _ in range(2))
    w, b = (1 + 0.1 * torch.randn(cols, device=DEV)).to(dtype), (0.1 * torch.randn(cols, device=DEV)).to(dtype)
    ours, exact = [[t.detach().clone().requires_grad_() for t in ts] for ts in ((x, w, b), (x.double(), w.double(), b.double()))]
    if kind == "ln":
        y, yr = OF.layer_norm(*ours, 1e-5), torch.nn.functional.layer_norm(exact[0], (cols,), exact[1], exact[2], 1e-5)
    else:
        y = OF.rms_norm(*ours, 1e-5)
        yr = exact[0] / (exact[0].pow(2).mean(-1, keepdim=True).sqrt() + 1e-5) * exact[1] + exact[2]
    got, want = torch.autograd.grad(y, ours, g), torch.autograd.grad(yr, exact, g.double())
    ulp = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -18}[dtype]
    _close(y, yr, ulp, rtol=ulp)
    _close(got[0], want[0], ulp, rtol=ulp)
    for a, e in zip(got[1:], want[1:]):
        _close(a, e, 1e-5 * math.sqrt(rows) + 1e-5, rtol=1e-5 + ulp)


@pytest.mark.parametrize("b,l,d", [(5, 2053, 520), (1, 40, 16), (2, 300, 1032)])
def test_causal_conv_long_and_short_runs(b, l, d):
    """Runs of 16 / 32 steps, where the machine is full with them, and of 4 / 8: outputs and all gradients against the library
    convolution in fp32.  Outputs round once; the weight gradient rounds once after b l fp32 products."""
    from gpt_neox_b200.ops import selective_scan as SS
    torch.manual_seed(l)
    leaves = [torch.randn(b, l, d, device=DEV).to(torch.bfloat16), (torch.randn(d, 4, device=DEV) * 0.5).to(torch.bfloat16),
              torch.randn(d, device=DEV).to(torch.bfloat16)]
    g = torch.randn(b, l, d, device=DEV).to(torch.bfloat16)
    ours, ref = [[t.to(ty).requires_grad_() for t in leaves] for ty in (torch.bfloat16, torch.float64)]
    y, yr = SS.causal_conv1d(*ours), SS.causal_conv1d(*ref)
    for a, e in zip([y, *torch.autograd.grad(y, ours, g)], [yr, *torch.autograd.grad(yr, ref, g.double())]):
        _close(a, e, 2e-4 + 2.0 ** -9 * e.abs().mean().item(), rtol=2.0 ** -8)


def test_loss_statistics_of_a_split_vocabulary():
    """Raw statistics of one rank's share, rebased on a larger maximum: the formula in fp64 (one rounding of each factor), rows whose
    own share is all -inf, targets of other ranks."""
    torch.manual_seed(0)
    rows, cols, v0 = 300, 1000, 2000
    x = (torch.randn(rows, cols, device=DEV) * 3).to(torch.float16)
    x[7] = -float("inf")
    tgt = torch.randint(0, 3 * cols, (rows,), device=DEV) + 1000
    local, stats = torch.empty(rows, device=DEV), torch.empty(rows, 2, device=DEV)
    L = native.lib()
    native.check(L.neox_ce_online_16(native.ptr(x), native.ptr(tgt), native.ptr(local), native.ptr(stats), rows, cols, v0, 2, 0, OF._s()), "online")
    raw, top = stats.clone(), torch.maximum(local, torch.randn(rows, device=DEV) * 20)
    native.check(L.neox_ce_rebase(native.ptr(tgt), native.ptr(local), native.ptr(top), native.ptr(stats), rows, cols, v0, OF._s()), "rebase")
    owned = (tgt >= v0) & (tgt < v0 + cols)
    assert 50 < int(owned.sum()) < 250
    picked = x.float()[torch.arange(rows, device=DEV), (tgt - v0).clamp(0, cols - 1)]
    assert torch.equal(raw[:, 1], torch.where(owned, picked, torch.zeros_like(picked)))
    _close(stats[:, 0], raw[:, 0].double() * (local - top).double().exp(), 0.0, rtol=2.0 ** -22)
    assert torch.equal(stats[:, 1], torch.where(owned, raw[:, 1] - top, torch.zeros_like(top)))
    assert float(stats[7, 0]) == 0.0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("s,b,hq,hk,d,rot", [(2049, 1, 5, 5, 64, 64), (9001, 2, 5, 2, 64, 64), (9001, 1, 3, 1, 96, 24), (33001, 1, 5, 2, 96, 24)])
def test_rope_in_place_vectors_of_one_and_four_heads(s, b, hq, hk, d, rot, dtype):
    """Sizes that take the vector forms (8 and 4 elements; one and four heads a thread, the last group part full): the bits of the
    element-wise form, which a slice of fewer tokens takes, and the rest of the projection untouched."""
    import ctypes
    torch.manual_seed(rot)
    packed = torch.randn(s, b, hq + 2 * hk, d, device=DEV).to(dtype)
    cos, sin = torch.randn(s, rot, device=DEV), torch.randn(s, rot, device=DEV)
    ll = ctypes.c_longlong

    def run(p, c, sn, inverse):
        q, k = p[:, :, :hq], p[:, :, hq:hq + hk]
        native.check(native.lib().neox_rope_qk_inplace(
            native.ptr(q), native.ptr(k), native.ptr(c), native.ptr(sn), p.shape[0], b, hq, hk, rot, ll(q.stride(0)),
            ll(q.stride(1)), ll(q.stride(2)), ll(k.stride(0)), ll(k.stride(1)), ll(k.stride(2)), inverse, OF._DT[dtype],
            OF._s()), "rope")
    for inverse in (0, 1):
        whole, parts = packed.clone(), packed.clone()
        run(whole, cos, sin, inverse)
        for i in range(0, s, 997):
            run(parts[i:i + 997], cos[i:i + 997], sin[i:i + 997], inverse)
        want = OF.rope_ref(packed[:, :, :hq + hk], cos.view(s, 1, 1, rot), (-sin if inverse else sin).view(s, 1, 1, rot))
        # one rounding after two products that may cancel
        _close(whole[:, :, :hq + hk], want, 2.0 ** -7, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
        assert ((whole != parts).float().mean().item()) < 1e-3          # the two forms may contract the products differently
        assert torch.equal(whole[:, :, hq + hk:], packed[:, :, hq + hk:])
        assert torch.equal(whole[..., rot:], packed[..., rot:])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,offset", [(700000, 0), (700003, 4), (700003, 1), (700001, 2)])
def test_adam_vectors_equal_single_elements(n, offset, dtype):
    """Shards large enough for four elements at a time, aligned and not, against the update in fp64 and nothing outside the shard."""
    import ctypes
    torch.manual_seed(n)
    full = n + offset + 8
    p, m, g = (torch.randn(full, device=DEV) for _ in range(3))
    v, out = torch.rand(full, device=DEV), torch.zeros(full, device=DEV, dtype=dtype)
    keep = [t.clone() for t in (p, m, v, out)]
    sl = slice(offset, offset + n)
    f = ctypes.c_float
    native.check(native.lib().neox_adam_step(
        native.ptr(p[sl]), native.ptr(m[sl]), native.ptr(v[sl]), native.ptr(g[sl]), native.ptr(out[sl]), OF._DT[dtype],
        ctypes.c_longlong(n), f(1e-2), f(0.9), f(0.95), f(1e-8), f(0.1), f(0.1), f(0.05), f(0.5), 1, OF._s()), "adam")
    P, M, V, Gr = (t[sl].double() for t in (*keep[:3], g))
    Gr = Gr * 0.5
    M, V = 0.9 * M + 0.1 * Gr, 0.95 * V + 0.05 * Gr * Gr
    P = P - (1e-2 / 0.1 * M / (V.sqrt() / 0.05 ** 0.5 + 1e-8) + 1e-2 * 0.1 * P)
    for have, want in ((p, P), (m, M), (v, V)):
        _close(have[sl], want, 1e-6, rtol=2e-6)
    assert torch.equal(out[sl], p[sl].to(dtype))
    for have, was in zip((p, m, v, out), keep):
        assert torch.equal(have[:offset], was[:offset]) and torch.equal(have[offset + n:], was[offset + n:])

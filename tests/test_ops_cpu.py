"""Operator-level checks that run on CPU (eager statements of the kernels' math)."""
import pytest
import torch




def test_fp8_linear_gelu_split_matches_plain_composition():
    """fc1 (GeLU, split pre-activation) -> fc2 (GeLU' folded into dgrad) in fp8 gives the gradients of the plain
    composition ``fc2(gelu(fc1(x)))`` evaluated on the same quantised operands' math (loose: fp8 rounding)."""
    import torch
    from gpt_neox_b200.ops import fp8 as F8
    torch.manual_seed(0)
    x = torch.randn(64, 32).bfloat16().requires_grad_(True)
    w1 = torch.nn.Parameter((torch.randn(48, 32) * 0.2).bfloat16())
    w2 = torch.nn.Parameter((torch.randn(32, 48) * 0.2).bfloat16())
    rec = F8.Fp8Recipe(hybrid=False)
    h, pre = F8.fp8_linear(x, w1, None, rec, act="gelu", split_pre=True)
    y = F8.fp8_linear(h, w2, None, rec, residual=x, dgelu_aux=pre)
    y.float().pow(2).sum().backward()
    got = [t.grad.float().clone() for t in (x, w1, w2)]
    for t in (x, w1, w2):
        t.grad = None
    yr = torch.nn.functional.gelu(x.float() @ w1.float().t(), approximate="tanh") @ w2.float().t() + x.float()
    yr.pow(2).sum().backward()
    assert ((y.float() - yr).norm() / yr.norm()).item() < 0.05
    for g, t in zip(got, (x, w1, w2)):
        assert ((g - t.grad.float()).norm() / t.grad.float().norm()).item() < 0.12


def test_fp8_delayed_scaling_history_and_weight_cache():
    import torch
    from gpt_neox_b200.ops import fp8 as F8
    m = F8.DelayedMeta(torch.device("cpu"), length=3, e5m2=False, margin=1, most_recent=False)
    m.update()
    assert float(m.buf[0]) == 1.0 and float(m.buf[1]) == 1.0            # nothing seen yet: scale 1
    x = torch.tensor([[0.5, -2.0], [1.0, 0.25]]).bfloat16()
    F8.cast(x, meta=m)
    assert float(m.buf[2]) == 2.0                                        # recorded amax
    m.update()
    assert abs(float(m.buf[0]) - 448.0 / (2.0 * 2.0)) < 1e-6             # fp8_max / (amax * 2^margin)
    F8.cast(x * 0.25, meta=m)
    m.update()
    assert abs(float(m.buf[0]) - 448.0 / (2.0 * 2.0)) < 1e-6             # 'max' over the history keeps the larger amax
    mr = F8.DelayedMeta(torch.device("cpu"), length=3, most_recent=True)
    mr.update(); F8.cast(x, meta=mr); mr.update(); F8.cast(x * 0.25, meta=mr); mr.update()
    assert abs(float(mr.buf[0]) - 448.0 / 0.5) < 1e-4                    # 'most_recent' follows the last amax

    w = torch.nn.Parameter(torch.randn(16, 16).bfloat16())
    rec = F8.Fp8Recipe()
    a = F8._cast_weight(w, rec)
    assert F8._cast_weight(w, rec) is a                                  # cached
    F8.invalidate_weight_cache()
    assert F8._cast_weight(w, rec) is not a                              # the engine's optimizer step invalidates
    with torch.no_grad():
        w.add_(1.0)                                                      # so does an in-place update autograd can see
    b = F8._cast_weight(w, rec)
    assert not torch.equal(b.q, a.q)


def test_pair_kernel_selection(monkeypatch):
    from gpt_neox_b200.ops import gemm as G
    monkeypatch.setattr(G, "_PAIR", "auto")
    assert G.use_pair_kernel(8192, 6144, 6144)                           # fills the machine with 256 x 256 tiles
    assert not G.use_pair_kernel(512, 512, 4096)                         # 4 tiles: one-CTA kernel
    assert not G.use_pair_kernel(8192, 6144, 128)                        # short K: nothing to pipeline
    monkeypatch.setattr(G, "_PAIR", "0")
    assert not G.use_pair_kernel(8192, 6144, 6144)
    monkeypatch.setattr(G, "_PAIR", "1")
    assert G.use_pair_kernel(64, 64, 64)


@pytest.mark.parametrize("kind,cfg", [
    ("local", {"block": 16, "num_sliding_window_blocks": 3}),
    ("sparse_fixed", {"block": 8, "num_local_blocks": 4, "num_global_blocks": 1}),
    ("sparse_variable", {"block": 16, "num_local_blocks": 2}),
    ("bigbird", {"block": 16, "num_sliding_window_blocks": 3, "num_global_blocks": 1, "num_random_blocks": 2}),
    ("bslongformer", {"block": 16, "num_sliding_window_blocks": 3, "global_block_indices": [0, 2]}),
])
def test_block_sparse_attention_matches_the_dense_masked_statement(kind, cfg):
    """Gathering only the kept tiles gives the same output and gradients as masking a dense score matrix."""
    from gpt_neox_b200.models.transformer import sparse_layout_mask
    from gpt_neox_b200.ops.sparse_attention import block_sparse_attention
    torch.manual_seed(0)
    s, b, h, hkv, d = 100, 2, 4, 2, 8                      # s is not a multiple of the block; grouped-query heads
    q = torch.randn(s, b, h, d, requires_grad=True)
    k = torch.randn(s, b, hkv, d, requires_grad=True)
    v = torch.randn(s, b, hkv, d, requires_grad=True)
    scale = d ** -0.5
    out = block_sparse_attention(q, k, v, kind, cfg, scale)
    g = torch.randn_like(out)
    out.backward(g)
    got = (out.detach(), q.grad.clone(), k.grad.clone(), v.grad.clone())
    for t in (q, k, v):
        t.grad = None
    mask = sparse_layout_mask(kind, s, s, cfg, q.device) | (torch.arange(s)[None, :] > torch.arange(s)[:, None])
    kf = k.repeat_interleave(h // hkv, dim=2)
    vf = v.repeat_interleave(h // hkv, dim=2)
    scores = torch.einsum("sbhd,tbhd->bhst", q, kf) * scale
    probs = torch.softmax(scores.masked_fill(mask[None, None], float("-inf")), dim=-1)
    ref = torch.einsum("bhst,tbhd->sbhd", probs, vf)
    ref.backward(g)
    for a, r in zip(got, (ref.detach(), q.grad, k.grad, v.grad)):
        torch.testing.assert_close(a, r, atol=2e-5, rtol=1e-4)


@pytest.mark.parametrize("adamw", [True, False])
def test_cpu_adam_host_kernel_matches_torch(adamw):
    """The OpenMP / AVX2 host kernel against torch's Adam / AdamW: host parameters are updated in place, the bf16
    copy is the rounded parameter, a gradient scale is folded in."""
    from gpt_neox_b200.optim.cpu_adam import CPUAdam
    torch.manual_seed(0)
    n = 1000 + 37
    p = torch.nn.Parameter(torch.randn(n))
    q = torch.nn.Parameter(p.detach().clone())
    p.model_out = torch.zeros(n, dtype=torch.bfloat16)
    kw = dict(lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    ours = CPUAdam([p], adamw_mode=adamw, **kw)
    ref = (torch.optim.AdamW if adamw else torch.optim.Adam)([q], **kw)
    ours.param_groups[0]["grad_scale"] = 0.5
    storage = p.data_ptr()
    for _ in range(5):
        g = torch.randn(n)
        p.grad, q.grad = g * 2.0, g.clone()               # the scale of 0.5 undoes the factor
        ours.step()
        ref.step()
    assert p.data_ptr() == storage and "host_param" not in ours.state[p]
    torch.testing.assert_close(p.detach(), q.detach(), atol=2e-6, rtol=1e-5)
    assert torch.equal(p.model_out, p.detach().bfloat16())


def test_plain_calls_leave_transforms_to_autograd():
    """Operators pass autograd.Function by only where nothing can tell the difference: gradients off, no functorch transform,
    no forward-mode level, plain tensors."""
    from torch.autograd import forward_ad
    from gpt_neox_b200.ops import native

    class Sub(torch.Tensor):
        pass
    x = torch.randn(3)
    assert not native.plain_call(x)
    seen = []
    with torch.no_grad():
        assert native.plain_call(x, None, torch.nn.Parameter(x))
        assert not native.plain_call(x, x.as_subclass(Sub))
        torch.func.vmap(lambda t: seen.append(native.plain_call(x)) or t)(x)
        with forward_ad.dual_level():
            seen.append(native.plain_call(x))
        torch.jit.trace(lambda t: (seen.append(native.plain_call(x)), t * 2)[1], (x,), check_trace=False)
    assert seen == [False] * len(seen) and len(seen) >= 3


def test_linear_without_gradients_equals_the_recorded_one():
    """The direct path of ``linear`` (no autograd node) gives the values of the recorded one, for every epilogue."""
    from gpt_neox_b200.ops.linear import linear
    torch.manual_seed(0)
    x, w, b, r = torch.randn(2, 5, 16), torch.randn(24, 16, requires_grad=True), torch.randn(24), torch.randn(2, 5, 24)
    for kw in ({}, {"bias": b}, {"bias": b, "act": "gelu"}, {"bias": b, "residual": r}, {"bias": b, "act": "gelu", "split_pre": True}):
        with_graph = linear(x, w, **kw)
        with torch.no_grad():
            without = linear(x, w, **kw)
        if kw.get("split_pre"):
            assert without[1] is None
            with_graph, without = with_graph[0], without[0]
        assert with_graph.requires_grad and not without.requires_grad and torch.equal(with_graph, without)


@pytest.fixture
def conv_routes(monkeypatch):
    """Lets CPU tensors take the routing of GPU tensors in ``causal_conv1d``: the returned list collects the calls that would
    have launched the kernel (whose result here is zeros)."""
    from gpt_neox_b200.ops import native, selective_scan as SS
    taken = []

    def kernel(xz, weight, bias, silu):
        taken.append(tuple(xz.shape))
        return torch.zeros(*xz.shape[:2], weight.shape[0], dtype=xz.dtype), xz[..., weight.shape[0]:]
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True), raising=False)
    monkeypatch.setattr(native, "available", lambda: True)
    monkeypatch.setattr(SS._CausalConv, "apply", kernel)
    return taken


@pytest.mark.parametrize("channels,bias,kernel", [
    (128, 128, True), (128, None, True), (64, 128, False), (256, 128, False), (136, 128, False), (128, 64, False),
    (128, 256, False), (128, "strided", False), (128, "matrix", False)])
def test_causal_conv_kernel_takes_only_matching_shapes(conv_routes, channels, bias, kernel):
    """The kernel reads ``weight.shape[0]`` channels of every row and as many bias elements, whatever the operands hold: a
    call with other counts is left to the library convolution, which refuses it (a strided bias it accepts)."""
    from gpt_neox_b200.ops.selective_scan import causal_conv1d
    x, w = torch.randn(2, 9, channels).bfloat16(), torch.randn(128, 4).bfloat16()
    if bias == "strided":
        b = torch.randn(256).bfloat16()[::2]
    elif bias == "matrix":
        b = torch.randn(1, 128).bfloat16()
    else:
        b = None if bias is None else torch.randn(bias).bfloat16()
    if kernel or bias == "strided":
        assert causal_conv1d(x, w, b).shape == (2, 9, 128)
    else:
        with pytest.raises(RuntimeError):
            causal_conv1d(x, w, b)
    assert bool(conv_routes) == kernel


@pytest.mark.parametrize("channels,kernel", [(256, True), (128, False), (264, False), (512, False)])
def test_causal_conv_split_kernel_takes_only_two_halves(conv_routes, channels, kernel):
    from gpt_neox_b200.ops.selective_scan import causal_conv1d_split
    xz, w = torch.randn(2, 9, channels).bfloat16(), torch.randn(128, 4).bfloat16()
    if kernel:
        x, z = causal_conv1d_split(xz, w, None)
        assert x.shape == z.shape == (2, 9, 128)
    else:
        with pytest.raises(RuntimeError):
            causal_conv1d_split(xz, w, None)
    assert bool(conv_routes) == kernel


def test_causal_conv_under_transforms_takes_the_library_path(conv_routes):
    """vmap, forward mode and tracing follow the library convolution; an autograd function around the kernel they do not."""
    from torch.autograd import forward_ad
    from gpt_neox_b200.ops.selective_scan import causal_conv1d
    x, w, b = torch.randn(3, 2, 9, 16).bfloat16(), torch.randn(16, 4).bfloat16(), torch.randn(16).bfloat16()
    got = torch.func.vmap(lambda t: causal_conv1d(t, w, b))(x)
    assert got.shape == x.shape and bool(got.abs().sum() > 0)
    with forward_ad.dual_level():
        out = causal_conv1d(forward_ad.make_dual(x[0], torch.ones_like(x[0])), w, b)
        assert forward_ad.unpack_dual(out).tangent is not None
    traced = torch.jit.trace(lambda t: causal_conv1d(t, w, b), (x[0],), check_trace=False)
    assert torch.equal(traced(x[1]), got[1])
    assert not conv_routes
    causal_conv1d(x[0], w, b)
    assert conv_routes


@pytest.mark.parametrize("halves", [1, 2])
def test_causal_conv_gradients_can_be_differentiated(monkeypatch, halves):
    """``create_graph=True``: second derivatives through the autograd function around the convolution kernel, whose launch is
    replaced by the library convolution in fp64 here, against finite differences."""
    from gpt_neox_b200.ops import native, selective_scan as SS

    class Lib:
        @staticmethod
        def neox_causal_conv_fwd(x, w, bias, out, strides, b, l, d, silu, *rest):
            y = torch.nn.functional.conv1d(x[..., :d].transpose(1, 2), w.unsqueeze(1), bias, padding=3, groups=d)[..., :l]
            out.copy_(torch.nn.functional.silu(y.transpose(1, 2)))
            return 0
    monkeypatch.setattr(native, "lib", lambda: Lib)
    monkeypatch.setattr(native, "ptr", lambda t: t)
    monkeypatch.setattr(native, "stream_ptr", lambda: 0)
    torch.manual_seed(0)
    xz, w, b = (torch.randn(*s, dtype=torch.float64, requires_grad=True) for s in ((2, 5, 3 * halves), (3, 4), (3,)))
    run = lambda *t: SS._CausalConv.apply(*t, True)[:halves]
    assert torch.autograd.gradgradcheck(run, (xz, w, b))
    assert torch.autograd.gradgradcheck(lambda t: SS._CausalConv.apply(t, w.detach(), None, True)[:halves], (xz,))


def test_aligned_rows_moves_a_contiguous_gradient_off_its_odd_start():
    """A gradient may be any view: contiguous, but starting between two 16-byte boundaries."""
    from gpt_neox_b200.ops.selective_scan import _aligned_rows
    flat = torch.randn(2 * 5 * 16 + 24).bfloat16()
    shift = (-flat.data_ptr() // 2) % 8                          # elements up to the first boundary
    for off in range(8):
        t = flat[shift + off: shift + off + 160].view(2, 5, 16)
        got = _aligned_rows(t)
        assert torch.equal(got, t) and got.data_ptr() % 16 == 0 and got.stride() == (80, 16, 1)
        assert (got is t) == (off == 0)


@pytest.mark.parametrize("shape,stride", [((2, 4, 8), (40, 1, 1)), ((2, 8, 4), (40, 2, 1)), ((3, 6, 8), (16, 48, 1)),
                                          ((3, 6, 8), (0, 0, 1)), ((1, 6, 8), (96, 16, 1)), ((3, 6, 1), (1, 3, 1))])
def test_scan_results_have_contiguous_channels(shape, stride):
    """The scan kernels write the last dimension with unit stride, also for an input of overlapping windows, whose dense copy
    puts time innermost."""
    from gpt_neox_b200.ops.selective_scan import _like_rows
    new = _like_rows(torch.zeros(400).as_strided(shape, stride))
    assert new.shape == shape and (new.stride(2) == 1 or shape[2] == 1)
    assert new.is_contiguous() or new.transpose(0, 1).is_contiguous()


def _run_cpp(tmp_path, source, cuda_headers=False):
    """Compile ``source`` against the kernels' headers with the host compiler alone and run it; returns what it prints."""
    import shutil
    import subprocess
    from pathlib import Path
    import gpt_neox_b200.ops
    include = ["-I", str(Path(gpt_neox_b200.ops.__file__).parent / "csrc")]
    if cuda_headers:
        home = Path("/usr/local/cuda/include")
        if not (home / "cuda_runtime.h").exists():
            pytest.skip("no CUDA headers")
        include += ["-I", str(home)]
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", *include, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout


def test_dynamic_shared_memory_is_allowed_on_every_device(tmp_path):
    """The permission for large dynamic shared memory belongs to a device: asked for once per kernel and device, again after a
    failure, and on every device a process uses.  The runtime calls are stand-ins."""
    out = _run_cpp(tmp_path, r"""
#include "dynamic_smem.h"
#include <cstdio>
static int dev = 0, calls = 0;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { ++calls; return answer; }
static void first(int) {}
static void second(int) {}
int main() {
    auto show = [](bool ok) { std::printf("%d/%d ", (int)ok, calls); };
    answer = cudaErrorInvalidValue; show(allow_dynamic_smem<first>(70000));
    answer = cudaSuccess;
    show(allow_dynamic_smem<first>(70000)); show(allow_dynamic_smem<first>(70000));
    show(allow_dynamic_smem<second>(70000));
    dev = 1; show(allow_dynamic_smem<first>(70000)); show(allow_dynamic_smem<first>(70000));
    dev = 70; show(allow_dynamic_smem<first>(70000)); show(allow_dynamic_smem<first>(70000));
    dev = 0; show(allow_dynamic_smem<first>(70000));
}""", cuda_headers=True)
    assert out.split() == ["0/1", "1/2", "1/2", "1/3", "1/4", "1/4", "1/5", "1/6", "1/6"]


def test_kernels_that_start_early_use_no_read_only_loads():
    """A kernel that waits for the launch in front lives through that one's writes, so none of its loads may assume constant data:
    no read-only load instruction, and no ``const __restrict__`` parameter, of which the compiler makes such loads."""
    import re
    from pathlib import Path
    import gpt_neox_b200.ops
    seen = 0
    for path in sorted((Path(gpt_neox_b200.ops.__file__).parent / "csrc").glob("*.cu")):
        text = path.read_text()
        kernels = [k for k in re.split(r"(?=\n(?:static )?__global__ )", text)[1:] if "wait_for_predecessor()" in k.split("\n}\n")[0]]
        for k in kernels:
            body = k.split("\n}\n")[0]
            assert not re.search(r"const\s+\w+\s*\*\s*__restrict__|__ldg\(", body), (path.name, body[:200])
        if kernels:
            assert "ld.global.nc" not in text, path.name
        seen += len(kernels)
    assert seen >= 4


@pytest.mark.parametrize("M,N,K,few_rows", [
    (1, 50432, 6144, True), (8, 50432, 6144, True), (9, 12288, 4096, True), (9, 50432, 6144, False), (12, 32000, 4096, True),
    (12, 24576, 6144, False), (16, 50304, 2048, True), (16, 18432, 6144, False), (16, 6144, 24576, True), (17, 8192, 2048, True),
    (17, 12288, 4096, False), (32, 2048, 8192, True), (32, 50304, 1024, False), (33, 2048, 2048, False), (4, 2048, 2044, False)])
def test_few_row_products_take_the_faster_kernel(M, N, K, few_rows, monkeypatch):
    """Which products of few rows stream the weights: as measured on either side of the lines (8, 16 and 32 rows, 8192 columns, the
    size of a product of 9 to 16 rows)."""
    from gpt_neox_b200.ops import gemm as G
    monkeypatch.setattr(G, "_PAIR", "auto")
    assert G.use_skinny_kernel(M, N, K, False, False) == few_rows
    assert not G.use_skinny_kernel(M, N, K, True, False) and not G.use_skinny_kernel(M, N, K, False, True)


def test_attention_tile_order_starts_every_tile_once(tmp_path):
    """The order of the attention tiles: every (tile, head) exactly once, heads in groups of consecutive ones whose operands fit
    48 MB together, heaviest tile of all heads of a group first, the last group part full."""
    out = _run_cpp(tmp_path, r"""
#include <algorithm>
#include <cstdio>
using std::min;
#define __device__
#define __forceinline__ inline
static struct { unsigned x, y; } blockIdx;
#include "flash_order.cuh"
int main() {
    const int tiles[] = {1, 3, 16, 64}, heads[] = {1, 2, 8, 17, 256};
    const long long bytes[] = {0, 1000, 786432, 16ll << 20, 17ll << 20, 1ll << 40};
    for (int t : tiles) for (int h : heads) for (long long b : bytes) {
        const TileOrder o = tile_order(t, h, b);
        std::printf("%d %d %lld %d", t, h, b, o.group);
        unsigned gx, gy;
        if (!tile_grid(o, gx, gy)) return 1;
        for (blockIdx.y = 0; blockIdx.y < gy; ++blockIdx.y) for (blockIdx.x = 0; blockIdx.x < gx; ++blockIdx.x) {
            int rank, head;
            pick_tile(o, rank, head);
            std::printf(" %d,%d", rank, head);
        }
        std::printf("\n");
    }
}""")
    lines = out.strip().split("\n")
    assert len(lines) == 4 * 5 * 6
    several = 0
    for line in lines:
        t, h, b, group, *order = line.split()
        t, h, b, group = int(t), int(h), int(b), int(group)
        assert group == max(1, min(h, (48 << 20) // max(b, 1)))
        want = [f"{rank},{head}" for g in range(0, h, group) for rank in range(t) for head in range(g, min(g + group, h))]
        assert order == want
        several += group < h and h % group != 0
    assert several > 0

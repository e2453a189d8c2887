// Depth-wise causal convolution over time of width 4 with bias and SiLU, channel-last, forward and backward:
//     pre[t] = bias + sum_k w[k] * x[t - 3 + k],      out[t] = silu(pre[t]) or pre[t]
//
// A thread walks a run of time steps of 8 (forward) or 4 (backward) neighbouring channels with the last three inputs in
// registers, so every input is read once apart from the three steps in front of a run (backward also three behind it); any
// batch and time strides are taken, which lets the operands be slices of a wider projection.  The library convolution it
// replaces wanted [b, d, l] (a transposing copy each way), ran SiLU and the bias as passes of their own and took 168 us
// forward, 220 us backward at b 4, l 2048, d 1536, with about 400 us of copies around them; these kernels take 23 and 62 us
// there.  Their bytes (x in, out out; backward x and the gradient in, the gradient of x out) would take 7.7 and 11.5: what
// bounds them is the latency of a run's loads, with 20 % of an SM's warps resident at 112 and 96 registers a thread and
// most of them waiting for memory.  The weight gradient is summed in registers and shared memory and leaves as one partial sum
// per block, so results are bitwise repeatable.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "neox_b200.h"

namespace {

constexpr int W = 4;             // taps
constexpr int TX = 32, TY = 8;   // channel groups x runs per block
constexpr int FC = 8, FT = 16, FT_SHORT = 4;   // forward: channels and steps of a thread
constexpr int BC = 4, BT = 32, BT_SHORT = 8;   // backward

template <typename T> __device__ __forceinline__ float2 to_f2(uint32_t w);
template <> __device__ __forceinline__ float2 to_f2<__nv_bfloat16>(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
template <> __device__ __forceinline__ float2 to_f2<__half>(uint32_t w) { return __half22float2(*reinterpret_cast<__half2*>(&w)); }
template <typename T> __device__ __forceinline__ uint32_t from_f2(float a, float b);
template <> __device__ __forceinline__ uint32_t from_f2<__nv_bfloat16>(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t from_f2<__half>(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
template <typename T, int N>
__device__ __forceinline__ void load(const T* p, float (&f)[N]) {
    uint32_t w[N / 2];
    if constexpr (N == 8) *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(p);
    else *reinterpret_cast<uint2*>(w) = *reinterpret_cast<const uint2*>(p);
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const float2 v = to_f2<T>(w[i]);
        f[2 * i] = v.x;
        f[2 * i + 1] = v.y;
    }
}
template <typename T, int N>
__device__ __forceinline__ void store(T* p, const float (&f)[N]) {
    uint32_t w[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) w[i] = from_f2<T>(f[2 * i], f[2 * i + 1]);
    if constexpr (N == 8) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<uint4*>(w);
    else *reinterpret_cast<uint2*>(p) = *reinterpret_cast<uint2*>(w);
}
template <int N>
__device__ __forceinline__ void zero(float (&f)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = 0.f;
}
// taps and bias of N neighbouring channels
template <typename T, int N>
__device__ __forceinline__ void taps(const T* w, const T* bias, int c, float (&tw)[W][N], float (&tb)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
#pragma unroll
        for (int k = 0; k < W; ++k) tw[k][i] = (float)w[(c + i) * W + k];
        tb[i] = bias ? (float)bias[c + i] : 0.f;
    }
}

template <typename T, int FT>
__global__ void __launch_bounds__(TX * TY)
conv_fwd_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias, T* __restrict__ out, int l,
                int d, int cblk, long long xb, long long xt, long long ob, long long ot, int silu) {
    const int c = (blockIdx.x % cblk * TX + threadIdx.x) * FC, t0 = (blockIdx.x / cblk * TY + threadIdx.y) * FT;
    if (c >= d || t0 >= l) return;
    x += blockIdx.y * xb + c;
    out += blockIdx.y * ob + c;
    float tw[W][FC], tb[FC], win[W - 1][FC];
    taps<T, FC>(w, bias, c, tw, tb);
#pragma unroll
    for (int k = 0; k < W - 1; ++k) {
        const int t = t0 - (W - 1) + k;
        if (t >= 0) load<T, FC>(x + t * xt, win[k]);
        else zero(win[k]);
    }
#pragma unroll 4
    for (int t = t0; t < min(t0 + FT, l); ++t) {
        float cur[FC], o[FC];
        load<T, FC>(x + t * xt, cur);
#pragma unroll
        for (int i = 0; i < FC; ++i) {
            const float pre = tb[i] + tw[0][i] * win[0][i] + tw[1][i] * win[1][i] + tw[2][i] * win[2][i] + tw[3][i] * cur[i];
            o[i] = silu ? pre / (1.f + __expf(-pre)) : pre;
            win[0][i] = win[1][i];
            win[1][i] = win[2][i];
            win[2][i] = cur[i];
        }
        store<T, FC>(out + t * ot, o);
    }
}

// part: [blocks along batch and time][d][W + 1] partial sums of the tap and bias gradients
template <typename T, int BT>
__global__ void __launch_bounds__(TX * TY)
conv_bwd_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias, const T* __restrict__ g,
                T* __restrict__ gx, float* __restrict__ part, int l, int d, int cblk, long long xb, long long xt,
                long long gb, long long gt, long long db, long long dt, int silu) {
    __shared__ float red[TY][BC * (W + 1)][TX];
    const int c = (blockIdx.x % cblk * TX + threadIdx.x) * BC, tblk = blockIdx.x / cblk;
    const int t0 = (tblk * TY + threadIdx.y) * BT;
    float gw[W][BC], gbias[BC];
#pragma unroll
    for (int k = 0; k < W; ++k) zero(gw[k]);
    zero(gbias);
    if (c < d && t0 < l) {
        x += blockIdx.y * xb + c;
        g += blockIdx.y * gb + c;
        gx += blockIdx.y * db + c;
        float tw[W][BC], tb[BC], win[W - 1][BC], acc[W - 1][BC];        // acc[k]: gradient of x[t - 3 + k] so far
        taps<T, BC>(w, bias, c, tw, tb);
#pragma unroll
        for (int k = 0; k < W - 1; ++k) {
            const int t = t0 - (W - 1) + k;
            if (t >= 0) load<T, BC>(x + t * xt, win[k]);
            else zero(win[k]);
            zero(acc[k]);
        }
        // the run's own steps, and three more for what they send back into it
#pragma unroll 4
        for (int s = 0; s < BT + W - 1; ++s) {
            const int t = t0 + s;
            float gp[BC], cur[BC];
            zero(gp);
            zero(cur);
            if (t < l) {
                load<T, BC>(x + t * xt, cur);
                load<T, BC>(g + t * gt, gp);
                if (silu) {
#pragma unroll
                    for (int i = 0; i < BC; ++i) {
                        const float pre =
                            tb[i] + tw[0][i] * win[0][i] + tw[1][i] * win[1][i] + tw[2][i] * win[2][i] + tw[3][i] * cur[i];
                        const float sg = 1.f / (1.f + __expf(-pre));
                        gp[i] *= sg * (1.f + pre * (1.f - sg));
                    }
                }
            }
            float done[BC];
#pragma unroll
            for (int i = 0; i < BC; ++i) {
                if (s < BT) {
                    gw[0][i] += gp[i] * win[0][i];
                    gw[1][i] += gp[i] * win[1][i];
                    gw[2][i] += gp[i] * win[2][i];
                    gw[3][i] += gp[i] * cur[i];
                    gbias[i] += gp[i];
                }
                done[i] = acc[0][i] + tw[0][i] * gp[i];
                acc[0][i] = acc[1][i] + tw[1][i] * gp[i];
                acc[1][i] = acc[2][i] + tw[2][i] * gp[i];
                acc[2][i] = tw[3][i] * gp[i];
                win[0][i] = win[1][i];
                win[1][i] = win[2][i];
                win[2][i] = cur[i];
            }
            if (s >= W - 1 && t - (W - 1) < l) store<T, BC>(gx + (t - (W - 1)) * dt, done);
        }
    }
#pragma unroll
    for (int i = 0; i < BC; ++i) {
#pragma unroll
        for (int k = 0; k < W; ++k) red[threadIdx.y][i * (W + 1) + k][threadIdx.x] = gw[k][i];
        red[threadIdx.y][i * (W + 1) + W][threadIdx.x] = gbias[i];
    }
    __syncthreads();
    const int tblocks = gridDim.x / cblk;
    float* dst = part + ((long long)blockIdx.y * tblocks + tblk) * d * (W + 1);
    for (int e = threadIdx.y; e < BC * (W + 1); e += TY) {
        float v = 0.f;
#pragma unroll
        for (int y = 0; y < TY; ++y) v += red[y][e][threadIdx.x];
        if (c < d) dst[(long long)c * (W + 1) + e] = v;
    }
}

bool aligned(const void* p, int bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

}  // namespace

// Steps of a thread.  A run re-reads the three inputs in front of it (backward also the three steps behind it), so runs are long
// where the machine has a block for every SM all the same, and short where a run's serial chain is all there is: forward
// at b 1, l 128, d 512 10.8 us with the long runs and 6.8 with the short ones, both passes 29.5 and 18.7.
static int run_length(int b, int l, int d, int channels, int run, int short_run) {
    const long long blocks = (long long)b * ((d / channels + TX - 1) / TX) * ((l + run * TY - 1) / (run * TY));
    return blocks < neox_sm_count() ? short_run : run;
}
static int time_blocks(int l, int run) { return (l + run * TY - 1) / (run * TY); }

extern "C" int neox_causal_conv_blocks(int b, int l, int d) { return b * time_blocks(l, run_length(b, l, d, BC, BT, BT_SHORT)); }

// strides: element strides (batch, time) of x and out; d and the strides multiples of 8.  w: [d][4].  bias may be NULL.
extern "C" int neox_causal_conv_fwd(const void* x, const void* w, const void* bias, void* out, const long long* strides, int b,
                                    int l, int d, int silu, int h16, void* stream) {
    if (b <= 0 || l <= 0 || d <= 0) return 0;
    if (d % 8 || b > 65535) return NEOX_ERR_SHAPE;
    for (int i = 0; i < 4; ++i)
        if (strides[i] % 8) return NEOX_ERR_ALIGN;
    if (!aligned(x, 16) || !aligned(out, 16)) return NEOX_ERR_ALIGN;
    const int run = run_length(b, l, d, FC, FT, FT_SHORT), cblk = (d / FC + TX - 1) / TX, tblk = time_blocks(l, run);
    dim3 grid(cblk * tblk, b), block(TX, TY);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define CONV_FWD(T, RUN)                                                                                                      \
    conv_fwd_kernel<T, RUN><<<grid, block, 0, s>>>((const T*)x, (const T*)w, (const T*)bias, (T*)out, l, d, cblk, strides[0], \
                                                   strides[1], strides[2], strides[3], silu)
    if (run == FT) {
        if (h16) CONV_FWD(__half, FT);
        else CONV_FWD(__nv_bfloat16, FT);
    } else {
        if (h16) CONV_FWD(__half, FT_SHORT);
        else CONV_FWD(__nv_bfloat16, FT_SHORT);
    }
#undef CONV_FWD
    return cudaGetLastError() == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
}

// strides: of x, g (gradient of out) and gx.  part: neox_causal_conv_blocks(b, l, d) x d x 5 floats (4 taps, bias).
extern "C" int neox_causal_conv_bwd(const void* x, const void* w, const void* bias, const void* g, void* gx, float* part,
                                    const long long* strides, int b, int l, int d, int silu, int h16, void* stream) {
    if (b <= 0 || l <= 0 || d <= 0) return 0;
    if (d % 8 || b > 65535) return NEOX_ERR_SHAPE;
    for (int i = 0; i < 6; ++i)
        if (strides[i] % 8) return NEOX_ERR_ALIGN;
    if (!aligned(x, 8) || !aligned(g, 8) || !aligned(gx, 8)) return NEOX_ERR_ALIGN;
    const int run = run_length(b, l, d, BC, BT, BT_SHORT), cblk = (d / BC + TX - 1) / TX, tblk = time_blocks(l, run);
    dim3 grid(cblk * tblk, b), block(TX, TY);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define CONV_BWD(T, RUN)                                                                                                       \
    conv_bwd_kernel<T, RUN><<<grid, block, 0, s>>>((const T*)x, (const T*)w, (const T*)bias, (const T*)g, (T*)gx, part, l, d,  \
                                                   cblk, strides[0], strides[1], strides[2], strides[3], strides[4], strides[5], \
                                                   silu)
    if (run == BT) {
        if (h16) CONV_BWD(__half, BT);
        else CONV_BWD(__nv_bfloat16, BT);
    } else {
        if (h16) CONV_BWD(__half, BT_SHORT);
        else CONV_BWD(__nv_bfloat16, BT_SHORT);
    }
#undef CONV_BWD
    return cudaGetLastError() == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
}

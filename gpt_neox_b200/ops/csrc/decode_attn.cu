// Attention of one new token per sequence against its key / value cache (a decoding step): rotary embedding of the new
// query and key, append of the new key and value to the cache, softmax over everything cached, in one launch.
//
// Bound: the cache rows, read once (2 n d 2 bytes per sequence and head); at the cache lengths of ordinary requests the
// launch itself.  The path it replaces took 5 launches per layer with the growing cache (two rotary, two copies, the
// flash kernel, whose 128-row query tile held one row) and 13 with the fixed-capacity one (index_select, index_copy,
// einsum over the whole capacity, mask, softmax, einsum).  Per layer, 16 heads of 128 and batch 4 over 520 to 580 tokens of a
// 2048-token cache: 50 us before, 9.0 us here.  Growing cache, batch 8 x 16 x 128 over 100 tokens: 19 us before, 5.6 us here.
//
// A cluster of CTAs owns one (sequence, query head); its warps take the cached keys in turn.  A key is read by 8 or 16
// neighbouring lanes, 16 bytes each, so every load instruction covers whole rows; four keys and four values per lane are
// in flight at a time.  Each lane group keeps its own running maximum, sum and fp32 accumulator; they meet in shared
// memory in a fixed order (across the cluster through distributed shared memory), so results are bitwise repeatable.
// The number of cached rows may come from the device (`pos`), so the same launch can be replayed from a CUDA graph.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "launch.cuh"
#include "neox_b200.h"

namespace {

namespace cg = cooperative_groups;

constexpr int DA_WARPS = 8;
constexpr int DA_THREADS = DA_WARPS * 32;
constexpr int DA_KEYS = 4;          // keys of one lane group in flight
constexpr float LOG2E = 1.4426950408889634f;

struct DecodeParams {
    const void *q, *k, *v;          // [b, heads, d], any batch and head strides
    void* out;                      // [b, heads_q, d] contiguous
    void *kc, *vc;                  // cache: [capacity, b, heads_kv, d] each, contiguous
    const float *cos_t, *sin_t;     // [rows, rot] (rot = 0: no rotary embedding)
    const long long* pos;           // rows already cached, on the device; nullptr: n
    const float* slopes;            // ALiBi, or nullptr
    long long qb, qh, kb, kh, vb, vh;
    int n, cap, b, hq, hkv, rot, window;
    float scale;
};

template <bool H16>
__device__ __forceinline__ float ld16(const void* p, long long i) {
    if constexpr (H16) return __half2float(static_cast<const __half*>(p)[i]);
    else return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
template <bool H16>
__device__ __forceinline__ float round16(float x) {
    if constexpr (H16) return __half2float(__float2half(x));
    else return __bfloat162float(__float2bfloat16(x));
}
template <bool H16>
__device__ __forceinline__ void st16(void* p, long long i, float x) {
    if constexpr (H16) static_cast<__half*>(p)[i] = __float2half(x);
    else static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16(x);
}
template <bool H16>
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (H16) {
            const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            f[2 * i] = t.x;
            f[2 * i + 1] = t.y;
        } else {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
}

// Element i of a head after the rotary embedding of row `row`, rounded to 16 bits as the cache holds it.
template <bool H16>
__device__ __forceinline__ float rotated(const void* x, long long base, int i, const DecodeParams& p, int row) {
    const float xi = ld16<H16>(x, base + i);
    if (i >= p.rot) return xi;
    const int half = p.rot / 2;
    const float other = i < half ? -ld16<H16>(x, base + i + half) : ld16<H16>(x, base + i - half);
    return round16<H16>(xi * p.cos_t[(long long)row * p.rot + i] + other * p.sin_t[(long long)row * p.rot + i]);
}

template <int D, bool H16>
__global__ void __launch_bounds__(DA_THREADS) decode_attn_kernel(const DecodeParams p) {
    constexpr int G = D == 64 ? 8 : 16;           // lanes per key
    constexpr int KPW = 32 / G;                   // keys per warp and load
    constexpr int NG = DA_WARPS * KPW;            // lane groups per CTA
    __shared__ float sq[D], skn[D], svn[D];
    __shared__ float acc_s[NG][D], m_s[NG + 1], l_s[NG];
    __shared__ float o_c[D], ml_c[2];
    cg::cluster_group cluster = cg::this_cluster();
    const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
    const int h = blockIdx.y, bi = blockIdx.z, rep = p.hq / p.hkv, hk = h / rep;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    launch::let_successor_start();
    launch::wait_for_predecessor();
    // the host keeps the position inside the cache; the clamp only bounds what a wrong one could touch
    const int n = p.pos ? (int)min(max(*p.pos, 0ll), (long long)p.cap - 1) : p.n;
    const float cs = p.scale * LOG2E;

    if (tid < D) {
        sq[tid] = rotated<H16>(p.q, bi * p.qb + h * p.qh, tid, p, n);
    } else if (tid >= 128 && tid < 128 + D) {
        const int i = tid - 128;
        const float kn = rotated<H16>(p.k, bi * p.kb + hk * p.kh, i, p, n), vn = ld16<H16>(p.v, bi * p.vb + hk * p.vh + i);
        skn[i] = kn;
        svn[i] = vn;
        if (crank == 0 && h % rep == 0) {         // read by later launches only: this one takes the row from skn / svn
            const long long o = (((long long)n * p.b + bi) * p.hkv + hk) * D + i;
            st16<H16>(p.kc, o, kn);
            st16<H16>(p.vc, o, vn);
        }
    }
    __syncthreads();

    const int sub = lane % G, grp = lane / G;
    const bool act = sub * 8 < D;
    const float slope = p.slopes ? p.slopes[h] * LOG2E : 0.f;
    float qr[8], acc[8], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        qr[i] = act ? sq[sub * 8 + i] : 0.f;
        acc[i] = 0.f;
    }
    const long long row = (long long)p.b * p.hkv * D;
    const long long head = ((long long)bi * p.hkv + hk) * D + sub * 8;
    const char* kc = static_cast<const char*>(p.kc) + head * 2;
    const char* vc = static_cast<const char*>(p.vc) + head * 2;
    const int first = p.window >= 0 ? max(0, n - p.window) : 0;
    const int stride = csize * NG;
    for (int j0 = first + (crank * DA_WARPS + warp) * KPW; j0 < n; j0 += stride * DA_KEYS) {
        uint4 kr[DA_KEYS], vr[DA_KEYS];
#pragma unroll
        for (int u = 0; u < DA_KEYS; ++u) {
            const int j = j0 + grp + u * stride;
            const bool in = act && j < n;
            kr[u] = in ? *reinterpret_cast<const uint4*>(kc + j * row * 2) : make_uint4(0, 0, 0, 0);
            vr[u] = in ? *reinterpret_cast<const uint4*>(vc + j * row * 2) : make_uint4(0, 0, 0, 0);
        }
        float s[DA_KEYS], top = m;
#pragma unroll
        for (int u = 0; u < DA_KEYS; ++u) {
            const int j = j0 + grp + u * stride;
            float f[8], d = 0.f;
            unpack8<H16>(kr[u], f);
#pragma unroll
            for (int i = 0; i < 8; ++i) d += qr[i] * f[i];
#pragma unroll
            for (int off = G / 2; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
            s[u] = j < n ? d * cs - slope * (float)(n - j) : -INFINITY;
            top = fmaxf(top, s[u]);
        }
        const float base = top == -INFINITY ? 0.f : top;          // nothing seen yet: every weight is 0
        const float keep = exp2f(m - base);
        m = top;
        l *= keep;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] *= keep;
#pragma unroll
        for (int u = 0; u < DA_KEYS; ++u) {
            const float w = exp2f(s[u] - base);
            float f[8];
            unpack8<H16>(vr[u], f);
            l += w;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] += w * f[i];
        }
    }
    const int gi = warp * KPW + grp;
    if (act) {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc_s[gi][sub * 8 + i] = acc[i];
    }
    if (sub == 0) {
        m_s[gi] = m;
        l_s[gi] = l;
    }
    if (warp == 0) {                                    // the new token's own score
        float d = 0.f;
        for (int i = lane; i < D; i += 32) d += sq[i] * skn[i];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
        if (lane == 0) m_s[NG] = crank == 0 ? d * cs : -INFINITY;
    }
    __syncthreads();
    if (tid < D) {
        float top = m_s[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) top = fmaxf(top, m_s[g]);
        const float base = top == -INFINITY ? 0.f : top;
        const float wn = exp2f(m_s[NG] - base);
        float o = crank == 0 ? wn * svn[tid] : 0.f, ls = crank == 0 ? wn : 0.f;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const float w = exp2f(m_s[g] - base);
            o += w * acc_s[g][tid];
            ls += w * l_s[g];
        }
        o_c[tid] = o;
        if (tid == 0) {
            ml_c[0] = top;
            ml_c[1] = ls;
        }
        if (csize == 1) st16<H16>(p.out, ((long long)bi * p.hq + h) * D + tid, o / ls);
    }
    if (csize > 1) {
        cluster.sync();
        if (crank == 0 && tid < D) {
            float top = -INFINITY;
            for (int c = 0; c < csize; ++c) top = fmaxf(top, *cluster.map_shared_rank(&ml_c[0], c));
            const float base = top == -INFINITY ? 0.f : top;
            float o = 0.f, ls = 0.f;
            for (int c = 0; c < csize; ++c) {
                const float w = exp2f(*cluster.map_shared_rank(&ml_c[0], c) - base);
                o += w * *cluster.map_shared_rank(&o_c[tid], c);
                ls += w * *cluster.map_shared_rank(&ml_c[1], c);
            }
            st16<H16>(p.out, ((long long)bi * p.hq + h) * D + tid, o / ls);
        }
        cluster.sync();
    }
}

}  // namespace

// strides: element strides (batch, head) of q, k, v.  n: rows cached so far (the new row's index), or with `pos` an upper
// bound of it.  kc / vc rows must be 16-byte aligned (d = 64, 96 or 128 and an aligned base).
extern "C" int neox_decode_attn(const void* q, const void* k, const void* v, void* out, void* kc, void* vc, const float* cos_t,
                                const float* sin_t, const long long* pos, const float* slopes, const long long* strides,
                                int n, int cap, int b, int hq, int hkv, int d, int rot, int window, float scale, int h16,
                                void* stream) {
    if (b <= 0 || hq <= 0) return 0;
    if (hkv <= 0 || hq % hkv || b > 65535 || hq > 65535 || n < 0 || n >= cap || rot < 0 || rot > d || rot % 2) return NEOX_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(kc) & 15) || (reinterpret_cast<uintptr_t>(vc) & 15)) return NEOX_ERR_ALIGN;
    DecodeParams p{q, k, v, out, kc, vc, cos_t, sin_t, pos, slopes, strides[0], strides[1], strides[2], strides[3],
                   strides[4], strides[5], n, cap, b, hq, hkv, rot, window, scale};
    // More CTAs per head while there is not one for every SM and each still has a full turn of its lane groups (128 keys).
    const int keys = window >= 0 && window < n ? window : n;
    int csize = 1;
    while (csize < 8 && (long long)b * hq * csize < neox_sm_count() && keys > 128 * csize) csize *= 2;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define DA_CASE(D_)  \
    case D_:         \
        return launch::overlapped(h16 ? decode_attn_kernel<D_, true> : decode_attn_kernel<D_, false>, dim3(csize, hq, b), \
                                  dim3(DA_THREADS), csize, s, p);
    switch (d) {
        DA_CASE(64)
        DA_CASE(96)
        DA_CASE(128)
        default: return NEOX_ERR_SHAPE;
    }
#undef DA_CASE
}

// RWKV-6 "wkv" linear-attention recurrence, forward and backward.
//
// Per (batch, head) with head size N, time t, key channel j, value channel i:
//     y_t[i]     = sum_j r_t[j] * ( u[j] * k_t[j] * v_t[i] + S_t[j][i] )
//     S_{t+1}[j][i] = S_t[j][i] * d_t[j] + k_t[j] * v_t[i],          d_t = exp(ew_t),  ew_t = -exp(w_t)
//
// Backward is organised as three independent single-direction scans, none of which needs stored states:
//   A (forward in time, thread = key channel j, registers hold S[j][.]):   gr, the partial sums for gu, and
//     grS_t[j] = sum_i S_t[j][i] gy_t[i];
//   B (reverse, thread = j, registers hold G[j][.] with G_{t-1} = d_t G_t + r_t gy_t^T):   gk and
//     gkG_t[j] = sum_i v_t[i] G_t[j][i];
//   C (reverse, thread = value channel i, registers hold G[.][i]):   gv.
// The decay gradient then follows from a scalar identity, d_t * dL/dd_t = sum_{s>t} r_s grS_s - sum_{s>=t} k_s gkG_s,
// i.e. two reverse cumulative sums; gw_t = ew_t * that.
// (The reference kernel, megatron/model/rwkv/v6/cuda/wkv6_cuda.cu, needs the sequence length as a compile-time
// constant for its decay-gradient pass; this formulation does not.)
//
// B has the form of A and C the form of the forward, with the operands exchanged and time reversed, so there are two scan
// bodies.  What bounds them is issue: four fp32 operations and most of a shared-memory read per step and state element,
// on as many SMs as there are (batch, head) pairs.  One block of N threads with a whole row of the state each, a barrier
// on both sides of every step and the step's global loads in between, paid those latencies 512 times over: 403 us forward
// at b 4, t 512, 12 heads of 64, and 1165 us backward in three launches plus 400 us of flips and cumulative sums.
//
// Here a row of the state is cut into SLICES pieces held by different warps.  A step's sum runs through the pieces in order:
// piece g works on the staged group of steps that piece g - 1 worked on one turn earlier and continues its partial
// sums.  There is one barrier per group of STEPS steps, whose operands were requested a turn ahead, and every sum is still
// taken over the channels one after the other, with the rounding it always had.  (Cutting time into chunks instead was
// faster still, 80 us forward, but a sum taken in another order changes the last bit of some of the 16-bit results, and
// twelve layers turn that into differences of 2 % between two training steps.)  The three backward scans share one
// launch, so they run side by side.  Now 108 us forward, 108 us for the three scans and 29 us for the decay gradient.
#include "dynamic_smem.h"
#include "neox_b200.h"
#include <cuda_bf16.h>

namespace {

typedef __nv_bfloat16 bf16;
constexpr int SLICES = 4;         // pieces of a state row
constexpr int STEPS = 8;          // steps staged at a time
constexpr int RING = SLICES + 1;  // staged groups: one per piece, and the one being filled

struct Shape {
    int T, C, H;
};

template <int N> struct ValueSmem {
    float p[RING][STEPS][N], q[RING][STEPS][N], own[RING][STEPS][N], d[RING][STEPS][N];
    float hand[SLICES - 1][2][STEPS][N];                  // partial sums on their way to the next piece
};
template <int N> struct KeySmem {
    float a[RING][STEPS][N], b[RING][STEPS][N], e[RING][STEPS][N], f[RING][STEPS][N], d[RING][STEPS][N];
    float dot[SLICES - 1][2][STEPS][N], ab[SLICES - 1][2][STEPS][N];
};

// Time of step s of group st in scan order.
template <bool REV>
__device__ __forceinline__ int when(int T, int st, int s) {
    const int t = st * STEPS + s;
    return REV ? T - 1 - t : t;
}

// The turns of the pipeline: `fetch(st)` requests a group's operands, `put(slot)` stores them to the ring, `work(st, slot,
// parity)` advances this thread's piece by one group.
template <typename Fetch, typename Put, typename Work>
__device__ __forceinline__ void pipeline(int groups, int piece, Fetch fetch, Put put, Work work) {
    fetch(0);
    put(0);
    __syncthreads();
    for (int turn = 0; turn < groups + SLICES - 1; ++turn) {
        const bool more = turn + 1 < groups;
        if (more) fetch(turn + 1);
        const int st = turn - piece;
        if (st >= 0 && st < groups) work(st, st % RING, turn & 1);
        if (more) put((turn + 1) % RING);
        __syncthreads();
    }
}

// ------------------------------------------------------------------ thread = value channel i (forward; backward C)
// x = q[j] * own;   out = sum_j p[j] * (u[j] * x + X[j]);   X[j] <- X[j] * d[j] + x
template <int N, bool REV>
__device__ __forceinline__ void value_scan(const Shape& sh, const bf16* __restrict__ p, const bf16* __restrict__ q,
                                           const bf16* __restrict__ own, const float* __restrict__ ew,
                                           const bf16* __restrict__ u, bf16* __restrict__ out, void* smem) {
    constexpr int PART = N / SLICES, PER = STEPS / SLICES;      // channels of a piece; staged steps per thread
    ValueSmem<N>& sm = *static_cast<ValueSmem<N>*>(smem);
    const int i = threadIdx.x % N, piece = threadIdx.x / N, h = blockIdx.x % sh.H;
    const size_t base = (size_t)(blockIdx.x / sh.H) * sh.T * sh.C + h * N + i;
    float X[PART], us[PART];
#pragma unroll
    for (int j = 0; j < PART; ++j) {
        X[j] = 0.f;
        us[j] = __bfloat162float(u[h * N + piece * PART + j]);
    }
    bf16 rp[PER], rq[PER], ro[PER];
    float rw[PER];
    auto fetch = [&](int st) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int s = piece * PER + k;
            if (st * STEPS + s < sh.T) {
                const size_t o = base + (size_t)when<REV>(sh.T, st, s) * sh.C;
                rp[k] = p[o];
                rq[k] = q[o];
                ro[k] = own[o];
                rw[k] = ew[o];
            }
        }
    };
    auto put = [&](int slot) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int s = piece * PER + k;
            sm.p[slot][s][i] = __bfloat162float(rp[k]);
            sm.q[slot][s][i] = __bfloat162float(rq[k]);
            sm.own[slot][s][i] = __bfloat162float(ro[k]);
            sm.d[slot][s][i] = __expf(rw[k]);
        }
    };
    auto work = [&](int st, int slot, int parity) {
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            if (st * STEPS + s >= sh.T) break;
            const float oi = sm.own[slot][s][i];
            float acc = piece ? sm.hand[piece - 1][parity ^ 1][s][i] : 0.f;
#pragma unroll
            for (int j = 0; j < PART; j += 4) {
                const float4 p4 = *reinterpret_cast<const float4*>(&sm.p[slot][s][piece * PART + j]);
                const float4 q4 = *reinterpret_cast<const float4*>(&sm.q[slot][s][piece * PART + j]);
                const float4 d4 = *reinterpret_cast<const float4*>(&sm.d[slot][s][piece * PART + j]);
                const float pv[4] = {p4.x, p4.y, p4.z, p4.w}, qv[4] = {q4.x, q4.y, q4.z, q4.w}, dv[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const float x = __fmul_rn(qv[m], oi);
                    acc = __fmaf_rn(pv[m], __fmaf_rn(us[j + m], x, X[j + m]), acc);
                    X[j + m] = __fmaf_rn(X[j + m], dv[m], x);
                }
            }
            if (piece < SLICES - 1) sm.hand[piece][parity][s][i] = acc;
            else out[base + (size_t)when<REV>(sh.T, st, s) * sh.C] = __float2bfloat16(acc);
        }
    };
    pipeline((sh.T + STEPS - 1) / STEPS, piece, fetch, put, work);
}

// ------------------------------------------------------------------ thread = key channel j (backward A, B)
// dot = sum_i a[i] X[i];   ab = sum_i a[i] b[i];   X[i] <- X[i] * d_j + e_j * b[i]
// grad = e_j u_j ab + dot;   cum = f_j dot;   gu += f_j e_j ab
template <int N, bool REV>
__device__ __forceinline__ void key_scan(const Shape& sh, const bf16* __restrict__ a, const bf16* __restrict__ b,
                                         const bf16* __restrict__ e, const bf16* __restrict__ f,
                                         const float* __restrict__ ew, const bf16* __restrict__ u, bf16* __restrict__ grad,
                                         float* __restrict__ cum, float* __restrict__ gu_part, void* smem) {
    constexpr int PART = N / SLICES, PER = STEPS / SLICES;
    KeySmem<N>& sm = *static_cast<KeySmem<N>*>(smem);
    const int j = threadIdx.x % N, piece = threadIdx.x / N, h = blockIdx.x % sh.H;
    const size_t base = (size_t)(blockIdx.x / sh.H) * sh.T * sh.C + h * N + j;
    const float uj = __bfloat162float(u[h * N + j]);
    float X[PART], gu = 0.f;
#pragma unroll
    for (int i = 0; i < PART; ++i) X[i] = 0.f;
    bf16 ra[PER], rb[PER], re[PER], rf[PER];
    float rw[PER];
    auto fetch = [&](int st) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int s = piece * PER + k;
            if (st * STEPS + s < sh.T) {
                const size_t o = base + (size_t)when<REV>(sh.T, st, s) * sh.C;
                ra[k] = a[o];
                rb[k] = b[o];
                re[k] = e[o];
                rf[k] = f[o];
                rw[k] = ew[o];
            }
        }
    };
    auto put = [&](int slot) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int s = piece * PER + k;
            sm.a[slot][s][j] = __bfloat162float(ra[k]);
            sm.b[slot][s][j] = __bfloat162float(rb[k]);
            sm.e[slot][s][j] = __bfloat162float(re[k]);
            sm.f[slot][s][j] = __bfloat162float(rf[k]);
            sm.d[slot][s][j] = __expf(rw[k]);
        }
    };
    auto work = [&](int st, int slot, int parity) {
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            if (st * STEPS + s >= sh.T) break;
            const float ej = sm.e[slot][s][j], dj = sm.d[slot][s][j];
            float dot = piece ? sm.dot[piece - 1][parity ^ 1][s][j] : 0.f, ab = piece ? sm.ab[piece - 1][parity ^ 1][s][j] : 0.f;
#pragma unroll
            for (int i = 0; i < PART; i += 4) {
                const float4 a4 = *reinterpret_cast<const float4*>(&sm.a[slot][s][piece * PART + i]);
                const float4 b4 = *reinterpret_cast<const float4*>(&sm.b[slot][s][piece * PART + i]);
                const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    dot = __fmaf_rn(X[i + m], av[m], dot);
                    ab = __fmaf_rn(bv[m], av[m], ab);
                    X[i + m] = __fmaf_rn(ej, bv[m], __fmul_rn(X[i + m], dj));
                }
            }
            if (piece < SLICES - 1) {
                sm.dot[piece][parity][s][j] = dot;
                sm.ab[piece][parity][s][j] = ab;
            } else {
                const float fj = sm.f[slot][s][j];
                const size_t o = base + (size_t)when<REV>(sh.T, st, s) * sh.C;
                grad[o] = __float2bfloat16(__fmaf_rn(__fmul_rn(uj, ej), ab, dot));
                cum[o] = __fmul_rn(fj, dot);
                gu = __fmaf_rn(__fmul_rn(fj, ej), ab, gu);
            }
        }
    };
    pipeline((sh.T + STEPS - 1) / STEPS, piece, fetch, put, work);
    if (gu_part && piece == SLICES - 1) gu_part[(size_t)blockIdx.x * N + j] = gu;
}

template <int N>
__global__ void __launch_bounds__(N * SLICES) wkv6_fwd_kernel(Shape sh, const bf16* __restrict__ r,
                                                              const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                              const float* __restrict__ ew, const bf16* __restrict__ u,
                                                              bf16* __restrict__ y) {
    extern __shared__ __align__(16) unsigned char smem[];
    value_scan<N, false>(sh, r, k, v, ew, u, y, smem);
}

// The three scans are independent: y selects one, so that few heads still fill the machine.
template <int N>
__global__ void __launch_bounds__(N * SLICES) wkv6_bwd_kernel(Shape sh, const bf16* __restrict__ r,
                                                              const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                              const float* __restrict__ ew, const bf16* __restrict__ u,
                                                              const bf16* __restrict__ gy, bf16* __restrict__ gr,
                                                              bf16* __restrict__ gk, bf16* __restrict__ gv,
                                                              float* __restrict__ cumA, float* __restrict__ cumB,
                                                              float* __restrict__ gu_part) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (blockIdx.y == 0) key_scan<N, false>(sh, gy, v, k, r, ew, u, gr, cumA, gu_part, smem);
    else if (blockIdx.y == 1) key_scan<N, true>(sh, v, gy, r, k, ew, u, gk, cumB, nullptr, smem);
    else value_scan<N, true>(sh, k, r, gy, ew, u, gv, smem);
}

// gw_t = ew_t * ((sum_{s>=t} a_s - a_t) - sum_{s>=t} b_s), the sums taken from the last step backwards.  A serial chain of
// additions per channel; the next AHEAD steps are requested before the present ones are added.
constexpr int AHEAD = 16;
__global__ void __launch_bounds__(64) wkv6_decay_kernel(int T, int C, long long channels, const float* __restrict__ cumA,
                                                        const float* __restrict__ cumB, const float* __restrict__ ew,
                                                        bf16* __restrict__ gw) {
    const long long ch = blockIdx.x * 64ll + threadIdx.x;
    if (ch >= channels) return;
    const size_t base = (size_t)(ch / C) * T * C + ch % C;
    float na[AHEAD], nb[AHEAD], ne[AHEAD], sa = 0.f, sb = 0.f;
    auto fetch = [&](int t1) {                     // steps t1 - 1 down to t1 - AHEAD
#pragma unroll
        for (int s = 0; s < AHEAD; ++s) {
            if (t1 - 1 - s >= 0) {
                const size_t o = base + (size_t)(t1 - 1 - s) * C;
                na[s] = cumA[o];
                nb[s] = cumB[o];
                ne[s] = ew[o];
            }
        }
    };
    fetch(T);
    for (int t1 = T; t1 > 0; t1 -= AHEAD) {
        float a[AHEAD], b[AHEAD], e[AHEAD];
#pragma unroll
        for (int s = 0; s < AHEAD; ++s) {
            a[s] = na[s];
            b[s] = nb[s];
            e[s] = ne[s];
        }
        fetch(t1 - AHEAD);
#pragma unroll
        for (int s = 0; s < AHEAD; ++s) {
            if (t1 - 1 - s >= 0) {
                sa = __fadd_rn(sa, a[s]);
                sb = __fadd_rn(sb, b[s]);
                gw[base + (size_t)(t1 - 1 - s) * C] = __float2bfloat16(__fmul_rn(__fadd_rn(__fadd_rn(sa, -a[s]), -sb), e[s]));
            }
        }
    }
}

#define WKV_DISPATCH(N_, ...)                                       \
    switch (N_) {                                                   \
        case 32: { constexpr int N = 32; __VA_ARGS__; break; }             \
        case 64: { constexpr int N = 64; __VA_ARGS__; break; }             \
        case 128: { constexpr int N = 128; __VA_ARGS__; break; }           \
        default: return NEOX_ERR_SHAPE;                             \
    }

}  // namespace

extern "C" int neox_wkv6_fwd(int B, int T, int C, int H, const void* r, const void* k, const void* v, const float* ew,
                             const void* u, void* y, void* stream) {
    if (C % H) return NEOX_ERR_SHAPE;
    if (B <= 0 || T <= 0) return 0;
    const int n = C / H;
    cudaStream_t st = (cudaStream_t)stream;
    const Shape sh{T, C, H};
    WKV_DISPATCH(n, {
        const size_t bytes = sizeof(ValueSmem<N>);
        if (!allow_dynamic_smem<wkv6_fwd_kernel<N>>(bytes)) return NEOX_ERR_LAUNCH;
        wkv6_fwd_kernel<N><<<B * H, N * SLICES, bytes, st>>>(sh, (const bf16*)r, (const bf16*)k, (const bf16*)v, ew,
                                                             (const bf16*)u, (bf16*)y);
    });
    return cudaGetLastError() == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
}

// cum: two of [B, T, C] floats of scratch; gu_part: [B, H, N] floats.
extern "C" int neox_wkv6_bwd(int B, int T, int C, int H, const void* r, const void* k, const void* v, const float* ew,
                             const void* u, const void* gy, void* gr, void* gk, void* gv, void* gw, float* cum,
                             float* gu_part, void* stream) {
    if (C % H) return NEOX_ERR_SHAPE;
    if (B <= 0) return 0;
    const int n = C / H;
    cudaStream_t st = (cudaStream_t)stream;
    if (T <= 0) return cudaMemsetAsync(gu_part, 0, (size_t)B * C * sizeof(float), st) == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
    const Shape sh{T, C, H};
    float* cumB = cum + (size_t)B * T * C;
    WKV_DISPATCH(n, {
        const size_t bytes = sizeof(KeySmem<N>) > sizeof(ValueSmem<N>) ? sizeof(KeySmem<N>) : sizeof(ValueSmem<N>);
        if (!allow_dynamic_smem<wkv6_bwd_kernel<N>>(bytes)) return NEOX_ERR_LAUNCH;
        wkv6_bwd_kernel<N><<<dim3(B * H, 3), N * SLICES, bytes, st>>>(sh, (const bf16*)r, (const bf16*)k, (const bf16*)v, ew,
                                                                     (const bf16*)u, (const bf16*)gy, (bf16*)gr, (bf16*)gk,
                                                                     (bf16*)gv, cum, cumB, gu_part);
    });
    const long long channels = (long long)B * C;
    wkv6_decay_kernel<<<(int)((channels + 63) / 64), 64, 0, st>>>(T, C, channels, cum, cumB, ew, (bf16*)gw);
    return cudaGetLastError() == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
}

// Mamba selective scan (S6), forward and backward, channel-last layouts, state size 16.
//
//     delta = softplus(dt + dt_bias)
//     h_t[j] = exp(delta_t * A[c][j]) * h_{t-1}[j] + delta_t * B_t[j] * u_t        (c = channel, j = state index)
//     y_t    = sum_j C_t[j] * h_t[j] + D[c] * u_t,      out_t = y_t * silu(z_t)
//
// The recurrence is linear in h, so time is cut into chunks of 32 steps that run side by side.  Forward:
//   state    every chunk from h = 0: its final state and the sum of its deltas (the decay of a whole chunk is
//            exp(A * sum delta));
//   combine  one short pass over the chunks turns these into the state at the start of every chunk;
//   output   every chunk again from its start state, writing out.
// The chunk start states are also the checkpoints of the backward, which runs the same three steps on the adjoint:
// adjoint (every chunk backwards from 0), combine (over the chunks in reverse), gradient.
//
// What bounds it: one exponential per step, channel and state on the special-function units (16 a clock and SM) and the
// arithmetic around it; the bytes are a tenth of that.  One thread per channel walking all of time serially, as this
// file did before, left most SMs without a block (6144 channels = 48 blocks forward, 96 of two warps backward) and paid
// the latency of every step: 1987 us forward, 7232 us backward at b 4, l 2048, d 1536.  The chunked form computes the
// exponentials twice and has 64 times the threads: 181 us forward (state 67, combine 10, output 104) and 514 us backward
// (adjoint 82, combine 15, gradient 417).  Exponentials alone would take 45 us a pass.
#include "dynamic_smem.h"
#include "neox_b200.h"
#include <cuda_bf16.h>

#include <cstring>

namespace {

typedef __nv_bfloat16 bf16;
constexpr int NS = 16;            // state size
constexpr int CHUNK = 32;         // steps per chunk = steps between checkpoints
constexpr int THREADS = 128;      // channels per block of the thread-per-channel kernels
constexpr int GROUP = 8;          // steps whose loads are issued together
constexpr float LOG2E = 1.4426950408889634f;

// Element strides (batch, time) of the [b, l, ...] operands; the last dimension is contiguous in all of them.
struct Strides {
    long long ub, ut, db, dt, zb, zt, ob, ot, bb, bt, cb, ct;       // u, dt, z, out or its gradient, B, C
    long long gub, gut, gdb, gdt, gzb, gzt, gsb, gst;               // gradients of u, dt, z and of B and C
};

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(__expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }

// ckpt and the adjoint's counterpart are [b][chunk][state][channel]: a warp's accesses are whole lines.
__device__ __forceinline__ size_t slot(int b, int ck, int nchk, int d) { return ((size_t)b * nchk + ck) * NS * d; }

__device__ __forceinline__ void stage_rows(float (*dst)[NS], const float* __restrict__ src, int steps, long long stride) {
    for (int i = threadIdx.x; i < CHUNK * NS; i += blockDim.x) {
        const int s = i / NS, j = i % NS;
        dst[s][j] = s < steps ? src[s * stride + j] : 0.f;
    }
}

// ------------------------------------------------------------------ forward: chunk states from h = 0
__global__ void __launch_bounds__(THREADS)
scan_state_kernel(const bf16* __restrict__ u, const bf16* __restrict__ dt, const float* __restrict__ A,
                  const float* __restrict__ B, const float* __restrict__ bias, float* __restrict__ ckpt,
                  float* __restrict__ sumd, int l, int d, int nchk, int dblk, Strides st) {
    __shared__ alignas(16) float sB[CHUNK][NS];
    const int b = blockIdx.y, ck = blockIdx.x / dblk, t0 = ck * CHUNK;        // never the last chunk: always full
    const int c = blockIdx.x % dblk * THREADS + threadIdx.x;
    stage_rows(sB, B + b * st.bb + t0 * st.bt, CHUNK, st.bt);
    __syncthreads();
    if (c >= d) return;
    float a[NS], h[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        a[j] = A[(size_t)c * NS + j] * LOG2E;
        h[j] = 0.f;
    }
    const float bc = bias[c];
    const bf16* up = u + b * st.ub + t0 * st.ut + c;
    const bf16* dp = dt + b * st.db + t0 * st.dt + c;
    float total = 0.f;
    for (int s0 = 0; s0 < CHUNK; s0 += GROUP) {
        bf16 ur[GROUP], dr[GROUP];
#pragma unroll
        for (int s = 0; s < GROUP; ++s) {
            ur[s] = up[(s0 + s) * st.ut];
            dr[s] = dp[(s0 + s) * st.dt];
        }
#pragma unroll
        for (int s = 0; s < GROUP; ++s) {
            const float delta = softplus_f(__bfloat162float(dr[s]) + bc);
            const float du = delta * __bfloat162float(ur[s]);
            total += delta;
#pragma unroll
            for (int j = 0; j < NS; j += 4) {
                const float4 bv = *reinterpret_cast<const float4*>(&sB[s0 + s][j]);
                h[j] = exp2f(delta * a[j]) * h[j] + du * bv.x;
                h[j + 1] = exp2f(delta * a[j + 1]) * h[j + 1] + du * bv.y;
                h[j + 2] = exp2f(delta * a[j + 2]) * h[j + 2] + du * bv.z;
                h[j + 3] = exp2f(delta * a[j + 3]) * h[j + 3] + du * bv.w;
            }
        }
    }
    float* cp = ckpt + slot(b, ck + 1, nchk, d) + c;
#pragma unroll
    for (int j = 0; j < NS; ++j) cp[(size_t)j * d] = h[j];
    sumd[((size_t)b * nchk + ck) * d + c] = total;
}

// An exponent as far as 2^x stays a normal number.  The decay of 32 steps may leave the range of fp32 although the state, taken
// step by step, does not: what is left of the exponent is then applied as a second factor, which is 1 otherwise.  Neither
// factor is ever 0 or inf, so a state of 0 stays 0 and one that has overflowed stays so.
__device__ __forceinline__ float within_range(float x) { return fminf(fmaxf(x, -126.f), 126.f); }

// ------------------------------------------------------------------ combine over the chunks, in place
// Forward: slot k + 1 holds the state that chunk k adds; afterwards the state at the start of chunk k + 1.
// Reverse: slot k - 1 holds the adjoint that chunk k adds; afterwards the adjoint arriving at the end of chunk k - 1.
template <bool REVERSE>
__global__ void __launch_bounds__(THREADS)
scan_combine_kernel(const float* __restrict__ A, const float* __restrict__ sumd, float* __restrict__ st, int d, int nchk) {
    const int b = blockIdx.y, j = blockIdx.x % NS, c = blockIdx.x / NS * THREADS + threadIdx.x;
    if (c >= d) return;
    const float a = A[(size_t)c * NS + j] * LOG2E;
    float h = 0.f;
    for (int k0 = 0; k0 < nchk - 1; k0 += GROUP) {
        float loc[GROUP], x[GROUP];
#pragma unroll
        for (int i = 0; i < GROUP; ++i) {
            if (k0 + i < nchk - 1) {
                const int k = REVERSE ? nchk - 1 - (k0 + i) : k0 + i;
                loc[i] = st[slot(b, REVERSE ? k - 1 : k + 1, nchk, d) + (size_t)j * d + c];
                x[i] = sumd[((size_t)b * nchk + k) * d + c];
            }
        }
#pragma unroll
        for (int i = 0; i < GROUP; ++i) {
            if (k0 + i < nchk - 1) {
                const int k = REVERSE ? nchk - 1 - (k0 + i) : k0 + i;
                const float e = a * x[i], e1 = within_range(e);
                h = __fmaf_rn(exp2f(e1), exp2f(within_range(e - e1)) * h, loc[i]);
                st[slot(b, REVERSE ? k - 1 : k + 1, nchk, d) + (size_t)j * d + c] = h;
            }
        }
    }
}

// ------------------------------------------------------------------ forward: outputs
// A block runs `span` chunks in a row.  span 1: the start state comes from ckpt.  span = all: it starts at 0 and writes
// the checkpoints itself.
__global__ void __launch_bounds__(THREADS)
scan_out_kernel(const bf16* __restrict__ u, const bf16* __restrict__ dt, const float* __restrict__ A,
                const float* __restrict__ B, const float* __restrict__ C, const float* __restrict__ D,
                const bf16* __restrict__ z, const float* __restrict__ bias, bf16* __restrict__ out,
                float* __restrict__ ckpt, int l, int d, int nchk, int span, int dblk, Strides st) {
    __shared__ alignas(16) float sB[CHUNK][NS], sC[CHUNK][NS];
    const int b = blockIdx.y;
    const int c = blockIdx.x % dblk * THREADS + threadIdx.x;
    const bool live = c < d;
    const int first = blockIdx.x / dblk * span, last = min(first + span, nchk);
    float a[NS], h[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        a[j] = live ? A[(size_t)c * NS + j] * LOG2E : 0.f;
        h[j] = live && first > 0 ? ckpt[slot(b, first, nchk, d) + (size_t)j * d + c] : 0.f;
    }
    const float Dc = live ? D[c] : 0.f, bc = live ? bias[c] : 0.f;
    for (int ck = first; ck < last; ++ck) {
        const int t0 = ck * CHUNK, steps = min(CHUNK, l - t0);
        __syncthreads();
        stage_rows(sB, B + b * st.bb + t0 * st.bt, steps, st.bt);
        stage_rows(sC, C + b * st.cb + t0 * st.ct, steps, st.ct);
        __syncthreads();
        if (!live) continue;
        if (ck > first) {
            float* cp = ckpt + slot(b, ck, nchk, d) + c;
#pragma unroll
            for (int j = 0; j < NS; ++j) cp[(size_t)j * d] = h[j];
        }
        const bf16* up = u + b * st.ub + t0 * st.ut + c;
        const bf16* dp = dt + b * st.db + t0 * st.dt + c;
        const bf16* zp = z + b * st.zb + t0 * st.zt + c;
        bf16* op = out + b * st.ob + t0 * st.ot + c;
        for (int s0 = 0; s0 < steps; s0 += GROUP) {
            bf16 ur[GROUP], dr[GROUP], zr[GROUP];
#pragma unroll
            for (int s = 0; s < GROUP; ++s) {
                if (s0 + s < steps) {
                    ur[s] = up[(s0 + s) * st.ut];
                    dr[s] = dp[(s0 + s) * st.dt];
                    zr[s] = zp[(s0 + s) * st.zt];
                }
            }
#pragma unroll
            for (int s = 0; s < GROUP; ++s) {
                if (s0 + s >= steps) break;
                const float uv = __bfloat162float(ur[s]);
                const float delta = softplus_f(__bfloat162float(dr[s]) + bc);
                const float du = delta * uv;
                float y0 = Dc * uv, y1 = 0.f, y2 = 0.f, y3 = 0.f;
#pragma unroll
                for (int j = 0; j < NS; j += 4) {
                    const float4 bv = *reinterpret_cast<const float4*>(&sB[s0 + s][j]);
                    const float4 cv = *reinterpret_cast<const float4*>(&sC[s0 + s][j]);
                    h[j] = exp2f(delta * a[j]) * h[j] + du * bv.x;
                    h[j + 1] = exp2f(delta * a[j + 1]) * h[j + 1] + du * bv.y;
                    h[j + 2] = exp2f(delta * a[j + 2]) * h[j + 2] + du * bv.z;
                    h[j + 3] = exp2f(delta * a[j + 3]) * h[j + 3] + du * bv.w;
                    y0 += cv.x * h[j];
                    y1 += cv.y * h[j + 1];
                    y2 += cv.z * h[j + 2];
                    y3 += cv.w * h[j + 3];
                }
                const float zv = __bfloat162float(zr[s]);
                op[(s0 + s) * st.ot] = __float2bfloat16(((y0 + y1) + (y2 + y3)) * zv * sigmoid_f(zv));
            }
        }
    }
}

// ------------------------------------------------------------------ backward: chunk adjoints from 0
__global__ void __launch_bounds__(THREADS)
scan_adjoint_kernel(const bf16* __restrict__ dt, const float* __restrict__ A, const float* __restrict__ C,
                    const bf16* __restrict__ z, const float* __restrict__ bias, const bf16* __restrict__ gout,
                    float* __restrict__ gst, float* __restrict__ sumd, int l, int d, int nchk, int dblk, Strides st) {
    __shared__ alignas(16) float sC[CHUNK][NS];
    const int b = blockIdx.y, ck = blockIdx.x / dblk + 1, t0 = ck * CHUNK, steps = min(CHUNK, l - t0);
    const int c = blockIdx.x % dblk * THREADS + threadIdx.x;
    stage_rows(sC, C + b * st.cb + t0 * st.ct, steps, st.ct);
    __syncthreads();
    if (c >= d) return;
    float a[NS], gh[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        a[j] = A[(size_t)c * NS + j] * LOG2E;
        gh[j] = 0.f;
    }
    const float bc = bias[c];
    const bf16* dp = dt + b * st.db + t0 * st.dt + c;
    const bf16* zp = z + b * st.zb + t0 * st.zt + c;
    const bf16* gp = gout + b * st.ob + t0 * st.ot + c;
    float total = 0.f;
    for (int s0 = (steps - 1) / GROUP * GROUP; s0 >= 0; s0 -= GROUP) {
        bf16 dr[GROUP], zr[GROUP], gr[GROUP];
#pragma unroll
        for (int s = 0; s < GROUP; ++s) {
            if (s0 + s < steps) {
                dr[s] = dp[(s0 + s) * st.dt];
                zr[s] = zp[(s0 + s) * st.zt];
                gr[s] = gp[(s0 + s) * st.ot];
            }
        }
#pragma unroll
        for (int s = GROUP - 1; s >= 0; --s) {
            if (s0 + s >= steps) continue;
            const float delta = softplus_f(__bfloat162float(dr[s]) + bc);
            const float zv = __bfloat162float(zr[s]);
            const float gy = __bfloat162float(gr[s]) * zv * sigmoid_f(zv);
            total += delta;
#pragma unroll
            for (int j = 0; j < NS; j += 4) {
                const float4 cv = *reinterpret_cast<const float4*>(&sC[s0 + s][j]);
                gh[j] = exp2f(delta * a[j]) * (gh[j] + gy * cv.x);
                gh[j + 1] = exp2f(delta * a[j + 1]) * (gh[j + 1] + gy * cv.y);
                gh[j + 2] = exp2f(delta * a[j + 2]) * (gh[j + 2] + gy * cv.z);
                gh[j + 3] = exp2f(delta * a[j + 3]) * (gh[j + 3] + gy * cv.w);
            }
        }
    }
    float* gp2 = gst + slot(b, ck - 1, nchk, d) + c;
#pragma unroll
    for (int j = 0; j < NS; ++j) gp2[(size_t)j * d] = gh[j];
    sumd[((size_t)b * nchk + ck) * d + c] = total;
}

// ------------------------------------------------------------------ backward: gradients of one chunk
// A block takes one chunk of 64 channels; four threads share a channel and hold four states each (lane = 8 * state group
// + channel of the warp), so that the states and decays of a few steps fit into registers: a sub-chunk of four steps is
// recomputed forwards from its start state and walked backwards at once, and no per-step state leaves the registers.
// Sub-chunks of four and results written over the staged operands keep it to 80 registers and 68 KB, three blocks on an SM:
// 491 us with sub-chunks of eight on two blocks, 417 us so (b 4, l 2048, d 1536).
// Per-element quantities that do not depend on the state index (softplus, SiLU) are computed once and shared through
// shared memory.  Sums over the states of a channel and over the channels of a warp are reduced "transposed" (every
// shuffle step halves the number of values a lane carries): 3 + 7 shuffles per step instead of 6 + 24.
constexpr int GCH = 64;                       // channels per block
constexpr int GTH = GCH * 4;                  // threads per block
constexpr int GSTEP = 4;                      // steps per sub-chunk
constexpr int NSUB = CHUNK / GSTEP;

struct GradSmem {
    // staged per-element inputs; once a step has been walked, in their places the step's sums over the states: gd * a, g * B, y
    float delta[CHUNK][GCH], u[CHUNK][GCH], gy[CHUNK][GCH];
    alignas(16) float B[CHUNK][NS];
    alignas(16) float C[CHUNK][NS];
    float start[NSUB][4][GTH];                                    // state at the start of every sub-chunk
    float red[2][GTH / 32][GSTEP][32];                            // dB | dC partial sums per warp, of two sub-chunks in turn
};

// SHORT: a chunk of fewer steps walks only the sub-chunks it has.  A form of its own, as the loops of a known length are 5 % faster.
template <bool SHORT>
__global__ void __launch_bounds__(GTH, 3)
scan_grad_kernel(const bf16* __restrict__ u, const bf16* __restrict__ dt, const float* __restrict__ A,
                 const float* __restrict__ B, const float* __restrict__ C, const float* __restrict__ D,
                 const bf16* __restrict__ z, const float* __restrict__ bias, const float* __restrict__ ckpt,
                 const float* __restrict__ gst, const bf16* __restrict__ gout, bf16* __restrict__ gu,
                 bf16* __restrict__ gdt, bf16* __restrict__ gz, float* __restrict__ gA, float* __restrict__ gB,
                 float* __restrict__ gC, float* __restrict__ gD, float* __restrict__ gbias, int l, int d, int nchk,
                 int dblk, Strides st) {
    extern __shared__ __align__(16) unsigned char raw[];
    GradSmem& sm = *reinterpret_cast<GradSmem*>(raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.y, ck = blockIdx.x / dblk, t0 = ck * CHUNK, steps = min(CHUNK, l - t0);
    const int c0 = blockIdx.x % dblk * GCH;

    // ---- per-element inputs; rows past the end and channels past the last one are zero: decay 1, no contribution
    {
        const int cc = tid % GCH, c = c0 + cc;
        const bool live = c < d;
        const float bc = live ? bias[c] : 0.f;
#pragma unroll
        for (int i = 0; i < CHUNK / 4; ++i) {
            const int s = tid / GCH + 4 * i;
            float delta = 0.f, uv = 0.f, gy = 0.f;
            if (live && s < steps) {
                uv = __bfloat162float(u[b * st.ub + (t0 + s) * st.ut + c]);
                delta = softplus_f(__bfloat162float(dt[b * st.db + (t0 + s) * st.dt + c]) + bc);
                const float zv = __bfloat162float(z[b * st.zb + (t0 + s) * st.zt + c]);
                gy = __bfloat162float(gout[b * st.ob + (t0 + s) * st.ot + c]) * zv * sigmoid_f(zv);
            }
            sm.delta[s][cc] = delta;
            sm.u[s][cc] = uv;
            sm.gy[s][cc] = gy;
        }
        stage_rows(sm.B, B + b * st.bb + t0 * st.bt, steps, st.bt);
        stage_rows(sm.C, C + b * st.cb + t0 * st.ct, steps, st.ct);
    }
    __syncthreads();

    const int sg = lane >> 3;                          // states 4 sg .. 4 sg + 3
    const int cc = warp * 8 + (lane & 7), c = c0 + cc;
    const bool live = c < d;
    float a[4], gh[4], ga[4], h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        a[j] = live ? A[(size_t)c * NS + sg * 4 + j] : 0.f;
        h[j] = live && ck > 0 ? ckpt[slot(b, ck, nchk, d) + (size_t)(sg * 4 + j) * d + c] : 0.f;
        gh[j] = live && ck + 1 < nchk ? gst[slot(b, ck, nchk, d) + (size_t)(sg * 4 + j) * d + c] : 0.f;
        ga[j] = 0.f;
    }
    // ---- states at the starts of the sub-chunks
    const int nsub = SHORT ? (steps + GSTEP - 1) / GSTEP : NSUB;
#pragma unroll 1
    for (int sub = 0; sub < nsub; ++sub) {
#pragma unroll
        for (int j = 0; j < 4; ++j) sm.start[sub][j][tid] = h[j];
        if (sub == nsub - 1) break;
#pragma unroll
        for (int i = 0; i < GSTEP; ++i) {
            const int s = sub * GSTEP + i;
            const float delta = sm.delta[s][cc], du = delta * sm.u[s][cc], d2 = delta * LOG2E;
            const float4 bv = *reinterpret_cast<const float4*>(&sm.B[s][sg * 4]);
            h[0] = exp2f(d2 * a[0]) * h[0] + du * bv.x;
            h[1] = exp2f(d2 * a[1]) * h[1] + du * bv.y;
            h[2] = exp2f(d2 * a[2]) * h[2] + du * bv.z;
            h[3] = exp2f(d2 * a[3]) * h[3] + du * bv.w;
        }
    }
    // ---- sub-chunks from the last to the first: recompute, then walk backwards
#pragma unroll 1
    for (int sub = nsub - 1; sub >= 0; --sub) {
        float hp[GSTEP + 1][4], dA[GSTEP][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) hp[0][j] = sm.start[sub][j][tid];
#pragma unroll
        for (int i = 0; i < GSTEP; ++i) {
            const int s = sub * GSTEP + i;
            const float delta = sm.delta[s][cc], du = delta * sm.u[s][cc], d2 = delta * LOG2E;
            const float4 bv = *reinterpret_cast<const float4*>(&sm.B[s][sg * 4]);
            const float bj[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                dA[i][j] = exp2f(d2 * a[j]);
                hp[i + 1][j] = dA[i][j] * hp[i][j] + du * bj[j];
            }
        }
#pragma unroll
        for (int i = GSTEP - 1; i >= 0; --i) {
            const int s = sub * GSTEP + i;
            const float delta = sm.delta[s][cc], du = delta * sm.u[s][cc], gy = sm.gy[s][cc];
            const float4 bv = *reinterpret_cast<const float4*>(&sm.B[s][sg * 4]);
            const float4 cv = *reinterpret_cast<const float4*>(&sm.C[s][sg * 4]);
            const float bj[4] = {bv.x, bv.y, bv.z, bv.w}, cj[4] = {cv.x, cv.y, cv.z, cv.w};
            float y = 0.f, sa = 0.f, sb = 0.f, pb[4], pc[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float g = gh[j] + gy * cj[j];              // adjoint of h_t[j]
                gh[j] = g * dA[i][j];
                const float gd = gh[j] * hp[i][j];               // d / d(delta * a[j])
                y += cj[j] * hp[i + 1][j];
                sa += gd * a[j];
                sb += g * bj[j];
                ga[j] += gd * delta;
                pb[j] = g * du;
                pc[j] = gy * hp[i + 1][j];
            }
            // over the four state groups of a channel (lane bits 3 and 4): group 0 ends with y, 1 with sa, 2 with sb
            {
                const bool hi = lane & 16, odd = lane & 8;
                const float k0 = (hi ? sb : y) + __shfl_xor_sync(0xffffffffu, hi ? y : sb, 16);
                const float k1 = (hi ? 0.f : sa) + __shfl_xor_sync(0xffffffffu, hi ? sa : 0.f, 16);
                // groups 0, 1: exchange y against sa; groups 2, 3: sb (group 3's result is not used)
                const float r = __shfl_xor_sync(0xffffffffu, odd ? k0 : (hi ? k0 : k1), 8);
                const float v = (odd ? (hi ? k0 : k1) : k0) + r;
                __syncwarp();               // every lane has read what this replaces; no other warp uses these channels
                if (sg < 3) (sg == 0 ? sm.gy : sg == 1 ? sm.delta : sm.u)[s][cc] = v;
            }
            // over the eight channels of the warp (lane bits 0 .. 2): every lane ends with one of pb[0..3], pc[0..3]
            {
                const bool b2 = lane & 4, b1 = lane & 2, b0 = lane & 1;
                float q[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    q[j] = (b2 ? pc[j] : pb[j]) + __shfl_xor_sync(0xffffffffu, b2 ? pb[j] : pc[j], 4);
                float r0 = (b1 ? q[2] : q[0]) + __shfl_xor_sync(0xffffffffu, b1 ? q[0] : q[2], 2);
                float r1 = (b1 ? q[3] : q[1]) + __shfl_xor_sync(0xffffffffu, b1 ? q[1] : q[3], 2);
                const float v = (b0 ? r1 : r0) + __shfl_xor_sync(0xffffffffu, b0 ? r0 : r1, 1);
                sm.red[sub & 1][warp][i][(b2 ? 16 : 0) + sg * 4 + (lane & 3)] = v;
            }
        }
        __syncthreads();                    // (the other buffer's sums were read before this barrier was reached)
        if (warp < GSTEP) {
            const int s = sub * GSTEP + warp;
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < GTH / 32; ++w) v += sm.red[sub & 1][w][warp][lane];
            if (s < steps) atomicAdd((lane < 16 ? gB : gC) + b * st.gsb + (t0 + s) * st.gst + (lane & 15), v);
        }
    }
    if (live) {
#pragma unroll
        for (int j = 0; j < 4; ++j) atomicAdd(gA + (size_t)c * NS + sg * 4 + j, ga[j]);
    }
    // ---- per-element gradients (the last __syncthreads() above made the sums over the states visible)
    {
        const int ce = tid % GCH, ch = c0 + ce;
        float gDc = 0.f, gbc = 0.f;
        if (ch < d) {
            const float Dc = D[ch], bc = bias[ch];
#pragma unroll
            for (int i = 0; i < CHUNK / 4; ++i) {
                const int s = tid / GCH + 4 * i;
                if (s >= steps) break;
                const float uv = __bfloat162float(u[b * st.ub + (t0 + s) * st.ut + ch]);
                const float x = __bfloat162float(dt[b * st.db + (t0 + s) * st.dt + ch]) + bc;
                const float zv = __bfloat162float(z[b * st.zb + (t0 + s) * st.zt + ch]);
                const float go = __bfloat162float(gout[b * st.ob + (t0 + s) * st.ot + ch]);
                const float sz = sigmoid_f(zv), gy = go * zv * sz, sb = sm.u[s][ce];
                const float g_dt = (sm.delta[s][ce] + uv * sb) * sigmoid_f(x);          // softplus'
                gDc += gy * uv;
                gbc += g_dt;
                gz[b * st.gzb + (t0 + s) * st.gzt + ch] =
                    __float2bfloat16(go * (Dc * uv + sm.gy[s][ce]) * sz * (1.f + zv * (1.f - sz)));
                gu[b * st.gub + (t0 + s) * st.gut + ch] = __float2bfloat16(gy * Dc + softplus_f(x) * sb);
                gdt[b * st.gdb + (t0 + s) * st.gdt + ch] = __float2bfloat16(g_dt);
            }
        }
        __syncthreads();                    // the last sub-chunk's sums have been read
        float* red = &sm.red[0][0][0][0];
        red[tid] = gDc;
        red[GTH + tid] = gbc;
        __syncthreads();
        if (tid < GCH && ch < d) {
            atomicAdd(gD + ch, (red[tid] + red[tid + GCH]) + (red[tid + 2 * GCH] + red[tid + 3 * GCH]));
            float* rb = red + GTH;
            atomicAdd(gbias + ch, (rb[tid] + rb[tid + GCH]) + (rb[tid + 2 * GCH] + rb[tid + 3 * GCH]));
        }
    }
}

// Chunks side by side, or all chunks of a channel in one block?  Side by side costs the exponentials twice and two launches
// more, and pays where the blocks of 128 channels alone leave the machine idle.  Measured at 148 SMs: a block that walks all of
// time takes 0.28 us a step, and a little longer with more of them (0.28 + 0.0005 a block up to four an SM); side by side a
// block's chunk takes 0.053 us of the machine, and the launches some 20.  Equating the two gives the line below, r blocks an
// SM.  In one block / side by side, us: 16 blocks 2048 steps 565 / 74, 144 blocks 512 steps 173 / 136, 221 blocks 512 steps
// 204 / 199, 288 blocks 2048 steps 804 / 994, 592 blocks 256 steps 149 / 257, 4 blocks 64 steps 21 / 22.
int forward_span(int b, int d, int nchk) {
    const double r = (double)b * ((d + THREADS - 1) / THREADS) / neox_sm_count();
    return nchk * (9.0 - 5.5 * r) > 20.0 ? 1 : nchk;
}

Strides make_strides(const long long* s, int operands) {
    Strides st{};
    memcpy(&st, s, operands * 2 * sizeof(long long));
    return st;
}

}  // namespace

// strides: (batch, time) element strides of u, dt, z, out, B, C.  ckpt: [b][chunks][16][d] floats; sumd: [b][chunks][d]
// floats of scratch.
extern "C" int neox_selective_scan_fwd(const void* u, const void* dt, const float* A, const float* B, const float* C,
                                       const float* D, const void* z, const float* bias, void* out, float* ckpt,
                                       float* sumd, const long long* strides, int b, int l, int d, int n, void* stream) {
    if (n != NS) return NEOX_ERR_SHAPE;
    if (b <= 0 || l <= 0 || d <= 0) return 0;
    const int nchk = (l + CHUNK - 1) / CHUNK;
    const Strides st = make_strides(strides, 6);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    const int dblk = (d + THREADS - 1) / THREADS;
    const int span = forward_span(b, d, nchk);
    if (span < nchk) {
        scan_state_kernel<<<dim3(dblk * (nchk - 1), b), THREADS, 0, cs>>>(
            static_cast<const bf16*>(u), static_cast<const bf16*>(dt), A, B, bias, ckpt, sumd, l, d, nchk, dblk, st);
        scan_combine_kernel<false><<<dim3(dblk * NS, b), THREADS, 0, cs>>>(A, sumd, ckpt, d, nchk);
    }
    scan_out_kernel<<<dim3(dblk * ((nchk + span - 1) / span), b), THREADS, 0, cs>>>(
        static_cast<const bf16*>(u), static_cast<const bf16*>(dt), A, B, C, D, static_cast<const bf16*>(z), bias,
        static_cast<bf16*>(out), ckpt, l, d, nchk, span, dblk, st);
    return cudaGetLastError() == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
}

// gA, gB, gC, gD, gbias must be zero on entry (they are accumulated with atomics).  gst, sumd: scratch of the sizes of ckpt and
// of the forward's sumd.  strides: as above with gout in the place of out, then gu, gdt, gz and gB (= gC).
extern "C" int neox_selective_scan_bwd(const void* u, const void* dt, const float* A, const float* B, const float* C,
                                       const float* D, const void* z, const float* bias, const float* ckpt,
                                       const void* gout, void* gu, void* gdt, void* gz, float* gA, float* gB, float* gC,
                                       float* gD, float* gbias, float* gst, float* sumd, const long long* strides, int b,
                                       int l, int d, int n, void* stream) {
    if (n != NS) return NEOX_ERR_SHAPE;
    if (b <= 0 || l <= 0 || d <= 0) return 0;
    const int nchk = (l + CHUNK - 1) / CHUNK;
    // sub-chunks past the end of the sequence: skipped where they are more than a tenth of all
    const bool skip = 10 * ((nchk * CHUNK - l) / GSTEP) > nchk * NSUB;
    if (!(skip ? allow_dynamic_smem<scan_grad_kernel<true>>(sizeof(GradSmem)) : allow_dynamic_smem<scan_grad_kernel<false>>(sizeof(GradSmem))))
        return NEOX_ERR_LAUNCH;
    const Strides st = make_strides(strides, 10);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    const int dblk = (d + THREADS - 1) / THREADS, gblk = (d + GCH - 1) / GCH;
    if (nchk > 1) {
        scan_adjoint_kernel<<<dim3(dblk * (nchk - 1), b), THREADS, 0, cs>>>(
            static_cast<const bf16*>(dt), A, C, static_cast<const bf16*>(z), bias, static_cast<const bf16*>(gout), gst, sumd,
            l, d, nchk, dblk, st);
        scan_combine_kernel<true><<<dim3(dblk * NS, b), THREADS, 0, cs>>>(A, sumd, gst, d, nchk);
    }
    auto* grad = skip ? scan_grad_kernel<true> : scan_grad_kernel<false>;
    grad<<<dim3(gblk * nchk, b), GTH, sizeof(GradSmem), cs>>>(
        static_cast<const bf16*>(u), static_cast<const bf16*>(dt), A, B, C, D, static_cast<const bf16*>(z), bias, ckpt, gst,
        static_cast<const bf16*>(gout), static_cast<bf16*>(gu), static_cast<bf16*>(gdt), static_cast<bf16*>(gz), gA, gB, gC,
        gD, gbias, l, d, nchk, gblk, st);
    return cudaGetLastError() == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
}

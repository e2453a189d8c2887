// GEMM of a few rows (M <= 32) against a large weight matrix: D[M, N] = epilogue(alpha * X[M, K] W[N, K]^T).
//
// This is the linear layer of a decoding step: W is read once and dominates (2 N K bytes against 2 M K + 2 M N), so the
// kernel is a stream over W bound by HBM, and what counts is how many bytes are in flight.  The 128 x 256-tile tcgen05
// kernel puts N / 256 CTAs on the machine (8 of 148 SMs for N = 2048), each walking all of K behind a 4-stage ring:
// 29 us per call in a 1.4B model's decoding step at batch 4 and 8, 18.5 us at hidden 1024, batch 1; here 6.6 and 4.2 us in
// a replayed graph (15 and 3.8 us of bytes for the four products of a layer).
//
// Split: a CTA owns 16 rows of W (one mma tile), its 8 warps take the 64-wide k-blocks in turn and, when N / 16 CTAs do
// not fill the machine, a cluster of 2 to 8 CTAs splits K further.  Partial sums meet in shared memory (distributed
// shared memory across the cluster) in a fixed order, so results are bitwise repeatable.  Every lane loads 16 bytes of a
// row at a time straight into registers: the contraction index may be permuted freely as long as W and X use the same
// permutation, so the 8 consecutive elements a lane holds serve as its fragments of two m16n8k16 products, with no pass
// through shared memory.  The tensor-core products only keep the arithmetic out of the way of the loads (at 16 rows
// packed-fp32 FMAs would already take longer than the bytes); a tcgen05 tile would be 1 / 4 to 1 / 128 full.
//
// A CTA asks for its whole share of W in L2 before it waits for the kernel in front (launch.cuh), so registers do not have
// to hold what is in flight; they are kept few instead, and four CTAs share an SM.  The four products of a layer, batch 1,
// replayed, hidden 1024 / 2048 / 4096: 29.9 / 42.4 / 100 us with two CTAs an SM and plain launches, 27.7 / 39.7 / 91 with
// the early request, 16.7 / 26.1 / 83 with four CTAs as well (3.8 / 15.1 / 60.5 of bytes).
#include <cooperative_groups.h>

#include "gemm_common.cuh"
#include "launch.cuh"
#include "neox_b200.h"

namespace {

namespace cg = cooperative_groups;
using namespace gemm;

constexpr int SK_ROWS = 16;       // rows of W per CTA
constexpr int SK_WARPS = 8;
constexpr int SK_THREADS = SK_WARPS * 32;
constexpr int SK_BK = 64;         // one k-block: a 128-byte line of every row
constexpr int SK_MAX_M = 32;

struct SkinnyParams {
    const void* X;
    const void* W;
    long long ldx, ldw;
    GemmParams e;                 // shape and epilogue
};

// W: used once.  A coherent load, as for X: the second operand of a product may be what the kernel in front has just written.
__device__ __forceinline__ uint4 load_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

template <bool H16>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
    if constexpr (H16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// CTAs an SM holds of the kernel for NT groups of 8 rows of X (its accumulators and fragments take twice the registers at 4).
constexpr int resident_ctas(int nt) { return nt == 4 ? 2 : 4; }

// U: k-blocks of a warp whose loads are issued together.
template <bool H16, int NT, int U>
__global__ void __launch_bounds__(SK_THREADS, resident_ctas(NT)) gemm_skinny_kernel(const SkinnyParams p) {
    __shared__ float part[SK_WARPS][NT * 8][SK_ROWS + 1];
    __shared__ float mine[NT * 8][SK_ROWS + 1];
    cg::cluster_group cluster = cg::this_cluster();
    const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (int)(blockIdx.x / csize) * SK_ROWS;
    const int M = p.e.M, N = p.e.N, K = p.e.K;
    const int nblk = (K + SK_BK - 1) / SK_BK, slices = SK_WARPS * csize;
    const int lr = lane >> 2, lk = (lane & 3) * 8;          // row within 8, first of this lane's 8 elements within 32
    const char* W0 = static_cast<const char*>(p.W) + ((long long)(n0 + lr) * p.ldw + lk) * 2;
    const char* W1 = W0 + 8 * p.ldw * 2;
    const char* X0 = static_cast<const char*>(p.X) + ((long long)lr * p.ldx + lk) * 2;
    const bool w0 = n0 + lr < N, w1 = n0 + lr + 8 < N;
    // the weights do not depend on the kernel in front: ask for this CTA's share while that one finishes
    launch::let_successor_start();
    if (lane < SK_ROWS && n0 + lane < N)
        for (int kb = crank * SK_WARPS + warp; kb < nblk; kb += slices)
            launch::prefetch_l2(static_cast<const char*>(p.W) + ((long long)(n0 + lane) * p.ldw + kb * SK_BK) * 2);
    launch::wait_for_predecessor();
    float acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    const uint4 zero = make_uint4(0, 0, 0, 0);

    for (int kb = crank * SK_WARPS + warp; kb < nblk; kb += slices * U) {
        uint4 a[U][2][2], x[U][2][NT];
#pragma unroll
        for (int i = 0; i < U; ++i) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const long long k = (long long)(kb + i * slices) * SK_BK + half * 32;
                const bool in = k + lk < K;                  // K is a multiple of 8: a lane's 8 elements are in or out
                a[i][half][0] = in && w0 ? load_stream(W0 + k * 2) : zero;
                a[i][half][1] = in && w1 ? load_stream(W1 + k * 2) : zero;
            }
        }
#pragma unroll
        for (int i = 0; i < U; ++i) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const long long k = (long long)(kb + i * slices) * SK_BK + half * 32;
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    x[i][half][t] = k + lk < K && t * 8 + lr < M
                                        ? launch::load_16(X0 + (t * 8 * p.ldx + k) * 2)
                                        : zero;
            }
        }
#pragma unroll
        for (int i = 0; i < U; ++i) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const uint4 u = a[i][half][0], v = a[i][half][1], b = x[i][half][t];
                    mma_16816<H16>(acc[t], u.x, v.x, u.y, v.y, b.x, b.y);
                    mma_16816<H16>(acc[t], u.z, v.z, u.w, v.w, b.z, b.w);
                }
            }
        }
    }
    // accumulator layout: c0, c1 = row lr, columns 2 (lane % 4) and the next; c2, c3 = row lr + 8
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const int m = t * 8 + (lane & 3) * 2;
        part[warp][m][lr] = acc[t][0];
        part[warp][m + 1][lr] = acc[t][1];
        part[warp][m][lr + 8] = acc[t][2];
        part[warp][m + 1][lr + 8] = acc[t][3];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < NT * 8 * SK_ROWS; e += SK_THREADS) {
        const int m = e / SK_ROWS, r = e % SK_ROWS;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) v += part[w][m][r];
        mine[m][r] = v;
    }
    if (csize > 1) cluster.sync();
    else __syncthreads();
    if (crank == 0) {
        const GemmParams& g = p.e;
        for (int e = threadIdx.x; e < NT * 8 * SK_ROWS; e += SK_THREADS) {
            const int m = e / SK_ROWS, r = e % SK_ROWS, n = n0 + r;
            if (m >= M || n >= N) continue;
            float v = mine[m][r];
            for (int c = 1; c < csize; ++c) v += *cluster.map_shared_rank(&mine[m][r], c);
            v *= g.alpha;
            if (g.bias) v += ld_16<H16>(g.bias, n);
            if (g.preact) st_16<H16>(g.preact, m * g.ldpre + n, v);
            if (g.act == 1) v = gelu_tanh(v);
            else if (g.act == 2) v *= dgelu_tanh(ld_16<H16>(g.aux, m * g.ldaux + n));
            if (g.add) {
                if (g.add_fp32) v += static_cast<const float*>(g.add)[m * g.ldadd + n];
                else v += ld_16<H16>(g.add, m * g.ldadd + n);
            }
            if (g.d_fp32) static_cast<float*>(g.D)[m * g.ldd + n] = v;
            else st_16<H16>(g.D, m * g.ldd + n, v);
        }
    }
    if (csize > 1) cluster.sync();        // the leader has read this CTA's sums
}

template <bool H16, int NT, int U>
int run(const SkinnyParams& p, int tiles, int csize, cudaStream_t stream) {
    return launch::overlapped(gemm_skinny_kernel<H16, NT, U>, dim3(tiles * csize), dim3(SK_THREADS), csize, stream, p);
}

}  // namespace

// Both operands K-major, M <= 32; the arguments and the epilogue of neox_gemm_16 otherwise.
extern "C" int neox_gemm_skinny_16(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb,
                                   long long ldd, int d_fp32, const void* bias, const void* add, long long ldadd,
                                   int add_fp32, void* preact, long long ldpre, const void* aux, long long ldaux, int act,
                                   float alpha, int h16, void* stream_) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if (M > SK_MAX_M || K % 8) return NEOX_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda % 8) || (ldb % 8))
        return NEOX_ERR_ALIGN;
    SkinnyParams p;
    p.X = A; p.W = B; p.ldx = lda; p.ldw = ldb;
    GemmParams& e = p.e;
    e.M = M; e.N = N; e.K = K; e.a_mn = e.b_mn = 0;
    e.D = D; e.ldd = ldd; e.d_fp32 = d_fp32;
    e.bias = static_cast<const __nv_bfloat16*>(bias);
    e.add = add; e.ldadd = ldadd; e.add_fp32 = add_fp32;
    e.preact = static_cast<__nv_bfloat16*>(preact); e.ldpre = ldpre;
    e.aux = static_cast<const __nv_bfloat16*>(aux); e.ldaux = ldaux;
    e.act = act; e.alpha = alpha; e.vec_ok = 0; e.status = nullptr; e.row_ptrs = nullptr;
    const int tiles = (N + SK_ROWS - 1) / SK_ROWS, nblk = (K + SK_BK - 1) / SK_BK;
    // Split K over a cluster while one wave still holds them all and no warp runs out of k-blocks.  (Counting four CTAs an SM also
    // for more than 16 rows made two waves of some products: 17 rows 2048 x 2048 9.3 us against 5.6, 2048 x 8192 16.8 / 13.3.)
    const int wave = resident_ctas(M <= 8 ? 1 : M <= 16 ? 2 : 4) * neox_sm_count();
    int csize = 1;
    while (csize < 8 && tiles * csize * 2 <= wave && nblk >= 2 * csize * SK_WARPS) csize *= 2;
    cudaStream_t s = static_cast<cudaStream_t>(stream_);
#define SK_LAUNCH(H)                                                  \
    return M <= 8    ? run<H, 1, 2>(p, tiles, csize, s)            \
           : M <= 16 ? run<H, 2, 1>(p, tiles, csize, s)            \
                     : run<H, 4, 1>(p, tiles, csize, s)
    if (h16) SK_LAUNCH(true);
    SK_LAUNCH(false);
#undef SK_LAUNCH
}

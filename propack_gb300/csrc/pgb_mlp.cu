// pgb_mlp.cu -- the learned start vector: a row-wise MLP that stands in for
// dgetu0's random start (double/dgetu0.F:11-89) on families of related
// matrices.  No reference counterpart; the random start stays the fallback.
//
// Per row i of A the network reads MLP_IN features
//   f0 = log1p(nnz of row i) / 4,
//   f1 = ||y_i|| / rho,  f2..f17 = 2 y_i / rho,
// where y = A Omega is a 16-column Gaussian sketch (Omega from a counter-based
// generator, so the sketch is reproducible) and rho the RMS of ||y_i||; it
// outputs one entry of the start vector u0:
//   h1 = relu(W1 f + b1), h2 = relu(W2 h1 + b2), u0_i = w3 . h2 + b3
// (18 -> 256 -> 256 -> 1).  Weights are held in FP32 (Adam master copy) and
// used as BF16; every product accumulates in FP32.  The 256 x 256 layer runs
// on the 5th-generation tensor cores (tcgen05.mma, FP32 accumulators in
// tensor memory), forward and backward through its input; the mma.sync
// kernel it replaced stays selectable (propack_mlp_set_impl) as the
// reference implementation.
//
// Training (propack_mlp_train_step) minimises, for a matrix whose leading k
// left singular vectors U are known,
//   L(u0) = -(1/k) sum_j log(c_j^2 + eps ||u0||^2 / k) + log ||u0||^2,
//   c = U' u0,
// which is small when u0 lies in span(U) with every c_j of similar size, the
// property that makes every wanted Ritz value converge early.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <map>
#include <vector>

#include <atomic>

#include "../../include/propack_gb300.h"
#include "pgb.cuh"
#include "pgb_spmv.cuh"
#include "pgb_tc.cuh"

namespace pgb {

constexpr int MLP_IN = 18, MLP_H = 256, MLP_SK = 16;
constexpr int OW1 = 0, OB1 = OW1 + MLP_H * MLP_IN, OW2 = OB1 + MLP_H, OB2 = OW2 + MLP_H * MLP_H,
              OW3 = OB2 + MLP_H, OB3 = OW3 + MLP_H, MLP_NP = OB3 + 1;
constexpr int W2S = MLP_H + 8;  // padded row stride of the BF16 W2 copies in shared memory
constexpr double MLP_EPS = 1e-4;
constexpr int64_t MLP_OM_KEPT = 1 << 23;  // sketch numbers that a model holds between calls (64 MB)
constexpr int MLP_LOSS_AT = 4095;  // the loss in the coefficient array (k <= 4000)

typedef __nv_bfloat16 bf16;

struct Mlp {
    float *p = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;  // MLP_NP each
    bf16 *W1b = nullptr, *W2b = nullptr, *W2Tb = nullptr, *w3b = nullptr;
    int64_t step = 0;
    int cap = 0;
    int64_t ucap = 0, omcap = 0;
    float *F = nullptr, *out = nullptr, *gout = nullptr, *D1 = nullptr;
    bf16 *H1 = nullptr, *H2 = nullptr, *D2 = nullptr;
    double *Y = nullptr, *om = nullptr, *U = nullptr, *red = nullptr, *coef = nullptr;
    float *part = nullptr;  // per-CTA partial sums of the reductions
    int *err = nullptr;     // set by the tensor-core kernel when a bounded wait runs out
    int device = 0;
    cudaStream_t s = nullptr, s2 = nullptr;  // s2: uploads of U
    cudaEvent_t ev = nullptr;
};

// ------------------------------------------------------------- helpers
__device__ __forceinline__ unsigned long long mix64(unsigned long long z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
// Omega(j, c): standard normal from two counter-based uniforms (Box-Muller),
// row-major n x MLP_SK, so that one entry of A meets its 16 numbers in one
// 128-byte line.  Bound by the FP64 pipe (log, sqrt and cospi of every
// element; 105 us of it at n = 50,000).
__global__ void k_mlp_omega(int n, unsigned long long seed, double *om)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)n * MLP_SK;
         t += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(t / MLP_SK), col = (int)(t % MLP_SK);
        const unsigned long long a = mix64(seed ^ mix64(((unsigned long long)col << 40) ^ (unsigned long long)j));
        const unsigned long long b = mix64(a);
        const double u1 = ((double)(a >> 11) + 0.5) * (1.0 / 9007199254740992.0);
        const double u2 = (double)(b >> 11) * (1.0 / 9007199254740992.0);
        om[t] = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
    }
}

// sum over entries e0 .. e1 of val[e] X[idx[e]][c] by a half warp (lane c of
// 16); columns from n0 on read the rows of Z
constexpr int SK_UNROLL = 4;
__device__ __forceinline__ double sketch_sum(const int *__restrict__ idx, const double *__restrict__ val, int e0,
                                             int e1, int step, int n0, const double *X, const double *Z, int c)
{
    double acc = 0.0;
    int e = e0;
    for (; e + (SK_UNROLL - 1) * step < e1; e += SK_UNROLL * step) {
        int ci[SK_UNROLL];
        double v[SK_UNROLL], x[SK_UNROLL];
#pragma unroll
        for (int u = 0; u < SK_UNROLL; u++) { ci[u] = idx[e + u * step]; v[u] = val[e + u * step]; }
#pragma unroll
        for (int u = 0; u < SK_UNROLL; u++)
            x[u] = ci[u] < n0 ? X[(size_t)ci[u] * MLP_SK + c] : Z[(size_t)(ci[u] - n0) * MLP_SK + c];
#pragma unroll
        for (int u = 0; u < SK_UNROLL; u++) acc = fma(v[u], x[u], acc);
    }
    for (; e < e1; e += step) {
        const int ci = idx[e];
        acc = fma(val[e], ci < n0 ? X[(size_t)ci * MLP_SK + c] : Z[(size_t)(ci - n0) * MLP_SK + c], acc);
    }
    return acc;
}

// Z = diag(w) R' Omega (r x MLP_SK): a warp per segment of `seg` entries of a
// row of Th = R' (its halves take alternate entries); the warp that
// completes a row adds its partials in order.  zpart: rows * nseg * MLP_SK,
// tick: rows zeroed counters, left zeroed.  seg is as short as it takes to
// give every resident warp a segment (64 at least, 512 at most): a segment's
// entries are a chain of gathers.
__global__ void __launch_bounds__(256) k_mlp_thin(Csr Th, const double *om, const double *w, int seg, int nseg,
                                                  double *zpart, double *Z, unsigned int *tick)
{
    const unsigned F = 0xffffffffu;
    const int lane = threadIdx.x & 31, h = lane >> 4, c = lane & 15;
    const int nw = gridDim.x * 8;
    for (int t = blockIdx.x * 8 + (threadIdx.x >> 5); t < Th.rows * nseg; t += nw) {
        const int row = t / nseg, sg = t % nseg;
        const int p0 = Th.ptr[row], p1 = Th.ptr[row + 1];
        const int used = max(1, (p1 - p0 + seg - 1) / seg);
        if (sg >= used) continue;
        const int e0 = p0 + sg * seg;
        double acc = sketch_sum(Th.idx, Th.val, e0 + h, min(p1, e0 + seg), 2, INT_MAX, om, nullptr, c);
        acc += __shfl_xor_sync(F, acc, 16);
        if (h == 0) zpart[(size_t)t * MLP_SK + c] = acc;
        __threadfence();
        __syncwarp();
        unsigned old = 0;
        if (lane == 0) old = atomicAdd(tick + row, 1u);
        if (__shfl_sync(F, old, 0) + 1 == (unsigned)used) {
            __threadfence();
            double s0 = 0.0, s1 = 0.0;
            int q = h;
            for (; q + 2 < used; q += 4) {
                s0 += __ldcg(zpart + ((size_t)row * nseg + q) * MLP_SK + c);
                s1 += __ldcg(zpart + ((size_t)row * nseg + q + 2) * MLP_SK + c);
            }
            if (q < used) s0 += __ldcg(zpart + ((size_t)row * nseg + q) * MLP_SK + c);
            double s = s0 + s1;
            s += __shfl_xor_sync(F, s, 16);
            if (h == 0) Z[(size_t)row * MLP_SK + c] = w[row] * s;
            if (lane == 0) tick[row] = 0u;
        }
    }
}

// Y = A Omega (row-major m x MLP_SK) in one pass over A, a half warp per row
// and column c per lane, and the CTAs' partial sums of ||y_i||^2.  As sixteen
// products by one column each it read A sixteen times behind 48 launches (830
// us at 200,000 x 50,000 with 14 entries per row, 500 us at a quarter of it).
// Bound by the FP64 pipe: one FMA per entry and column.
// Rows longer than SK_LONG are left to the whole CTA (its half warps take every
// 16th entry), so that no half warp walks one alone; the CTA takes its long
// rows in the order of their index, so that Y and the sums of squares are the
// same bits on every call.  Rows are dealt round-robin, so that few long rows
// reach all CTAs.
constexpr int SK_LONG = 256;
__global__ void __launch_bounds__(256, 8) k_mlp_sketch(Csr A, const double *om, const double *Z, double *Y,
                                                    double *part)
{
    __shared__ double buf[256];
    __shared__ unsigned longs[8];
    const int c = threadIdx.x & 15, hw = threadIdx.x >> 4, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double sq = 0.0;
    int seen = 0;
    for (long long rr = blockIdx.x + (long long)gridDim.x * hw; rr < A.rows; rr += (long long)gridDim.x * 16) {
        const int r = (int)rr, e0 = A.ptr[r], e1 = A.ptr[r + 1];
        if (e1 - e0 > SK_LONG) {
            seen = 1;
            continue;
        }
        const double y = sketch_sum(A.idx, A.val, e0, e1, 1, A.ncol0, om, Z, c);
        Y[(size_t)r * MLP_SK + c] = y;
        sq = fma(y, y, sq);
    }
    if (__syncthreads_or(seen)) {
        // the CTA's rows, 256 at a time: bit l of longs[w] marks the long ones
        for (long long base = blockIdx.x; base < A.rows; base += (long long)gridDim.x * 256) {
            const long long rr = base + (long long)gridDim.x * threadIdx.x;
            const bool lg = rr < A.rows && A.ptr[rr + 1] - A.ptr[rr] > SK_LONG;
            const unsigned bits = __ballot_sync(0xffffffffu, lg);
            if (lane == 0) longs[w] = bits;
            __syncthreads();
            for (int q = 0; q < 8; q++)
                for (unsigned mask = longs[q]; mask; mask &= mask - 1) {
                    const int r = (int)(base + (long long)gridDim.x * (32 * q + __ffs(mask) - 1));
                    double y = sketch_sum(A.idx, A.val, A.ptr[r] + hw, A.ptr[r + 1], 16, A.ncol0, om, Z, c);
                    y += __shfl_xor_sync(0xffffffffu, y, 16);
                    if (lane < 16) buf[16 * w + c] = y;
                    __syncthreads();
                    if (hw == 0) {
                        y = buf[c];
                        for (int i = 1; i < 8; i++) y += buf[16 * i + c];
                        Y[(size_t)r * MLP_SK + c] = y;
                        sq = fma(y, y, sq);
                    }
                    __syncthreads();
                }
            __syncthreads();
        }
    }
    block_sums<256, 1>({sq}, buf, {part + blockIdx.x});
}

__global__ void __launch_bounds__(256) k_mlp_features(int m, const int *rowptr, const double *Y, const double *part,
                                                      int nparts, float *F)
{
    __shared__ double buf[256], tot, irho;
    double s = 0.0;
    for (int b = threadIdx.x; b < nparts; b += 256) s += part[b];
    block_sums<256, 1>({s}, buf, {&tot});
    __syncthreads();
    if (threadIdx.x == 0) {
        double rho = sqrt(tot / (double)m);
        if (!(rho > 0.0)) rho = 1.0;
        irho = 1.0 / rho;
    }
    __syncthreads();
    const double ir = irho;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        float *f = F + (size_t)i * MLP_IN;
        const double2 *y2 = reinterpret_cast<const double2 *>(Y + (size_t)i * MLP_SK);
        double nn = 0.0;
#pragma unroll
        for (int c = 0; c < MLP_SK / 2; c++) {
            const double2 v = y2[c];
            const double a = v.x * ir, b = v.y * ir;
            nn = fma(a, a, nn);
            nn = fma(b, b, nn);
            f[2 + 2 * c] = (float)(2.0 * a);
            f[3 + 2 * c] = (float)(2.0 * b);
        }
        f[0] = (float)(log1p((double)(rowptr[i + 1] - rowptr[i])) / 4.0);
        f[1] = (float)sqrt(nn);
    }
}

// h1 = relu(W1 f + b1) as BF16, row-major m x 256: a thread holds the weights
// of two units and takes every other row of a 32-row tile of features in
// shared memory (five 16-byte broadcasts and 36 FMAs a row); as one row
// per CTA at a time it waited on a global load per 18 FMAs (186 us at 200,000
// rows).
constexpr int L1_TR = 32, L1_FS = 20;  // rows per tile, padded row of features
__global__ void __launch_bounds__(256) k_mlp_l1(int m, const float *F, const bf16 *W1b, const float *b1, bf16 *H1)
{
    __shared__ __align__(16) float f[L1_TR * L1_FS];
    const int u = threadIdx.x & 127, g = threadIdx.x >> 7;
    float w0[MLP_IN], w1[MLP_IN];
#pragma unroll
    for (int q = 0; q < MLP_IN; q++) {
        w0[q] = __bfloat162float(W1b[(2 * u) * MLP_IN + q]);
        w1[q] = __bfloat162float(W1b[(2 * u + 1) * MLP_IN + q]);
    }
    const float c0 = b1[2 * u], c1 = b1[2 * u + 1];
    for (long long i0 = (long long)blockIdx.x * L1_TR; i0 < m; i0 += (long long)gridDim.x * L1_TR) {
        const int nr = (int)min((long long)L1_TR, m - i0);
        for (int t = threadIdx.x; t < nr * MLP_IN; t += 256)
            f[(t / MLP_IN) * L1_FS + t % MLP_IN] = F[i0 * MLP_IN + t];
        __syncthreads();
        for (int r = g; r < nr; r += 2) {
            float fv[L1_FS];
#pragma unroll
            for (int q = 0; q < L1_FS / 4; q++) {
                const float4 v = *reinterpret_cast<const float4 *>(f + r * L1_FS + 4 * q);
                fv[4 * q] = v.x; fv[4 * q + 1] = v.y; fv[4 * q + 2] = v.z; fv[4 * q + 3] = v.w;
            }
            float z0 = c0, z1 = c1;
#pragma unroll
            for (int q = 0; q < MLP_IN; q++) {
                z0 = fmaf(w0[q], fv[q], z0);
                z1 = fmaf(w1[q], fv[q], z1);
            }
            __nv_bfloat162 h;
            h.x = __float2bfloat16_rn(fmaxf(z0, 0.f));
            h.y = __float2bfloat16_rn(fmaxf(z1, 0.f));
            *reinterpret_cast<__nv_bfloat162 *>(H1 + (i0 + r) * MLP_H + 2 * u) = h;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void mma16816(float c[4], const unsigned a[4], unsigned b0, unsigned b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Z = X Wt' (X: m x 256 BF16 row-major; Wt: 256 x 256 BF16 [n][k]) on the
// tensor cores, one warp per 16 rows and all 256 columns.  MODE 0 (forward
// layer 2): out = bf16(relu(Z + bias)) -> Ob.  MODE 1 (backward through
// layer 2): out = Z * (mask > 0) -> Of (FP32), mask = H1.
template <int MODE>
__global__ void __launch_bounds__(256) k_mlp_mm(int m, const bf16 *X, const bf16 *Wt, const float *bias,
                                               const bf16 *mask, bf16 *Ob, float *Of)
{
    extern __shared__ __align__(16) unsigned short wsm[];  // 256 x W2S
    for (int t = threadIdx.x; t < MLP_H * MLP_H / 2; t += blockDim.x) {
        const int n = t / (MLP_H / 2), k2 = t % (MLP_H / 2);
        reinterpret_cast<unsigned *>(wsm)[(n * W2S) / 2 + k2] = reinterpret_cast<const unsigned *>(Wt)[t];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int nw = blockDim.x / 32;
    for (int r0 = (blockIdx.x * nw + (threadIdx.x >> 5)) * 16; r0 < m; r0 += gridDim.x * nw * 16) {
        const int ra = r0 + gid, rb = ra + 8;
        float acc[32][4];
#pragma unroll
        for (int t = 0; t < 32; t++) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
        for (int k0 = 0; k0 < MLP_H; k0 += 16) {
            unsigned a[4];
            const unsigned *xa = reinterpret_cast<const unsigned *>(X + (size_t)ra * MLP_H + k0 + 2 * tig);
            const unsigned *xb = reinterpret_cast<const unsigned *>(X + (size_t)rb * MLP_H + k0 + 2 * tig);
            a[0] = ra < m ? xa[0] : 0u;
            a[1] = rb < m ? xb[0] : 0u;
            a[2] = ra < m ? xa[4] : 0u;
            a[3] = rb < m ? xb[4] : 0u;
#pragma unroll
            for (int t = 0; t < 32; t++) {
                const unsigned short *bp = wsm + (8 * t + gid) * W2S + k0 + 2 * tig;
                mma16816(acc[t], a, *reinterpret_cast<const unsigned *>(bp), *reinterpret_cast<const unsigned *>(bp + 8));
            }
        }
#pragma unroll
        for (int t = 0; t < 32; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = h ? rb : ra;
                if (r >= m) continue;
                const int c = 8 * t + 2 * tig;
                float z0 = acc[t][2 * h], z1 = acc[t][2 * h + 1];
                if (MODE == 0) {
                    z0 = fmaxf(z0 + bias[c], 0.f);
                    z1 = fmaxf(z1 + bias[c + 1], 0.f);
                    __nv_bfloat162 v;
                    v.x = __float2bfloat16_rn(z0);
                    v.y = __float2bfloat16_rn(z1);
                    *reinterpret_cast<__nv_bfloat162 *>(Ob + (size_t)r * MLP_H + c) = v;
                } else {
                    const __nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162 *>(mask + (size_t)r * MLP_H + c);
                    Of[(size_t)r * MLP_H + c] = __bfloat162float(mk.x) > 0.f ? z0 : 0.f;
                    Of[(size_t)r * MLP_H + c + 1] = __bfloat162float(mk.y) > 0.f ? z1 : 0.f;
                }
            }
    }
}

// The same product on the 5th-generation tensor cores.  A persistent CTA
// (256 threads, one per SM: 192 KB of shared memory) keeps Wt in shared
// memory in the no-swizzle K-major layout of pgb_tc.cuh (16 K steps of 256
// rows x 16 K) and takes tiles of 128 rows of X in turn: the threads write
// the tile into the same layout (two lanes per 32-byte sector of a row, so
// that the loads are whole sectors and a warp's stores take the minimum
// four wavefronts), thread 0 issues the 16 MMAs (M = 128, N = 256, K = 16,
// BF16 x BF16 -> FP32) into TMEM columns 0..255 and commits them to an
// mbarrier, and every warp reads 32 TMEM lanes (rows; lanes 32 (w mod 4)..)
// x 128 columns (half w / 4) with tcgen05.ld and applies k_mlp_mm's
// epilogue.  Every wait is bounded; one that runs out sets *err and the CTA
// stops after its MMAs in flight are done.
constexpr int TM_BM = 128, TM_N = MLP_H, TM_KSTEPS = MLP_H / 16;
constexpr int TM_ATILE = TM_BM * 16 * 2;  // 4096 bytes per K step
constexpr int TM_BTILE = TM_N * 16 * 2;   // 8192 bytes per K step
constexpr int TM_SMEM = TM_KSTEPS * (TM_ATILE + TM_BTILE) + 128;
constexpr uint32_t TM_IDESC = tc_idesc_bf16(TM_BM, TM_N);
constexpr unsigned TM_TMEM_COLS = TM_N;
constexpr long TM_WAIT_LIMIT = 1L << 22;
constexpr int TM_PRE = TM_BM * (MLP_H / 8) / 256;  // 16-byte pieces of a tile per thread
static_assert(TM_SMEM <= 227 * 1024, "shared memory");

template <int MODE>
__global__ void __launch_bounds__(256, 1) k_mlp_mm_tc(int m, const bf16 *X, const bf16 *Wt, const float *bias,
                                                      const bf16 *mask, bf16 *Ob, float *Of, int *err)
{
    extern __shared__ __align__(1024) unsigned char tm_sm[];
    const uint32_t a_s = tc_smem(tm_sm), b_s = a_s + TM_KSTEPS * TM_ATILE;
    uint64_t *bar = reinterpret_cast<uint64_t *>(tm_sm + TM_KSTEPS * (TM_ATILE + TM_BTILE));
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 1);
    int *sbad = reinterpret_cast<int *>(tslot + 1);
    const uint32_t bar_s = tc_smem(bar);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int ntiles = (m + TM_BM - 1) / TM_BM;
    if (tid == 0) {
        tc_bar_init(bar_s, 1);
        *sbad = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (w == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tslot)),
                     "r"(TM_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // Wt (256 rows n x 256 K) into shared memory, once per CTA
    for (int q = tid; q < TM_N * (MLP_H / 8); q += blockDim.x) {
        const int n = (q >> 1) & (TM_N - 1), kc = ((q >> 9) << 1) | (q & 1);
        const uint4 v = *reinterpret_cast<const uint4 *>(Wt + (size_t)n * MLP_H + kc * 8);
        tc_st16(b_s + (kc >> 1) * TM_BTILE + (n >> 3) * 256 + (kc & 1) * 128 + (n & 7) * 16, v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    int it = 0;
    bool bad = false;
    // a tile of X in registers (rows past m read as zeros): the next tile's
    // loads are in flight while this tile's MMAs and epilogue run
    uint4 pre[TM_PRE];
    auto fetch = [&](int tile) {
#pragma unroll
        for (int i = 0; i < TM_PRE; i++) {
            const int q = tid + 256 * i;
            const int r = (q >> 1) & (TM_BM - 1), kc = ((q >> 8) << 1) | (q & 1);
            const long long row = (long long)tile * TM_BM + r;
            pre[i] = make_uint4(0u, 0u, 0u, 0u);
            if (row < m) pre[i] = *reinterpret_cast<const uint4 *>(X + row * MLP_H + kc * 8);
        }
    };
    if ((int)blockIdx.x < ntiles) fetch(blockIdx.x);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, it++) {
        const int row0 = t * TM_BM;
#pragma unroll
        for (int i = 0; i < TM_PRE; i++) {
            const int q = tid + 256 * i;
            const int r = (q >> 1) & (TM_BM - 1), kc = ((q >> 8) << 1) | (q & 1);
            tc_st16(a_s + (kc >> 1) * TM_ATILE + (r >> 3) * 256 + (kc & 1) * 128 + (r & 7) * 16, pre[i]);
        }
        tc_fence_proxy();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < TM_KSTEPS; ks++)
                tc_mma(tmem, tc_desc(a_s + ks * TM_ATILE), tc_desc(b_s + ks * TM_BTILE), TM_IDESC, ks > 0 ? 1u : 0u);
            tc_commit(bar_s);
        }
        if (t + (int)gridDim.x < ntiles) fetch(t + gridDim.x);
        const bool ok = tc_bar_wait(bar_s, (unsigned)(it & 1), TM_WAIT_LIMIT);
        if (__syncthreads_or(!ok)) {
            bad = true;
            break;
        }
        tc_fence_after();
        {
            const int L = 32 * (w & 3), cb = (w >> 2) * (TM_N / 2);
            const int row = row0 + L + lane;
#pragma unroll 1
            for (int cc = 0; cc < TM_N / 2; cc += 8) {
                uint32_t v[8];
                tc_ld8(tmem + ((uint32_t)L << 16) + (uint32_t)(cb + cc), v);
                tc_wait_ld();
                if (row >= m) continue;
                const int c = cb + cc;
                if (MODE == 0) {
                    uint32_t pk[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float z0 = fmaxf(__uint_as_float(v[2 * j]) + bias[c + 2 * j], 0.f);
                        const float z1 = fmaxf(__uint_as_float(v[2 * j + 1]) + bias[c + 2 * j + 1], 0.f);
                        __nv_bfloat162 h;
                        h.x = __float2bfloat16_rn(z0);
                        h.y = __float2bfloat16_rn(z1);
                        pk[j] = *reinterpret_cast<uint32_t *>(&h);
                    }
                    *reinterpret_cast<uint4 *>(Ob + (size_t)row * MLP_H + c) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                } else {
                    const uint4 mk = *reinterpret_cast<const uint4 *>(mask + (size_t)row * MLP_H + c);
                    const uint32_t mw[4] = {mk.x, mk.y, mk.z, mk.w};
                    float o[8];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&mw[j]);
                        o[2 * j] = __bfloat162float(h.x) > 0.f ? __uint_as_float(v[2 * j]) : 0.f;
                        o[2 * j + 1] = __bfloat162float(h.y) > 0.f ? __uint_as_float(v[2 * j + 1]) : 0.f;
                    }
                    float4 *dst = reinterpret_cast<float4 *>(Of + (size_t)row * MLP_H + c);
                    dst[0] = make_float4(o[0], o[1], o[2], o[3]);
                    dst[1] = make_float4(o[4], o[5], o[6], o[7]);
                }
            }
        }
        // the TMEM reads are done before the next tile's MMAs overwrite the
        // accumulators, and the MMAs before the next tile's X overwrites A
        tc_fence_before();
        __syncthreads();
    }
    if (bad) {
        if (tid == 0) atomicExch(err, 1);
        tc_bar_wait(bar_s, (unsigned)(it & 1), TM_WAIT_LIMIT);  // the MMAs in flight (bounded)
    }
    tc_fence_before();
    __syncthreads();
    if (w == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TM_TMEM_COLS) : "memory");
}

// u0_i = w3 . h2_i + b3, one warp per row
__global__ void k_mlp_l3(int m, const bf16 *H2, const bf16 *w3b, const float *b3, float *out)
{
    const int lane = threadIdx.x & 31;
    for (int i = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); i < m; i += gridDim.x * (blockDim.x / 32)) {
        float s = 0.f;
        for (int j = lane; j < MLP_H; j += 32) s = fmaf(__bfloat162float(w3b[j]), __bfloat162float(H2[(size_t)i * MLP_H + j]), s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[i] = s + b3[0];
    }
}

// partials of c = U' u0 (k values) and ||u0||^2 (column k): a warp per column
// and row segment, part[seg * (k+1) + j].  A block reduction per column had
// cost more than the columns (131 us for the 51 MB of 200,000 x 32).
__global__ void __launch_bounds__(256) k_mlp_proj(int m, int k, int nseg, const double *U, const float *out,
                                                  double *part)
{
    const int lane = threadIdx.x & 31, nw = gridDim.x * 8;
    const int len = (m + nseg - 1) / nseg;
    for (int t = blockIdx.x * 8 + (threadIdx.x >> 5); t < (k + 1) * nseg; t += nw) {
        const int j = t % (k + 1), sg = t / (k + 1);
        const long long i0 = (long long)sg * len, i1 = min((long long)m, i0 + len);
        const double *u = U + (size_t)min(j, k - 1) * m;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        long long i = i0 + lane;
        for (; i + 96 < i1; i += 128) {
            const double o0 = out[i], o1 = out[i + 32], o2 = out[i + 64], o3 = out[i + 96];
            s0 = fma(j < k ? u[i] : o0, o0, s0);
            s1 = fma(j < k ? u[i + 32] : o1, o1, s1);
            s2 = fma(j < k ? u[i + 64] : o2, o2, s2);
            s3 = fma(j < k ? u[i + 96] : o3, o3, s3);
        }
        for (; i < i1; i += 32) {
            const double o = out[i];
            s0 = fma(j < k ? u[i] : o, o, s0);
        }
        const double s = warp_sum((s0 + s1) + (s2 + s3));
        if (lane == 0) part[t] = s;
    }
}

// c, the loss and the coefficients of dL/du0 from the partials; one CTA.
// L = log ||u0||^2 - (1/k) sum_j log(c_j^2 + eps), eps = MLP_EPS ||u0||^2 / k:
// coef_j multiplies U_j, coef_k multiplies u0.
__global__ void __launch_bounds__(256) k_mlp_coef(int k, int nseg, const double *part, double *coef, double *loss)
{
    __shared__ double buf[512], tot[2], nrm;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // column k first: the others need eps
    if (w == 0) {
        double s = 0.0;
        for (int q = lane; q < nseg; q += 32) s += part[(size_t)q * (k + 1) + k];
        s = warp_sum(s);
        if (lane == 0) nrm = fmax(s, 1e-300);
    }
    __syncthreads();
    const double nrm2 = nrm, eps = MLP_EPS * nrm2 / k;
    double lg = 0.0, rec = 0.0;
    for (int j = w; j < k; j += 8) {
        double s = 0.0;
        for (int q = lane; q < nseg; q += 32) s += part[(size_t)q * (k + 1) + j];
        s = warp_sum(s);
        if (lane == 0) {
            const double d = s * s + eps;
            coef[j] = -2.0 * s / (d * k);
            lg += log(d);
            rec += (MLP_EPS / k) / d;
        }
    }
    block_sums<256, 2>({lg, rec}, buf, {tot, tot + 1});
    __syncthreads();
    if (threadIdx.x == 0) {
        coef[k] = 2.0 / nrm2 - 2.0 * tot[1] / k;
        *loss = log(nrm2) - tot[0] / k;
    }
}

// dL/du0_i = sum_j U_ij coef_j + coef_k u0_i
__global__ void k_mlp_gout(int m, int k, const double *U, const double *coef, const float *out, float *g)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        double s = coef[k] * (double)out[i];
        for (int j = 0; j < k; j++) s = fma(U[(size_t)j * m + i], coef[j], s);
        g[i] = (float)s;
    }
}

// layer 3 backward: D2 = bf16(g w3 [h2 > 0]) and partials of dw3, db2 (the
// column sums of D2) and db3: a thread takes two units of every other row of
// the CTA, four rows in flight.  part[b * B3_N]: dw3, db2, db3.
constexpr int B3_N = 2 * MLP_H + 1, B3_UNROLL = 4;
__global__ void __launch_bounds__(256) k_mlp_b3(int m, const float *g, const bf16 *H2, const bf16 *w3b, bf16 *D2,
                                                float *part)
{
    __shared__ float red[128][5];
    const int u = threadIdx.x & 127, gr = threadIdx.x >> 7;
    const float w0 = __bfloat162float(w3b[2 * u]), w1 = __bfloat162float(w3b[2 * u + 1]);
    float a0 = 0.f, a1 = 0.f, d0 = 0.f, d1 = 0.f, db = 0.f;
    const long long st = 2LL * gridDim.x;
    auto one = [&](long long i, float gi, __nv_bfloat162 h) {
        const float h0 = __bfloat162float(h.x), h1 = __bfloat162float(h.y);
        a0 = fmaf(gi, h0, a0);
        a1 = fmaf(gi, h1, a1);
        __nv_bfloat162 d;
        d.x = __float2bfloat16_rn(h0 > 0.f ? gi * w0 : 0.f);
        d.y = __float2bfloat16_rn(h1 > 0.f ? gi * w1 : 0.f);
        d0 += __bfloat162float(d.x);
        d1 += __bfloat162float(d.y);
        db += gi;
        *reinterpret_cast<__nv_bfloat162 *>(D2 + i * MLP_H + 2 * u) = d;
    };
    long long i = 2LL * blockIdx.x + gr;
    for (; i + (B3_UNROLL - 1) * st < m; i += B3_UNROLL * st) {
        float gi[B3_UNROLL];
        __nv_bfloat162 h[B3_UNROLL];
#pragma unroll
        for (int q = 0; q < B3_UNROLL; q++) {
            gi[q] = g[i + q * st];
            h[q] = *reinterpret_cast<const __nv_bfloat162 *>(H2 + (i + q * st) * MLP_H + 2 * u);
        }
#pragma unroll
        for (int q = 0; q < B3_UNROLL; q++) one(i + q * st, gi[q], h[q]);
    }
    for (; i < m; i += st) one(i, g[i], *reinterpret_cast<const __nv_bfloat162 *>(H2 + i * MLP_H + 2 * u));
    if (gr == 1) { red[u][0] = a0; red[u][1] = a1; red[u][2] = d0; red[u][3] = d1; red[u][4] = db; }
    __syncthreads();
    if (gr == 0) {
        float *P = part + (size_t)blockIdx.x * B3_N;
        P[2 * u] = a0 + red[u][0];
        P[2 * u + 1] = a1 + red[u][1];
        P[MLP_H + 2 * u] = d0 + red[u][2];
        P[MLP_H + 2 * u + 1] = d1 + red[u][3];
        if (u == 0) P[2 * MLP_H] = db + red[u][4];
    }
}

// dW2 = D2' H1 (256 x 256, summed over rows) on the tensor cores: CTA (tile,
// chunk) owns a 128 x 128 block over one row chunk, its eight warps 64 x 32
// each (mma.sync m16n8k16, BF16 products, FP32 accumulation).  Both operands
// are row-major with the rows as K, so ldmatrix.trans hands the fragments out;
// stages of 32 rows arrive by cp.async, three in flight.  The accumulators are
// added into a second set every DW_FLUSH rows, so that no sum passes through
// more than a few MMAs of the unit's own rounding.  Partials per chunk.  On
// FP32 FMAs the product had taken 1075 us at 200,000 rows.
constexpr int DW_TR = 32, DW_LD = 128 + 8, DW_STAGES = 3, DW_FLUSH = 64;
constexpr int DW_SMEM = DW_STAGES * 2 * DW_TR * DW_LD * 2;
__global__ void __launch_bounds__(256, 1) k_mlp_dw2(int m, int chunk, const bf16 *D2, const bf16 *H1, float *part)
{
    extern __shared__ __align__(16) unsigned short dws[];
    const int tj = (blockIdx.x >> 1) * 128, tl = (blockIdx.x & 1) * 128;
    const long long i0 = (long long)blockIdx.y * chunk, i1 = min((long long)m, i0 + chunk);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int wj = (w & 1) * 64, wl = (w >> 1) * 32;
    const uint32_t base = tc_smem(dws);
    const int nst = i1 > i0 ? (int)((i1 - i0 + DW_TR - 1) / DW_TR) : 0;
    // stage s: D2 rows [DW_TR][DW_LD], then H1 rows; rows past i1 are zeros
    auto issue = [&](int s) {
        if (s < nst) {
            const uint32_t st = base + (uint32_t)(s % DW_STAGES) * (2 * DW_TR * DW_LD * 2);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int t = tid + 256 * q;  // 2 operands x 32 rows x 16 pieces
                const int op = t >> 9, r = (t >> 4) & 31, c = t & 15;
                const long long i = i0 + (long long)s * DW_TR + r;
                const bf16 *src = (op ? H1 : D2) + (i < i1 ? i : i0) * MLP_H + (op ? tl : tj) + c * 8;
                const uint32_t dst = st + (uint32_t)(op * DW_TR * DW_LD + r * DW_LD + c * 8) * 2;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(i < i1 ? 16 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[4][4][4], tot[4][4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[a][b][q] = tot[a][b][q] = 0.f;
    auto flush = [&]() {
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    tot[a][b][q] += acc[a][b][q];
                    acc[a][b][q] = 0.f;
                }
    };
    auto ldm = [](uint32_t (&v)[4], uint32_t at) {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                     : "r"(at)
                     : "memory");
    };
    const int mt = lane >> 3, mr = lane & 7;
    for (int s = 0; s < DW_STAGES - 1; s++) issue(s);
    for (int s = 0; s < nst; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DW_STAGES - 2) : "memory");
        __syncthreads();  // stage s has arrived, stage s - 1 has been read by all
        issue(s + DW_STAGES - 1);
        const uint32_t st = base + (uint32_t)(s % DW_STAGES) * (2 * DW_TR * DW_LD * 2), sh = st + DW_TR * DW_LD * 2;
#pragma unroll
        for (int k0 = 0; k0 < DW_TR; k0 += 16) {
            uint32_t bf[2][4];
#pragma unroll
            for (int b = 0; b < 2; b++)
                ldm(bf[b], sh + (uint32_t)((k0 + (mt & 1) * 8 + mr) * DW_LD + wl + 16 * b + (mt >> 1) * 8) * 2);
#pragma unroll
            for (int a = 0; a < 4; a++) {
                uint32_t af[4];
                ldm(af, st + (uint32_t)((k0 + (mt >> 1) * 8 + mr) * DW_LD + wj + 16 * a + (mt & 1) * 8) * 2);
#pragma unroll
                for (int b = 0; b < 4; b++) mma16816(acc[a][b], af, bf[b >> 1][2 * (b & 1)], bf[b >> 1][2 * (b & 1) + 1]);
            }
        }
        if ((s + 1) % (DW_FLUSH / DW_TR) == 0) flush();
    }
    flush();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float *P = part + (size_t)blockIdx.y * (MLP_H * MLP_H);
    const int gid = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int j = tj + wj + 16 * a + gid + 8 * h, l = tl + wl + 8 * b + 2 * tig;
                *reinterpret_cast<float2 *>(P + (size_t)j * MLP_H + l) =
                    make_float2(tot[a][b][2 * h], tot[a][b][2 * h + 1]);
            }
}

// dW1 = D1' F (256 x 18) and db1 = sum D1: thread = unit, tiles of 32 rows of
// features in shared memory, eight rows of D1 in flight; partials per CTA
__global__ void __launch_bounds__(MLP_H) k_mlp_dw1(int m, const float *D1, const float *F, float *part)
{
    __shared__ __align__(16) float f[L1_TR * L1_FS];
    const int j = threadIdx.x;
    float acc[MLP_IN + 1] = {};
    for (long long i0 = (long long)blockIdx.x * L1_TR; i0 < m; i0 += (long long)gridDim.x * L1_TR) {
        const int nr = (int)min((long long)L1_TR, m - i0);
        for (int t = threadIdx.x; t < L1_TR * L1_FS; t += MLP_H) {
            const int r = t / L1_FS, q = t % L1_FS;
            f[t] = r < nr && q < MLP_IN ? F[(i0 + r) * MLP_IN + q] : 0.f;
        }
        __syncthreads();
        for (int r0 = 0; r0 < nr; r0 += 8) {
            float d[8];
#pragma unroll
            for (int q = 0; q < 8; q++) d[q] = r0 + q < nr ? D1[(i0 + r0 + q) * MLP_H + j] : 0.f;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                float fv[L1_FS];
#pragma unroll
                for (int c = 0; c < L1_FS / 4; c++) {
                    const float4 v = *reinterpret_cast<const float4 *>(f + (r0 + q) * L1_FS + 4 * c);
                    fv[4 * c] = v.x; fv[4 * c + 1] = v.y; fv[4 * c + 2] = v.z; fv[4 * c + 3] = v.w;
                }
#pragma unroll
                for (int c = 0; c < MLP_IN; c++) acc[c] = fmaf(d[q], fv[c], acc[c]);
                acc[MLP_IN] += d[q];
            }
        }
        __syncthreads();
    }
    float *P = part + (size_t)blockIdx.x * (MLP_H * (MLP_IN + 1));
#pragma unroll
    for (int q = 0; q <= MLP_IN; q++) P[(size_t)q * MLP_H + j] = acc[q];
}

// fixed-order sums of nb rows of n partials into the flat gradient: a CTA per
// 32 columns, eight row groups.  KIND 0: dw3, db2, db3; 1: dW2; 2: dW1, db1.
template <int KIND>
__global__ void __launch_bounds__(256) k_mlp_sum(int nb, int n, const float *part, float *g)
{
    __shared__ float red[8][33];
    const int c = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t = blockIdx.x * 32 + c;
    float s = 0.f;
    if (t < n)
#pragma unroll 4
        for (int b = w; b < nb; b += 8) s += part[(size_t)b * n + t];
    red[w][c] = s;
    __syncthreads();
    if (w != 0 || t >= n) return;
    for (int q = 1; q < 8; q++) s += red[q][c];
    if (KIND == 0) g[t < MLP_H ? OW3 + t : t < 2 * MLP_H ? OB2 + t - MLP_H : OB3] = s;
    else if (KIND == 1) g[OW2 + t] = s;
    else {
        const int q = t / MLP_H, j = t % MLP_H;
        g[q < MLP_IN ? OW1 + j * MLP_IN + q : OB1 + j] = s;
    }
}

// Adam (Kingma & Ba 2015) on the FP32 master copy
__global__ void k_mlp_adam(float *p, const float *g, float *m1, float *m2, float lr, float c1, float c2)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= MLP_NP) return;
    const float gt = g[t];
    const float a = 0.9f * m1[t] + 0.1f * gt;
    const float b = 0.999f * m2[t] + 0.001f * gt * gt;
    m1[t] = a;
    m2[t] = b;
    p[t] -= lr * (a / c1) / (sqrtf(b / c2) + 1e-8f);
}

// BF16 compute copies of the weights (W2 also transposed)
__global__ void k_mlp_cast(const float *p, bf16 *W1b, bf16 *W2b, bf16 *W2Tb, bf16 *w3b)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < MLP_H * MLP_IN) W1b[t] = __float2bfloat16_rn(p[OW1 + t]);
    if (t < MLP_H * MLP_H) {
        const int n = t / MLP_H, k = t % MLP_H;
        const bf16 v = __float2bfloat16_rn(p[OW2 + t]);
        W2b[t] = v;                       // [out n][in k]
        W2Tb[(size_t)k * MLP_H + n] = v;  // [in k][out n]
    }
    if (t < MLP_H) w3b[t] = __float2bfloat16_rn(p[OW3 + t]);
}

// ------------------------------------------------------------ host side
static std::mutex g_mlp_mu;
static std::map<int64_t, Mlp *> g_mlps;
static int64_t g_mlp_next = 1;

static Mlp *lookup_mlp(int64_t h)
{
    std::lock_guard<std::mutex> lk(g_mlp_mu);
    auto it = g_mlps.find(h);
    return it == g_mlps.end() ? nullptr : it->second;
}

static void mlp_reserve(Mlp &M, int m, int k)
{
    if (m > M.cap) {
        for (void *q : {(void *)M.F, (void *)M.out, (void *)M.gout, (void *)M.D1, (void *)M.H1, (void *)M.H2,
                        (void *)M.D2, (void *)M.Y})
            if (q) cudaFree(q);
        PGB_CUDA(cudaMalloc(&M.F, sizeof(float) * (size_t)m * MLP_IN));
        PGB_CUDA(cudaMalloc(&M.out, sizeof(float) * (size_t)m));
        PGB_CUDA(cudaMalloc(&M.gout, sizeof(float) * (size_t)m));
        PGB_CUDA(cudaMalloc(&M.D1, sizeof(float) * (size_t)m * MLP_H));
        PGB_CUDA(cudaMalloc(&M.H1, sizeof(bf16) * (size_t)m * MLP_H));
        PGB_CUDA(cudaMalloc(&M.H2, sizeof(bf16) * (size_t)m * MLP_H));
        PGB_CUDA(cudaMalloc(&M.D2, sizeof(bf16) * (size_t)m * MLP_H));
        PGB_CUDA(cudaMalloc(&M.Y, sizeof(double) * (size_t)m * MLP_SK));
        M.cap = m;
    }
    const size_t need = (size_t)m * (size_t)std::max(k, 1);
    if (need > (size_t)M.ucap) {
        if (M.U) cudaFree(M.U);
        PGB_CUDA(cudaMalloc(&M.U, sizeof(double) * need));
        M.ucap = (int64_t)need;
    }
}

constexpr int MLP_GRID = 608;          // CTAs of the row-parallel reductions at most
constexpr int MLP_SEGS = 64;           // row segments of the projections
constexpr int MLP_RED_GRID = 4096;     // partials that the reduction scratch holds at least
constexpr int MLP_DW2_CHUNKS = 38;     // row chunks of dW2 at most (four blocks each: one CTA per SM)

static void mlp_cast(Mlp &M)
{
    k_mlp_cast<<<(MLP_H * MLP_H + 255) / 256, 256, 0, M.s>>>(M.p, M.W1b, M.W2b, M.W2Tb, M.w3b);
    PGB_LAUNCHED();
}

// features of the operator's rows into M.F (m rows)
static void mlp_features(Mlp &M, const Operator &op, unsigned long long seed)
{
    const int m = op.m, n = op.n;
    mlp_reserve(M, m, 1);
    const int64_t nom = (int64_t)std::max(n, 1) * MLP_SK;
    // (the pool's memory where it is large, so that a wide operator's is not held
    // beside its solve; the model's up to MLP_OM_KEPT, which saves 4 of 304 us a call)
    const bool kept = nom <= MLP_OM_KEPT;
    if (kept && nom > M.omcap) {
        if (M.om) PGB_CUDA(cudaFree(M.om));
        M.om = nullptr;
        M.omcap = 0;
        PGB_CUDA(cudaMalloc(&M.om, sizeof(double) * (size_t)nom));
        M.omcap = nom;
    }
    double *om = kept ? M.om : (double *)pool_alloc(sizeof(double) * (size_t)nom, M.s);
    const int full = 8 * device_info().sms;  // CTAs of 256 threads that fit at once
    k_mlp_omega<<<std::min<int64_t>(full, (nom + 255) / 256), 256, 0, M.s>>>(n, seed, om);
    PGB_LAUNCHED();
    double *Z = nullptr, *zpart = nullptr;
    unsigned *tick = nullptr;
    if (op.r > 0) {
        const int64_t mx = (int64_t)op.thin_r.segs * NNZ_PB;  // bounds the longest row
        int64_t seg = (mx * op.thin_r.rows / (8 * (int64_t)full) + 31) / 32 * 32;
        seg = std::max<int64_t>(64, std::min<int64_t>(512, seg));
        const int nseg = (int)((mx + seg - 1) / seg), nt = op.thin_r.rows * nseg;
        Z = (double *)pool_alloc(sizeof(double) * MLP_SK * (size_t)op.r, M.s);
        zpart = (double *)pool_alloc(sizeof(double) * MLP_SK * (size_t)nt, M.s);
        tick = (unsigned *)pool_alloc(sizeof(unsigned) * (size_t)op.r, M.s);
        PGB_CUDA(cudaMemsetAsync(tick, 0, sizeof(unsigned) * (size_t)op.r, M.s));
        k_mlp_thin<<<std::max(1, std::min(full, (nt + 7) / 8)), 256, 0, M.s>>>(op.thin_r, om, op.w, (int)seg, nseg,
                                                                                         zpart, Z, tick);
        PGB_LAUNCHED();
    }
    const int64_t want = std::max<int64_t>((m + 15) / 16, std::min<int64_t>(m, op.fwd.nnz / 4096));
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>(std::min(full, MLP_RED_GRID), want));
    k_mlp_sketch<<<g, 256, 0, M.s>>>(op.fwd, om, Z, M.Y, M.red);
    PGB_LAUNCHED();
    k_mlp_features<<<std::max(1, std::min(full, (m + 255) / 256)), 256, 0, M.s>>>(m, op.fwd.ptr, M.Y, M.red, g, M.F);
    PGB_LAUNCHED();
    if (!kept) pool_free(om, M.s);
    pool_free(Z, M.s);
    pool_free(zpart, M.s);
    pool_free(tick, M.s);
}

static size_t mm_smem() { return sizeof(unsigned short) * MLP_H * W2S; }

// the 256 x 256 layer: 1 the tcgen05 kernel (default), 0 the mma.sync one
static std::atomic<int> g_mlp_impl{1};

// Z = X Wt' with the layer's epilogue (MODE 0 forward, 1 backward)
template <int MODE>
static void mlp_mm(Mlp &M, int m, const bf16 *X, const bf16 *Wt, const float *bias, const bf16 *mask, bf16 *Ob,
                   float *Of)
{
    if (g_mlp_impl.load() == 1) {
        const int g = std::max(1, std::min(device_info().sms, (m + TM_BM - 1) / TM_BM));
        k_mlp_mm_tc<MODE><<<g, 256, TM_SMEM, M.s>>>(m, X, Wt, bias, mask, Ob, Of, M.err);
    } else {
        const int g = std::min(device_info().sms, (m + 127) / 128);
        k_mlp_mm<MODE><<<g, 256, mm_smem(), M.s>>>(m, X, Wt, bias, mask, Ob, Of);
    }
    PGB_LAUNCHED();
}
// after the stream has been synchronised: a wait of the tensor-core kernel that ran out
static void mlp_check(Mlp &M)
{
    int e = 0;
    PGB_CUDA(cudaMemcpy(&e, M.err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) {
        PGB_CUDA(cudaMemsetAsync(M.err, 0, sizeof(int), M.s));
        set_error("learned start: a tensor-core wait ran out");
        throw WaitFailure();
    }
}

static void mlp_forward(Mlp &M, int m)
{
    const int g = std::max(1, std::min(4 * device_info().sms, (m + L1_TR - 1) / L1_TR));
    k_mlp_l1<<<g, 256, 0, M.s>>>(m, M.F, M.W1b, M.p + OB1, M.H1);
    PGB_LAUNCHED();
    mlp_mm<0>(M, m, M.H1, M.W2b, M.p + OB2, nullptr, M.H2, nullptr);
    k_mlp_l3<<<std::min(4096, (m + 7) / 8), 256, 0, M.s>>>(m, M.H2, M.w3b, M.p + OB3, M.out);
    PGB_LAUNCHED();
}

// flat gradient (M.g) and loss (device, M.coef[4095]) for the matrix whose
// features sit in M.F and whose leading left singular vectors (m x k,
// column-major) sit in M.U
static void mlp_backward(Mlp &M, int m, int k)
{
    const int sms = device_info().sms;
    k_mlp_proj<<<std::min(8 * sms, ((k + 1) * MLP_SEGS + 7) / 8), 256, 0, M.s>>>(m, k, MLP_SEGS, M.U, M.out, M.red);
    PGB_LAUNCHED();
    k_mlp_coef<<<1, 256, 0, M.s>>>(k, MLP_SEGS, M.red, M.coef, M.coef + MLP_LOSS_AT);
    PGB_LAUNCHED();
    k_mlp_gout<<<std::min(4096, (m + 255) / 256), 256, 0, M.s>>>(m, k, M.U, M.coef, M.out, M.gout);
    PGB_LAUNCHED();
    float *pf = reinterpret_cast<float *>(M.red);
    const int gb = std::max(1, std::min(std::min(MLP_GRID, 4 * sms), (m + 15) / 16));
    k_mlp_b3<<<gb, 256, 0, M.s>>>(m, M.gout, M.H2, M.w3b, M.D2, pf);
    PGB_LAUNCHED();
    k_mlp_sum<0><<<(B3_N + 31) / 32, 256, 0, M.s>>>(gb, B3_N, pf, M.g);
    PGB_LAUNCHED();
    // whole stages per chunk, at least a flush interval
    const int nch = std::max(1, std::min(MLP_DW2_CHUNKS, (m + DW_FLUSH - 1) / DW_FLUSH));
    const int chunk = ((m + nch - 1) / nch + DW_TR - 1) / DW_TR * DW_TR;
    k_mlp_dw2<<<dim3(4, nch), 256, DW_SMEM, M.s>>>(m, chunk, M.D2, M.H1, M.part);
    PGB_LAUNCHED();
    k_mlp_sum<1><<<MLP_H * MLP_H / 32, 256, 0, M.s>>>(nch, MLP_H * MLP_H, M.part, M.g);
    PGB_LAUNCHED();
    mlp_mm<1>(M, m, M.D2, M.W2Tb, nullptr, M.H1, nullptr, M.D1);
    const int g1 = std::max(1, std::min(std::min(MLP_GRID, 4 * sms), (m + L1_TR - 1) / L1_TR));
    k_mlp_dw1<<<g1, MLP_H, 0, M.s>>>(m, M.D1, M.F, pf);
    PGB_LAUNCHED();
    k_mlp_sum<2><<<MLP_H * (MLP_IN + 1) / 32, 256, 0, M.s>>>(g1, MLP_H * (MLP_IN + 1), pf, M.g);
    PGB_LAUNCHED();
}

// U (host, leading dimension ldu) to M.U on the copy stream, while the
// features and the forward pass run; M.s waits for it
static void mlp_upload(Mlp &M, const double *U, int ldu, int m, int k)
{
    if (ldu == m) h2d_bytes(M.U, U, sizeof(double) * (size_t)m * k, M.s2, 8);
    else
        PGB_CUDA(cudaMemcpy2DAsync(M.U, sizeof(double) * m, U, sizeof(double) * ldu, sizeof(double) * m, k,
                                   cudaMemcpyHostToDevice, M.s2));
    PGB_CUDA(cudaEventRecord(M.ev, M.s2));
    PGB_CUDA(cudaStreamWaitEvent(M.s, M.ev, 0));
}

static Operator *mlp_operator(int64_t op_handle)
{
    Operator *op = lookup_operator(op_handle);
    if (!op) {
        set_error("no live operator handle");
        throw ArgFailure();
    }
    if (op->cplx == 2) {
        set_error("the learned start takes real operators");
        throw ArgFailure();
    }
    return op;
}

}  // namespace pgb

using namespace pgb;

#define MLP_TRY(...)                        \
    try {                                   \
        __VA_ARGS__;                        \
        return 0;                           \
    } catch (const ArgFailure &) {          \
        return PROPACK_ERR_ARG;             \
    } catch (const CudaFailure &) {         \
        return PROPACK_ERR_CUDA;            \
    } catch (const WaitFailure &) {         \
        return PROPACK_ERR_WAIT;            \
    }

extern "C" int propack_mlp_create(uint64_t seed, int64_t *handle)
{
    MLP_TRY({
        if (!handle) { set_error("propack_mlp_create: null handle"); throw ArgFailure(); }
        Mlp *M = new Mlp();
        PGB_CUDA(cudaGetDevice(&M->device));
        PGB_CUDA(cudaStreamCreateWithFlags(&M->s, cudaStreamNonBlocking));
        PGB_CUDA(cudaStreamCreateWithFlags(&M->s2, cudaStreamNonBlocking));
        PGB_CUDA(cudaEventCreateWithFlags(&M->ev, cudaEventDisableTiming));
        // He-style initialisation, drawn on the host (small)
        std::vector<float> p(MLP_NP, 0.f);
        unsigned long long st = seed * 0x9E3779B97F4A7C15ull + 12345ull;
        auto nrm = [&]() {
            auto nx = [&]() {
                st = st * 6364136223846793005ull + 1442695040888963407ull;
                return ((double)(st >> 11) + 0.5) / 9007199254740992.0;
            };
            const double u1 = nx(), u2 = nx();
            return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
        };
        for (int t = 0; t < MLP_H * MLP_IN; t++) p[OW1 + t] = (float)(nrm() * std::sqrt(2.0 / MLP_IN));
        for (int t = 0; t < MLP_H * MLP_H; t++) p[OW2 + t] = (float)(nrm() * std::sqrt(2.0 / MLP_H));
        for (int t = 0; t < MLP_H; t++) p[OW3 + t] = (float)(nrm() * std::sqrt(1.0 / MLP_H));
        PGB_CUDA(cudaMalloc(&M->p, sizeof(float) * MLP_NP));
        PGB_CUDA(cudaMalloc(&M->g, sizeof(float) * MLP_NP));
        PGB_CUDA(cudaMalloc(&M->m1, sizeof(float) * MLP_NP));
        PGB_CUDA(cudaMalloc(&M->m2, sizeof(float) * MLP_NP));
        PGB_CUDA(cudaMemcpyAsync(M->p, p.data(), sizeof(float) * MLP_NP, cudaMemcpyHostToDevice, M->s));
        PGB_CUDA(cudaMemsetAsync(M->g, 0, sizeof(float) * MLP_NP, M->s));
        PGB_CUDA(cudaMemsetAsync(M->m1, 0, sizeof(float) * MLP_NP, M->s));
        PGB_CUDA(cudaMemsetAsync(M->m2, 0, sizeof(float) * MLP_NP, M->s));
        PGB_CUDA(cudaMalloc(&M->W1b, sizeof(bf16) * MLP_H * MLP_IN));
        PGB_CUDA(cudaMalloc(&M->W2b, sizeof(bf16) * MLP_H * MLP_H));
        PGB_CUDA(cudaMalloc(&M->W2Tb, sizeof(bf16) * MLP_H * MLP_H));
        PGB_CUDA(cudaMalloc(&M->w3b, sizeof(bf16) * MLP_H));
        const size_t red = std::max<size_t>((size_t)MLP_GRID * (MLP_H * (MLP_IN + 1)) * sizeof(float),
                                            (size_t)MLP_SEGS * 4096 * sizeof(double));
        PGB_CUDA(cudaMalloc(&M->red, red));
        PGB_CUDA(cudaMalloc(&M->coef, sizeof(double) * 4096));
        PGB_CUDA(cudaMalloc(&M->part, sizeof(float) * (size_t)MLP_DW2_CHUNKS * (MLP_H * MLP_H)));
        PGB_CUDA(cudaFuncSetAttribute(k_mlp_mm<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mm_smem()));
        PGB_CUDA(cudaFuncSetAttribute(k_mlp_mm<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mm_smem()));
        PGB_CUDA(cudaFuncSetAttribute(k_mlp_dw2, cudaFuncAttributeMaxDynamicSharedMemorySize, DW_SMEM));
        PGB_CUDA(cudaFuncSetAttribute(k_mlp_mm_tc<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, TM_SMEM));
        PGB_CUDA(cudaFuncSetAttribute(k_mlp_mm_tc<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, TM_SMEM));
        PGB_CUDA(cudaMalloc(&M->err, sizeof(int)));
        PGB_CUDA(cudaMemsetAsync(M->err, 0, sizeof(int), M->s));
        mlp_cast(*M);
        PGB_CUDA(cudaStreamSynchronize(M->s));
        std::lock_guard<std::mutex> lk(g_mlp_mu);
        *handle = g_mlp_next++;
        g_mlps[*handle] = M;
    })
}

extern "C" int propack_mlp_destroy(int64_t handle)
{
    Mlp *M = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mlp_mu);
        auto it = g_mlps.find(handle);
        if (it == g_mlps.end()) return PROPACK_ERR_HANDLE;
        M = it->second;
        g_mlps.erase(it);
    }
    cudaStreamSynchronize(M->s);
    for (void *q : {(void *)M->p, (void *)M->g, (void *)M->m1, (void *)M->m2, (void *)M->W1b, (void *)M->W2b,
                    (void *)M->W2Tb, (void *)M->w3b, (void *)M->F, (void *)M->out, (void *)M->gout, (void *)M->D1,
                    (void *)M->H1, (void *)M->H2, (void *)M->D2, (void *)M->Y, (void *)M->om, (void *)M->U,
                    (void *)M->red, (void *)M->coef, (void *)M->part, (void *)M->err})
        if (q) cudaFree(q);
    cudaStreamDestroy(M->s);
    cudaStreamDestroy(M->s2);
    cudaEventDestroy(M->ev);
    delete M;
    return 0;
}

extern "C" int propack_mlp_params(int64_t handle, float *get, const float *set)
{
    Mlp *M = lookup_mlp(handle);
    if (!M) return PROPACK_ERR_HANDLE;
    MLP_TRY({
        if (set) {
            PGB_CUDA(cudaMemcpyAsync(M->p, set, sizeof(float) * MLP_NP, cudaMemcpyHostToDevice, M->s));
            mlp_cast(*M);
        }
        if (get) PGB_CUDA(cudaMemcpyAsync(get, M->p, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost, M->s));
        PGB_CUDA(cudaStreamSynchronize(M->s));
    })
}

extern "C" int propack_mlp_nparams(void) { return MLP_NP; }

extern "C" int propack_mlp_set_impl(int impl)
{
    if (impl != 0 && impl != 1) return PROPACK_ERR_ARG;
    g_mlp_impl.store(impl);
    return 0;
}

extern "C" int propack_mlp_features(int64_t handle, int64_t op_handle, uint64_t seed, float *F)
{
    Mlp *M = lookup_mlp(handle);
    if (!M) return PROPACK_ERR_HANDLE;
    MLP_TRY({
        const Operator *op = mlp_operator(op_handle);
        mlp_features(*M, *op, seed);
        if (F) PGB_CUDA(cudaMemcpyAsync(F, M->F, sizeof(float) * (size_t)op->m * MLP_IN, cudaMemcpyDeviceToHost, M->s));
        PGB_CUDA(cudaStreamSynchronize(M->s));
    })
}

extern "C" int propack_mlp_start(int64_t handle, int64_t op_handle, uint64_t seed, double *u0)
{
    Mlp *M = lookup_mlp(handle);
    if (!M) return PROPACK_ERR_HANDLE;
    MLP_TRY({
        if (!u0) { set_error("propack_mlp_start: null output"); throw ArgFailure(); }
        const Operator *op = mlp_operator(op_handle);
        const int m = op->m;
        mlp_features(*M, *op, seed);
        mlp_forward(*M, m);
        std::vector<float> o(m);
        PGB_CUDA(cudaMemcpyAsync(o.data(), M->out, sizeof(float) * m, cudaMemcpyDeviceToHost, M->s));
        PGB_CUDA(cudaStreamSynchronize(M->s));
        mlp_check(*M);
        for (int i = 0; i < m; i++) u0[i] = o[i];
    })
}

// gradient of the loss for (operator, U) without an update; grad: MLP_NP floats
extern "C" int propack_mlp_grad(int64_t handle, int64_t op_handle, uint64_t seed, const double *U, int ldu, int k,
                                float *grad, double *loss)
{
    Mlp *M = lookup_mlp(handle);
    if (!M) return PROPACK_ERR_HANDLE;
    MLP_TRY({
        const Operator *op = mlp_operator(op_handle);
        const int m = op->m;
        if (!U || ldu < m || k < 1 || k > 4000) { set_error("propack_mlp_grad: invalid U"); throw ArgFailure(); }
        mlp_features(*M, *op, seed);
        mlp_reserve(*M, m, k);
        mlp_forward(*M, m);
        mlp_upload(*M, U, ldu, m, k);
        mlp_backward(*M, m, k);
        double L = 0.0;
        PGB_CUDA(cudaMemcpyAsync(&L, M->coef + MLP_LOSS_AT, sizeof(double), cudaMemcpyDeviceToHost, M->s));
        if (grad) PGB_CUDA(cudaMemcpyAsync(grad, M->g, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost, M->s));
        PGB_CUDA(cudaStreamSynchronize(M->s));
        mlp_check(*M);
        if (loss) *loss = L;
    })
}

// one Adam step on (operator, U)
extern "C" int propack_mlp_train_step(int64_t handle, int64_t op_handle, uint64_t seed, const double *U, int ldu,
                                      int k, double lr, double *loss)
{
    Mlp *M = lookup_mlp(handle);
    if (!M) return PROPACK_ERR_HANDLE;
    MLP_TRY({
        const Operator *op = mlp_operator(op_handle);
        const int m = op->m;
        if (!U || ldu < m || k < 1 || k > 4000) { set_error("propack_mlp_train_step: invalid U"); throw ArgFailure(); }
        mlp_features(*M, *op, seed);
        mlp_reserve(*M, m, k);
        mlp_forward(*M, m);
        mlp_upload(*M, U, ldu, m, k);
        mlp_backward(*M, m, k);
        double L = 0.0;
        PGB_CUDA(cudaMemcpyAsync(&L, M->coef + MLP_LOSS_AT, sizeof(double), cudaMemcpyDeviceToHost, M->s));
        M->step++;
        const float c1 = 1.f - std::pow(0.9f, (float)M->step), c2 = 1.f - std::pow(0.999f, (float)M->step);
        k_mlp_adam<<<(MLP_NP + 255) / 256, 256, 0, M->s>>>(M->p, M->g, M->m1, M->m2, (float)lr, c1, c2);
        PGB_LAUNCHED();
        mlp_cast(*M);
        PGB_CUDA(cudaStreamSynchronize(M->s));
        mlp_check(*M);
        if (loss) *loss = L;
    })
}

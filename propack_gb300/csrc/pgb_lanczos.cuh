// pgb_lanczos.cuh -- device-resident steps of dlanbpro (double/dlanbpro.F:283-546).
//
// One half step (V half: alpha_j v_j = A' u_j - beta_j v_{j-1}; U half:
// beta_{j+1} u_{j+1} = A v_j - alpha_j u_j) is a sequence of phases:
//
//   spmv   fused SpMV + axpy with the previous vector + partial sums of
//          ||y||^2 and <prev, y>  (dlanbpro.F:288-296, :420-424)
//   elr    one extended-local-reorthogonalisation pass (:301-316, :429-443)
//   dots   projections of one classical Gram-Schmidt pass (dreorth.F:174)
//   upd    v -= W h and ||v||^2 (dreorth.F:85-95, dcgs :199); further passes
//          (the iterated refinement) repeat the pair
//
// The run kernel executes them for a range of half steps in one launch.  A
// phase ends at a grid barrier whose master CTA reduces the partial sums in a
// fixed order and runs the scalar logic of dlanbpro: the alpha/beta
// bookkeeping, the ||A|| estimate, the omega recurrences (dupdate_nu/mu,
// parallel over k), dcompute_int, the reorthogonalisation decision and the
// invariant-subspace test; it then says which phase comes next.  The host
// reads no scalar before the run ends.  An invariant subspace that needs a
// fresh random vector sets status = 1 and ends the run; the host finishes
// the case and resumes.
//
// dsafescal (dsafescal.F:4-55) is deferred: the new vector is left
// unscaled, the product that reads it through the operator is scaled
// instead (A(v/a) = (Av)/a), and the next same-side SpMV, which reads it
// row by row, writes the scaled value back.
#pragma once
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "pgb.cuh"
#include "pgb_f3.cuh"
#include "pgb_planes.cuh"
#include "pgb_spmv.cuh"

namespace pgb {

// The scalar state of the tails: the control block, and the arrays of the
// recurrences, in the shared memory of the CTA that runs every tail or
// (launch_run decides) in global memory.
constexpr int TAIL_WORDS = 128;  // bit words of the interval search: up to 4096 columns
struct Tail {
    LbCtl c;
    int go;
    double red[16];
    double rinv;                // 1 / alpha_j (V half), 1 / beta_j (U half) of the omega update
    double *ba, *bb, *mu, *nu;  // B and the omega recurrences
    double *hA, *hB;            // hypot(alpha_k, beta_k), hypot(alpha_k, beta_{k-1}) kept per step (may be null)
    int *index;
    unsigned big[TAIL_WORDS], small[TAIL_WORDS];  // |mu_k| > delta, |mu_k| < eta of the latest update
};

__device__ __forceinline__ Pend make_scale(double a)
{
    Pend p;
    if (fabs(a) >= SFMIN) { p.mode = 1; p.val = 1.0 / a; }
    else { p.mode = 2; p.val = a; }
    return p;
}

// ---------------------------------------------------------------- tails
// fixed-order sums of N arrays of per-CTA partials into t.red[0 .. N)
// (visible to warp 0 after the barrier here); buf: N * BS doubles
template <int N>
__device__ inline void sum_parts(const double *const (&p)[N], int nb, double *buf, Tail &t)
{
    double s[N];
    double *out[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
        s[q] = 0.0;
        out[q] = t.red + q;
    }
    for (int b = threadIdx.x; b < nb; b += BS) {
#pragma unroll
        for (int q = 0; q < N; q++) s[q] += __ldcg(p[q] + b);
    }
    block_sums<BS, N>(s, buf, out);
    __syncthreads();
}

// dset_mu (dlanbpro.F:555-577), all threads
__device__ inline void set_mu(int k, double *mu, const int *index, double val)
{
    int i = 0;
    while (index[i] <= k && index[i] > 0) {
        const int p = index[i], q = index[i + 1];
        for (int j = p + threadIdx.x; j <= q; j += BS) mu[j - 1] = val;
        i += 2;
    }
}

// dcompute_int (dlanbpro.F:581-624), thread 0.  Fortran DO-variable exit
// values are reproduced (s = lo-1 and i = j+1 when a search runs out).
__device__ inline void compute_int_serial(const double *mu, int j, double delta, double eta, int *index)
{
    int ip = 0, i = 0, k, s;
    index[0] = 0;
    while (i < j) {
        for (k = i + 1; k <= j; k++)
            if (fabs(mu[k - 1]) > delta) break;
        if (k > j) break;
        const int lo = i > 1 ? i : 1;
        for (s = k; s >= lo; s--)
            if (fabs(mu[s - 1]) < eta) break;
        index[ip++] = s + 1;
        for (i = s + 1; i <= j; i++)
            if (fabs(mu[i - 1]) < eta) break;
        index[ip++] = i - 1;
    }
    index[ip] = j + 1;
}
// the first set bit k in [from, n] (bit k-1 of the words), n + 1 if none
__device__ __forceinline__ int next_bit(const unsigned *w, int from, int n)
{
    for (int k = from; k <= n; k = ((k - 1) | 31) + 2) {
        const unsigned m = w[(k - 1) >> 5] >> ((k - 1) & 31);
        if (m) return min(k + __ffs(m) - 1, n + 1);
    }
    return n + 1;
}
// the last set bit k in [lo, from], lo - 1 if none
__device__ __forceinline__ int prev_bit(const unsigned *w, int from, int lo)
{
    for (int k = from; k >= lo; k = ((k - 1) & ~31)) {
        const unsigned m = w[(k - 1) >> 5] << (31 - ((k - 1) & 31));
        if (m) return max(k - __clz(m), lo - 1);
    }
    return lo - 1;
}
// the same over the bit words that the omega update left (a search step is
// a word instead of an element)
__device__ inline void compute_int(Tail &t, const double *mu, int j)
{
    const double delta = t.c.delta, eta = t.c.eta;
    if (delta < eta) return;
    int *index = t.index;
    if (j > 32 * TAIL_WORDS) {
        compute_int_serial(mu, j, delta, eta, index);
        return;
    }
    int ip = 0, i = 0;
    index[0] = 0;
    while (i < j) {
        const int k = next_bit(t.big, i + 1, j);
        if (k > j) break;
        const int s = prev_bit(t.small, k, i > 1 ? i : 1);
        index[ip++] = s + 1;
        i = next_bit(t.small, s + 1, j);
        index[ip++] = i - 1;
    }
    index[ip] = j + 1;
}

// expand index[] into the 0-based column list walked by dcgs (CGS) or
// dmgs (MGS stops at an empty range); all threads.  Returns the ndot count
// of one pass and the number of columns.
__device__ inline int build_sel(const int *index, int kk, int icgs, int *sel, int *nsel)
{
    int ns = 0, nd = 0, i = 0;
    while (true) {
        const int p = index[i];
        if (!(p <= kk && p > 0)) break;
        const int q = index[i + 1];
        if (!icgs && p > q) break;
        nd += q - p + 1;
        for (int c = p + threadIdx.x; c <= q; c += BS) sel[ns + c - p] = c - 1;
        if (q >= p) ns += q - p + 1;
        i += 2;
    }
    *nsel = ns;
    return nd + kk;
}

__device__ __forceinline__ double tail_hypot(double a, double b)
{
    const double q = fma(a, a, b * b);
    return q > 1e-280 && q < 1e280 ? sqrt(q) : hypot(a, b);
}
// bit words of one round of an omega update (k = k0 + threadIdx.x)
__device__ __forceinline__ void set_bits(Tail &t, int k0, bool valid, double v)
{
    const unsigned b = __ballot_sync(0xffffffffu, valid && fabs(v) > t.c.delta);
    const unsigned s = __ballot_sync(0xffffffffu, valid && fabs(v) < t.c.eta);
    const int w = ((k0 - 1) >> 5) + (threadIdx.x >> 5);
    if ((threadIdx.x & 31) == 0 && w < TAIL_WORDS) {
        t.big[w] = b;
        t.small[w] = s;
    }
}

// dupdate_nu (dlanbpro.F:684-723), all threads; j > 1
__device__ inline void update_nu_par(Tail &t, int j)
{
    const double *ba = t.ba, *bb = t.bb;
    double *mu = t.mu, *nu = t.nu;
    const double e1 = t.c.epsn2, an = t.c.anorm;
    const double aj = ba[j - 1], bjm = bb[j - 2], ra = t.rinv;
    const double hj = t.hB ? t.hB[j - 1] : tail_hypot(aj, bjm);
    double loc = 0.0;
    for (int k0 = 1; k0 <= j - 1; k0 += BS) {
        const int k = k0 + threadIdx.x;
        double v = 0.0;
        if (k <= j - 1) {
            const double h = t.hA ? t.hA[k - 1] : tail_hypot(ba[k - 1], bb[k - 1]);
            v = bb[k - 1] * mu[k] + ba[k - 1] * mu[k - 1] - bjm * nu[k - 1];
            const double d = e1 * (h + hj) + e1 * an;
            v = (v + copysign(d, v)) * ra;
            nu[k - 1] = v;
            loc = fmax(loc, fabs(v));
        }
        set_bits(t, k0, k <= j - 1, v);
    }
    const double mx = block_max_pos<BS>(loc, t.red + 8);
    if (threadIdx.x == 0) {
        nu[j - 1] = 1.0;
        t.c.numax = mx;
    }
}

// dupdate_mu (dlanbpro.F:628-679), all threads
__device__ inline void update_mu_par(Tail &t, int j)
{
    const double *ba = t.ba, *bb = t.bb;
    double *mu = t.mu;
    const double *nu = t.nu;
    const double e1 = t.c.epsn2, an = t.c.anorm;
    double loc = 0.0;
    const double aj = ba[j - 1], bj = bb[j - 1], rb = t.rinv;
    const double hj = t.hA ? t.hA[j - 1] : tail_hypot(aj, bj);
    for (int k0 = 1; k0 <= j; k0 += BS) {
        const int k = k0 + threadIdx.x;
        double v = 0.0, d;
        if (k <= j) {
            if (j == 1) {
                v = e1 / bj;
            } else {
                const double hk = k == 1 ? ba[0] : t.hB ? t.hB[k - 1] : tail_hypot(ba[k - 1], bb[k - 2]);
                if (k == 1) v = ba[0] * nu[0] - aj * mu[0];
                else if (k < j) v = ba[k - 1] * nu[k - 1] + bb[k - 2] * nu[k - 2] - aj * mu[k - 1];
                else v = bb[j - 2] * nu[j - 2];
                d = e1 * (hj + hk) + e1 * an;
                v = (v + copysign(d, v)) * rb;
            }
            mu[k - 1] = v;
            loc = fmax(loc, fabs(v));
        }
        set_bits(t, k0, k <= j, v);
    }
    const double mx = block_max_pos<BS>(loc, t.red + 8);
    if (threadIdx.x == 0) {
        mu[j] = 1.0;
        t.c.mumax = mx;
    }
}

// ---------------------------------------------------------- V half logic
__device__ inline void v_post(Tail &t, int j)
{
    if (threadIdx.x != 0) return;
    LbCtl &c = t.c;
    if (c.alpha < c.anorm * c.epsn && j < c.k) {
        c.rnorm = c.alpha;
        c.alpha = 0.0;
        c.status = 1;
        c.susp_reason = 1;
        c.susp_side = 0;
        c.susp_j = j;
        return;
    } else if (j > 1 && !c.full_reorth && j < c.k && (c.delta * c.alpha < c.anorm * c.eps_vec)) {
        c.ierr = j;
    }
    t.ba[j - 1] = c.alpha;
    if (c.alpha != 0.0) c.pend_v = make_scale(c.alpha);
    else { c.pend_v.mode = c.collapsed ? 3 : 0; c.pend_v.val = 0.0; }
    c.pend_v_col = j - 1;
}
__device__ inline void v_post_reorth(Tail &t, int j)
{
    set_mu(j - 1, t.nu, t.index, t.c.eps_vec);
    if (threadIdx.x != 0) return;
    t.c.numax = t.c.eta;
    t.c.force_reorth = !t.c.force_reorth;
}
// dlanbpro.F:340-367: nu recurrence and the reorthogonalisation decision
__device__ inline void v_reorth_decide(Tail &t, const LbArgs &a, int j)
{
    __syncthreads();
    const bool do_nu = !t.c.full_reorth && t.c.alpha != 0.0;
    if (do_nu && j > 1) update_nu_par(t, j);
    if (threadIdx.x == 0) {
        LbCtl &c = t.c;
        t.go = 4;
        c.collapsed = 0;
        if ((c.full_reorth || c.numax > c.delta || c.force_reorth) && c.alpha != 0.0) {
            if (c.full_reorth || c.eta == 0.0) {
                t.index[0] = 1; t.index[1] = j - 1; t.index[2] = j;
            } else if (!c.force_reorth) {
                compute_int(t, t.nu, j - 1);
            }
            t.go = j - 1 <= 0 ? 3 : 0;  // dreorth returns at once for k <= 0
        }
    }
    __syncthreads();
    if (t.go == 3) { v_post_reorth(t, j); v_post(t, j); }
    else if (t.go == 4) v_post(t, j);
    else {
        int ns;
        const int nd = build_sel(t.index, j - 1, t.c.icgs, a.sel, &ns);
        if (threadIdx.x == 0) {
            LbCtl &c = t.c;
            c.ndot_iter = nd;
            c.nsel = ns;
            c.reorth_active = 1;
            c.reorth_iter = 0;
            c.reorth_nrm0 = c.alpha;
        }
    }
}
// B(j,1), amax and the ||A|| estimate (dlanbpro.F:318-334), then the
// decision.  The quotients by amax are formed by four lanes of warp 0 at
// once, the three square roots by three.
__device__ inline void v_finish_alpha(Tail &t, const LbArgs &a, int j)
{
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const double alpha = t.c.alpha, amax = fmax(t.c.amax, alpha);
        const double *ba = t.ba, *bb = t.bb;
        // alpha_{j-1}, beta_{j-1}, beta_{j-2} (j > 2), alpha_j
        double q = lane == 0 ? ba[j - 2] : lane == 1 ? bb[j - 2] : lane == 2 ? (j > 2 ? bb[j - 3] : 0.0) : alpha;
        // lane 4: the reciprocal that the nu update multiplies by
        q = (lane == 4 ? 1.0 : q) / (lane == 4 ? alpha : amax);
        const double q0 = __shfl_sync(0xffffffffu, q, 0), q1 = __shfl_sync(0xffffffffu, q, 1),
                     q2 = __shfl_sync(0xffffffffu, q, 2), q3 = __shfl_sync(0xffffffffu, q, 3);
        const double r = sqrt(lane == 0 ? q0 * q0 + q1 * q1 + q0 * q2 + q3 * q1
                                        : lane == 1 ? q0 * q0 + q1 * q1 : q3 * q3 + q1 * q1);
        const double h = amax > 0.0 ? amax * r : 0.0;
        if (lane == 1 && t.hA) t.hA[j - 2] = h;
        if (lane == 2 && t.hB) t.hB[j - 1] = h;
        if (lane == 4) t.rinv = q;
        if (lane == 0) {
            t.ba[j - 1] = alpha;
            t.c.amax = amax;
            t.c.anorm = fmax(t.c.anorm, FUDGE * amax * r);
        }
    }
    v_reorth_decide(t, a, j);
}

// ---------------------------------------------------------- U half logic
__device__ inline void u_post(Tail &t, int j)
{
    if (threadIdx.x != 0) return;
    LbCtl &c = t.c;
    if (c.beta < c.anorm * c.epsn && j < c.k) {
        c.rnorm = c.beta;
        c.beta = 0.0;
        c.status = 1;
        c.susp_reason = 1;
        c.susp_side = 1;
        c.susp_j = j;
        return;
    } else if (!c.full_reorth && j < c.k && (c.delta * c.beta < c.anorm * c.eps_vec)) {
        c.ierr = j;
    }
    t.bb[j - 1] = c.beta;
    if (c.beta != 0.0 && c.beta != 1.0) c.pend_u = make_scale(c.beta);
    else { c.pend_u.mode = c.collapsed ? 3 : 0; c.pend_u.val = 0.0; }
    c.pend_u_col = j;
    c.rnorm = c.beta;
    c.j = j + 1;
}
__device__ inline void u_post_reorth(Tail &t, int j)
{
    set_mu(j, t.mu, t.index, t.c.eps_vec);
    if (threadIdx.x != 0) return;
    t.c.mumax = t.c.eta;
    t.c.force_reorth = !t.c.force_reorth;
}
// dlanbpro.F:463-498
__device__ inline void u_reorth_decide(Tail &t, const LbArgs &a, int j)
{
    __syncthreads();
    const bool do_mu = !t.c.full_reorth && t.c.beta != 0.0;
    if (do_mu) update_mu_par(t, j);
    if (threadIdx.x == 0) {
        LbCtl &c = t.c;
        t.go = 4;
        c.collapsed = 0;
        if ((c.full_reorth || c.mumax > c.delta || c.force_reorth) && c.beta != 0.0) {
            if (c.full_reorth || c.eta == 0.0) {
                t.index[0] = 1; t.index[1] = j; t.index[2] = j + 1;
            } else if (!c.force_reorth) {
                compute_int(t, t.mu, j);
            } else {
                for (int i = 0; i < 2 * j + 1; i++)
                    if (t.index[i] == j) { t.index[i] = j + 1; break; }
            }
            t.go = 0;
        }
    }
    __syncthreads();
    if (t.go == 4) u_post(t, j);
    else {
        int ns;
        const int nd = build_sel(t.index, j, t.c.icgs, a.sel, &ns);
        if (threadIdx.x == 0) {
            LbCtl &c = t.c;
            c.ndot_iter = nd;
            c.nsel = ns;
            c.reorth_active = 1;
            c.reorth_iter = 0;
            c.reorth_nrm0 = c.beta;
        }
    }
}
// B(j,2), amax and the ||A|| estimate (dlanbpro.F:445-458); as above
__device__ inline void u_finish_beta(Tail &t, const LbArgs &a, int j)
{
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const double beta = t.c.beta, amax = fmax(t.c.amax, beta);
        // alpha_j, beta_j, beta_{j-1} (j > 1)
        double q = lane == 0 ? t.ba[j - 1] : lane == 1 ? beta : j > 1 ? t.bb[j - 2] : 0.0;
        // j = 1: hypot(alpha_1, beta_1), which amax (the largest alpha, beta) does not bound
        const double top = j > 1 ? amax : fmax(amax, fabs(t.ba[0]));
        q = (lane == 4 ? 1.0 : q) / (lane == 4 ? beta : top);
        const double q0 = __shfl_sync(0xffffffffu, q, 0), q1 = __shfl_sync(0xffffffffu, q, 1),
                     q2 = __shfl_sync(0xffffffffu, q, 2);
        const double r = sqrt(lane == 0 ? q0 * q0 + q1 * q1 + q0 * q2
                                        : lane == 1 ? q0 * q0 + q1 * q1 : q0 * q0 + q2 * q2);
        const double h = top > 0.0 ? top * r : 0.0;
        if (lane == 1 && t.hA) t.hA[j - 1] = h;
        if (lane == 2 && t.hB) t.hB[j - 1] = h;
        if (lane == 4) t.rinv = q;
        if (lane == 0) {
            t.bb[j - 1] = beta;
            t.c.amax = amax;
            t.c.anorm = fmax(t.c.anorm, h);
        }
    }
    u_reorth_decide(t, a, j);
}

// ------------------------------------------------ continuations by phase
// The sums of the phase are in t.red: ||y||^2, then the projection on the
// previous vector (real, or its real and imaginary parts).
// cdot: the launch formed the complex projection <prev, y> = (dotp,
// dotp_im) (the native complex SpMV), so the ELR needs no pass to form it
template <int SIDE>
__device__ inline void after_spmv(Tail &t, const LbArgs &a, int j, bool cdot = false)
{
    if (threadIdx.x == 0) {
        LbCtl &c = t.c;
        const double nrm = sqrt(t.red[0]), dotp = t.red[1], dotp_im = cdot ? t.red[2] : 0.0;
        c.nopx++;
        t.go = 1;
        if (SIDE == 0) {
            if (j > 1) c.pend_v.mode = 0;  // v_{j-1} was scaled in place by the SpMV
            c.alpha = nrm;
            if (j == 1) {
                c.anorm = fmax(c.anorm, FUDGE * c.alpha);
                t.go = 2;
            } else if (c.ielr > 0 && c.alpha < KAPPA * c.beta) {
                c.elr_active = 1;
                c.elr_iter = 1;
                if (c.cplx) {
                    c.elr_need_dot = cdot ? 0 : 1;
                    c.elr_s = dotp;
                    c.elr_s_im = dotp_im;
                } else {
                    c.elr_s = dotp;
                    if (c.beta != 0.0) { c.beta += dotp; t.bb[j - 2] = c.beta; }
                }
                t.go = 0;
            }
        } else {
            c.pend_u.mode = 0;  // u_j was scaled in place by the SpMV
            c.beta = nrm;
            if (c.ielr > 0 && c.beta < KAPPA * c.alpha) {
                c.elr_active = 1;
                c.elr_iter = 1;
                if (c.cplx) {
                    c.elr_need_dot = cdot ? 0 : 1;
                    c.elr_s = dotp;
                    c.elr_s_im = dotp_im;
                } else {
                    c.elr_s = dotp;
                    if (c.alpha != 0.0) { c.alpha += dotp; t.ba[j - 1] = c.alpha; }
                }
                t.go = 0;
            }
        }
    }
    __syncthreads();
    if (SIDE == 0) {
        if (t.go == 1) v_finish_alpha(t, a, j);
        else if (t.go == 2) v_reorth_decide(t, a, j);
    } else {
        if (t.go == 1) u_finish_beta(t, a, j);
    }
}

template <int SIDE>
__device__ inline void after_elr(Tail &t, const LbArgs &a, int j)
{
    if (threadIdx.x == 0) {
        LbCtl &c = t.c;
        const double snrm = sqrt(t.red[0]), dotp = t.red[1];
        double &cur = SIDE == 0 ? c.alpha : c.beta;
        double &oth = SIDE == 0 ? c.beta : c.alpha;
        t.go = 0;
        if (snrm >= KAPPA * cur || c.elr_iter >= c.ielr) {
            if (SIDE == 0) t.nu[j - 2] = c.eps_vec;
            else t.mu[j - 1] = c.eps_vec;
            cur = snrm;
            c.elr_active = 0;
            t.go = 1;
        } else {
            cur = snrm;
            c.elr_iter++;
            c.elr_s = dotp;
            if (c.cplx) c.elr_s_im = t.red[2];
            else if (oth != 0.0) {
                oth += dotp;
                if (SIDE == 0) t.bb[j - 2] = oth;
                else t.ba[j - 1] = oth;
            }
        }
    }
    __syncthreads();
    if (t.go == 1) {
        if (SIDE == 0) v_finish_alpha(t, a, j);
        else u_finish_beta(t, a, j);
    }
}

// h[c] = sum over CTAs of part_cols[c * nb + b], one warp per column: warp
// gw of nw warps, ncols columns, nparts partials each
__device__ __forceinline__ void reduce_cols(const LbArgs &a, int ncols, int nparts, int gw, int nw)
{
    const int lane = threadIdx.x & 31;
    for (int c = gw; c < ncols; c += nw) {
        const double *p = a.part_cols + (size_t)c * a.nb;
        double s = 0.0;
        for (int b = lane; b < nparts; b += 32) s += __ldcg(p + b);
        s = warp_sum(s);
        if (lane == 0) a.h[c] = s;
    }
}

template <int SIDE>
__device__ inline void after_cgs(Tail &t, const LbArgs &a, int j)
{
    if (threadIdx.x == 0) {
        LbCtl &c = t.c;
        const double nrm = sqrt(t.red[0]);
        double &cur = SIDE == 0 ? c.alpha : c.beta;
        c.ndot += c.ndot_iter;
        (SIDE == 1 ? c.cgs_cols_u : c.cgs_cols_v) += c.nsel;
        t.go = 2;
        if (nrm > KAPPA * c.reorth_nrm0) {
            cur = nrm;
            t.go = 1;
        } else {
            cur = nrm;
            c.reorth_nrm0 = nrm;
            if (++c.reorth_iter >= NTRY) {
                cur = 0.0;
                c.collapsed = 1;
                t.go = 1;
            }
        }
        if (t.go == 1) {
            c.nreorth++;
            c.reorth_active = 0;
        }
    }
    __syncthreads();
    if (t.go == 1) {
        if (SIDE == 0) { v_post_reorth(t, j); v_post(t, j); }
        else { u_post_reorth(t, j); u_post(t, j); }
    }
}

// ----------------------------------------------------------------- kernels
// T is the type of the Lanczos vectors: double (the reference's FP64
// method) or float (the mixed form: FP32 vectors, FP32 SpMV on the FP32
// copy of the values, compensated FP32 reductions; all scalars FP64).
template <typename T>
__device__ __forceinline__ const T *csr_vals(const Csr &A);
template <>
__device__ __forceinline__ const double *csr_vals<double>(const Csr &A) { return A.val; }
template <>
__device__ __forceinline__ const float *csr_vals<float>(const Csr &A) { return A.valf; }

// The scalars of the control block that every CTA of a phase reads.
struct LbPub {
    Pend pend_u, pend_v;
    double alpha, beta, elr_s, elr_s_im;
    int elr_need_dot, nsel;
};
__device__ __forceinline__ LbPub publish(const LbCtl &c)
{
    LbPub p;
    p.pend_u = c.pend_u;
    p.pend_v = c.pend_v;
    p.alpha = c.alpha;
    p.beta = c.beta;
    p.elr_s = c.elr_s;
    p.elr_s_im = c.elr_s_im;
    p.elr_need_dot = c.elr_need_dot;
    p.nsel = c.nsel;
    return p;
}

// Shared memory of the SpMV.  SHORT 1: the matrix uses the chunked schedule
// (compiled separately so that it carries neither the staged schedule's
// shared memory nor its registers, and fits more CTAs per SM); 2: either
// schedule, by the matrix (Csr::short_rows).
template <typename T, int SHORT>
struct SpmvShared {
    std::conditional_t<SHORT == 1, int, SpmvStage<T, T>[SPMV_WARPS]> st;
    ChunkStage<T> cst[SPMV_WARPS];
};

// The fused SpMV of one half step: the product (host_product: the caller's
// APROD already wrote it into the output column), the deferred scales, the
// axpy with the previous vector, and the CTA's partial sums of ||y||^2 and
// <prev, y> in part_sq, part_dot.  tb0, tb1: the warp's tiles (chunked).
template <int SIDE, typename T, int SHORT>
__device__ __forceinline__ void spmv_phase(const LbArgs &a, int j, int host_product, const Pend pin,
                                           const Pend pprev, const T coef, int tb0, int tb1,
                                           SpmvShared<T, SHORT> &sh, double *buf)
{
    const Csr &A = SIDE == 0 ? a.adj : a.fwd;
    const bool has_prev = SIDE == 1 || j > 1;
    const T *x = SIDE == 0 ? ucol<T>(a, j - 1) : vcol<T>(a, j - 1);
    T *out = SIDE == 0 ? vcol<T>(a, j - 1) : ucol<T>(a, j);
    T *prev = SIDE == 0 ? (j > 1 ? vcol<T>(a, j - 2) : nullptr) : ucol<T>(a, j - 1);
    const double *z = a.z;
    const int n0 = A.ncol0;
    // this phase rewrites the output column and (deferred scale) the
    // previous one: their FP32 planes no longer hold them
    if (a.okU && blockIdx.x == 0 && threadIdx.x == 0) {
        int *ok = SIDE == 0 ? a.okV : a.okU;
        ok[SIDE == 0 ? j - 1 : j] = 0;
        if (has_prev) ok[SIDE == 0 ? j - 2 : j - 1] = 0;
    }
    Acc<T> sq, dt;
    auto epi = [&](int r, double acc, double pvd) {
        T y = apply_pend((T)acc, pin);
        if (has_prev) {
            T pv = (T)pvd;
            if (pprev.mode) {
                pv = apply_pend(pv, pprev);
                prev[r] = pv;
            }
            y = fma(-coef, pv, y);
            dt.add_prod(pv, y);
        }
        out[r] = y;
        sq.add_prod(y, y);
    };
    auto pre = [&](int r) -> double { return has_prev ? (double)prev[r] : 0.0; };
    if (!host_product) {
        auto xl = [&](int c) -> T { return c < n0 ? x[c] : (T)z[c - n0]; };
        if (SHORT == 1 || A.short_rows)
            csr_rows_chunked<T, T>(A.ptr, A.tbase, A.cidx, chunk_vals<T>(A), A.rows, xl, pre, epi, sh.cst, tb0, tb1);
        else if constexpr (SHORT != 1)
            csr_rows_staged<T, T>(A.ptr, A.idx, csr_vals<T>(A), A.blk, A.nblk, xl, pre, epi, sh.st);
    } else {
        for (int r = blockIdx.x * BS + threadIdx.x; r < A.rows; r += gridDim.x * BS) epi(r, (double)out[r], pre(r));
    }
    __syncthreads();  // buf may share the stage's memory
    block_sums<BS, 2>({sq.value(), dt.value()}, buf, {a.part_sq + blockIdx.x, a.part_dot + blockIdx.x});
}

// one ELR pass (dlanbpro.F:301-316, :429-443): x -= s p, and the partial
// sums of ||x||^2 and of the next projection
template <int SIDE, typename T>
__device__ __forceinline__ void elr_phase(const LbArgs &a, int j, const T s, double *buf)
{
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    T *x = SIDE == 0 ? vcol<T>(a, j - 1) : ucol<T>(a, j);
    const T *p = SIDE == 0 ? vcol<T>(a, j - 2) : ucol<T>(a, j - 1);
    Acc<T> sq, dt;
    for (int r = blockIdx.x * BS + threadIdx.x; r < len; r += gridDim.x * BS) {
        const T pv = p[r];
        const T y = fma(-s, pv, x[r]);
        x[r] = y;
        sq.add_prod(y, y);
        dt.add_prod(pv, y);
    }
    block_sums<BS, 2>({sq.value(), dt.value()}, buf, {a.part_sq + blockIdx.x, a.part_dot + blockIdx.x});
}
// 16-byte vectors of the Lanczos type: 4 floats or 2 doubles
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    using V = float4;
    static constexpr int W = 4;
    __device__ static __forceinline__ float get(const V &v, int i)
    {
        return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
    }
    __device__ static __forceinline__ void fms(V &x, const V &w, float h)
    {
        x.x = fmaf(-w.x, h, x.x);
        x.y = fmaf(-w.y, h, x.y);
        x.z = fmaf(-w.z, h, x.z);
        x.w = fmaf(-w.w, h, x.w);
    }
};
template <>
struct Vec16<double> {
    using V = double2;
    static constexpr int W = 2;
    __device__ static __forceinline__ double get(const V &v, int i) { return i == 0 ? v.x : v.y; }
    __device__ static __forceinline__ void fms(V &x, const V &w, double h)
    {
        x.x = fma(-w.x, h, x.x);
        x.y = fma(-w.y, h, x.y);
    }
};

// projections h = W(:,sel)' x (dreorth.F:174, the dgemv('T') of dcgs):
// each CTA owns a contiguous chunk of 16-byte row vectors; each warp takes
// four columns at a time and streams the chunk once for them, so every x
// vector it loads serves four columns (ten 16-byte loads in flight per
// lane).  The last CTA also takes the rows past the last whole vector.
constexpr int DOT_COLS = 4;
// columns whose per-slice partials lie in shared memory at a time: what a CTA
// takes of it comes out of the L1 that holds the SpMV's gathers in flight
constexpr int WPART_COLS = 64;
// Selections of more columns (BIG instances: dimensions past GS_COLS) have their
// indices and, in an update, their coefficients in shared memory GS_COLS at a
// time.  x goes through memory once more per GS_COLS columns (1/256 of the pass),
// but no dimension takes more than 7 KB (complex 11) out of the L1 or is refused
// for its size: with all columns there (1000003 rows of 8 entries, kmax 2000, 989
// steps) product and adjoint took 153 and 137 us, projections 1166, updates 820,
// by blocks 79, 70, 937 and 689.  The smaller dimensions keep instances without
// the loop over blocks: with it the compiler gives the product's loads fewer
// registers (FP32, 500001 rows: 66 -> 80 us).
constexpr int GS_COLS = 512;
template <int SIDE>
__device__ __forceinline__ void dots_f64(const LbArgs &a, int j, int L)
{
    using T = double;
    using VT = Vec16<T>;
    using V = typename VT::V;
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ld = SIDE == 0 ? a.ldv : a.ldu;
    const T *W = (const T *)(SIDE == 0 ? a.V : a.U);
    const T *x = SIDE == 0 ? vcol<T>(a, j - 1) : ucol<T>(a, j);
    const int nvec = len / VT::W;
    const int chunk = (nvec + gridDim.x - 1) / gridDim.x;
    const int v0 = blockIdx.x * chunk, v1 = min(nvec, v0 + chunk);
    const bool tail_rows = blockIdx.x == gridDim.x - 1;
    const V *xv = reinterpret_cast<const V *>(x);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int c0 = w * DOT_COLS; c0 < L; c0 += (BS / 32) * DOT_COLS) {
        const int nc = min(DOT_COLS, L - c0);
        const T *col[DOT_COLS];
#pragma unroll
        for (int u = 0; u < DOT_COLS; u++) col[u] = W + (size_t)a.sel[c0 + (u < nc ? u : 0)] * ld;
        Acc<T> acc[DOT_COLS][2];
        int v = v0 + lane;
        for (; v + 32 < v1; v += 64) {
            const V x0 = xv[v], x1 = xv[v + 32];
            V w0[DOT_COLS], w1[DOT_COLS];
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++) {
                w0[u] = reinterpret_cast<const V *>(col[u])[v];
                w1[u] = reinterpret_cast<const V *>(col[u])[v + 32];
            }
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++)
#pragma unroll
                for (int q = 0; q < VT::W; q++) {
                    acc[u][0].add_prod(VT::get(w0[u], q), VT::get(x0, q));
                    acc[u][1].add_prod(VT::get(w1[u], q), VT::get(x1, q));
                }
        }
        if (v < v1) {
            const V x0 = xv[v];
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++) {
                const V w0 = reinterpret_cast<const V *>(col[u])[v];
#pragma unroll
                for (int q = 0; q < VT::W; q++) acc[u][0].add_prod(VT::get(w0, q), VT::get(x0, q));
            }
        }
        if (tail_rows)
            for (int r = nvec * VT::W + lane; r < len; r += 32)
#pragma unroll
                for (int u = 0; u < DOT_COLS; u++) acc[u][1].add_prod(col[u][r], x[r]);
#pragma unroll
        for (int u = 0; u < DOT_COLS; u++) {
            const double sum = warp_sum(acc[u][0].value() + acc[u][1].value());
            if (lane == 0 && u < nc) a.part_cols[(size_t)(c0 + u) * a.nb + blockIdx.x] = sum;
        }
    }
}

// Row slices of a CTA's chunk of `chunk` vectors in the projections: the
// eight warps are rs slices x 8 / rs column groups.  A long chunk gives
// every warp a slice and all columns; a short one (small problems) would
// leave most lanes without a vector, so its warps share slices and split the
// columns instead (20011 rows x 40 columns: 45 -> 9 us a pass).
__device__ __forceinline__ int dot_slices(int chunk)
{
    return chunk >= 256 ? 8 : chunk >= 128 ? 4 : chunk >= 64 ? 2 : 1;
}

// projections of the FP32 form: compensated sums, the work layout of dots_pl
// below (slices of 4-element vectors, groups of DOT_COLS columns)
template <int SIDE, bool BIG>
__device__ __forceinline__ void dots_f32(const LbArgs &a, int j, int L, double *wpart)
{
    int *ssel = reinterpret_cast<int *>(wpart + BS / 32 * WPART_COLS);
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ldq = (size_t)(SIDE == 0 ? a.ldv : a.ldu) / 4;
    const float *W = (const float *)(SIDE == 0 ? a.V : a.U);
    const float4 *Wv = reinterpret_cast<const float4 *>(W);
    const float *x = SIDE == 0 ? vcol<float>(a, j - 1) : ucol<float>(a, j);
    const float4 *xv = reinterpret_cast<const float4 *>(x);
    const int nvec = len / 4;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int chunk = (nvec + gridDim.x - 1) / gridDim.x;
    const int cb0 = min(nvec, blockIdx.x * chunk), cb1 = min(nvec, cb0 + chunk);
    const int rs = dot_slices(chunk), ws = w % rs, wg = w / rs, cgs = BS / 32 / rs;
    const int sl = (cb1 - cb0 + rs - 1) / rs;
    const int v0 = min(cb1, cb0 + ws * sl), v1 = min(cb1, v0 + sl);
    // the rows past the last whole vector: the last slice's warps of the last CTA
    const int r0 = blockIdx.x == gridDim.x - 1 && ws == rs - 1 ? nvec * 4 + lane : len;
    int s0 = 0;
    do {
        const int s1 = BIG ? min(L, s0 + GS_COLS) : L;
        for (int c = threadIdx.x; c < s1 - s0; c += BS) ssel[c] = a.sel[s0 + c];
        __syncthreads();
        for (int b0 = s0; b0 < s1; b0 += WPART_COLS) {
            const int b1 = min(s1, b0 + WPART_COLS);
            for (int cb = b0 + wg * DOT_COLS; cb < b1; cb += cgs * DOT_COLS) {
                const int nc = min(DOT_COLS, b1 - cb);
                const int *scol = ssel + (cb - s0);
                const float4 *Wq[DOT_COLS];
#pragma unroll
                for (int u = 0; u < DOT_COLS; u++) Wq[u] = Wv + (size_t)scol[u < nc ? u : 0] * ldq;
                Acc<float> acc[DOT_COLS];
                int v = v0 + lane;
#pragma unroll 1
                for (; v < v1; v += 32) {  // one vector of each column in flight: see dots_pl
                    float4 w0[DOT_COLS];
#pragma unroll
                    for (int u = 0; u < DOT_COLS; u++) w0[u] = __ldcs(Wq[u] + v);
                    const float4 x0 = xv[v];
#pragma unroll
                    for (int u = 0; u < DOT_COLS; u++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[u].add_prod(Vec16<float>::get(w0[u], q), Vec16<float>::get(x0, q));
                }
                if (r0 < len) {
                    const float xr = x[r0];
#pragma unroll
                    for (int u = 0; u < DOT_COLS; u++)
                        if (u < nc) acc[u].add_prod(W[(size_t)scol[u] * (4 * ldq) + r0], xr);
                }
                PlAcc p[DOT_COLS];
#pragma unroll
                for (int u = 0; u < DOT_COLS; u++) {
                    p[u].s = acc[u].s;
                    p[u].c = acc[u].c;
                }
                const PlAcc tot = pl_warp_sum4(p);
                if ((lane & 7) == 0 && (lane >> 3) < nc) wpart[ws * WPART_COLS + cb - b0 + (lane >> 3)] = tot.value();
            }
            __syncthreads();
            for (int c = threadIdx.x; c < b1 - b0; c += BS) {
                double sum = 0.0;
                for (int ww = 0; ww < rs; ww++) sum += wpart[ww * WPART_COLS + c];
                a.part_cols[(size_t)(b0 + c) * a.nb + blockIdx.x] = sum;
            }
            __syncthreads();
        }
        s0 += GS_COLS;
    } while (BIG && s0 < L);
}

// x -= W(:,sel) h (dreorth.F:85-95, the dgemv('N') of dcgs) and ||x||^2:
// one 16-byte row vector per thread and step, the selected columns streamed
// with CGS_UNROLL loads in flight; h and the selection sit in shared memory.
constexpr int CGS_UNROLL = 8;
template <int SIDE, typename T, bool BIG>
__device__ __forceinline__ void upd_full(const LbArgs &a, int j, int L, double *dyn, double *buf)
{
    using VT = Vec16<T>;
    using V = typename VT::V;
    // dyn: h (as T, one double slot each) | sel, of the block's columns
    T *hs = reinterpret_cast<T *>(dyn);
    int *ssel = reinterpret_cast<int *>(dyn + (BIG ? min(L, GS_COLS) : L));
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ld = SIDE == 0 ? a.ldv : a.ldu;
    const T *W = (const T *)(SIDE == 0 ? a.V : a.U);
    T *x = SIDE == 0 ? vcol<T>(a, j - 1) : ucol<T>(a, j);
    V *xv = reinterpret_cast<V *>(x);
    const int nvec = len / VT::W;
    Acc<T> sq;
    int b0 = 0;
    do {
        const int nb = BIG ? min(GS_COLS, L - b0) : L;
        const bool last = !BIG || b0 + nb >= L;
        if (BIG && b0 > 0) __syncthreads();
        for (int c = threadIdx.x; c < nb; c += BS) {
            hs[c] = (T)a.h[b0 + c];
            ssel[c] = a.sel[b0 + c];
        }
        __syncthreads();
        for (int v = blockIdx.x * BS + threadIdx.x; v < nvec; v += gridDim.x * BS) {
            V acc = xv[v];
            int c = 0;
            for (; c + CGS_UNROLL <= nb; c += CGS_UNROLL) {
                V wv[CGS_UNROLL];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++)
                    wv[u] = reinterpret_cast<const V *>(W + (size_t)ssel[c + u] * ld)[v];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) VT::fms(acc, wv[u], hs[c + u]);
            }
            for (; c < nb; c++) VT::fms(acc, reinterpret_cast<const V *>(W + (size_t)ssel[c] * ld)[v], hs[c]);
            xv[v] = acc;
            if (last)
#pragma unroll
                for (int q = 0; q < VT::W; q++) sq.add_prod(VT::get(acc, q), VT::get(acc, q));
        }
        if (blockIdx.x == gridDim.x - 1) {
            for (int r = nvec * VT::W + threadIdx.x; r < len; r += BS) {
                T y = x[r];
                for (int c = 0; c < nb; c++) y = fma(-W[(size_t)ssel[c] * ld + r], hs[c], y);
                x[r] = y;
                if (last) sq.add_prod(y, y);
            }
        }
        b0 += GS_COLS;
    } while (BIG && b0 < L);
    block_sums<BS, 1>({sq.value()}, buf, {a.part_sq + blockIdx.x});
}

// The FP64 form's projections on the FP32 pipe (pgb_f3.cuh): same layout
// of work and partial sums as dots_f64; each thread scales its own x
// values by a power of two (its largest exponent) and its partial sums
// back before the warp sum.
template <int SIDE>
__device__ __forceinline__ void dots_f3(const LbArgs &a, int j, int L)
{
    using V = double2;
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ld = SIDE == 0 ? a.ldv : a.ldu;
    const double *W = (const double *)(SIDE == 0 ? a.V : a.U);
    const double *x = SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j);
    const int nvec = len / 2;
    const int chunk = (nvec + gridDim.x - 1) / gridDim.x;
    const int v0 = blockIdx.x * chunk, v1 = min(nvec, v0 + chunk);
    const bool tail_rows = blockIdx.x == gridDim.x - 1;
    const V *xv = reinterpret_cast<const V *>(x);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // this thread's scale: |x 2^-xs| < 2
    int xe = 0;
    for (int v = v0 + lane; v < v1; v += 32) {
        const V xx = xv[v];
        xe = max(xe, max(f3_expo(xx.x), f3_expo(xx.y)));
    }
    if (tail_rows)
        for (int r = nvec * 2 + lane; r < len; r += 32) xe = max(xe, f3_expo(x[r]));
    const int xs = xe == 0 ? 0 : xe - 1023;
    const double back = f3_pow2(xs);
    for (int c0 = w * DOT_COLS; c0 < L; c0 += (BS / 32) * DOT_COLS) {
        const int nc = min(DOT_COLS, L - c0);
        const double *col[DOT_COLS];
#pragma unroll
        for (int u = 0; u < DOT_COLS; u++) col[u] = W + (size_t)a.sel[c0 + (u < nc ? u : 0)] * ld;
        F3Acc acc[DOT_COLS];
        for (int v = v0 + lane; v < v1; v += 32) {
            const V xx = xv[v];
            V wv[DOT_COLS];
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++) wv[u] = reinterpret_cast<const V *>(col[u])[v];
            const F3 x0 = f3_split(xx.x, xs), x1 = f3_split(xx.y, xs);
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++) {
                acc[u].add(f3_split(wv[u].x, 0), x0);
                acc[u].add(f3_split(wv[u].y, 0), x1);
            }
        }
        if (tail_rows)
            for (int r = nvec * 2 + lane; r < len; r += 32) {
                const F3 xr = f3_split(x[r], xs);
#pragma unroll
                for (int u = 0; u < DOT_COLS; u++) acc[u].add(f3_split(col[u][r], 0), xr);
            }
#pragma unroll
        for (int u = 0; u < DOT_COLS; u++) {
            const double sum = warp_sum(acc[u].value() * back);
            if (lane == 0 && u < nc) a.part_cols[(size_t)(c0 + u) * a.nb + blockIdx.x] = sum;
        }
    }
}

// The FP64 form's update on the FP32 pipe: sum_c W(i, c) h_c at three
// levels per row (h scaled by the power of two of its largest entry),
// then one FP64 FMA per row applies it to x.
template <int SIDE, bool BIG>
__device__ __forceinline__ void upd_f3(const LbArgs &a, int j, int L, double *dyn, double *buf)
{
    using V = double2;
    // dyn: h as F3 (one double2 slot each) | sel, of the block's columns
    __shared__ int hsh;
    F3 *h3 = reinterpret_cast<F3 *>(dyn);
    int *ssel = reinterpret_cast<int *>(dyn + 2 * (size_t)(BIG ? min(L, GS_COLS) : L));
    if (threadIdx.x == 0) hsh = 0;
    __syncthreads();
    int he = 0;
    for (int c = threadIdx.x; c < L; c += BS) he = max(he, f3_expo(a.h[c]));
    if (he) atomicMax(&hsh, he);
    __syncthreads();
    const int hs = hsh == 0 ? 0 : hsh - 1023;  // |h 2^-hs| < 2
    const double back = f3_pow2(hs);
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ld = SIDE == 0 ? a.ldv : a.ldu;
    const double *W = (const double *)(SIDE == 0 ? a.V : a.U);
    double *x = SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j);
    V *xv = reinterpret_cast<V *>(x);
    const int nvec = len / 2;
    Acc<double> sq;
    int b0 = 0;
    do {
        const int nb = BIG ? min(GS_COLS, L - b0) : L;
        const bool last = !BIG || b0 + nb >= L;
        if (BIG && b0 > 0) __syncthreads();
        for (int c = threadIdx.x; c < nb; c += BS) {
            h3[c] = f3_split(a.h[b0 + c], hs);
            ssel[c] = a.sel[b0 + c];
        }
        __syncthreads();
        for (int v = blockIdx.x * BS + threadIdx.x; v < nvec; v += gridDim.x * BS) {
            F3Acc s0, s1;
            int c = 0;
            for (; c + CGS_UNROLL <= nb; c += CGS_UNROLL) {
                V wv[CGS_UNROLL];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++)
                    wv[u] = reinterpret_cast<const V *>(W + (size_t)ssel[c + u] * ld)[v];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) {
                    const F3 hc = h3[c + u];
                    s0.add(f3_split(wv[u].x, 0), hc);
                    s1.add(f3_split(wv[u].y, 0), hc);
                }
            }
            for (; c < nb; c++) {
                const V wc = reinterpret_cast<const V *>(W + (size_t)ssel[c] * ld)[v];
                s0.add(f3_split(wc.x, 0), h3[c]);
                s1.add(f3_split(wc.y, 0), h3[c]);
            }
            V acc = xv[v];
            acc.x = fma(-s0.value(), back, acc.x);
            acc.y = fma(-s1.value(), back, acc.y);
            xv[v] = acc;
            if (last) {
                sq.add_prod(acc.x, acc.x);
                sq.add_prod(acc.y, acc.y);
            }
        }
        if (blockIdx.x == gridDim.x - 1) {
            for (int r = nvec * 2 + threadIdx.x; r < len; r += BS) {
                F3Acc sr;
                for (int c = 0; c < nb; c++) sr.add(f3_split(W[(size_t)ssel[c] * ld + r], 0), h3[c]);
                const double y = fma(-sr.value(), back, x[r]);
                x[r] = y;
                if (last) sq.add_prod(y, y);
            }
        }
        b0 += GS_COLS;
    } while (BIG && b0 < L);
    block_sums<BS, 1>({sq.value()}, buf, {a.part_sq + blockIdx.x});
}

// ------------------------------------------------ split-once planes
// The FP64 form's Gram-Schmidt on the FP32 pipe, reading each basis element
// as 8 bytes of FP32 planes: hi = the leading 24 bits of w, lo = the next
// 23, so that hi + lo holds w to 2^-47 relative (a Lanczos column has
// |w| <= 1; parts below 2^-74 are dropped, far below the column's unit norm).  A column is
// split by the first projection that selects it while its flag is clear;
// the update of the same pass and every later pass read its planes until
// the column is rewritten (the SpMV that writes a column, the flush and the
// deferred-scale kernel clear its flag; the host clears all flags whenever
// it writes columns itself).  One product w x costs 12 FP32 operations --
// hi*hi as an exact two-product folded into a two-sum, the cross terms
// hi*lo and lo*hi into the compensation -- for an error of a few 2^-48 of
// sum |w_i x_i|, the size of an FP64 dot product's own rounding over a
// few thousand terms.  A pass streams 8 bytes per element either way; on
// GB300 the FP64 pipe (2 lanes per clock per SM) holds one FMA per element
// below the HBM rate, 12 FP32 operations (128 lanes per clock) do not.

// projections h = W(:,sel)' x from the planes.  Each CTA owns a contiguous
// chunk of 2-element row vectors and each of its warps one eighth of the
// chunk.  A warp first splits its x values (scaled by a power of two per
// warp) into the x planes scratch and the rows of its slice of every
// selected column whose planes are stale (read in FP64, written as planes);
// it then streams its slice once per group of DOT_COLS columns, reading the
// planes only, so every warp has the same work whatever the column count.
// Each lane reads back only the vectors it wrote itself.  A group's sums
// are reduced over the warp as compensated FP32 pairs (no FP64 operation
// per group), then added over the warps in a fixed order, then over the
// CTAs by CTA 0 or the grid (reduce_cols).  The grid is one wave at the kernel's occupancy (<= nb CTAs).
constexpr int PL_WARPS = BS / 32;
constexpr int PL_SPLIT_UNROLL = 4;          // FP64 loads in flight per lane when a column is split
static_assert(GS_COLS % WPART_COLS == 0 && WPART_COLS % PL_WARPS == 0, "column groups stay with their warps");
template <int SIDE, bool BIG>
__device__ __forceinline__ void dots_pl(const LbArgs &a, int j, int L, double *wpart)
{
    // wpart: [PL_WARPS][WPART_COLS] per-slice partial projections | sel of GS_COLS columns and their stale flags
    int *ssel = reinterpret_cast<int *>(wpart + PL_WARPS * WPART_COLS);
    unsigned char *sstale = reinterpret_cast<unsigned char *>(ssel + min(a.kmax + 1, GS_COLS));
    const int *ok = SIDE == 0 ? a.okV : a.okU;
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ld = SIDE == 0 ? a.ldv : a.ldu;
    const size_t ldq = ld / 2;  // leading dimension in float4 (two elements)
    const double *W = (const double *)(SIDE == 0 ? a.V : a.U);
    float2 *Wp = SIDE == 0 ? a.Vp : a.Up;
    const double *x = SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j);
    const double2 *xv = reinterpret_cast<const double2 *>(x);
    float4 *xq = reinterpret_cast<float4 *>(a.xpl);
    const int nvec = len / 2;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int chunk = (nvec + gridDim.x - 1) / gridDim.x;
    const int cb0 = min(nvec, blockIdx.x * chunk), cb1 = min(nvec, cb0 + chunk);
    const int rs = dot_slices(chunk), ws = w % rs, wg = w / rs, cgs = PL_WARPS / rs;
    const int sl = (cb1 - cb0 + rs - 1) / rs;
    const int v0 = min(cb1, cb0 + ws * sl), v1 = min(cb1, v0 + sl);
    // the row past the last whole vector (odd lengths): lane 0 of the last slice's warps in the last CTA
    const bool tail_row = (len & 1) && blockIdx.x == gridDim.x - 1 && ws == rs - 1 && lane == 0;
    // this warp's scale (|x 2^-xs| < 2), then its x planes
    int xe = 0;
    for (int v = v0 + lane; v < v1; v += 32) {
        const double2 xx = xv[v];
        xe = max(xe, max(f3_expo(xx.x), f3_expo(xx.y)));
    }
    if (tail_row) xe = max(xe, f3_expo(x[len - 1]));
    xe = __reduce_max_sync(0xffffffffu, xe);
    const int xs = xe == 0 ? 0 : xe - 1023;
    const double back = f3_pow2(xs);
    for (int v = v0 + lane; v < v1; v += 32) {
        const double2 xx = xv[v];
        const float2 p = pl_xsplit(xx.x, xs), q = pl_xsplit(xx.y, xs);
        xq[v] = make_float4(p.x, p.y, q.x, q.y);
    }
    float2 xr = make_float2(0.f, 0.f);
    if (tail_row) xr = pl_xsplit(x[len - 1], xs);
    int s0 = 0;
    do {
        const int s1 = BIG ? min(L, s0 + GS_COLS) : L;
        for (int c = threadIdx.x; c < s1 - s0; c += BS) {
            const int col = a.sel[s0 + c];
            ssel[c] = col;
            sstale[c] = ok[col] == 0;
        }
        __syncthreads();
        // planes of the stale columns, on this lane's rows
        for (int c = 0; c < s1 - s0; c++) {
            if (!sstale[c] || (c / DOT_COLS) % cgs != wg) continue;
            const int col = ssel[c];
            float4 *Wq = reinterpret_cast<float4 *>(Wp) + (size_t)col * ldq;
            const double2 *Wd = reinterpret_cast<const double2 *>(W + (size_t)col * ld);
            int v = v0 + lane;
            for (; v + 32 * (PL_SPLIT_UNROLL - 1) < v1; v += 32 * PL_SPLIT_UNROLL) {
                double2 d[PL_SPLIT_UNROLL];
#pragma unroll
                for (int u = 0; u < PL_SPLIT_UNROLL; u++) d[u] = Wd[v + 32 * u];
#pragma unroll
                for (int u = 0; u < PL_SPLIT_UNROLL; u++) Wq[v + 32 * u] = pl_split2(d[u]);
            }
            for (; v < v1; v += 32) Wq[v] = pl_split2(Wd[v]);
            if (tail_row) Wp[(size_t)col * ld + len - 1] = pl_split(W[(size_t)col * ld + len - 1]);
        }
        for (int b0 = s0; b0 < s1; b0 += WPART_COLS) {
            const int b1 = min(s1, b0 + WPART_COLS);
            for (int cb = b0 + wg * DOT_COLS; cb < b1; cb += cgs * DOT_COLS) {
                const int nc = min(DOT_COLS, b1 - cb);
                const float4 *Wq[DOT_COLS];
#pragma unroll
                for (int u = 0; u < DOT_COLS; u++)
                    Wq[u] = reinterpret_cast<const float4 *>(Wp) + (size_t)ssel[cb - s0 + (u < nc ? u : 0)] * ldq;
                PlAcc acc[DOT_COLS];
                int v = v0 + lane;
                // The planes stream through once (evict-first), so that the x
                // planes, read again by every group, stay in L2.  One vector of each
                // column in flight per lane: a second one lets the warps' streams
                // thrash each other (1000003 x 250007, 120 columns: 141 us a pass
                // with two, 106 with one; 4M rows, 75 columns: 548 and 506), and
                // eight columns at a time or slices interleaved over the CTA's warps do
                // the same (146 and 151; 626 and 606).
#pragma unroll 1
                for (; v < v1; v += 32) {
                    float4 w0[DOT_COLS];
#pragma unroll
                    for (int u = 0; u < DOT_COLS; u++) w0[u] = __ldcs(Wq[u] + v);
                    const float4 x0 = xq[v];
#pragma unroll
                    for (int u = 0; u < DOT_COLS; u++) {
                        acc[u].add(w0[u].x, w0[u].y, x0.x, x0.y);
                        acc[u].add(w0[u].z, w0[u].w, x0.z, x0.w);
                    }
                }
                if (tail_row) {
#pragma unroll
                    for (int u = 0; u < DOT_COLS; u++) {
                        if (u >= nc) break;
                        const float2 wr = Wp[(size_t)ssel[cb - s0 + u] * ld + len - 1];
                        acc[u].add(wr.x, wr.y, xr.x, xr.y);
                    }
                }
                static_assert(DOT_COLS == 4, "pl_warp_sum4 sums four columns");
                const PlAcc tot = pl_warp_sum4(acc);
                if ((lane & 7) == 0 && (lane >> 3) < nc) wpart[ws * WPART_COLS + cb - b0 + (lane >> 3)] = tot.value() * back;
            }
            __syncthreads();
            for (int c = threadIdx.x; c < b1 - b0; c += BS) {
                double s = 0.0;
                for (int ww = 0; ww < rs; ww++) s += wpart[ww * WPART_COLS + c];
                a.part_cols[(size_t)(b0 + c) * a.nb + blockIdx.x] = s;
            }
            __syncthreads();
        }
        s0 += GS_COLS;
    } while (BIG && s0 < L);
}

// x -= W(:,sel) h from the planes, and ||x||^2: one 2-element row vector
// per thread and step, the selected columns streamed with CGS_UNROLL
// 16-byte loads in flight.  h (scaled by the power of two of its largest
// entry) sits in shared memory as (hi, lo) planes; each row's sum of
// products is formed on the FP32 pipe and applied with one FP64 FMA.
template <int SIDE, bool BIG>
__device__ __forceinline__ void upd_pl(const LbArgs &a, int j, int L, double *dyn, double *buf)
{
    // dyn: h as float2 planes (one double slot each) | sel, of the block's columns
    __shared__ int hsh;
    float2 *hp = reinterpret_cast<float2 *>(dyn);
    int *ssel = reinterpret_cast<int *>(dyn + (BIG ? min(L, GS_COLS) : L));
    if (threadIdx.x == 0) hsh = 0;
    __syncthreads();
    int he = 0;
    for (int c = threadIdx.x; c < L; c += BS) he = max(he, f3_expo(a.h[c]));
    if (he) atomicMax(&hsh, he);
    __syncthreads();
    const int hs = hsh == 0 ? 0 : hsh - 1023;  // |h 2^-hs| < 2
    const double hscale = f3_pow2(-hs), back = f3_pow2(hs);
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ld = SIDE == 0 ? a.ldv : a.ldu;
    const size_t ldq = ld / 2;
    const float4 *Wq = reinterpret_cast<const float4 *>(SIDE == 0 ? a.Vp : a.Up);
    const float2 *Wp = SIDE == 0 ? a.Vp : a.Up;
    double *x = SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j);
    double2 *xv = reinterpret_cast<double2 *>(x);
    const int nvec = len / 2;
    double sq = 0.0;
    int b0 = 0;
    do {
        const int nb = BIG ? min(GS_COLS, L - b0) : L;
        const bool last = !BIG || b0 + nb >= L;
        if (BIG && b0 > 0) __syncthreads();
        for (int c = threadIdx.x; c < nb; c += BS) {
            hp[c] = pl_split(a.h[b0 + c] * hscale);
            ssel[c] = a.sel[b0 + c];
        }
        __syncthreads();
        for (int v = blockIdx.x * BS + threadIdx.x; v < nvec; v += gridDim.x * BS) {
            const double2 x0 = xv[v];
            PlAcc s0, s1;
            int c = 0;
            for (; c + CGS_UNROLL <= nb; c += CGS_UNROLL) {
                float4 wv[CGS_UNROLL];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) wv[u] = Wq[(size_t)ssel[c + u] * ldq + v];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) {
                    const float2 hc = hp[c + u];
                    s0.add(wv[u].x, wv[u].y, hc.x, hc.y);
                    s1.add(wv[u].z, wv[u].w, hc.x, hc.y);
                }
            }
            for (; c < nb; c++) {
                const float4 wc = Wq[(size_t)ssel[c] * ldq + v];
                const float2 hc = hp[c];
                s0.add(wc.x, wc.y, hc.x, hc.y);
                s1.add(wc.z, wc.w, hc.x, hc.y);
            }
            double2 y;
            y.x = fma(-pl_f2d(s0.c), back, fma(-pl_f2d(s0.s), back, x0.x));
            y.y = fma(-pl_f2d(s1.c), back, fma(-pl_f2d(s1.s), back, x0.y));
            xv[v] = y;
            if (last) {
                sq = fma(y.x, y.x, sq);
                sq = fma(y.y, y.y, sq);
            }
        }
        if (blockIdx.x == gridDim.x - 1 && (len & 1) && threadIdx.x == 0) {
            const int r = len - 1;
            PlAcc sr;
            for (int c = 0; c < nb; c++) {
                const float2 wc = Wp[(size_t)ssel[c] * ld + r];
                sr.add(wc.x, wc.y, hp[c].x, hp[c].y);
            }
            const double y = fma(-sr.value(), back, x[r]);
            x[r] = y;
            if (last) sq = fma(y, y, sq);
        }
        b0 += GS_COLS;
    } while (BIG && b0 < L);
    block_sums<BS, 1>({sq}, buf, {a.part_sq + blockIdx.x});
}

// ------------------------------------------------- complex*16 vectors
// The complex form (complex16/zlanbpro.F) keeps alpha, beta and the omega
// recurrences real.  Its vectors are (re, im) pairs of doubles and its
// operator is the real 2x2-block form of A (pgb_operator.cu), so the fused
// SpMV, the norms, the deferred scaling and the flush above serve it as
// they are.  What differs are the inner products, which are conjugated and
// complex: in the ELR (zlanbpro.F:318-331, :451-464) and in Gram-Schmidt
// (zreorth.F, zcgs: zgemv 'C' then 'N').

// conj(w) x added to (re, im)
__device__ __forceinline__ void zdot_acc(double &re, double &im, const double2 &w, const double2 &x)
{
    re = fma(w.x, x.x, re);
    re = fma(w.y, x.y, re);
    im = fma(w.x, x.y, im);
    im = fma(-w.y, x.x, im);
}
// acc -= w h
__device__ __forceinline__ void zfms(double2 &acc, const double2 &w, const double2 &h)
{
    acc.x = fma(-w.x, h.x, acc.x);
    acc.x = fma(w.y, h.y, acc.x);
    acc.y = fma(-w.x, h.y, acc.y);
    acc.y = fma(-w.y, h.x, acc.y);
}

// One complex ELR pass: x -= s p, ||x||^2 and the next projection <p, x>.
// The fused SpMV cannot form the complex <p, x> (the real and imaginary
// rows of an element are different rows of the 2x2-block operator), so the
// first pass after it (elr_need_dot set) forms <p, x> alone.
template <int SIDE>
__device__ __forceinline__ void zelr_phase(const LbArgs &a, int j, bool dot_only, double sr, double si, double *buf)
{
    const int len = (SIDE == 0 ? a.adj.rows : a.fwd.rows) / 2;
    double2 *x = reinterpret_cast<double2 *>(SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j));
    const double2 *p =
        reinterpret_cast<const double2 *>(SIDE == 0 ? vcol<double>(a, j - 2) : ucol<double>(a, j - 1));
    double sq = 0.0, dr = 0.0, di = 0.0;
    for (int r = blockIdx.x * BS + threadIdx.x; r < len; r += gridDim.x * BS) {
        const double2 pv = p[r];
        double2 y = x[r];
        if (!dot_only) {
            y.x = fma(-sr, pv.x, y.x);
            y.x = fma(si, pv.y, y.x);
            y.y = fma(-sr, pv.y, y.y);
            y.y = fma(-si, pv.x, y.y);
            x[r] = y;
            sq = fma(y.x, y.x, sq);
            sq = fma(y.y, y.y, sq);
        }
        zdot_acc(dr, di, pv, y);
    }
    // Gram-Schmidt is idle while the ELR runs: its partials hold the imaginary part
    block_sums<BS, 3>({sq, dr, di}, buf, {a.part_sq + blockIdx.x, a.part_dot + blockIdx.x, a.part_cols + blockIdx.x});
}

// The fused complex SpMV of one half step on a native complex operator
// (zlanbpro.F:297-311 and :442-450): y = op(A) x with complex
// accumulation (one index and one 16-byte value per entry, 16-byte gathers),
// the deferred scale of x and of the previous vector, y -= coef prev (coef
// real), and the partial sums of ||y||^2 and of the complex projection
// <prev, y> = sum conj(prev) y that the first ELR pass subtracts
// (pzdotc), in the same launch.  host_product: the caller's ZAPROD already
// wrote y.
constexpr int ZSPMV_UNROLL = 4;  // its (index, value) pairs and gathers in flight per lane
template <int SIDE>
__device__ __forceinline__ void zspmv_phase(const LbArgs &a, int j, int host_product, const Pend pin, const Pend pprev,
                                            double coef, int tb0, int tb1, ChunkStage<double2> *cst, double *buf)
{
    const Csr &A = SIDE == 0 ? a.zadj : a.zfwd;
    const bool has_prev = SIDE == 1 || j > 1;
    const double2 *x = reinterpret_cast<const double2 *>(SIDE == 0 ? ucol<double>(a, j - 1) : vcol<double>(a, j - 1));
    double2 *out = reinterpret_cast<double2 *>(SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j));
    double2 *prev = has_prev ? reinterpret_cast<double2 *>(SIDE == 0 ? vcol<double>(a, j - 2) : ucol<double>(a, j - 1))
                             : nullptr;
    // this phase rewrites the output column and (deferred scale) the
    // previous one: their planes no longer hold them
    if (a.okU && blockIdx.x == 0 && threadIdx.x == 0) {
        int *ok = SIDE == 0 ? a.okV : a.okU;
        ok[SIDE == 0 ? j - 1 : j] = 0;
        if (has_prev) ok[SIDE == 0 ? j - 2 : j - 1] = 0;
    }
    double sq = 0.0, dr = 0.0, di = 0.0;
    auto scale = [](double2 v, const Pend &p) { return make_double2(apply_pend(v.x, p), apply_pend(v.y, p)); };
    auto epi = [&](int r, double2 acc, double2 pv) {
        double2 y = scale(acc, pin);
        if (has_prev) {
            if (pprev.mode) {
                pv = scale(pv, pprev);
                prev[r] = pv;
            }
            y.x = fma(-coef, pv.x, y.x);
            y.y = fma(-coef, pv.y, y.y);
            zdot_acc(dr, di, pv, y);
        }
        out[r] = y;
        sq = fma(y.x, y.x, sq);
        sq = fma(y.y, y.y, sq);
    };
    auto pre = [&](int r) -> double2 { return has_prev ? prev[r] : make_double2(0.0, 0.0); };
    if (!host_product) {
        auto xl = [&](int c) -> double2 { return x[c]; };
        csr_rows_chunked<double2, double2, ZSPMV_UNROLL>(A.ptr, A.tbase, A.cidx, A.czval, A.rows, xl, pre, epi, cst,
                                                         tb0, tb1);
    } else {
        const int rows = (SIDE == 0 ? a.adj.rows : a.fwd.rows) / 2;
        for (int r = blockIdx.x * BS + threadIdx.x; r < rows; r += gridDim.x * BS) epi(r, out[r], pre(r));
    }
    __syncthreads();  // buf may share the stage's memory
    // Gram-Schmidt is idle while the SpMV runs: its partials hold the imaginary part
    block_sums<BS, 3>({sq, dr, di}, buf, {a.part_sq + blockIdx.x, a.part_dot + blockIdx.x, a.part_cols + blockIdx.x});
}

// projections h = W(:,sel)^H x (the zgemv('C') of zcgs): the work layout of
// dots_f64 with one complex element per 16-byte vector; column c's
// partials go to part_cols rows 2c (re) and 2c+1 (im), and h comes out as
// (re, im) pairs
template <int SIDE>
__device__ __forceinline__ void zdots_f64(const LbArgs &a, int j, int L)
{
    const int len = (SIDE == 0 ? a.adj.rows : a.fwd.rows) / 2;
    const size_t ld = (size_t)(SIDE == 0 ? a.ldv : a.ldu) / 2;
    const double2 *W = reinterpret_cast<const double2 *>(SIDE == 0 ? a.V : a.U);
    const double2 *x =
        reinterpret_cast<const double2 *>(SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j));
    const int chunk = (len + gridDim.x - 1) / gridDim.x;
    const int v0 = blockIdx.x * chunk, v1 = min(len, v0 + chunk);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int c0 = w * DOT_COLS; c0 < L; c0 += (BS / 32) * DOT_COLS) {
        const int nc = min(DOT_COLS, L - c0);
        const double2 *col[DOT_COLS];
#pragma unroll
        for (int u = 0; u < DOT_COLS; u++) col[u] = W + (size_t)a.sel[c0 + (u < nc ? u : 0)] * ld;
        double re[DOT_COLS][2], im[DOT_COLS][2];
#pragma unroll
        for (int u = 0; u < DOT_COLS; u++) re[u][0] = re[u][1] = im[u][0] = im[u][1] = 0.0;
        int v = v0 + lane;
        for (; v + 32 < v1; v += 64) {
            const double2 x0 = x[v], x1 = x[v + 32];
            double2 w0[DOT_COLS], w1[DOT_COLS];
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++) {
                w0[u] = col[u][v];
                w1[u] = col[u][v + 32];
            }
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++) {
                zdot_acc(re[u][0], im[u][0], w0[u], x0);
                zdot_acc(re[u][1], im[u][1], w1[u], x1);
            }
        }
        if (v < v1) {
            const double2 x0 = x[v];
#pragma unroll
            for (int u = 0; u < DOT_COLS; u++) zdot_acc(re[u][0], im[u][0], col[u][v], x0);
        }
#pragma unroll
        for (int u = 0; u < DOT_COLS; u++) {
            const double sr = warp_sum(re[u][0] + re[u][1]);
            const double si = warp_sum(im[u][0] + im[u][1]);
            if (lane == 0 && u < nc) {
                a.part_cols[(size_t)(2 * (c0 + u)) * a.nb + blockIdx.x] = sr;
                a.part_cols[(size_t)(2 * (c0 + u) + 1) * a.nb + blockIdx.x] = si;
            }
        }
    }
}

// x -= W(:,sel) h (the zgemv('N') of zcgs) and ||x||^2, one complex element
// per thread and step; h (as double2) and the selection in shared memory
template <int SIDE, bool BIG>
__device__ __forceinline__ void zupd_f64(const LbArgs &a, int j, int L, double *dyn, double *buf)
{
    // dyn: h as (re, im) | sel, of the block's columns
    double2 *hs = reinterpret_cast<double2 *>(dyn);
    int *ssel = reinterpret_cast<int *>(dyn + 2 * (size_t)(BIG ? min(L, GS_COLS) : L));
    const int len = (SIDE == 0 ? a.adj.rows : a.fwd.rows) / 2;
    const size_t ld = (size_t)(SIDE == 0 ? a.ldv : a.ldu) / 2;
    const double2 *W = reinterpret_cast<const double2 *>(SIDE == 0 ? a.V : a.U);
    double2 *x = reinterpret_cast<double2 *>(SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j));
    double sq = 0.0;
    int b0 = 0;
    do {
        const int nb = BIG ? min(GS_COLS, L - b0) : L;
        const bool last = !BIG || b0 + nb >= L;
        if (BIG && b0 > 0) __syncthreads();
        for (int c = threadIdx.x; c < nb; c += BS) {
            hs[c] = make_double2(a.h[2 * (b0 + c)], a.h[2 * (b0 + c) + 1]);
            ssel[c] = a.sel[b0 + c];
        }
        __syncthreads();
        for (int v = blockIdx.x * BS + threadIdx.x; v < len; v += gridDim.x * BS) {
            double2 acc = x[v];
            int c = 0;
            for (; c + CGS_UNROLL <= nb; c += CGS_UNROLL) {
                double2 wv[CGS_UNROLL];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) wv[u] = W[(size_t)ssel[c + u] * ld + v];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) zfms(acc, wv[u], hs[c + u]);
            }
            for (; c < nb; c++) zfms(acc, W[(size_t)ssel[c] * ld + v], hs[c]);
            x[v] = acc;
            if (last) {
                sq = fma(acc.x, acc.x, sq);
                sq = fma(acc.y, acc.y, sq);
            }
        }
        b0 += GS_COLS;
    } while (BIG && b0 < L);
    block_sums<BS, 1>({sq}, buf, {a.part_sq + blockIdx.x});
}

// ------------------------------------ complex Gram-Schmidt on the planes
// The complex basis read as its real (re, im) arrays: one complex element is
// one float4 of planes (re hi, re lo, im hi, im lo), split, flagged and
// scaled exactly as in the real kernels above.  The projection
// h = sum conj(w) x has Re h = sum (w.re x.re + w.im x.im), the real dot of
// the two arrays, and Im h = sum (w.re x.im - w.im x.re), the same loaded
// values with the parts of x swapped and one negated: two compensated sums
// per column, four plane products per element, on the FP32 pipe where the
// FP64 kernels spend four FP64 FMAs per 16 bytes.

// projections h = W(:,sel)^H x (zgemv 'C' of zcgs, zreorth.F) from the
// planes: the work layout of dots_pl with two columns per group
// (their re and im sums are the four sums of pl_warp_sum4); partials of
// column c go to part_cols rows 2c (re) and 2c+1 (im), h comes out as
// (re, im) pairs
constexpr int ZPL_COLS = 2;
template <int SIDE, bool BIG>
__device__ __forceinline__ void zdots_pl(const LbArgs &a, int j, int L, double *wpart)
{
    // wpart: [PL_WARPS][2 WPART_COLS] per-slice partials | sel of GS_COLS columns and their stale flags
    int *ssel = reinterpret_cast<int *>(wpart + PL_WARPS * 2 * WPART_COLS);
    unsigned char *sstale = reinterpret_cast<unsigned char *>(ssel + min(a.kmax + 1, GS_COLS));
    const int *ok = SIDE == 0 ? a.okV : a.okU;
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;  // real scalars: twice the complex length
    const size_t ld = SIDE == 0 ? a.ldv : a.ldu;
    const size_t ldq = ld / 2;  // leading dimension in float4 (one complex element)
    const double *W = (const double *)(SIDE == 0 ? a.V : a.U);
    float2 *Wp = SIDE == 0 ? a.Vp : a.Up;
    const double *x = SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j);
    const double2 *xv = reinterpret_cast<const double2 *>(x);
    float4 *xq = reinterpret_cast<float4 *>(a.xpl);
    const int nvec = len / 2;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int chunk = (nvec + gridDim.x - 1) / gridDim.x;
    const int cb0 = min(nvec, blockIdx.x * chunk), cb1 = min(nvec, cb0 + chunk);
    const int rs = dot_slices(chunk), ws = w % rs, wg = w / rs, cgs = PL_WARPS / rs;
    const int sl = (cb1 - cb0 + rs - 1) / rs;
    const int v0 = min(cb1, cb0 + ws * sl), v1 = min(cb1, v0 + sl);
    int xe = 0;
    for (int v = v0 + lane; v < v1; v += 32) {
        const double2 xx = xv[v];
        xe = max(xe, max(f3_expo(xx.x), f3_expo(xx.y)));
    }
    xe = __reduce_max_sync(0xffffffffu, xe);
    const int xs = xe == 0 ? 0 : xe - 1023;
    const double back = f3_pow2(xs);
    for (int v = v0 + lane; v < v1; v += 32) {
        const double2 xx = xv[v];
        const float2 p = pl_xsplit(xx.x, xs), q = pl_xsplit(xx.y, xs);
        xq[v] = make_float4(p.x, p.y, q.x, q.y);
    }
    // conj(w) x into (re, im): w = (w.x + w.y, w.z + w.w), x likewise
    auto zacc = [](PlAcc &re, PlAcc &im, const float4 &wv, const float4 &xq4) {
        re.add(wv.x, wv.y, xq4.x, xq4.y);
        re.add(wv.z, wv.w, xq4.z, xq4.w);
        im.add(wv.x, wv.y, xq4.z, xq4.w);
        im.add(wv.z, wv.w, -xq4.x, -xq4.y);
    };
    int s0 = 0;
    do {
        const int s1 = BIG ? min(L, s0 + GS_COLS) : L;
        for (int c = threadIdx.x; c < s1 - s0; c += BS) {
            const int col = a.sel[s0 + c];
            ssel[c] = col;
            sstale[c] = ok[col] == 0;
        }
        __syncthreads();
        // planes of the stale columns, on this lane's rows
        for (int c = 0; c < s1 - s0; c++) {
            if (!sstale[c] || (c / ZPL_COLS) % cgs != wg) continue;
            const int col = ssel[c];
            float4 *Wq = reinterpret_cast<float4 *>(Wp) + (size_t)col * ldq;
            const double2 *Wd = reinterpret_cast<const double2 *>(W + (size_t)col * ld);
            int v = v0 + lane;
            for (; v + 32 * (PL_SPLIT_UNROLL - 1) < v1; v += 32 * PL_SPLIT_UNROLL) {
                double2 d[PL_SPLIT_UNROLL];
#pragma unroll
                for (int u = 0; u < PL_SPLIT_UNROLL; u++) d[u] = Wd[v + 32 * u];
#pragma unroll
                for (int u = 0; u < PL_SPLIT_UNROLL; u++) Wq[v + 32 * u] = pl_split2(d[u]);
            }
            for (; v < v1; v += 32) Wq[v] = pl_split2(Wd[v]);
        }
        for (int b0 = s0; b0 < s1; b0 += WPART_COLS) {
            const int b1 = min(s1, b0 + WPART_COLS);
            for (int cb = b0 + wg * ZPL_COLS; cb < b1; cb += cgs * ZPL_COLS) {
                const int nc = min(ZPL_COLS, b1 - cb);
                const float4 *Wq[ZPL_COLS];
#pragma unroll
                for (int u = 0; u < ZPL_COLS; u++)
                    Wq[u] = reinterpret_cast<const float4 *>(Wp) + (size_t)ssel[cb - s0 + (u < nc ? u : 0)] * ldq;
                PlAcc acc[2 * ZPL_COLS];  // re, im of column cb, then of column cb + 1
                int v = v0 + lane;
                for (; v + 32 < v1; v += 64) {
                    float4 w0[ZPL_COLS], w1[ZPL_COLS];
#pragma unroll
                    for (int u = 0; u < ZPL_COLS; u++) {
                        w0[u] = __ldcs(Wq[u] + v);
                        w1[u] = __ldcs(Wq[u] + v + 32);
                    }
                    const float4 x0 = xq[v], x1 = xq[v + 32];
#pragma unroll
                    for (int u = 0; u < ZPL_COLS; u++) {
                        zacc(acc[2 * u], acc[2 * u + 1], w0[u], x0);
                        zacc(acc[2 * u], acc[2 * u + 1], w1[u], x1);
                    }
                }
                if (v < v1) {
                    const float4 x0 = xq[v];
#pragma unroll
                    for (int u = 0; u < ZPL_COLS; u++) zacc(acc[2 * u], acc[2 * u + 1], __ldcs(Wq[u] + v), x0);
                }
                static_assert(2 * ZPL_COLS == 4, "pl_warp_sum4 sums four accumulators");
                const PlAcc tot = pl_warp_sum4(acc);
                const int q = lane >> 3;  // accumulator q: column cb + q / 2, part q % 2
                if ((lane & 7) == 0 && (q >> 1) < nc) wpart[(ws * WPART_COLS + cb - b0) * 2 + q] = tot.value() * back;
            }
            __syncthreads();
            for (int c = threadIdx.x; c < 2 * (b1 - b0); c += BS) {
                double s = 0.0;
                for (int ww = 0; ww < rs; ww++) s += wpart[ww * 2 * WPART_COLS + c];
                a.part_cols[(size_t)(2 * b0 + c) * a.nb + blockIdx.x] = s;
            }
            __syncthreads();
        }
        s0 += GS_COLS;
    } while (BIG && s0 < L);
}

// x -= W(:,sel) h (zgemv 'N' of zcgs) from the planes, and ||x||^2: one
// complex element per thread and step; h (scaled by the power of two of its
// largest part) in shared memory as float4 planes (re hi, re lo, im hi,
// im lo); Re and Im of each row's sum formed on the FP32 pipe and applied
// with FP64 FMAs
template <int SIDE, bool BIG>
__device__ __forceinline__ void zupd_pl(const LbArgs &a, int j, int L, double *dyn, double *buf)
{
    // dyn: h as float4 planes (two double slots each) | sel, of the block's columns
    __shared__ int hsh;
    float4 *hp = reinterpret_cast<float4 *>(dyn);
    int *ssel = reinterpret_cast<int *>(dyn + 2 * (size_t)(BIG ? min(L, GS_COLS) : L));
    if (threadIdx.x == 0) hsh = 0;
    __syncthreads();
    int he = 0;
    for (int c = threadIdx.x; c < 2 * L; c += BS) he = max(he, f3_expo(a.h[c]));
    if (he) atomicMax(&hsh, he);
    __syncthreads();
    const int hs = hsh == 0 ? 0 : hsh - 1023;  // |h 2^-hs| < 2
    const double hscale = f3_pow2(-hs), back = f3_pow2(hs);
    const int len = SIDE == 0 ? a.adj.rows : a.fwd.rows;
    const size_t ldq = (size_t)(SIDE == 0 ? a.ldv : a.ldu) / 2;
    const float4 *Wq = reinterpret_cast<const float4 *>(SIDE == 0 ? a.Vp : a.Up);
    double2 *xv = reinterpret_cast<double2 *>(SIDE == 0 ? vcol<double>(a, j - 1) : ucol<double>(a, j));
    const int nvec = len / 2;
    // w h into (re, im)
    auto zmul = [](PlAcc &re, PlAcc &im, const float4 &wv, const float4 &h) {
        re.add(wv.x, wv.y, h.x, h.y);
        re.add(wv.z, wv.w, -h.z, -h.w);
        im.add(wv.x, wv.y, h.z, h.w);
        im.add(wv.z, wv.w, h.x, h.y);
    };
    double sq = 0.0;
    int b0 = 0;
    do {
        const int nb = BIG ? min(GS_COLS, L - b0) : L;
        const bool last = !BIG || b0 + nb >= L;
        if (BIG && b0 > 0) __syncthreads();
        for (int c = threadIdx.x; c < nb; c += BS) {
            const float2 hr = pl_split(a.h[2 * (b0 + c)] * hscale), hi = pl_split(a.h[2 * (b0 + c) + 1] * hscale);
            hp[c] = make_float4(hr.x, hr.y, hi.x, hi.y);
            ssel[c] = a.sel[b0 + c];
        }
        __syncthreads();
        for (int v = blockIdx.x * BS + threadIdx.x; v < nvec; v += gridDim.x * BS) {
            const double2 x0 = xv[v];
            PlAcc sr, si;
            int c = 0;
            for (; c + CGS_UNROLL <= nb; c += CGS_UNROLL) {
                float4 wv[CGS_UNROLL];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) wv[u] = Wq[(size_t)ssel[c + u] * ldq + v];
#pragma unroll
                for (int u = 0; u < CGS_UNROLL; u++) zmul(sr, si, wv[u], hp[c + u]);
            }
            for (; c < nb; c++) zmul(sr, si, Wq[(size_t)ssel[c] * ldq + v], hp[c]);
            double2 y;
            y.x = fma(-pl_f2d(sr.c), back, fma(-pl_f2d(sr.s), back, x0.x));
            y.y = fma(-pl_f2d(si.c), back, fma(-pl_f2d(si.s), back, x0.y));
            xv[v] = y;
            if (last) {
                sq = fma(y.x, y.x, sq);
                sq = fma(y.y, y.y, sq);
            }
        }
        b0 += GS_COLS;
    } while (BIG && b0 < L);
    block_sums<BS, 1>({sq}, buf, {a.part_sq + blockIdx.x});
}

// --------------------------------------------------------- the run kernel
// Lanczos steps j0 .. k in one cooperative launch: the phases of each half
// step follow one another behind a grid barrier, and a phase that is not due
// (no ELR, no reorthogonalisation, its passes converged) costs nothing.  As
// one kernel per phase, a half step was six launches (ELR and two
// Gram-Schmidt passes enqueued ahead, most of which found nothing to do, at
// ~2.6 us each) whose tails each reloaded the scalar state.
//
// The barrier has one master, CTA 0: the others add to an arrival counter;
// CTA 0 waits for them, runs the tail -- the fixed-order sums of the phase's
// partials and dlanbpro's scalar logic, its state and the recurrences'
// arrays staying in CTA 0's shared memory for the whole run -- and releases
// the grid with a word that carries what comes next.  All CTAs are
// co-resident (cooperative launch); every wait is bounded and reports
// through sync[2].
enum { GO_NEXT = 0, GO_ELR = 1, GO_CGS = 2, GO_STOP = 3 };
enum { GS_PL = 0, GS_F64 = 1, GS_F3 = 2 };  // Gram-Schmidt arithmetic of the instance
constexpr unsigned RUN_SPIN_LIMIT = 1u << 24;
constexpr size_t RUN_SMEM_L1 = 15 * 1024;  // a CTA's shared memory, so that four (and 1 KB each) fit in 64 KB
constexpr int RUN_SMEM_KMAX = 300;  // recurrences in shared memory up to this dimension (17 KB of it)

__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct Run {
    unsigned gen = 0;
    unsigned *word;  // shared: the word of the latest release
};
// One grid barrier; tail() runs in CTA 0 between the last arrival and the
// release (all its threads) and returns what comes next (in every thread or
// in thread 0).  Returns that in every thread of the grid.
template <typename F>
__device__ __forceinline__ int grid_step(const RunArgs &R, Run &rn, F tail)
{
    __syncthreads();  // every thread's writes of the phase have been issued
    const unsigned gen = ++rn.gen & 0x3fffffffu;
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            const unsigned want = rn.gen * (gridDim.x - 1);
            unsigned n = 0;
            while (ld_relaxed(R.sync) != want && ++n < RUN_SPIN_LIMIT) {}
            if (n >= RUN_SPIN_LIMIT) R.sync[2] = 1u;
            *rn.word = n >= RUN_SPIN_LIMIT ? 1u : 0u;
            __threadfence();
        }
        __syncthreads();
        int go = GO_STOP;
        if (*rn.word == 0u) go = tail();
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned v = gen << 2 | (unsigned)go;
            __threadfence();
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(R.sync + 1), "r"(v) : "memory");
            *rn.word = v;
        }
    } else if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(R.sync), "r"(1u) : "memory");
        unsigned n = 0, v;
        while (((v = ld_relaxed(R.sync + 1)) >> 2) != gen && ++n < RUN_SPIN_LIMIT)
            if (n > 256) __nanosleep(64);
        if (n >= RUN_SPIN_LIMIT) {
            R.sync[2] = 1u;
            v = GO_STOP;
        }
        __threadfence();
        *rn.word = v;
    }
    __syncthreads();
    return (int)(*rn.word & 3u);
}

// what comes next, by the control block (CTA 0 after a tail); publishes the
// scalars that the next phase reads
__device__ __forceinline__ int tail_end(const RunArgs &R, Tail &t, int kind, unsigned long long &mark)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        *R.pub = publish(t.c);
        if (R.prof) {
            const unsigned long long now = global_ns();
            t.c.prof_ns[kind] += now - mark;
            t.c.prof_n[kind] += 1;
            mark = now;
        }
    }
    return t.c.status ? GO_STOP : t.c.elr_active ? GO_ELR : t.c.reorth_active ? GO_CGS : GO_NEXT;
}

template <typename T, int SHORT>
struct RunShared {
    union {
        SpmvShared<T, SHORT> spmv;
        // partial sums of the closing reductions (three with complex products)
        double buf[(SHORT == 1 && !std::is_same<T, double2>::value ? 2 : 3) * BS];
    };
    Tail t;  // CTA 0
    unsigned word;
    int tiles[2][SPMV_WARPS][2];  // chunked schedule: each warp's tiles of A' and A
};

// The phases of one half step; returns true when the run stops.
// T double2: a native complex operator (or a host product); BLOCK: complex
// vectors with the real 2x2-block operator (T double).
template <int SIDE, typename T, int SHORT, int GS, bool BLOCK, bool BIG>
__device__ __forceinline__ bool run_half(const LbArgs &a, const RunArgs &R, RunShared<T, SHORT> &sh, double *dyn,
                                         Run &rn, int j, unsigned long long &mark)
{
    constexpr bool ZV = std::is_same<T, double2>::value;  // complex products
    constexpr bool CPLX = ZV || BLOCK;                    // complex inner products
    Tail &t = sh.t;
    const int w = threadIdx.x >> 5;
    if (R.r > 0 && !R.host_product) {
        // low-rank prepass z = w .* (R' v) or w .* (L' u)
        if constexpr (!ZV && !BLOCK) {
            thin_phase<T>(SIDE == 0 ? R.thin_l : R.thin_r, SIDE == 0 ? ucol<T>(a, j - 1) : vcol<T>(a, j - 1), R.w,
                          R.zpart, R.z, R.ztick);
            if (grid_step(R, rn, [&]() { return tail_end(R, t, 5, mark) & 0; }) == GO_STOP) return true;
        }
    }
    const LbPub *pub = R.pub;
    const Pend pin = SIDE == 0 ? pub->pend_u : pub->pend_v;
    const Pend pprev = SIDE == 0 ? pub->pend_v : pub->pend_u;
    const double coef = SIDE == 0 ? pub->beta : pub->alpha;
    const int tb0 = sh.tiles[SIDE][w][0], tb1 = sh.tiles[SIDE][w][1];
    int go;
    if constexpr (ZV) {
        zspmv_phase<SIDE>(a, j, R.host_product, pin, pprev, coef, tb0, tb1, sh.spmv.cst, sh.buf);
        go = grid_step(R, rn, [&]() {
            sum_parts<3>({a.part_sq, a.part_dot, a.part_cols}, gridDim.x, sh.buf, t);
            after_spmv<SIDE>(t, a, j, true);
            return tail_end(R, t, SIDE, mark);
        });
    } else {
        spmv_phase<SIDE, T, SHORT>(a, j, R.host_product, pin, pprev, (T)coef, tb0, tb1, sh.spmv, sh.buf);
        go = grid_step(R, rn, [&]() {
            sum_parts<2>({a.part_sq, a.part_dot}, gridDim.x, sh.buf, t);
            after_spmv<SIDE>(t, a, j);
            return tail_end(R, t, SIDE, mark);
        });
    }
    while (go == GO_ELR) {
        if constexpr (CPLX) {
            const bool dot_only = pub->elr_need_dot != 0;
            zelr_phase<SIDE>(a, j, dot_only, pub->elr_s, pub->elr_s_im, sh.buf);
            go = grid_step(R, rn, [&]() {
                sum_parts<3>({a.part_sq, a.part_dot, a.part_cols}, gridDim.x, sh.buf, t);
                if (dot_only) {
                    if (threadIdx.x == 0) {
                        t.c.elr_s = t.red[1];
                        t.c.elr_s_im = t.red[2];
                        t.c.elr_need_dot = 0;
                    }
                } else {
                    after_elr<SIDE>(t, a, j);
                }
                return tail_end(R, t, 2, mark);
            });
        } else {
            elr_phase<SIDE, T>(a, j, (T)pub->elr_s, sh.buf);
            go = grid_step(R, rn, [&]() {
                sum_parts<2>({a.part_sq, a.part_dot}, gridDim.x, sh.buf, t);
                after_elr<SIDE>(t, a, j);
                return tail_end(R, t, 2, mark);
            });
        }
    }
    while (go == GO_CGS) {
        const int L = pub->nsel, ncols = CPLX ? 2 * L : L;
        if constexpr (CPLX && GS == GS_PL) zdots_pl<SIDE, BIG>(a, j, L, dyn);
        else if constexpr (CPLX) zdots_f64<SIDE>(a, j, L);
        else if constexpr (std::is_same<T, float>::value) dots_f32<SIDE, BIG>(a, j, L, dyn);
        else if constexpr (GS == GS_PL) dots_pl<SIDE, BIG>(a, j, L, dyn);
        else if constexpr (GS == GS_F3) dots_f3<SIDE>(a, j, L);
        else dots_f64<SIDE>(a, j, L);
        // the CTAs' partials: few by CTA 0, many by one warp of the grid per
        // column behind a second barrier (all of them through one SM would
        // take longer than that barrier)
        const bool wide = (long long)ncols * gridDim.x > 8192;
        if (grid_step(R, rn, [&]() {
                if (GS == GS_PL && a.okU) {
                    int *ok = SIDE == 0 ? a.okV : a.okU;
                    for (int c = threadIdx.x; c < L; c += BS) ok[a.sel[c]] = 1;
                }
                if (wide) return (int)GO_CGS;
                reduce_cols(a, ncols, gridDim.x, w, BS / 32);
                return tail_end(R, t, 3, mark);
            }) == GO_STOP)
            return true;
        if (wide) {
            reduce_cols(a, ncols, gridDim.x, blockIdx.x * (BS / 32) + w, gridDim.x * (BS / 32));
            if (grid_step(R, rn, [&]() { return tail_end(R, t, 3, mark); }) == GO_STOP) return true;
        }
        if constexpr (CPLX && GS == GS_PL) zupd_pl<SIDE, BIG>(a, j, L, dyn, sh.buf);
        else if constexpr (CPLX) zupd_f64<SIDE, BIG>(a, j, L, dyn, sh.buf);
        else if constexpr (std::is_same<T, double>::value && GS == GS_PL) upd_pl<SIDE, BIG>(a, j, L, dyn, sh.buf);
        else if constexpr (std::is_same<T, double>::value && GS == GS_F3) upd_f3<SIDE, BIG>(a, j, L, dyn, sh.buf);
        else upd_full<SIDE, T, BIG>(a, j, L, dyn, sh.buf);
        go = grid_step(R, rn, [&]() {
            sum_parts<1>({a.part_sq}, gridDim.x, sh.buf, t);
            after_cgs<SIDE>(t, a, j);
            return tail_end(R, t, 4, mark);
        });
    }
    return go == GO_STOP;
}

// CTAs per SM the instances are compiled for: 64 registers for the chunked
// real products (four CTAs: the gathers in flight are what the SpMV needs),
// 80 for complex values and for the staged schedule
template <typename T, int SHORT>
constexpr int run_minb() { return SHORT == 1 && !std::is_same<T, double2>::value ? 4 : 3; }

template <typename T, int SHORT, int GS, bool BLOCK, bool BIG>
__global__ void __launch_bounds__(BS, run_minb<T, SHORT>()) k_lb_run(const __grid_constant__ LbArgs a,
                                                                     const __grid_constant__ RunArgs R)
{
    constexpr bool ZV = std::is_same<T, double2>::value;
    extern __shared__ __align__(16) double dyn[];  // float4 and double2 in the complex updates
    __shared__ RunShared<T, SHORT> sh;
    Run rn;
    rn.word = &sh.word;
    const int w = threadIdx.x >> 5;
    unsigned long long mark = 0;
    if (!R.host_product) {
        const Csr &A0 = ZV ? a.zadj : a.adj, &A1 = ZV ? a.zfwd : a.fwd;
        int q[2][2] = {{0, 0}, {0, 0}};
        if (SHORT == 1 || A0.short_rows) chunk_warp_tiles(A0.tbase, A0.rows, q[0][0], q[0][1]);
        if (SHORT == 1 || A1.short_rows) chunk_warp_tiles(A1.tbase, A1.rows, q[1][0], q[1][1]);
        if ((threadIdx.x & 31) == 0)
            for (int i = 0; i < 4; i++) sh.tiles[i >> 1][w][i & 1] = q[i >> 1][i & 1];
    }
    if (blockIdx.x == 0) {
        Tail &t = sh.t;
        const int n = a.kmax + 2;
        if (threadIdx.x == 0) {
            t.c = *a.ctl;
            double *p = dyn + R.smem_tail;
            const bool in = R.smem_tail > 0;
            t.ba = in ? p : a.balpha;
            t.bb = in ? p + n : a.bbeta;
            t.mu = in ? p + 2 * n : a.mu;
            t.nu = in ? p + 3 * n : a.nu;
            t.hA = in ? p + 4 * n : nullptr;
            t.hB = in ? p + 5 * n : nullptr;
            t.index = in ? reinterpret_cast<int *>(p + 6 * n) : a.index;
            if (R.prof) mark = global_ns();
        }
        __syncthreads();
        if (R.smem_tail > 0) {
            for (int i = threadIdx.x; i < n; i += BS) {
                t.ba[i] = a.balpha[i];
                t.bb[i] = a.bbeta[i];
                t.mu[i] = a.mu[i];
                t.nu[i] = a.nu[i];
                t.hA[i] = tail_hypot(a.balpha[i], a.bbeta[i]);
                t.hB[i] = i > 0 ? tail_hypot(a.balpha[i], a.bbeta[i - 1]) : 0.0;
            }
            for (int i = threadIdx.x; i < 2 * a.kmax + 8; i += BS) t.index[i] = a.index[i];
        }
    }
    // the scalars of the first phase
    grid_step(R, rn, [&]() {
        if (threadIdx.x == 0) *R.pub = publish(sh.t.c);
        return (int)GO_NEXT;
    });
    for (int j = R.j0; j <= R.j1; j++) {
        if (j > R.j0 || R.side0 == 0)
            if (run_half<0, T, SHORT, GS, BLOCK, BIG>(a, R, sh, dyn, rn, j, mark)) break;
        if (j < R.j1 || R.side1 == 1)
            if (run_half<1, T, SHORT, GS, BLOCK, BIG>(a, R, sh, dyn, rn, j, mark)) break;
    }
    if (blockIdx.x == 0) {
        Tail &t = sh.t;
        const int n = a.kmax + 2;
        __syncthreads();
        if (R.smem_tail > 0) {
            for (int i = threadIdx.x; i < n; i += BS) {
                a.balpha[i] = t.ba[i];
                a.bbeta[i] = t.bb[i];
                a.mu[i] = t.mu[i];
                a.nu[i] = t.nu[i];
            }
            for (int i = threadIdx.x; i < 2 * a.kmax + 8; i += BS) a.index[i] = t.index[i];
        }
        if (threadIdx.x == 0) *a.ctl = t.c;
    }
}

// ------------------------------------------------------------ host side
// shared memory of the projections (with planes, or of the FP32 form): the
// slices' partials (complex: re, im), the selection and its stale flags
inline size_t dots_smem(int kmax, bool cplx)
{
    return sizeof(double) * PL_WARPS * (cplx ? 2 : 1) * WPART_COLS + (sizeof(int) + 1) * (size_t)std::min(kmax + 1, GS_COLS);
}
// of the update: h (wide: two double slots per column) and the selection
inline size_t upd_smem(int kmax, bool wide)
{
    return ((wide ? 2 : 1) * sizeof(double) + sizeof(int)) * (size_t)std::min(kmax + 1, GS_COLS) + 16;
}

template <typename T, int SHORT, int GS, bool BLOCK, bool BIG>
static void launch_run_as(LbArgs a, RunArgs R, int want, cudaStream_t s)
{
    // dynamic shared memory: the Gram-Schmidt phases', then (CTA 0) the recurrences
    const int K = a.kmax;
    constexpr bool cplx = BLOCK || std::is_same<T, double2>::value;
    const bool wp = GS == GS_PL || std::is_same<T, float>::value;
    size_t sm = std::max(upd_smem(K, cplx || GS == GS_F3), wp ? dots_smem(K, cplx) : (size_t)0);
    sm = (sm + 15) / 16 * 16;
    const Dev &d = device_info();
    const size_t tail = sizeof(double) * 6 * (size_t)(K + 2) + sizeof(int) * (2 * (size_t)K + 8);
    // A grid that fills the chip keeps the recurrences in global memory where
    // they would take the CTAs past RUN_SMEM_L1: one scalar tail a half step is
    // a microsecond longer, but the L1 that holds the gathers grows (4M rows,
    // dimension 150, product and adjoint: 211 and 190 us with 100 KB of shared
    // memory per SM, 207 and 184 with 64 KB, 233 and 214 with 132 KB).
    const bool fills = want >= run_minb<T, SHORT>() * d.sms;
    R.smem_tail = 0;
    if (K <= RUN_SMEM_KMAX &&
        !(SHORT == 1 && fills && sizeof(RunShared<T, SHORT>) + sm + tail > RUN_SMEM_L1)) {
        R.smem_tail = (int)(sm / sizeof(double));
        sm += tail;
    }
    // the smallest carve-out for this size, left to L1 what it leaves (the
    // runtime's own choice is larger: 64 KB asked for, 4M rows, dimension
    // 150: 195 and 217 us with its choice, 188 and 211 with this one)
    const size_t need = run_minb<T, SHORT>() * (sm + sizeof(RunShared<T, SHORT>) + 1024);
    int kb = 228;
    for (int c : {196, 164, 132, 100, 64, 32})
        if (need <= (size_t)c * 1024) kb = c;
    const void *fn = (const void *)k_lb_run<T, SHORT, GS, BLOCK, BIG>;
    PGB_CUDA(cudaMemsetAsync(R.sync, 0, 3 * sizeof(unsigned), s));
    // The carve-out belongs to the kernel, not to the caller's thread, and a
    // cooperative launch may not exceed the occupancy under it: hint, occupancy
    // and launch are one critical section, and a call finds the hint of
    // whichever thread launched last.
    struct Hint {
        int kb = 0, per = 0;
        size_t smem = 0;
    };
    static std::mutex mu;
    static std::map<int, Hint> hints;  // by device
    std::lock_guard<std::mutex> lk(mu);
    Hint &h = hints[d.device];
    if (h.kb != kb || h.smem != sm) {
        if (h.kb == 0) allow_dynamic_smem(fn);
        if (h.kb != kb)
            PGB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, (kb * 100 + 227) / 228));
        h = Hint();  // a failed question leaves nothing behind
        int per = 0;
        PGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, BS, sm));
        h.kb = kb;
        h.per = per;
        h.smem = sm;
    }
    const int g = std::max(1, std::min(want, std::min(d.nb, std::max(1, h.per) * d.sms)));
    a.nb = g;
    void *args[] = {&a, &R};
    PGB_CUDA(cudaLaunchCooperativeKernel(fn, dim3(g), dim3(BS), args, sm, s));
    PGB_LAUNCHED();
}
template <typename T, int SHORT, int GS, bool BLOCK>
static void launch_run(const LbArgs &a, const RunArgs &R, int want, cudaStream_t s)
{
    if (a.kmax + 1 > GS_COLS) launch_run_as<T, SHORT, GS, BLOCK, true>(a, R, want, s);
    else launch_run_as<T, SHORT, GS, BLOCK, false>(a, R, want, s);
}

}  // namespace pgb

// pgb_bidiag.cuh -- lane-parallel numerics for the small upper bidiagonal R
// (diagonal d[0..n-1], superdiagonal e[0..n-2]) that the IRL analysis and
// the Ritz-vector step need.
//
// Why not the QR iteration the reference uses (Lapack_Util/dbdsqr.f):
// its rotation chain is one dependent sequence of FP64 operations, and on
// this GPU an FP64 instruction issued for one thread occupies the FP64 pipe
// as long as one issued for a full warp (2 FP64 lanes per clock per SM), so
// a thread-serial chain runs ~30x slower than on a CPU core.  The methods
// here keep every lane of a warp busy instead:
//
//   singular values   warp multisection on the Golub-Kahan tridiagonal
//                     TGK = tridiag(b; 0; b), b = (d1, e1, d2, e2, ..., dn),
//                     whose eigenvalues are +-sigma_i.  The Sturm count of
//                     TGK - x I (LDL' pivots of a zero-diagonal matrix)
//                     locates sigma_i to high relative accuracy (Demmel &
//                     Kahan 1990, section 7); 32 lanes evaluate 31 points per
//                     round, 5 bits per round.
//   vectors           the twisted factorization of TGK - sigma I (Parlett &
//                     Dhillon 1997; the "getvec" step of MRRR): forward and
//                     backward pivot sequences, twist index r = argmin
//                     |gamma_r|, then z from both ends.  z = (x1, y1, x2,
//                     y2, ...)/sqrt(2) with R x = sigma y; one warp per value.
//
// All functions are plain arithmetic on caller-provided storage, so the same
// code serves any dimension.
#pragma once
#include "pgb.cuh"
#include "pgb_scalar.cuh"

namespace pgb {

// number of negative pivots of TGK - lam I (size N = 2n)
__device__ __forceinline__ int tgk_negcount(int N, const double *b2, double lam, double pivmin)
{
    double D = -lam;
    if (fabs(D) < pivmin) D = -pivmin;
    int cnt = D < 0.0;
    for (int j = 1; j < N; j++) {
        D = -lam - b2[j - 1] / D;
        if (fabs(D) < pivmin) D = -pivmin;
        cnt += D < 0.0;
    }
    return cnt;
}

// The same count without a division in the chain: p_j = -lam p_{j-1} -
// b2_{j-1} p_{j-2} are the leading principal minors (Wilkinson's Sturm
// sequence; the pivots above are p_j / p_{j-1}, so a negative pivot is a sign
// change).  Two FP64 instructions per step (128 cycles: one warp gets one per
// 64 on this GPU), where the pivot recurrence waited for a division (~1000).
// The roundings of a step move the b2 it uses by a few eps relative, as those
// of the pivot recurrence do (divide by p_{j-1}), so the count is as accurate.
// The caller scales the matrix (tgk_scale) so that |b| <= 1 and lam <= 1:
// |p| then grows by less than 2^12 in TGK_RESCALE steps, and shrinks by no
// more than lam^TGK_RESCALE >= 2^-640, and is brought back to exponent 0
// after them.  A p of exactly 0 takes the sign opposite to its predecessor's
// (the pivot guard's); two in a row (an exact eigenvalue of a decoupled
// leading block) leave no sign to count, and the caller falls back on the
// pivots.  lam < TGK_POLY_MIN (values below 1e-12 sigma_1) keeps the pivots.
constexpr int TGK_RESCALE = 16;
constexpr double TGK_POLY_MIN = 9.094947017729282e-13;  // 2^-40

__device__ __forceinline__ bool tgk_is_zero(double p)
{
    return ((unsigned)__double2hiint(p) << 1 | (unsigned)__double2loint(p)) == 0u;
}
__device__ __forceinline__ void tgk_rescale(double &p1, double &p0)
{
    const int e1 = (__double2hiint(p1) >> 20) & 0x7ff, e0 = (__double2hiint(p0) >> 20) & 0x7ff;
    const int k = 1023 - max(e1, e0);
    const double f = __hiloint2double((min(max(k, -1000), 1000) + 1023) << 20, 0);
    p1 *= f;
    p0 *= f;
}
// the count, or -1 when two successive minors vanish
__device__ __forceinline__ int tgk_negcount_sturm(int N, const double *b2, double lam)
{
    double p0 = 1.0, p1 = -lam;
    int cnt = 1, j = 1;
    int sg = -1;  // sign word of p1
    auto step = [&](double b) {
        const double p2 = fma(-lam, p1, -(b * p0));
        const int s2 = tgk_is_zero(p2) ? ~sg : __double2hiint(p2);
        cnt += (int)((unsigned)(s2 ^ sg) >> 31);
        sg = s2;
        p0 = p1;
        p1 = p2;
    };
    for (; j + TGK_RESCALE <= N; j += TGK_RESCALE) {
#pragma unroll
        for (int q = 0; q < TGK_RESCALE; q++) step(b2[j + q - 1]);
        tgk_rescale(p1, p0);
    }
    for (; j < N; j++) step(b2[j - 1]);
    return tgk_is_zero(p1) && tgk_is_zero(p0) ? -1 : cnt;
}
// the count in FP32 (b2 rounded to FP32, lam >= TGK_F32_MIN): exact for a
// matrix whose entries moved by a few 2^-24 relative, so the values it locates
// are right to about 4 N 2^-24; at a tenth of the FP64 count's time
constexpr float TGK_F32_MIN = 0.000244140625f;  // 2^-12: lam^8 stays far from underflow
__device__ __forceinline__ int tgk_negcount_f32(int N, const float *b2, float lam)
{
    float p0 = 1.f, p1 = -lam;
    int cnt = 1, j = 1;
    while (j < N) {
        const int je = min(N, j + 8);
        for (; j < je; j++) {
            float p2 = fmaf(-lam, p1, -(b2[j - 1] * p0));
            if (p2 == 0.f) p2 = p1 * -1.f;  // any value of the guard's sign
            cnt += (int)((unsigned)(__float_as_int(p2) ^ __float_as_int(p1)) >> 31);
            p0 = p1;
            p1 = p2;
        }
        const int k = 127 - max((__float_as_int(p1) >> 23) & 0xff, (__float_as_int(p0) >> 23) & 0xff);
        const float f = __int_as_float((min(max(k, -120), 120) + 127) << 23);
        p1 *= f;
        p0 *= f;
    }
    return cnt;
}

// The power of two that brings the Gershgorin bound into [1/2, 1); 0 when
// the matrix is too small, too large or not finite to be scaled (the pivot
// recurrence then works on the matrix as it is).
__device__ __forceinline__ double tgk_scale(double gersh)
{
    const int e = (__double2hiint(gersh) >> 20) & 0x7ff;
    return e > 1023 - 400 && e < 1023 + 400 ? __hiloint2double((2045 - e) << 20, 0) : 0.0;
}

// sigma_t (t = 1: largest) of R by warp multisection; all lanes return it.
// b2: the squares of the off-diagonals times sc^2 (sc = 0: unscaled), b2f the
// same in FP32 (scaled only), hi0 an upper bound of sigma_max (Gershgorin of
// TGK) of the unscaled matrix.  Three rounds of FP32 counts find a bracket of
// ~2^-13, which one round of FP64 counts at its widened ends confirms (or the
// search starts from [0, hi0]); FP64 rounds finish, 5 bits each.
__device__ inline double warp_sigma(int n, const double *b2, const float *b2f, int t, double hi0, double pivmin,
                                    double sc)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, N = 2 * n;
    const double guard = sc != 0.0 ? SFMIN : pivmin;
    // #(sigma > p) = 2n - negcount(p) for p > 0
    auto above = [&](double p) {
        int c = -1;
        if (sc != 0.0 && __all_sync(FULL, p >= TGK_POLY_MIN)) c = tgk_negcount_sturm(N, b2, p);
        if (__any_sync(FULL, c < 0)) c = tgk_negcount(N, b2, p, guard);
        return N - c;
    };
    double lo = 0.0, hi = sc != 0.0 ? hi0 * sc : hi0;
    if (sc != 0.0) {
        float fl = 0.f, fh = (float)hi;
        for (int round = 0; round < 3; round++) {
            const float p = fl + (fh - fl) * ((float)(lane + 1) / 33.f);
            if (!__all_sync(FULL, p >= TGK_F32_MIN)) break;
            const unsigned bal = __ballot_sync(FULL, N - tgk_negcount_f32(N, b2f, p) >= t);
            const int q = __popc(bal);
            const float plo = __shfl_sync(FULL, p, q > 0 ? q - 1 : 0), phi = __shfl_sync(FULL, p, q < 32 ? q : 31);
            if (q > 0) fl = plo;
            if (q < 32) fh = phi;
        }
        if (fl > 0.f) {
            const double w = 4.0 * N * 5.9604644775390625e-08;
            const double a = (double)fl * (1.0 - w), z = fmin((double)fh * (1.0 + w), hi);
            const double p = a + (z - a) * ((double)lane / 31.0);
            const unsigned bal = __ballot_sync(FULL, above(p) >= t);
            const int q = __popc(bal);
            if (q > 0 && q < 32) {
                lo = __shfl_sync(FULL, p, q - 1);
                hi = __shfl_sync(FULL, p, q);
            }
        }
    }
    const double frac = (double)(lane + 1) / 33.0;
    for (int round = 0; round < 64; round++) {
        if (hi - lo <= 2.0 * EPS * hi) break;
        const double p = lo + (hi - lo) * frac;
        const unsigned bal = __ballot_sync(FULL, above(p) >= t);
        const int q = __popc(bal);  // counts are monotone: lanes 0..q-1 satisfy
        const double plo = __shfl_sync(FULL, p, q > 0 ? q - 1 : 0);
        const double phi = __shfl_sync(FULL, p, q < 32 ? q : 31);
        const double nlo = q > 0 ? plo : lo, nhi = q < 32 ? phi : hi;
        if (nlo == lo && nhi == hi) break;  // no representable progress
        lo = nlo;
        hi = nhi;
    }
    const double s = 0.5 * (lo + hi);
    return sc != 0.0 ? s / sc : s;
}

// Product of v over the lanes up to this one.
__device__ __forceinline__ double warp_scan_mul(double v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v *= u;
    }
    return v;
}

// Twisted factorization of TGK - lam I by one warp: the unit eigenvector
// goes to bd, |z_N| is returned.  b: off-diagonals, b2 their squares, both
// scaled like lam (scaled: |b| <= 1, see above).  The forward and backward
// minors run in lanes 0 and 1 (one dependent FMA per step); the pivots,
// their ratios, the twist index and the products z_j from it are then formed
// by all lanes.  fn, fd, bn, bd: N doubles of scratch each.
__device__ inline double warp_twisted(int N, const double *b, const double *b2, double lam, double pivmin,
                                      bool scaled, double *fn, double *fd, double *bn, double *bd)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (lane < 2) {
        double *num = lane ? bn : fn, *den = lane ? bd : fd;
        const int i0 = lane ? N - 1 : 0, st = lane ? -1 : 1;
        if (scaled && lam >= TGK_POLY_MIN) {
            double p0 = 1.0, p1 = -lam;
            num[i0] = p1;
            den[i0] = 1.0;
            for (int j = 1; j < N; j++) {
                const int at = i0 + st * j;
                // forward: b2[j-1]; backward: b2[N-1-j]
                double p2 = fma(-lam, p1, -(b2[lane ? at : at - 1] * p0));
                if (tgk_is_zero(p2)) p2 = p1 * -7.888609052210118e-31;  // 2^-100: far below eps lam
                num[at] = p2;
                den[at] = p1;
                p0 = p1;
                p1 = p2;
                if ((j & (TGK_RESCALE - 1)) == 0) tgk_rescale(p1, p0);
            }
        } else {
            double D = -lam;
            if (fabs(D) < pivmin) D = -pivmin;
            num[i0] = D;
            den[i0] = 1.0;
            for (int j = 1; j < N; j++) {
                const int at = i0 + st * j;
                D = -lam - b2[lane ? at : at - 1] / D;
                if (fabs(D) < pivmin) D = -pivmin;
                num[at] = D;
                den[at] = 1.0;
            }
        }
    }
    __syncwarp();
    // pivots; gamma_j = Dp_j + Dm_j - (T - lam I)_jj = Dp_j + Dm_j + lam
    int r = 0;
    double gmin = INFINITY;
    for (int j = lane; j < N; j += 32) {
        const double dp = fn[j] / fd[j], dm = bn[j] / bd[j];
        fn[j] = dp;
        bn[j] = dm;
        const double g = fabs(dp + dm + lam);
        if (g < gmin) { gmin = g; r = j; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double g = __shfl_xor_sync(FULL, gmin, o);
        const int q = __shfl_xor_sync(FULL, r, o);
        if (g < gmin || (g == gmin && q < r)) { gmin = g; r = q; }
    }
    __syncwarp();
    // z_r = 1; z_j = -(b_j / Dp_j) z_{j+1} above r, -(b_{j-1} / Dm_j) z_{j-1} below
    double nrm2 = 0.0, carry = 1.0, zN = 1.0;
    for (int base = r - 1; base >= 0; base -= 32) {
        const int j = base - lane;
        double v = j >= 0 ? -(b[j] / fn[j]) : 1.0;
        v = warp_scan_mul(v) * carry;
        if (j >= 0) {
            bd[j] = v;
            nrm2 += v * v;
        }
        carry = __shfl_sync(FULL, v, 31);
    }
    carry = 1.0;
    for (int base = r + 1; base < N; base += 32) {
        const int j = base + lane;
        double v = j < N ? -(b[j - 1] / bn[j]) : 1.0;
        v = warp_scan_mul(v) * carry;
        if (j < N) {
            bd[j] = v;
            nrm2 += v * v;
        }
        carry = __shfl_sync(FULL, v, 31);
        zN = __shfl_sync(FULL, v, min(31, N - 1 - base));
    }
    nrm2 = warp_sum(nrm2) + 1.0;
    const double inv = 1.0 / sqrt(nrm2);
    __syncwarp();
    if (lane == 0) bd[r] = 1.0;
    __syncwarp();
    for (int j = lane; j < N; j += 32) bd[j] *= inv;
    __syncwarp();
    return fabs(zN) * inv;
}

// dbdqr (double/dbsvd.F:87-157) of the lower bidiagonal with diagonal al
// and subdiagonal be by one warp: R's diagonal to b[0], b[2], ..., its
// superdiagonal to b[1], b[3], ... (the off-diagonals of TGK in order), the
// rotations to c, s.  last: the last row is rotated too (dim != min(m, n));
// otherwise s[n-1] = 0.  The diagonal before rotation i, dt_i, obeys
//   1/dt_{i+1}^2 = (1 + be_i^2 / dt_i^2) / al_{i+1}^2,
// a recurrence of positive terms with one FMA per step (each error is damped
// by the next step's weight < 1); everything else is formed by all lanes.
// Zeros and values whose squares leave the FP64 range take the rotations
// one after the other (dlartg's sequence).
__device__ inline void warp_bdqr(int n, const double *al, const double *be, bool last, double *c, double *s,
                                 double *b)
{
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < n; i += 32) {
        const double g = 1.0 / (al[i] * al[i]);
        c[i] = g;
        s[i] = i > 0 ? be[i - 1] * be[i - 1] * g : 0.0;
    }
    __syncwarp();
    if (lane == 0) {
        double r = c[0];
        b[0] = r;
        for (int i = 1; i < n; i++) {
            r = fma(s[i], r, c[i]);
            b[2 * i] = r;
        }
    }
    __syncwarp();
    bool ok = true;
    for (int i = lane; i < n; i += 32) ok = ok && b[2 * i] > 1e-280 && b[2 * i] < 1e280 && fabs(be[i]) < 1e140;
    if (__all_sync(0xffffffffu, ok)) {
        unsigned par = 0;  // sign of dt_i: the product of the signs of al_0 .. al_i
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const unsigned neg = __ballot_sync(0xffffffffu, i < n && al[i] < 0.0);
            if (i < n) {
                const unsigned q = (__popc(neg & (0xffffffffu >> (31 - lane))) + par) & 1u;
                const double r = b[2 * i], bi = be[i];
                const double dt = q ? -rsqrt(r) : rsqrt(r);
                if (i < n - 1 || last) {
                    const double h = sqrt(fma(bi, bi, 1.0 / r));
                    c[i] = dt / h;
                    s[i] = bi / h;
                    b[2 * i] = h;
                } else {
                    c[i] = 1.0;
                    s[i] = 0.0;
                    b[2 * i] = dt;
                }
                if (i < n - 1) b[2 * i + 1] = s[i] * al[i + 1];
            }
            par += __popc(neg);
        }
    } else if (lane == 0) {
        double dt = al[0], cs, sn, r;
        for (int i = 0; i < n; i++) {
            if (i < n - 1 || last) lartg(dt, be[i], cs, sn, r);
            else { cs = 1.0; sn = 0.0; r = dt; }
            c[i] = cs;
            s[i] = sn;
            b[2 * i] = r;
            if (i < n - 1) {
                b[2 * i + 1] = sn * al[i + 1];
                dt = cs * al[i + 1];
            }
        }
    }
    __syncwarp();
}

// w = Q [y; 0] for the rotations of warp_bdqr (Q' B = [R; 0]), n + 1 entries:
// y at y[t * sy], t < n; w to w[t * sw].  t0: n + 1 doubles of scratch.  The
// chain is one FMA per step in lane 0.
__device__ inline void warp_apply_q(int n, const double *c, const double *s, const double *y, int sy, double *t0,
                                    double *w, size_t sw)
{
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        double t = 0.0;
        t0[n] = 0.0;
        for (int i = n - 1; i >= 0; i--) {
            t = fma(-s[i], t, c[i] * y[i * sy]);
            t0[i] = t;
        }
        w[0] = t;
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) w[(size_t)(i + 1) * sw] = fma(c[i], t0[i + 1], s[i] * y[i * sy]);
    __syncwarp();
}

// Gershgorin bound and pivot guard of TGK from its off-diagonals, one warp
__device__ inline void warp_tgk_bounds(int N, const double *b, double &gersh, double &pivmin)
{
    const int lane = threadIdx.x & 31;
    double g = 0.0, m2 = 0.0;
    for (int j = lane; j < N; j += 32) {
        const double left = j > 0 ? fabs(b[j - 1]) : 0.0, right = j < N - 1 ? fabs(b[j]) : 0.0;
        g = fmax(g, left + right);
        m2 = fmax(m2, right * right);
    }
    gersh = warp_max(g) * (1.0 + 4.0 * EPS) + SFMIN;
    pivmin = SFMIN * fmax(1.0, warp_max(m2));
}

// The off-diagonals of TGK and their squares (b2f: in FP32), scaled by the
// power of two of the Gershgorin bound; one warp.
__device__ inline void stage_tgk(int N, double *b, double *b2, float *b2f, double &gersh, double &pivmin, double &sc)
{
    warp_tgk_bounds(N, b, gersh, pivmin);
    sc = tgk_scale(gersh);
    const double f = sc != 0.0 ? sc : 1.0;
    __syncwarp();
    for (int j = threadIdx.x & 31; j < N - 1; j += 32) {
        const double v = b[j] * f;
        b[j] = v;
        b2[j] = v * v;
        if (b2f) b2f[j] = (float)(v * v);
    }
    __syncwarp();
}

}  // namespace pgb

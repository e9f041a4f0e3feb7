// pgb_lanczos.cu -- the run kernel of the FP64 form (planes), its dispatch, the flush
#include "pgb_lanczos.cuh"

namespace pgb {

// Gram-Schmidt arithmetic of the FP64 form (propack_set_cgs_arith)
thread_local int g_cgs_arith = CGS_PLANES;

// The planes are used when the driver allocated them: FP64 form up to dimension
// 2843, complex vectors 1504.  They take the memory of a second basis on each
// side; beyond these dimensions the bases go without (a solve whose bases fill
// the device still fits) and Gram-Schmidt runs on FP64 FMAs.
bool lb_planes_fit(int kmax, bool cplx) { return kmax <= (cplx ? 1504 : 2843); }

// device words of the barrier, the published scalars
size_t lb_run_scratch() { return 64 + sizeof(LbPub); }

// steps (j0, side0) .. (j1, side1) of dlanbpro on at most `want` CTAs
template <>
void lb_run<double>(const LbArgs &a, RunArgs R, bool, int want, cudaStream_t s)
{
    const bool both_short = R.host_product || (a.fwd.short_rows && a.adj.short_rows);
    if (a.Up && both_short) launch_run<double, 1, GS_PL, false>(a, R, want, s);
    else if (a.Up) launch_run<double, 2, GS_PL, false>(a, R, want, s);
    else lb_run_fp64(a, R, want, s);
}

// apply the deferred scaling of the newest u and v columns
template <typename T>
__global__ void __launch_bounds__(BS) k_lb_flush(LbArgs a)
{
    if (a.ctl->status != 0) return;
    const Pend pu = a.ctl->pend_u, pv = a.ctl->pend_v;
    const int cu = a.ctl->pend_u_col, cv = a.ctl->pend_v_col;
    const int m = a.fwd.rows, n = a.adj.rows;
    const int len = m > n ? m : n;
    T *uc = cu >= 0 ? ucol<T>(a, cu) : nullptr;
    T *vc = cv >= 0 ? vcol<T>(a, cv) : nullptr;
    if (a.okU && blockIdx.x == 0 && threadIdx.x == 0) {
        if (pu.mode && cu >= 0) a.okU[cu] = 0;
        if (pv.mode && cv >= 0) a.okV[cv] = 0;
    }
    for (int r = blockIdx.x * BS + threadIdx.x; r < len; r += gridDim.x * BS) {
        if (pu.mode && uc && r < m) uc[r] = apply_pend(uc[r], pu);
        if (pv.mode && vc && r < n) vc[r] = apply_pend(vc[r], pv);
    }
    if (last_cta(&a.ctl->ticket)) {
        if (threadIdx.x == 0) {
            a.ctl->pend_u.mode = 0;
            a.ctl->pend_v.mode = 0;
            __threadfence();
        }
    }
}

// (complex: the flush of the real scalars, whose lengths LbArgs counts)
template <typename T>
void lb_enqueue_flush(const LbArgs &a, cudaStream_t s)
{
    using E = typename std::conditional<VecW<T>::w == 2, double, T>::type;
    k_lb_flush<E><<<a.nb, BS, 0, s>>>(a);
    PGB_LAUNCHED();
}

template void lb_enqueue_flush<double>(const LbArgs &, cudaStream_t);
template void lb_enqueue_flush<float>(const LbArgs &, cudaStream_t);
template void lb_enqueue_flush<double2>(const LbArgs &, cudaStream_t);

}  // namespace pgb

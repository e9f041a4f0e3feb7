// pgb_lanczos_alt.cu -- the run kernel of the FP32 form and of the FP64 form without planes
#include "pgb_lanczos.cuh"

namespace pgb {

template <>
void lb_run<float>(const LbArgs &a, RunArgs R, bool, int want, cudaStream_t s)
{
    if (R.host_product || (a.fwd.short_rows && a.adj.short_rows)) launch_run<float, 1, GS_F64, false>(a, R, want, s);
    else launch_run<float, 2, GS_F64, false>(a, R, want, s);
}

// the FP64 form on FP64 FMAs or on three-way splits
void lb_run_fp64(const LbArgs &a, RunArgs R, int want, cudaStream_t s)
{
    if (g_cgs_arith == CGS_F3) launch_run<double, 2, GS_F3, false>(a, R, want, s);
    else launch_run<double, 2, GS_F64, false>(a, R, want, s);
}

}  // namespace pgb

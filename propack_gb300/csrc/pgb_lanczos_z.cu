// pgb_lanczos_z.cu -- the run kernel of the complex*16 form
#include "pgb_lanczos.cuh"

namespace pgb {

// block: the operator is held as its real 2x2-block form
template <>
void lb_run<double2>(const LbArgs &a, RunArgs R, bool block, int want, cudaStream_t s)
{
    if (block) {
        if (a.Up) launch_run<double, 2, GS_PL, true>(a, R, want, s);
        else launch_run<double, 2, GS_F64, true>(a, R, want, s);
    } else if (a.Up) {
        launch_run<double2, 1, GS_PL, false>(a, R, want, s);
    } else {
        launch_run<double2, 1, GS_F64, false>(a, R, want, s);
    }
}

}  // namespace pgb

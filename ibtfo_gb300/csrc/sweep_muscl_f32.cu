// Instantiations of the FP32 compensated sweep for Scheme=MUSCL (HLL/HLLC, HLLC_Toro and
// Steger-Warming; compiled with contraction on).
#include "sweep_f32_impl.cuh"

namespace ibtfo {

SweepLaunch sweep_launcher_muscl_f32(int riemann, int limiter)
{
    return select_f32<MUSCL>(riemann, limiter == VANLEER);
}

} // namespace ibtfo

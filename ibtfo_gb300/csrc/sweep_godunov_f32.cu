// Instantiations of the FP32 compensated sweep for Scheme=GODUNOV (HLL/HLLC, HLLC_Toro and
// Steger-Warming; compiled with contraction on).
#include "sweep_f32_impl.cuh"

namespace ibtfo {

SweepLaunch sweep_launcher_godunov_f32(int riemann, int limiter)
{
    return select_f32<GODUNOV>(riemann, limiter == VANLEER);
}

} // namespace ibtfo

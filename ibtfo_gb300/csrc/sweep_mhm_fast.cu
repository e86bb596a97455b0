// Instantiations of the fused sweep for Scheme=MHM, fp64_fast (compiled with contraction).
// One translation unit per scheme and precision so the library builds in parallel.
#include "sweep_impl.cuh"

namespace ibtfo {

SweepLaunch sweep_launcher_mhm_fast(int riemann, int limiter, bool fine)
{
    return select_sweep<MHM, 1>(riemann, limiter, fine);
}

} // namespace ibtfo

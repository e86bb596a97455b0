// Instantiations of the fused sweep for Scheme=MHM, strict FP64 (compiled without contraction).
// One translation unit per scheme and precision so the library builds in parallel.
#include "sweep_impl.cuh"

namespace ibtfo {

SweepLaunch sweep_launcher_mhm(int riemann, int limiter, bool fine)
{
    return select_sweep<MHM, 0>(riemann, limiter, fine);
}

} // namespace ibtfo

// Instantiations of the fused sweep for Scheme=Godunov, fp64_fast (compiled with contraction).
// One translation unit per scheme and precision so the library builds in parallel.
#include "sweep_impl.cuh"

namespace ibtfo {

SweepLaunch sweep_launcher_godunov_fast(int riemann, int limiter, bool fine)
{
    return select_sweep<GODUNOV, 1>(riemann, limiter, fine);
}

} // namespace ibtfo

// k_win_weight.cu -- the windowed sweep kernels of weight estimation (k_sweep_win.cuh).
#include "k_sweep_win.cuh"

namespace muca {

cudaError_t launch_sweep_win_weight(const SweepPlan &p, const SweepArgs &a, cudaStream_t s)
{
    return p.rounds == 10 ? launch_sweep_win<kModeWeight, 10>(p, a, s) : launch_sweep_win<kModeWeight, 7>(p, a, s);
}

}  // namespace muca

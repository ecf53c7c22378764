// k_win_produce.cu -- the windowed sweep kernels of production (k_sweep_win.cuh).
#include "k_sweep_win.cuh"

namespace muca {

cudaError_t launch_sweep_win_produce(const SweepPlan &p, const SweepArgs &a, cudaStream_t s)
{
    return p.rounds == 10 ? launch_sweep_win<kModeProduce, 10>(p, a, s) : launch_sweep_win<kModeProduce, 7>(p, a, s);
}

}  // namespace muca

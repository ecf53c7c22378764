// k_batch_place7.cu -- batch sweeps of 7 rounds, all lattices in shared or in global memory.
#define MUCA_BATCH_INSTANCES
#include "k_batch_sweep.cuh"

template muca::BatchKernel muca::batch_kernel_of<7, muca::kLatShared>(bool, bool);
template muca::BatchKernel muca::batch_kernel_of<7, muca::kLatGlobal>(bool, bool);

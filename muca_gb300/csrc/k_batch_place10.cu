// k_batch_place10.cu -- batch sweeps of 10 rounds, all lattices in shared or in global memory.
#define MUCA_BATCH_INSTANCES
#include "k_batch_sweep.cuh"

template muca::BatchKernel muca::batch_kernel_of<10, muca::kLatShared>(bool, bool);
template muca::BatchKernel muca::batch_kernel_of<10, muca::kLatGlobal>(bool, bool);

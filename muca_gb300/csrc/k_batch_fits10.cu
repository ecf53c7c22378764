// k_batch_fits10.cu -- batch sweeps of 10 rounds, each lattice in shared memory where it fits.
#define MUCA_BATCH_INSTANCES
#include "k_batch_sweep.cuh"

template muca::BatchKernel muca::batch_kernel_of<10, muca::kLatWhereFits>(bool, bool);

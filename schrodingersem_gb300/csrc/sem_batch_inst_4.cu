// Explicit instantiation of the batched kernels for N = 4 (p = 3).
#define SEM_BATCH_DEFINE_KERNELS
#include "sem_batch.cuh"
SEM_BATCH_INSTANTIATE(4)

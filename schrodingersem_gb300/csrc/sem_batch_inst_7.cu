// Explicit instantiation of the batched kernels for N = 7 (p = 6).
#define SEM_BATCH_DEFINE_KERNELS
#include "sem_batch.cuh"
SEM_BATCH_INSTANTIATE(7)

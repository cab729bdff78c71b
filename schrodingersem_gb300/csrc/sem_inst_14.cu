// Explicit instantiation of the kernel launchers for N = 14 (p = 13); one degree
// per unit, so that the degrees compile in parallel.
#include "sem_kernels.cuh"
SEM_INSTANTIATE(14)

// Explicit instantiation of the kernel launchers for N = 13 (p = 12); one degree
// per unit, so that the degrees compile in parallel.
#include "sem_kernels.cuh"
SEM_INSTANTIATE(13)

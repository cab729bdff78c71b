// Explicit instantiation of the kernel launchers for N = 8 (p = 7); one degree
// per unit, so that the degrees compile in parallel.
#include "sem_kernels.cuh"
SEM_INSTANTIATE(8)

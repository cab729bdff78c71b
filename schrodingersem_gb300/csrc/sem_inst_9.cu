// Explicit instantiation of the kernel launchers for N = 9 (p = 8); one degree
// per unit, so that the degrees compile in parallel.
#include "sem_kernels.cuh"
SEM_INSTANTIATE(9)

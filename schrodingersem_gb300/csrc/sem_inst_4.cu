// Explicit instantiation of the kernel launchers for N = 4 (p = 3); one degree
// per unit, so that the degrees compile in parallel.
#include "sem_kernels.cuh"
SEM_INSTANTIATE(4)

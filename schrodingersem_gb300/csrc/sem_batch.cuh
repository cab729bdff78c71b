// Batched ensembles (device side): many independent Schroedinger instances (each its own
// mesh, degree, potential and state) advanced by BDF2 together.  No
// counterpart in the reference, whose drivers step one mesh
// (include/openmp_impl/schrodinger.hpp:22-128); each instance follows that
// driver exactly, with the library's mixed-precision stage solve (FP32 inner
// iterations, FP64 refinement judged on the true residual).
//
// Execution: one persistent launch per time step and group of instances (same
// degree and cluster size) on forked streams.  A cluster of 1, 2, 4 or 8 blocks
// takes an instance from its group's device work queue (largest first) and
// advances it by one step on its own -- projection, right-hand side, the
// complete refined stage solve with cluster barriers and reductions through
// distributed shared memory, unmask -- so instances never wait for one another
// and each records its own convergence flag and iteration count.  The cluster
// size grows with the instance (batch_cluster), so that the largest ones do not
// set the length of a step from a single SM.  The step (queue resets + kernels)
// is captured once as a CUDA graph and replayed; every per-step quantity
// (history slot, BDF coefficient) is derived on the device from the instance's
// own step counter, so the same graph serves every step.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "sem_internal.h"

namespace semgb {

// threads per block: with the element preconditioner two blocks per SM, without
// (one block per instance, MINRES) one
constexpr int BATCH_TPB = 256, BATCH_TPB_PLAIN = 512;
constexpr int BATCH_MIN_N = 3;  // p = 2
constexpr int BATCH_MAX_N = 9;  // p = 8
constexpr size_t BATCH_SMEM_BUDGET = 108 * 1024;  // two blocks per SM
// blocks that share an instance of this many element-local nodes: at least 2,048
// nodes each.  Two steps of 160 instances of 4^2..32^2 elements, p = 4, 6, 8 (the
// largest has 83 k nodes) take 24.8 ms, with one block per instance 152 ms: there
// the largest instance sets the time
inline int batch_cluster(long long nodes) { return nodes >= 16384 ? 8 : nodes >= 8192 ? 4 : nodes >= 4096 ? 2 : 1; }

struct BatchInst {
    DevMesh m;
    double* p;         // state, 2 planes, continuous format
    double* hist[2];   // projected states [M p_re; -M p_im] (masked), 2 planes each
    double* b;         // right-hand side, 2 planes
    const double* V;   // potential
    const float* pot32;
    KrylovWork<float> w;
    double* r64;       // 2 planes
    double* Y64;       // 2 planes
    float* x32;        // 2 planes
    const float4* fac4;  // per-node data of the stage solver (k_cg_prep)
    const float* nnw;
    SolveOut* out;
    int* step;         // steps taken
    int* status;       // 0 running, 1 stopped (a stage solve failed)
    long long* iters;  // inner iterations over all steps
    int kmax, kmax64;  // elements per pass of the stage solver and of its FP64 residual
};

struct BatchArgs {
    const BatchInst* inst;
    const int* order;  // this launch's instances (one degree), largest first
    int n;
    int* queue;
    double dt, tol;
    int maxit;
    double inner_tol, outer_scale;
    int max_sweeps, fdm;
};

// elements per pass for an instance of E elements in clusters of C blocks
template <int N>
void batch_pass(int E, int C, int* kmax, int* kmax64);
template <int N>
size_t batch_smem_n(int kmax, int kmax64);
template <int N>
cudaError_t batch_prepare(size_t smem, bool fdm, int* per_sm);
template <int N>
cudaError_t batch_prep_instance(const DevMesh& m, void* fac, float* wt, cudaStream_t st);
template <int N>
cudaError_t batch_launch_step(const BatchArgs& ba, const DevMesh& m0, int grid, int cluster, size_t smem,
                              cudaStream_t st);

}  // namespace semgb

// definitions: compiled only in the instantiation units
#ifdef SEM_BATCH_DEFINE_KERNELS
#include "sem_device.cuh"
#include "sem_solvers.cuh"

namespace semgb {

template <int N>
__device__ void bdf2_instance(const BatchInst& I, const BatchArgs& ba, unsigned char* smraw, double* red,
                              MinresScal<float>& sc, double* sweep_state, float* fdmS, float* fdmL, Team& tm,
                              const EoD<N, double>& et, const CgTab<N>& tab)
{
    constexpr int NN = N * N;
    const DevMesh& m = I.m;
    const long long n = m.n;
    const int k = *I.step;
    if (*I.status) return;  // the same in every block of the cluster
    // this block's elements
    const int eb = (int)((long long)tm.rank * m.E / tm.size), ee = (int)((long long)(tm.rank + 1) * m.E / tm.size);
    const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
    double* hnew = I.hist[k & 1];
    const double* hold = I.hist[(k + 1) & 1];
    // proj(p) (galerkin.hpp:42-57 via schrodinger.hpp:69-78): mass * p per
    // element, assembled and masked; the imaginary plane negated
    for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
        const double ms = m.mass[idx];
        I.Y64[idx] = ms * I.p[idx];
        I.Y64[n + idx] = ms * I.p[n + idx];
    }
    team_barrier<TEAM_CLUSTER>(tm);
    const double c0 = -1.0 / 3.0, c1 = 4.0 / 3.0;  // schrodinger.hpp:102
    for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
        const int e = (int)(idx / NN);
        const int node = (int)(idx - (long long)e * NN);
        const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            double v = dss_value<N, double, DSS_MASK>(m, I.Y64 + c * n, ni, e, idx);
            if (c == 1) v = -1.0 * v;
            hnew[c * n + idx] = v;
            I.b[c * n + idx] = (k == 0) ? v : c0 * hold[c * n + idx] + c1 * v;
        }
    }
    team_barrier<TEAM_CLUSTER>(tm);
    // stage solve Res(alpha) p = b from p (schrodinger.hpp:97,104), alpha = dt
    // on the first step, 2 dt / 3 after (schrodinger.hpp:98-99)
    SolveArgs a{};
    a.op = OP_RES;
    a.nc = 2;
    a.pot = I.V;
    a.alpha = (k == 0) ? ba.dt : (2.0 / 3.0) * ba.dt;
    a.b[0] = I.b;
    a.b[1] = I.b + n;
    a.x[0] = I.p;
    a.x[1] = I.p + n;
    a.maxit = ba.maxit;
    a.tol = ba.tol;
    a.x_is_zero = 0;
    a.kmax = I.kmax;
    a.kmax64 = I.kmax64;
    a.rel_to_b = 0;
    a.timeout_ns = 0;
    a.sync = nullptr;  // block-local MINRES
    a.out = I.out;
    MixedArgs mx{};
    mx.inner_tol = ba.inner_tol;
    mx.max_sweeps = ba.max_sweeps;
    mx.inner_maxit = ba.maxit;
    mx.r64[0] = I.r64;
    mx.r64[1] = I.r64 + n;
    mx.Y64[0] = I.Y64;
    mx.Y64[1] = I.Y64 + n;
    mx.x32[0] = I.x32;
    mx.x32[1] = I.x32 + n;
    mx.pot32 = I.pot32;
    mx.fac4 = I.fac4;
    mx.nnw = I.nnw;
    mx.pinv32 = nullptr;
    mx.fdm = ba.fdm;
    mx.fused = 0;
    mx.outer_scale = ba.outer_scale;
    mx.adaptive = 1;
    int done = 0;
    bool minres = !ba.fdm;
    if (ba.fdm) {
        CgRefine r{};
        cg_refine<N, TEAM_CLUSTER>(m, a, I.w, mx, eb, ee, smraw, fdmL, et, tab, tm, r);
        done = r.inner;
        minres = r.fallback;
        a.maxit -= done;
        mx.max_sweeps -= r.sweeps;
        a.r0_given = r.r0;
        if (tm.rank == 0 && threadIdx.x == 0) {
            I.out->success = r.conv ? 1 : 0;
            I.out->n_iter = r.inner;
            I.out->residual = r.rn;
            I.out->inner_iters = r.inner;
            I.out->sweeps = r.sweeps;
        }
    }
    if (minres) {  // no preconditioner, or the conjugate gradients gave up: the whole instance on one block
        if (tm.rank == 0) {
            a.kmax = a.kmax64 = I.kmax64;
            mixed_solve<N, OP_RES, MIXED_BATCH>(m, a, I.w, mx, 0, m.E, true, smraw, red, sc, sweep_state, fdmS, fdmL,
                                                et);
        }
        team_barrier<TEAM_CLUSTER>(tm);
    }
    // unmask(p) (schrodinger.hpp:105-106): owner copies are never written here
    for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
        const int e = (int)(idx / NN);
        const int node = (int)(idx - (long long)e * NN);
        const long long src = ni_gather_src(m, node_info<N>(m, e, node % N, node / N), e, idx);
        if (src != idx) {
            I.p[idx] = __ldcg(I.p + src);
            I.p[n + idx] = __ldcg(I.p + n + src);
        }
    }
    team_barrier<TEAM_CLUSTER>(tm);
    if (tm.rank == 0 && threadIdx.x == 0) {
        *I.iters += I.out->n_iter + (minres ? done : 0);
        if (!I.out->success) *I.status = 1;
        *I.step = k + 1;
    }
}

// one time step of every instance in ba.order (all of degree N)
template <int N>
__global__ void __launch_bounds__(BATCH_TPB_PLAIN, 1)
    k_batch_bdf2(BatchArgs ba, const __grid_constant__ EoD<N, double> et, const __grid_constant__ CgTab<N> tab)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[34];
    __shared__ MinresScal<float> sc;
    __shared__ double sweep_state[3];
    __shared__ float fdmS[N * N], fdmL[N];
    __shared__ __align__(16) unsigned char ibuf[sizeof(BatchInst)];
    __shared__ unsigned long long next;
    BatchInst& I = *reinterpret_cast<BatchInst*>(ibuf);
    Team tm{nullptr, 0, nullptr, 0, cluster_rank(), cluster_size()};
    // a block's shared memory may be written by another one only once the block
    // is known to run: the barrier comes before rank 0's first store
    team_barrier<TEAM_CLUSTER>(tm);
    for (;;) {
        if (tm.rank == 0 && threadIdx.x == 0) {
            const int q = atomicAdd(ba.queue, 1);
            next = (unsigned long long)q;
            for (int r = 1; r < tm.size; ++r) cluster_put(&next, r, (unsigned long long)q);
        }
        team_barrier<TEAM_CLUSTER>(tm);
        const int q = (int)next;
        if (q >= ba.n) break;
        if (threadIdx.x == 0) I = ba.inst[ba.order[q]];
        __syncthreads();
        bdf2_instance<N>(I, ba, smraw, red, sc, sweep_state, fdmS, fdmL, tm, et, tab);
        team_barrier<TEAM_CLUSTER>(tm);  // `next` and the instance read, before rank 0 takes another
    }
    team_barrier<TEAM_CLUSTER>(tm);  // no block leaves while another may still write its shared memory
}

template <int N>
void batch_pass(int E, int C, int* kmax, int* kmax64)
{
    const int share = (E + C - 1) / C;
    int k = std::max(1, std::min(share, BATCH_TPB / N));  // a line per thread
    while (k > 1 && cg_smem_bytes<N>(k) > BATCH_SMEM_BUDGET) --k;
    const int passes = (share + k - 1) / k;
    *kmax = (share + passes - 1) / passes;
    int k6 = std::max(1, std::min(share, BATCH_TPB / N));
    while (k6 > 1 && range_smem_bytes<N, double, OP_RES>(k6) > BATCH_SMEM_BUDGET) --k6;
    *kmax64 = k6;
}

template <int N>
size_t batch_smem_n(int kmax, int kmax64)
{
    return std::max(range_smem_bytes<N, double, OP_RES>(kmax64), cg_smem_bytes<N>(kmax));
}

// shared-memory opt-in and resident blocks per SM of the step kernel
template <int N>
cudaError_t batch_prepare(size_t smem, bool fdm, int* per_sm)
{
    size_t limit = 0;
    if (!smem_opt_in_all((const void*)k_batch_bdf2<N>, &limit) || smem > limit) return cudaErrorInvalidConfiguration;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_batch_bdf2<N>, fdm ? BATCH_TPB : BATCH_TPB_PLAIN,
                                                         smem);
}

template <int N>
cudaError_t batch_prep_instance(const DevMesh& m, void* fac, float* wt, cudaStream_t st)
{
    k_cg_prep<N><<<(int)std::min<long long>((m.n + 255) / 256, 1024), 256, 0, st>>>(m, (float4*)fac, wt);
    return cudaGetLastError();
}

template <int N>
cudaError_t batch_launch_step(const BatchArgs& ba, const DevMesh& m0, int grid, int cluster, size_t smem,
                              cudaStream_t st)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid * cluster);
    cfg.blockDim = dim3(ba.fdm ? BATCH_TPB : BATCH_TPB_PLAIN);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_batch_bdf2<N>, ba, eo_d_table<N, double>(m0.Dh), cg_table<N>(m0));
}

}  // namespace semgb

#endif  // SEM_BATCH_DEFINE_KERNELS

#define SEM_BATCH_INSTANTIATE(NV)                                                                        \
    namespace semgb {                                                                                    \
    template void batch_pass<NV>(int, int, int*, int*);                                                  \
    template size_t batch_smem_n<NV>(int, int);                                                          \
    template cudaError_t batch_prepare<NV>(size_t, bool, int*);                                          \
    template cudaError_t batch_prep_instance<NV>(const DevMesh&, void*, float*, cudaStream_t);           \
    template cudaError_t batch_launch_step<NV>(const BatchArgs&, const DevMesh&, int, int, size_t,       \
                                                 cudaStream_t);                                          \
    }

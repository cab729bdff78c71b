// FP64 Krylov solvers in one cooperative launch: MINRES (include/minres.hpp:19-107
// with the identity preconditioner) on the stage and Helmholtz operators and
// PCG (include/pcg.hpp:59-97) on the Poisson operator.  One block per SM, each
// owning a contiguous element range; every iteration has two grid all-reduces.
//
// What an iteration costs beside the FP64 arithmetic (one warp instruction per
// 16 cycles and SM) is latency, so:
//  - when the block's elements fit in one pass (27 elements of p = 8: 223 KB),
//    the element factors w_i w_j {A, B, C, J, J V}, the Lanczos vectors r1, r2, y
//    (PCG: r, p) and the operator output stay in shared memory for the whole
//    solve; only ring copies of the output go through global memory, and w and
//    x, which are off the critical path (k_minres64r, k_pcg64r).  Larger shares
//    stream everything through passes (k_minres64, k_pcg64);
//  - an all-reduce is one round trip: a block publishes its partial as tagged
//    words on its own line and polls every block's, instead of a counter
//    barrier followed by a read of the partials;
//  - the reductions are split (arrive, work, wait): MINRES updates w and x and
//    forms the previous iteration's Givens rotation, PCG updates x, between
//    arrival and wait, so the stopping test is taken half an iteration later
//    (on the same numbers);
//  - PCG's p.Ap is summed over element-local values, p_e.(A_e p_e), which needs
//    no assembled vector: the reduction is also the barrier in front of the
//    assembly (two round trips per iteration, was three).
// Vectors are kept in the continuous format (every copy of a shared node holds
// the assembled value, boundary zero); dots weight owner copies, so they equal
// the reference's masked-vector dots, and x is updated on owner copies only.
#pragma once
#include "sem_device.cuh"

namespace semgb {

// threads, at most.  At 128 registers the line contractions spill from N = 10 on,
// but half as many threads with 255 leave the loads of a pass and the vector updates
// to 8 warps, which costs more: 60 iterations on 75 x 75 elements of p = 11 took 16.4 ms
// (MINRES, stage operator; 13.2 now) and 8.46 (Helmholtz; 7.26), on 62 x 62 of p = 14
// 19.6 (15.8), on 32 x 32 of p = 12 2.29 (2.22, Helmholtz); only shares of one element
// at p = 12 to 15 were 3 to 5 % faster
constexpr int K64_TPB = 512;
constexpr int K64_MAXQ = 5;  // lines polled per lane: grids up to 160 blocks
constexpr int K64_WSTRIDE = RESIDENT_SLOT_STRIDE;
constexpr int K64_PART = K64_TPB / 2 + 4;  // block sum: half-warp partials, then four

// operator planes (u, s1, s2), factor planes and (resident) one more vector of
// kmax elements
template <int N, int OP>
__host__ __device__ constexpr int k64_planes(bool resident)
{
    return (resident ? 4 : 3) * op_nc<OP>() + 3 + (OP == OP_RES ? 2 : OP == OP_HELM ? 1 : 0);
}
template <int N, int OP>
__host__ __device__ constexpr size_t k64_smem_bytes(int kmax, bool resident)
{
    return sizeof(double) * ((size_t)N * N + (size_t)k64_planes<N, OP>(resident) * kmax * line_es(N));
}

// One double as two words {32 bits, tag}; a lost half shows in its tag.
__device__ __forceinline__ ulonglong2 k64_words(double v, unsigned tag)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
    return make_ulonglong2(t | (b >> 32), t | (b & 0xffffffffull));
}
__device__ __forceinline__ double k64_value(const ulonglong2& w)
{
    return __longlong_as_double((long long)((w.x << 32) | (w.y & 0xffffffffull)));
}
__device__ __forceinline__ bool k64_ready(const ulonglong2& w, unsigned tag)
{
    return (unsigned)(w.x >> 32) == tag && (unsigned)(w.y >> 32) == tag;
}
__device__ __forceinline__ ulonglong2 k64_ld(const unsigned long long* p)
{
    ulonglong2 v;
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}

// Split grid all-reduce of K doubles (also the barrier that orders the blocks'
// global stores before arrive against their loads after wait).
struct K64Sync {
    unsigned long long* slots;  // [2][grid][K64_WSTRIDE]
    unsigned epoch;
    GridSync* gs;
    long long tmo;
};
// (An FP64 addition occupies its warp's pipe for 64 cycles.  With 16 warps the
// block sum is a tree with few additions per pipe: one per warp, then two or
// three values and five shuffle steps on one warp per pipe, then three; smaller
// blocks have a warp or two per pipe and reduce by warps.  Fixed order.)
template <int K>
__device__ __forceinline__ void k64_publish(const double (&a)[K], K64Sync& y)
{
    unsigned long long* own = y.slots + ((size_t)(y.epoch & 1u) * gridDim.x + blockIdx.x) * K64_WSTRIDE;
    __threadfence();  // the block's stores (ordered before by the barrier) ahead of the words
#pragma unroll
    for (int k = 0; k < K; ++k) __stcg((ulonglong2*)own + k, k64_words(a[k], y.epoch));
}
template <int K>
__device__ __forceinline__ void k64_arrive(const double (&v)[K], K64Sync& y, double (*part)[K64_PART])
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double a[K];
    ++y.epoch;
    if (nw <= 8) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            a[k] = v[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_down_sync(0xffffffffu, a[k], o);
            if (lane == 0) part[k][wid] = a[k];
        }
        __syncthreads();
        if (wid == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                a[k] = lane < nw ? part[k][lane] : 0.0;
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) a[k] += __shfl_down_sync(0xffffffffu, a[k], o);
            }
            if (lane == 0) k64_publish<K>(a, y);
        }
        return;
    }
    const int nv = blockDim.x >> 1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        a[k] = v[k] + __shfl_down_sync(0xffffffffu, v[k], 16);
        if (lane < 16) part[k][wid * 16 + lane] = a[k];
    }
    __syncthreads();
    if (wid < 4) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double b = part[k][threadIdx.x];
            if ((int)threadIdx.x + 128 < nv) b += part[k][threadIdx.x + 128];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) b += __shfl_down_sync(0xffffffffu, b, o);
            if (lane == 0) part[k][256 + wid] = b;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (threadIdx.x == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                a[k] = (part[k][256] + part[k][257]) + (part[k][258] + part[k][259]);
            k64_publish<K>(a, y);
        }
    }
}
// first warp only: the sums, on every lane; false when the wait ran out
template <int K>
__device__ __forceinline__ bool k64_poll(K64Sync& y, double (&out)[K])
{
    const int lane = threadIdx.x & 31, G = gridDim.x;
    const unsigned long long* sl = y.slots + (size_t)(y.epoch & 1u) * G * K64_WSTRIDE;
    ulonglong2 u[K64_MAXQ][K];
    const ulonglong2 none = k64_words(0.0, y.epoch);
    const unsigned long long t0 = global_ns();
#pragma unroll
    for (int q = 0; q < K64_MAXQ; ++q)
#pragma unroll
        for (int k = 0; k < K; ++k) u[q][k] = lane + 32 * q < G ? k64_ld(sl + (lane + 32 * q) * K64_WSTRIDE + 2 * k) : none;
    bool ok = true;
    for (unsigned polls = 1;; ++polls) {
        bool ready = true;
#pragma unroll
        for (int q = 0; q < K64_MAXQ; ++q)
#pragma unroll
            for (int k = 0; k < K; ++k) ready &= k64_ready(u[q][k], y.epoch);
        if (ready) break;
        if ((polls & 31u) == 1 && (*(volatile int*)&y.gs->err || (long long)(global_ns() - t0) > y.tmo)) {
            atomicExch(&y.gs->err, 1);
            ok = false;
            break;
        }
#pragma unroll
        for (int q = 0; q < K64_MAXQ; ++q)
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (!k64_ready(u[q][k], y.epoch)) u[q][k] = k64_ld(sl + (lane + 32 * q) * K64_WSTRIDE + 2 * k);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < K64_MAXQ; ++q) s += k64_value(u[q][k]);
        out[k] = s;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < K; ++k) out[k] += __shfl_xor_sync(0xffffffffu, out[k], o);
    __threadfence();
    return __all_sync(0xffffffffu, ok) != 0;
}
// wait: fn(sums) runs on one thread between the poll and the block barrier;
// false (on every thread) when the wait ran out
template <int K, class Fn>
__device__ __forceinline__ bool k64_wait(K64Sync& y, Fn&& fn)
{
    bool ok = true;
    if (threadIdx.x < 32) {
        double s[K];
        ok = k64_poll<K>(y, s);
        if (threadIdx.x == 0) fn(s);
    }
    return !__syncthreads_or(!ok);
}

// The operator of one pass over ne elements: shared planes laid out for kmax
template <int N, int OP>
struct K64Op {
    static constexpr int NC = op_nc<OP>();
    static constexpr int ES = line_es(N);
    double *D, *su, *s1, *s2, *g, *ms, *mv, *sr;
    int st;
    __device__ __forceinline__ K64Op(unsigned char* sm, int kmax)
    {
        st = kmax * ES;
        D = (double*)sm;
        su = D + N * N;
        s1 = su + NC * st;
        s2 = s1 + NC * st;
        g = s2 + NC * st;   // g11, g12, g22
        mv = g + 3 * st;    // w_i w_j J V (or c)
        ms = mv + st;       // w_i w_j J
        // resident kernels: one more vector behind the factor planes in use
        sr = OP == OP_RES ? ms + st : OP == OP_HELM ? ms : mv;
    }
    // factors of elements [e0, e0 + ne) (visible after the next block barrier)
    __device__ __forceinline__ void load(const DevMesh& m, const double* __restrict__ pot, int e0, int ne)
    {
#pragma unroll 2
        for (int t = threadIdx.x; t < ne * N * N; t += blockDim.x) {
            const int le = t / (N * N), node = t - le * (N * N);
            const long long flat = (long long)(e0 + le) * (N * N) + node;
            const int q = le * ES + node;
            const double a = __ldg(m.g11 + flat), b = __ldg(m.g12 + flat), c = __ldg(m.g22 + flat);
            double w = 0.0, v = 0.0;
            if (OP != OP_LAPLACE) {
                w = __ldg(m.mass + flat);
                v = __ldg(pot + flat);
            }
            g[q] = a;
            g[st + q] = b;
            g[2 * st + q] = c;
            if (OP != OP_LAPLACE) mv[q] = w * v;
            if (OP == OP_RES) ms[q] = w;
        }
    }
    // s1 + s2 = weak Laplacian of su (block barriers inside, one at the end)
    __device__ __forceinline__ void laplace(const EoD<N, double>& et, int ne)
    {
        const Gs64<N> gs{g, st};
        if (laplace64_nodes(N, NC, ne, blockDim.x))
            laplace64_small<N, NC>(D, su, s1, s2, st, gs, ne);
        else
            laplace64<N, NC>(et, su, s1, s2, st, gs, ne);
    }
    // operator output of staged node q
    __device__ __forceinline__ void combine(int q, double alpha, double (&o)[NC]) const
    {
        if (OP == OP_RES) {
            const double u0 = su[q], u1 = su[st + q], w = ms[q], v = mv[q];
            const double Lv = (s1[st + q] + s2[st + q]) + v * u1;
            const double Lu = (s1[q] + s2[q]) + v * u0;
            o[0] = w * u0 + alpha * Lv;
            o[NC - 1] = alpha * Lu - w * u1;
        } else {
            o[0] = s1[q] + s2[q];
            if (OP == OP_HELM) o[0] = o[0] + mv[q] * su[q];
        }
    }
};

// One operator pass structure over the block's range: load(flat, ni, e, u, q)
// fills the inputs of a node, fin(flat, q, o) takes its output.
template <int N, int OP, class Load, class Fin>
__device__ __forceinline__ void k64_pass(K64Op<N, OP>& op, const EoD<N, double>& et, const DevMesh& m,
                                         const double* __restrict__ pot, double alpha, int eb, int ee, int kmax,
                                         Load&& load, Fin&& fin)
{
    constexpr int NN = N * N, NC = op_nc<OP>();
    for (int e0 = eb; e0 < ee; e0 += kmax) {
        const int ne = min(kmax, ee - e0);
        op.load(m, pot, e0, ne);
#pragma unroll 2
        for (int t = threadIdx.x; t < ne * NN; t += blockDim.x) {
            const int le = t / NN, node = t - le * NN;
            double u[NC];
            load(e0 + le, node, (long long)(e0 + le) * NN + node, u);
#pragma unroll
            for (int c = 0; c < NC; ++c) op.su[c * op.st + le * op.ES + node] = u[c];
        }
        __syncthreads();
        op.laplace(et, ne);
        for (int t = threadIdx.x; t < ne * NN; t += blockDim.x) {
            const int le = t / NN, node = t - le * NN;
            const int q = le * op.ES + node;
            double o[NC];
            op.combine(q, alpha, o);
            fin((long long)(e0 + le) * NN + node, q, o);
        }
        if (e0 + kmax < ee) __syncthreads();
    }
}

// coefficients of one w / x update and the stopping test, thread 0 to all
struct K64Rot {
    double g, eps, delta, phi, inv_b;
    int stop;
};
// thread 0's MINRES recurrence (minres.hpp:28-40, 65-92)
struct K64Givens {
    double bnorm, beta, inv, beta_k, inv_k, phibar, cs, sn, dbar, eps;
    bool conv;
    __device__ __forceinline__ void start(double b2)
    {
        bnorm = beta = phibar = sqrt(b2);
        inv = 1.0 / beta;
        cs = -1.0;
        sn = dbar = eps = 0.0;
        conv = false;
    }
    // beta of the next iteration from its square
    __device__ __forceinline__ void next(double b2, double& inv_b, double& c1)
    {
        beta_k = beta;
        inv_k = inv;
        beta = sqrt(b2);
        inv = 1.0 / beta;
        inv_b = inv;
        c1 = beta / beta_k;
    }
    // rotation of iteration k (its alpha, beta_k; this->beta is the next)
    __device__ __forceinline__ void rotate(double alpha_i, int k, double tol, int maxit, K64Rot& r)
    {
        const double eps_old = eps;
        const double delta = cs * dbar + sn * alpha_i;
        const double gbar = sn * dbar - cs * alpha_i;
        eps = sn * beta;
        dbar = -cs * beta;
        double gamma = sqrt(gbar * gbar + beta * beta);
        if (gamma < DBL_EPSILON) gamma = DBL_EPSILON;
        cs = gbar / gamma;
        sn = beta / gamma;
        const double phi = cs * phibar;
        phibar *= sn;
        conv = phibar < tol * bnorm + tol;  // minres.hpp:92
        r.g = 1.0 / gamma;
        r.eps = eps_old;
        r.delta = delta;
        r.phi = phi;
        r.inv_b = inv_k;
        r.stop = conv || k >= maxit ? 1 : 0;
    }
};

template <int N, int OP>
__global__ void __launch_bounds__(K64_TPB, 1)
    k_minres64(DevMesh m, SolveArgs a, KrylovWork<double> w, const __grid_constant__ EoD<N, double> et,
               unsigned long long* slots, unsigned epoch0)
{
    constexpr int NN = N * N, NC = op_nc<OP>();
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double part[1][K64_PART];
    // scalars: thread 0 writes, every thread reads after a block barrier
    __shared__ double inv_b, c1, c2;
    __shared__ K64Rot rot;
    K64Op<N, OP> op(smraw, a.kmax);
    load_dmat_raw<N, double>(op.D, m);
    const long long n = m.n;
    const double* pot = (const double*)a.pot;
    const double alpha = a.alpha;
    const double* const b0 = (const double*)a.b[0];
    const double* const b1 = (const double*)a.b[1];
    double* const x0 = (double*)a.x[0];
    double* const x1 = (double*)a.x[1];
    int eb, ee;
    block_range(m.E, eb, ee);
    const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
    const int kmax = a.kmax;
    K64Sync sy{slots, epoch0, a.sync, a.timeout_ns};
    // x0 != 0: Y1 = A_local(unmask(x0))
    double* const Y1 = w.Y[1];
    const bool xz = a.x_is_zero != 0;
    if (!xz) {
        k64_pass<N, OP>(
            op, et, m, pot, alpha, eb, ee, kmax,
            [&](int e, int node, long long flat, double (&u)[NC]) {
                const long long src = ni_gather_src(m, node_info<N>(m, e, node % N, node / N), e, flat);
                u[0] = x0[src];
                if (NC == 2) u[NC - 1] = x1[src];
            },
            [&](long long flat, int, const double (&o)[NC]) {
#pragma unroll
                for (int c = 0; c < NC; ++c) Y1[c * n + flat] = o[c];
            });
        const double z[1] = {0.0};
        k64_arrive<1>(z, sy, part);
        if (!k64_wait<1>(sy, [](const double (&)[1]) {})) return;
    }
    // r0 = unmask(b) - DSS(Y1) (minres.hpp:28-31); Y = A_local(r0)
    double *r1 = w.L[0], *r2 = w.L[1], *ly = w.L[2];
    double *w1 = w.W[0], *w2 = w.W[1], *wn = w.W[2];
    double* const Y = w.Y[0];
    double acc[1] = {0.0};
    k64_pass<N, OP>(
        op, et, m, pot, alpha, eb, ee, kmax,
        [&](int e, int node, long long flat, double (&u)[NC]) {
            const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
            const long long src = ni_gather_src(m, ni, e, flat);
            const bool own = ni_owner(ni);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                double r = (c == 0 ? b0 : b1)[src];
                if (!xz) r = r - dss_value<N, double, DSS_CONT>(m, Y1 + c * n, ni, e, flat);
                r2[c * n + flat] = r;
                w1[c * n + flat] = 0.0;
                w2[c * n + flat] = 0.0;
                u[c] = r;
                if (own) acc[0] = fma(r, r, acc[0]);
            }
        },
        [&](long long flat, int, const double (&o)[NC]) {
#pragma unroll
            for (int c = 0; c < NC; ++c) Y[c * n + flat] = o[c];
        });
    K64Givens gv{};
    double alpha_i = 0.0;
    k64_arrive<1>(acc, sy, part);
    if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
            gv.start(s[0]);
            inv_b = gv.inv;
            c1 = 0.0;
            rot.stop = 0;
        }))
        return;
    int it = 1;
    if (a.maxit >= 1) {
        for (;; ++it) {
            // ---- Phase B: y = A v - c1 r1; alpha = v.y
            {
                const double ib = inv_b, cc = c1;
                const bool hist = it >= 2;
                double s1[1] = {0.0};
#pragma unroll 2
                for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
                    const int e = (int)(idx / NN);
                    const int node = (int)(idx - (long long)e * NN);
                    const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
                    const bool own = ni_owner(ni);
                    double av[NC], rv[NC], zv[NC];
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        rv[c] = hist ? r1[c * n + idx] : 0.0;
                        zv[c] = r2[c * n + idx];
                        av[c] = dss_value<N, double, DSS_CONT>(m, Y + c * n, ni, e, idx);
                    }
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const double y3 = fma(-cc, rv[c], av[c] * ib);
                        ly[c * n + idx] = y3;
                        if (own) s1[0] = fma(ib * zv[c], y3, s1[0]);
                    }
                }
                k64_arrive<1>(s1, sy, part);
            }
            // ---- between arrival and wait: the previous iteration's Givens
            // rotation (minres.hpp:65-92) and its w / x update
            if (it > 1) {
                if (threadIdx.x == 0) gv.rotate(alpha_i, it - 1, a.tol, a.maxit, rot);
                __syncthreads();
                const double g = rot.g, ep = rot.eps, de = rot.delta, ph = rot.phi, pb = rot.inv_b;
#pragma unroll 2
                for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
                    const int e = (int)(idx / NN);
                    const int node = (int)(idx - (long long)e * NN);
                    const bool own = ni_owner(node_info<N>(m, e, node % N, node / N));
                    double rv[NC], a1[NC], a2[NC], xv[NC];
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        rv[c] = r1[c * n + idx];
                        a1[c] = w1[c * n + idx];
                        a2[c] = w2[c * n + idx];
                        xv[c] = own ? (c == 0 ? x0 : x1)[idx] : 0.0;
                    }
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const double wv = g * ((pb * rv[c] - ep * a1[c]) - de * a2[c]);
                        wn[c * n + idx] = wv;
                        if (own) (c == 0 ? x0 : x1)[idx] = fma(ph, wv, xv[c]);
                    }
                }
                double* t = w1;
                w1 = w2;
                w2 = wn;
                wn = t;
            }
            if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
                    alpha_i = s[0];
                    c2 = s[0] / gv.beta;
                }))
                return;
            if (rot.stop) break;
            // ---- Phase A: y -= c2 r2; beta^2 = y.y; Y = A_local(y)
            const double cc = c2;
            double ss[1] = {0.0};
            k64_pass<N, OP>(
                op, et, m, pot, alpha, eb, ee, kmax,
                [&](int e, int node, long long flat, double (&u)[NC]) {
                    const bool own = ni_owner(node_info<N>(m, e, node % N, node / N));
#pragma unroll
                    for (int c = 0; c < NC; ++c) u[c] = fma(-cc, r2[c * n + flat], ly[c * n + flat]);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        ly[c * n + flat] = u[c];
                        if (own) ss[0] = fma(u[c], u[c], ss[0]);
                    }
                },
                [&](long long flat, int, const double (&o)[NC]) {
#pragma unroll
                    for (int c = 0; c < NC; ++c) Y[c * n + flat] = o[c];
                });
            k64_arrive<1>(ss, sy, part);
            double* t = r1;
            r1 = r2;
            r2 = ly;
            ly = t;
            if (!k64_wait<1>(sy, [&](const double (&s)[1]) { gv.next(s[0], inv_b, c1); }))
                return;
        }
        --it;  // the iteration that stopped
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->success = gv.conv ? 1 : 0;
        a.out->n_iter = gv.conv ? it : (a.maxit >= 1 ? a.maxit + 1 : 1);
        a.out->residual = gv.phibar;
        a.out->status = 0;
        a.out->epoch = sy.epoch;
    }
}

// square of the stopping threshold tol |b| (pcg.hpp:84): a tolerance that is not
// positive is met by no residual, as it is before squaring
__device__ __forceinline__ double pcg64_threshold(double tol, double b2) { return tol > 0.0 ? tol * tol * b2 : 0.0; }

// PCG on the Poisson operator (pcg.hpp:59-97, identity preconditioner)
template <int N>
__global__ void __launch_bounds__(K64_TPB, 1)
    k_pcg64(DevMesh m, SolveArgs a, KrylovWork<double> w, const __grid_constant__ EoD<N, double> et,
            unsigned long long* slots, unsigned epoch0)
{
    constexpr int NN = N * N;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double part[2][K64_PART];
    __shared__ double rho, rho_prev, thr2, inv_rho, al, be;
    __shared__ int done;
    K64Op<N, OP_LAPLACE> op(smraw, a.kmax);
    load_dmat_raw<N, double>(op.D, m);
    const double* const b = (const double*)a.b[0];
    double* const x = (double*)a.x[0];
    double* const R = w.L[0];
    double* const P = w.L[1];
    double* const Y = w.Y[0];
    double* const Y1 = w.Y[1];
    int eb, ee;
    block_range(m.E, eb, ee);
    const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
    const int kmax = a.kmax;
    K64Sync sy{slots, epoch0, a.sync, a.timeout_ns};
    if (!a.x_is_zero) {
        k64_pass<N, OP_LAPLACE>(
            op, et, m, nullptr, 0.0, eb, ee, kmax,
            [&](int e, int node, long long flat, double (&u)[1]) {
                u[0] = x[ni_gather_src(m, node_info<N>(m, e, node % N, node / N), e, flat)];
            },
            [&](long long flat, int, const double (&o)[1]) { Y1[flat] = o[0]; });
        const double z[1] = {0.0};
        k64_arrive<1>(z, sy, part);
        if (!k64_wait<1>(sy, [](const double (&)[1]) {})) return;
    }
    double v2[2] = {0.0, 0.0};
#pragma unroll 2
    for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
        const int e = (int)(idx / NN);
        const int node = (int)(idx - (long long)e * NN);
        const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
        const double bv = b[ni_gather_src(m, ni, e, idx)];
        double r = bv;
        if (!a.x_is_zero) r = bv - dss_value<N, double, DSS_CONT>(m, Y1, ni, e, idx);
        R[idx] = r;
        if (ni_owner(ni)) {
            v2[0] = fma(bv, bv, v2[0]);
            v2[1] = fma(r, r, v2[1]);
        }
    }
    k64_arrive<2>(v2, sy, part);
    if (!k64_wait<2>(sy, [&](const double (&s)[2]) {
            thr2 = pcg64_threshold(a.tol, s[0]);
            rho = s[1];
            rho_prev = 0.0;
            be = 0.0;
        }))
        return;
    bool conv = false;
    int it = 0;
    for (it = 0; it < a.maxit; ++it) {
        // p = r + beta p; Y = A_local p; p.Ap over element-local values
        const double bt = be;
        double pap[1] = {0.0};
        k64_pass<N, OP_LAPLACE>(
            op, et, m, nullptr, 0.0, eb, ee, kmax,
            [&](int, int, long long flat, double (&u)[1]) {
                u[0] = it == 0 ? R[flat] : fma(bt, P[flat], R[flat]);
                P[flat] = u[0];
            },
            [&](long long flat, int q, const double (&o)[1]) {
                Y[flat] = o[0];
                pap[0] = fma(op.su[q], o[0], pap[0]);
            });
        k64_arrive<1>(pap, sy, part);
        if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
                al = rho / s[0];
                rho_prev = rho;
                done = rho < thr2;  // sqrt(rho) < tol |b|, pcg.hpp:84, rho of this iteration's start
            }))
            return;
        conv = done != 0;
        const double alv = al;
        double rr[1] = {0.0};
#pragma unroll 2
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const int e = (int)(idx / NN);
            const int node = (int)(idx - (long long)e * NN);
            const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
            const double rv = R[idx];
            const double r = fma(-alv, dss_value<N, double, DSS_CONT>(m, Y, ni, e, idx), rv);
            R[idx] = r;
            if (ni_owner(ni)) rr[0] = fma(r, r, rr[0]);
        }
        k64_arrive<1>(rr, sy, part);
        if (threadIdx.x == 0) inv_rho = 1.0 / rho_prev;
#pragma unroll 4
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const int e = (int)(idx / NN);
            const int node = (int)(idx - (long long)e * NN);
            if (ni_owner(node_info<N>(m, e, node % N, node / N))) x[idx] = fma(alv, P[idx], x[idx]);
        }
        if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
                be = s[0] * inv_rho;
                rho = s[0];
            }))
            return;
        if (conv) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->success = conv ? 1 : 0;
        a.out->n_iter = it;
        a.out->residual = sqrt(rho_prev);  // rho of the last iteration's start (pcg.hpp:93)
        a.out->status = 0;
        a.out->epoch = sy.epoch;
    }
}

// ------------------------------------------------------------ resident forms
// assembled value (continuous format) at staged node (e, i, j): the block's
// own element output v, ring copies of other elements from Y (every ring copy
// is stored there, this block's too, so corner sums run over the same list in
// every copy: dss_value's sums)
template <int N>
__device__ __forceinline__ double k64_dss(const DevMesh& m, const double* Y, double v, int e, int i, int j,
                                          long long flat, bool& own)
{
    const NodeInfo ni = node_info<N>(m, e, i, j);
    own = ni_owner(ni);
    if (ni.kind == 0) return v;
    if (ni.kind == 1) {
        const int sb = __ldg(m.side_base + 4 * e + ni.sc), ss = __ldg(m.side_step + 4 * e + ni.sc);
        if (ni_boundary(ni)) return 0.0;
        if (ni_lone(ni)) return v;
        return v + __ldcg(Y + ((long long)sb + (long long)ni.k * ss));
    }
    return dss_value<N, double, DSS_CONT>(m, Y, ni, e, flat);
}

// staged operator of the whole share: su -> s1 (element output), ring copies to
// Y; fin(q, o) takes each node's output.  One block barrier first, none last
template <int N, int OP, class Fin>
__device__ __forceinline__ void k64_apply_r(K64Op<N, OP>& op, const EoD<N, double>& et, double alpha, int eb, int ne,
                                            long long n, double* __restrict__ Y, Fin&& fin)
{
    constexpr int NN = N * N, NC = op_nc<OP>();
    __syncthreads();
    op.laplace(et, ne);
    for (int t = threadIdx.x; t < ne * NN; t += blockDim.x) {
        const int le = t / NN, node = t - le * NN, i = node % N, j = node / N;
        const int q = le * op.ES + node;
        double o[NC];
        op.combine(q, alpha, o);
        const bool ring = i == 0 || i == N - 1 || j == 0 || j == N - 1;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            op.s1[c * op.st + q] = o[c];
            if (ring) __stcg(Y + c * n + (long long)eb * NN + t, o[c]);
        }
        fin(q, o);
    }
}

template <int N, int OP>
__global__ void __launch_bounds__(K64_TPB, 1)
    k_minres64r(DevMesh m, SolveArgs a, KrylovWork<double> w, const __grid_constant__ EoD<N, double> et,
                unsigned long long* slots, unsigned epoch0)
{
    constexpr int NN = N * N, NC = op_nc<OP>();
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double part[1][K64_PART];
    __shared__ double inv_b, c1, c2;
    __shared__ K64Rot rot;
    K64Op<N, OP> op(smraw, a.kmax);
    load_dmat_raw<N, double>(op.D, m);
    const long long n = m.n;
    const double alpha = a.alpha;
    const double* const b0 = (const double*)a.b[0];
    const double* const b1 = (const double*)a.b[1];
    double* const x0 = (double*)a.x[0];
    double* const x1 = (double*)a.x[1];
    int eb, ee;
    block_range(m.E, eb, ee);
    const int ne = ee - eb, nodes = ne * NN;
    const long long nb = (long long)eb * NN;
    const int st = op.st;
    op.load(m, (const double*)a.pot, eb, ne);
    K64Sync sy{slots, epoch0, a.sync, a.timeout_ns};
    double* const Y = w.Y[0];
    double* const Y1 = w.Y[1];
    const bool xz = a.x_is_zero != 0;
    if (!xz) {  // Y1 = A_local(unmask(x0)): ring copies in Y1, the rest in s1
        for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
            const int le = t / NN, node = t - le * NN;
            const long long src = ni_gather_src(m, node_info<N>(m, eb + le, node % N, node / N), eb + le, nb + t);
            op.su[le * op.ES + node] = x0[src];
            if (NC == 2) op.su[st + le * op.ES + node] = x1[src];
        }
        k64_apply_r<N, OP>(op, et, alpha, eb, ne, n, Y1, [](int, const double (&)[NC]) {});
        const double z[1] = {0.0};
        k64_arrive<1>(z, sy, part);
        if (!k64_wait<1>(sy, [](const double (&)[1]) {})) return;
    }
    double *w1 = w.W[0], *w2 = w.W[1], *wn = w.W[2];
    double acc[1] = {0.0};
    for (int t = threadIdx.x; t < nodes; t += blockDim.x) {  // r0 (minres.hpp:28-31)
        const int le = t / NN, node = t - le * NN, i = node % N, j = node / N;
        const int e = eb + le, q = le * op.ES + node;
        const NodeInfo ni = node_info<N>(m, e, i, j);
        const long long src = ni_gather_src(m, ni, e, nb + t);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            double r = (c == 0 ? b0 : b1)[src];
            bool own = ni_owner(ni);
            if (!xz) r = r - k64_dss<N>(m, Y1 + c * n, op.s1[c * st + q], e, i, j, nb + t, own);
            op.su[c * st + q] = r;
            w1[c * n + nb + t] = 0.0;
            w2[c * n + nb + t] = 0.0;
            if (own) acc[0] = fma(r, r, acc[0]);
        }
    }
    k64_apply_r<N, OP>(op, et, alpha, eb, ne, n, Y, [](int, const double (&)[NC]) {});
    K64Givens gv{};
    double alpha_i = 0.0;
    k64_arrive<1>(acc, sy, part);
    if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
            gv.start(s[0]);
            inv_b = gv.inv;
            c1 = 0.0;
            rot.stop = 0;
        }))
        return;
    int it = 1;
    if (a.maxit >= 1) {
        for (;; ++it) {
            // ---- Phase B (s1, Y: A r2): y = A v - c1 r1 into s2; alpha = v.y
            {
                const double ib = inv_b, cc = c1;
                const bool hist = it >= 2;
                double s1[1] = {0.0};
#pragma unroll 4
                for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
                    const int le = t / NN, node = t - le * NN, i = node % N, j = node / N;
                    const int q = le * op.ES + node;
                    bool own = true;
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const double av = k64_dss<N>(m, Y + c * n, op.s1[c * st + q], eb + le, i, j, nb + t, own);
                        const double a0 = av * ib;
                        const double y3 = hist ? fma(-cc, op.sr[c * st + q], a0) : a0;
                        op.s2[c * st + q] = y3;
                        if (own) s1[0] = fma(ib * op.su[c * st + q], y3, s1[0]);
                    }
                }
                k64_arrive<1>(s1, sy, part);
            }
            // ---- between arrival and wait: the previous iteration's Givens
            // rotation and its w / x update
            if (it > 1) {
                if (threadIdx.x == 0) gv.rotate(alpha_i, it - 1, a.tol, a.maxit, rot);
                __syncthreads();
                const double g = rot.g, ep = rot.eps, de = rot.delta, ph = rot.phi, pb = rot.inv_b;
#pragma unroll 2
                for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
                    const int le = t / NN, node = t - le * NN;
                    const int q = le * op.ES + node;
                    const long long idx = nb + t;
                    const bool own = ni_owner(node_info<N>(m, eb + le, node % N, node / N));
                    double a1[NC], a2[NC], xv[NC];
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        a1[c] = w1[c * n + idx];
                        a2[c] = w2[c * n + idx];
                        xv[c] = own ? (c == 0 ? x0 : x1)[idx] : 0.0;
                    }
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const double wv = g * ((pb * op.sr[c * st + q] - ep * a1[c]) - de * a2[c]);
                        wn[c * n + idx] = wv;
                        if (own) (c == 0 ? x0 : x1)[idx] = fma(ph, wv, xv[c]);
                    }
                }
                double* t = w1;
                w1 = w2;
                w2 = wn;
                wn = t;
            }
            if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
                    alpha_i = s[0];
                    c2 = s[0] / gv.beta;
                }))
                return;
            if (rot.stop) break;
            // ---- Phase A: r1 = r2, r2 = y - c2 r2; beta^2 = r2.r2; A_local(r2)
            const double cc = c2;
            double ss[1] = {0.0};
            for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
                const int le = t / NN, node = t - le * NN;
                const int q = le * op.ES + node;
                const bool own = ni_owner(node_info<N>(m, eb + le, node % N, node / N));
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const double r = op.su[c * st + q];
                    const double u = fma(-cc, r, op.s2[c * st + q]);
                    op.sr[c * st + q] = r;
                    op.su[c * st + q] = u;
                    if (own) ss[0] = fma(u, u, ss[0]);
                }
            }
            k64_apply_r<N, OP>(op, et, alpha, eb, ne, n, Y, [](int, const double (&)[NC]) {});
            k64_arrive<1>(ss, sy, part);
            if (!k64_wait<1>(sy, [&](const double (&s)[1]) { gv.next(s[0], inv_b, c1); }))
                return;
        }
        --it;  // the iteration that stopped
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->success = gv.conv ? 1 : 0;
        a.out->n_iter = gv.conv ? it : (a.maxit >= 1 ? a.maxit + 1 : 1);
        a.out->residual = gv.phibar;
        a.out->status = 0;
        a.out->epoch = sy.epoch;
    }
}

template <int N>
__global__ void __launch_bounds__(K64_TPB, 1)
    k_pcg64r(DevMesh m, SolveArgs a, KrylovWork<double> w, const __grid_constant__ EoD<N, double> et,
             unsigned long long* slots, unsigned epoch0)
{
    constexpr int NN = N * N;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double part[2][K64_PART];
    __shared__ double rho, rho_prev, thr2, inv_rho, al, be;
    __shared__ int done;
    K64Op<N, OP_LAPLACE> op(smraw, a.kmax);
    load_dmat_raw<N, double>(op.D, m);
    const long long n = m.n;
    const double* const b = (const double*)a.b[0];
    double* const x = (double*)a.x[0];
    double* const Y = w.Y[0];
    double* const Y1 = w.Y[1];
    int eb, ee;
    block_range(m.E, eb, ee);
    const int ne = ee - eb, nodes = ne * NN;
    const long long nb = (long long)eb * NN;
    op.load(m, nullptr, eb, ne);
    K64Sync sy{slots, epoch0, a.sync, a.timeout_ns};
    if (!a.x_is_zero) {
        for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
            const int le = t / NN, node = t - le * NN;
            op.su[le * op.ES + node] =
                x[ni_gather_src(m, node_info<N>(m, eb + le, node % N, node / N), eb + le, nb + t)];
        }
        k64_apply_r<N, OP_LAPLACE>(op, et, 0.0, eb, ne, n, Y1, [](int, const double (&)[1]) {});
        const double z[1] = {0.0};
        k64_arrive<1>(z, sy, part);
        if (!k64_wait<1>(sy, [](const double (&)[1]) {})) return;
    }
    double v2[2] = {0.0, 0.0};
    for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
        const int le = t / NN, node = t - le * NN, i = node % N, j = node / N;
        const int e = eb + le, q = le * op.ES + node;
        const NodeInfo ni = node_info<N>(m, e, i, j);
        const double bv = b[ni_gather_src(m, ni, e, nb + t)];
        double r = bv;
        bool own = ni_owner(ni);
        if (!a.x_is_zero) r = bv - k64_dss<N>(m, Y1, op.s1[q], e, i, j, nb + t, own);
        op.sr[q] = r;
        if (own) {
            v2[0] = fma(bv, bv, v2[0]);
            v2[1] = fma(r, r, v2[1]);
        }
    }
    k64_arrive<2>(v2, sy, part);
    if (!k64_wait<2>(sy, [&](const double (&s)[2]) {
            thr2 = pcg64_threshold(a.tol, s[0]);
            rho = s[1];
            rho_prev = 0.0;
            be = 0.0;
        }))
        return;
    bool conv = false;
    int it = 0;
    for (it = 0; it < a.maxit; ++it) {
        const double bt = be;
        for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
            const int le = t / NN, q = le * op.ES + (t - le * NN);
            op.su[q] = it == 0 ? op.sr[q] : fma(bt, op.su[q], op.sr[q]);
        }
        double pap[1] = {0.0};
        k64_apply_r<N, OP_LAPLACE>(op, et, 0.0, eb, ne, n, Y,
                                   [&](int q, const double (&o)[1]) { pap[0] = fma(op.su[q], o[0], pap[0]); });
        k64_arrive<1>(pap, sy, part);
        if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
                al = rho / s[0];
                rho_prev = rho;
                done = rho < thr2;  // sqrt(rho) < tol |b|, pcg.hpp:84, rho of this iteration's start
            }))
            return;
        conv = done != 0;
        const double alv = al;
        double rr[1] = {0.0};
#pragma unroll 4
        for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
            const int le = t / NN, node = t - le * NN;
            const int q = le * op.ES + node;
            bool own = true;
            const double ap = k64_dss<N>(m, Y, op.s1[q], eb + le, node % N, node / N, nb + t, own);
            const double r = fma(-alv, ap, op.sr[q]);
            op.sr[q] = r;
            if (own) rr[0] = fma(r, r, rr[0]);
        }
        k64_arrive<1>(rr, sy, part);
        if (threadIdx.x == 0) inv_rho = 1.0 / rho_prev;
#pragma unroll 4
        for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
            const int le = t / NN, node = t - le * NN;
            if (ni_owner(node_info<N>(m, eb + le, node % N, node / N)))
                x[nb + t] = fma(alv, op.su[le * op.ES + node], x[nb + t]);
        }
        if (!k64_wait<1>(sy, [&](const double (&s)[1]) {
                be = s[0] * inv_rho;
                rho = s[0];
            }))
            return;
        if (conv) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->success = conv ? 1 : 0;
        a.out->n_iter = it;
        a.out->residual = sqrt(rho_prev);  // rho of the last iteration's start (pcg.hpp:93)
        a.out->status = 0;
        a.out->epoch = sy.epoch;
    }
}

}  // namespace semgb

// Persistent (cooperative) FP64 iterative refinement around an FP32 inner solve:
// MINRES, or the conjugate gradients of sem_cg.cuh with the element
// preconditioner (k_cg_mixed, its own block shape).  One block per SM, SOLVER_TPB
// threads; each block owns a contiguous element range and stages
// up to kmax of its elements per pass in dynamic shared memory
// (apply_range).  Grid-wide phases are separated by bounded grid barriers.
//
// Scalar recurrences (Givens rotations, step lengths, stopping tests) run in
// FP64 on one thread per block and are broadcast through shared memory, with
// T-typed copies of the per-pass coefficients: GB300's FP64 pipe is 1/58 of
// FP32, so redundant per-thread scalar FP64 code would dominate small passes.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <limits>

#include "sem_cg.cuh"
#include "sem_device.cuh"
#include "sem_krylov64.cuh"

namespace semgb {

constexpr int SOLVER_TPB = 512;

struct MinresOut {
    int it;
    double phibar;
    bool conv;
};

// block sum of per-thread T partials: warp shuffles in T, then FP64 across
// warps (fixed order); result returned to every thread
template <typename T>
__device__ __forceinline__ double block_sum_t(T v, double* red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = (double)v;
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        double s = lane < nw ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) red[32] = s;
    }
    __syncthreads();
    return red[32];
}

// grid all-reduce of up to two T partials behind one barrier: block sums to
// partials[slot][2][grid], then every block sums them in the same fixed order
template <typename T>
__device__ __forceinline__ void grid_sum2_t(T v0, T v1, double* partials, int slot, GridSync* gs, long long tmo,
                                            double* red, bool& ok, double& r0, double& r1)
{
    const double b0 = block_sum_t<T>(v0, red);
    const double b1 = block_sum_t<T>(v1, red);
    if (!gs) {  // block-local solve: the block sums are the sums
        ok = true;
        r0 = b0;
        r1 = b1;
        return;
    }
    const int G = gridDim.x;
    double* p0 = partials + (size_t)(slot * 2) * G;
    double* p1 = p0 + G;
    if (threadIdx.x == 0) {
        p0[blockIdx.x] = b0;
        p1[blockIdx.x] = b1;
    }
    ok = grid_barrier(gs, tmo);
    if (threadIdx.x < 32) {
        double s0 = 0.0, s1 = 0.0;
        for (int q = threadIdx.x; q < G; q += 32) {
            s0 += __ldcg(p0 + q);
            s1 += __ldcg(p1 + q);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, o);
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        }
        if (threadIdx.x == 0) {
            red[33] = s0;
            red[32] = s1;
        }
    }
    __syncthreads();
    r0 = red[33];
    r1 = red[32];
    __syncthreads();
}

// MINRES scalar state (minres.hpp:28-40, 65-84), shared memory, thread 0 only
template <typename T>
struct MinresScal {
    double bnorm, beta, beta_old, phibar, cs, sn, dbar, eps, inv_beta;
    double pg, peps, pdelta, pphi, pinvb, alpha_i;
    int pending, conv, stop;
    // coefficients of the next vector pass, in T
    T inv_b, c1, c2, cq, tpg, tpeps, tpdelta, tpphi, tpinvb;
};

template <typename T>
__device__ __forceinline__ void scal_init(MinresScal<T>& sc, double bnorm, double beta1)
{
    sc.bnorm = bnorm;
    sc.beta = beta1;
    sc.inv_beta = 1.0 / beta1;
    sc.beta_old = 0.0;
    sc.phibar = beta1;
    sc.cs = -1.0;
    sc.sn = 0.0;
    sc.dbar = 0.0;
    sc.eps = 0.0;
    sc.pg = sc.peps = sc.pdelta = sc.pphi = sc.pinvb = sc.alpha_i = 0.0;
    sc.pending = 0;
    sc.conv = 0;
    sc.stop = 0;
}

// coefficients of pass `it` (Phase B / fused pass)
template <typename T>
__device__ __forceinline__ void scal_publish(MinresScal<T>& sc, int it, double cq)
{
    sc.inv_b = (T)(1.0 / sc.beta);
    sc.c1 = (T)(it >= 2 ? sc.beta / sc.beta_old : 0.0);
    sc.cq = (T)cq;
    sc.tpg = (T)sc.pg;
    sc.tpeps = (T)sc.peps;
    sc.tpdelta = (T)sc.pdelta;
    sc.tpphi = (T)sc.pphi;
    sc.tpinvb = (T)sc.pinvb;
}

// Givens rotation of one iteration (minres.hpp:65-92)
template <typename T>
__device__ __forceinline__ void scal_givens(MinresScal<T>& sc, double alpha_i, double beta_new, double eps_mach,
                                            double tol_rel, double tol_abs)
{
    const double eps_old = sc.eps;
    const double delta = sc.cs * sc.dbar + sc.sn * alpha_i;
    const double gbar = sc.sn * sc.dbar - sc.cs * alpha_i;
    sc.eps = sc.sn * beta_new;
    sc.dbar = -sc.cs * beta_new;
    double gamma = sqrt(gbar * gbar + beta_new * beta_new);
    if (gamma < eps_mach) gamma = eps_mach;
    sc.cs = gbar / gamma;
    sc.sn = beta_new / gamma;
    const double phi = sc.cs * sc.phibar;
    sc.phibar *= sc.sn;
    sc.pending = 1;
    sc.pg = 1.0 / gamma;
    sc.peps = eps_old;
    sc.pdelta = delta;
    sc.pphi = phi;
    sc.pinvb = 1.0 / sc.beta;
    sc.beta_old = sc.beta;
    sc.beta = beta_new;
    sc.conv = sc.phibar < tol_rel * sc.bnorm + tol_abs;  // minres.hpp:92
}

// scal_givens + scal_publish of one iteration (it_next >= 2) for the FP32
// inner solver, with the square roots and reciprocals taken from two FP64
// reciprocal square roots: on one thread, GB300's FP64 division and square
// root are long dependent sequences on the critical path of every iteration.
template <typename T>
__device__ __forceinline__ void scal_step_rsqrt(MinresScal<T>& sc, double alpha_i, double bnew2, double eps_mach,
                                                double tol_rel, double tol_abs)
{
    const double inv_beta_new = bnew2 > 0.0 ? rsqrt(bnew2) : 1.0 / bnew2;
    const double beta_new = bnew2 > 0.0 ? bnew2 * inv_beta_new : 0.0;
    const double eps_old = sc.eps;
    const double delta = sc.cs * sc.dbar + sc.sn * alpha_i;
    const double gbar = sc.sn * sc.dbar - sc.cs * alpha_i;
    sc.eps = sc.sn * beta_new;
    sc.dbar = -sc.cs * beta_new;
    const double g2 = gbar * gbar + beta_new * beta_new;
    double ig = rsqrt(g2), gamma = g2 * ig;
    if (!(gamma >= eps_mach)) {
        gamma = eps_mach;
        ig = 1.0 / eps_mach;
    }
    sc.cs = gbar * ig;
    sc.sn = beta_new * ig;
    const double phi = sc.cs * sc.phibar;
    sc.phibar *= sc.sn;
    sc.pending = 1;
    sc.pg = ig;
    sc.peps = eps_old;
    sc.pdelta = delta;
    sc.pphi = phi;
    sc.pinvb = sc.inv_beta;
    const double c1 = beta_new * sc.inv_beta;
    sc.beta_old = sc.beta;
    sc.beta = beta_new;
    sc.inv_beta = inv_beta_new;
    sc.conv = sc.phibar < tol_rel * sc.bnorm + tol_abs;  // minres.hpp:92
    sc.inv_b = (T)inv_beta_new;
    sc.c1 = (T)c1;
    sc.cq = T(0);
    sc.tpg = (T)sc.pg;
    sc.tpeps = (T)sc.peps;
    sc.tpdelta = (T)sc.pdelta;
    sc.tpphi = (T)sc.pphi;
    sc.tpinvb = (T)sc.pinvb;
}

// One node of MINRES Phase B: Av = DSS(Y)/beta, y = Av - c1 r1, the
// alpha partial v.y, and (pending) the w / x update of the previous
// iteration.  The vectors arrive as restrict pointers (distinct buffers), so
// that once inlined into an unrolled node loop the loads of the next node
// can be issued before the stores of this one.
template <int N, typename T, int NC, int PRE>
__device__ __forceinline__ void phase_b_node(const DevMesh& m, long long n, long long idx, int it, bool pending,
                                             T inv_b, T c1, T tpg, T tpeps, T tpdelta, T tpphi, T tpinvb,
                                             const T* __restrict__ Ycur, const T* __restrict__ Lr1,
                                             const T* __restrict__ Zc, const T* __restrict__ Zq,
                                             const T* __restrict__ W1, const T* __restrict__ W2,
                                             const T* __restrict__ pinv, T* __restrict__ Ly, T* __restrict__ Wn,
                                             T* __restrict__ x0, T* __restrict__ x1, T& s1)
{
    constexpr int NN = N * N;
    const int e = (int)(idx / NN);
    const int node = (int)(idx - (long long)e * NN);
    const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
    const bool own = ni_owner(ni);
    const T pv = PRE == 1 ? pinv[idx] : T(1);
    T av[NC], r1v[NC], zc[NC], zp[NC], w1v[NC], w2v[NC], xv[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const long long q = c * n + idx;
        av[c] = dss_value<N, T, DSS_CONT>(m, Ycur + c * n, ni, e, idx);
        r1v[c] = it >= 2 ? Lr1[q] : T(0);
        zc[c] = Zc[q];
        if (pending) {
            zp[c] = PRE == 2 ? Zq[q] : T(0);
            w1v[c] = W1[q];
            w2v[c] = W2[q];
            if (own) xv[c] = (c == 0 ? x0 : x1)[idx];
        }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const long long q = c * n + idx;
        const T a = av[c] * inv_b;
        const T y3 = it >= 2 ? a - c1 * r1v[c] : a;
        const T vv = inv_b * (PRE == 1 ? pv * zc[c] : zc[c]);
        if (own) s1 = fma(vv, y3, s1);
        Ly[q] = y3;
        if (pending) {
            const T vprev = tpinvb * (PRE == 2 ? zp[c] : PRE == 1 ? pv * r1v[c] : r1v[c]);
            const T wn = tpg * ((vprev - tpeps * w1v[c]) - tpdelta * w2v[c]);
            Wn[q] = wn;
            if (own) (c == 0 ? x0 : x1)[idx] = xv[c] + tpphi * wn;
        }
    }
}

// include/minres.hpp:19-107 inside a cooperative kernel.  Lanczos vectors
// are kept in the continuous format (every copy of a shared node holds the
// assembled value, boundary zero) so the operator needs no gather; dots
// weight owner copies only, which makes them equal to the reference's
// masked-vector dots.  Per iteration two grid barriers:
//   Phase B_i:   Av = DSS(Y)/beta_i; y = Av - (beta_i/beta_{i-1}) r1;
//                alpha_i = v.y;  pending w_{i-1} / x update
//   Phase A_i+1: y -= (alpha_i/beta_i) r2; z = P^-1 y; beta_{i+1}^2 = y.z;
//                Y = A_local(z)
// x is updated on owner copies only, reproducing x += phi*w with the
// reference's masked w.  Stops when phibar < tol_rel*|r0| + tol_abs.  With
// PRE a diagonal preconditioner P^-1 (continuous format) is applied in the
// Paige-Saunders form beta = sqrt(r2 . P^-1 r2).
// rhs(ni, e, flat, c) gives the initial residual (continuous format) at a
// node.  Returns false when a grid barrier timed out.
template <int N, typename T, int OP, int PRE, class Rhs>
__device__ __forceinline__ bool minres_core(T* sm, int kmax, double* red, MinresScal<T>& sc, const DevMesh& m,
                                            const T* pot, T alpha, int eb, int ee,
                                            const KrylovWork<T>& w, GridSync* gs, long long tmo,
                                            int& slot, Rhs&& rhs, T* const* xp, int maxit,
                                            double tol_rel, double tol_abs, MinresOut& res,
                                            const T* __restrict__ pinv, const T* fS = nullptr,
                                            const T* fL = nullptr)
{
    constexpr int NN = N * N;
    constexpr int NC = op_nc<OP>();
    const Fac<T> fac = fac_of<T>(m);
    const long long n = m.n;
    const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
    const double eps_mach = (double)std::numeric_limits<T>::epsilon();
    bool ok = true;
    T* L[3] = {w.L[0], w.L[1], w.L[2]};
    T* W[3] = {w.W[0], w.W[1], w.W[2]};
    int ir1 = 0, ir2 = 1, iy = 2;
    int iw1 = 0, iw2 = 1, iw = 2;
    auto store_y = [&](T* Yb) {
        return [=](int, int, int, long long flat, const T* o) {
#pragma unroll
            for (int c = 0; c < NC; ++c) Yb[c * n + flat] = o[c];
        };
    };
    // P1: r; |r|^2 and r.z (z = P^-1 r); W[0] = W[1] = 0; Y[0] = A_local(z)
    T part = T(0), partz = T(0);
    if constexpr (PRE == 2) {
        // element preconditioner: weighted local solves into Y[1], then
        // z = DSS (continuous) kept in Z[0]
        T* Zl = w.Y[1];
        for (int e0 = eb; e0 < ee; e0 += kmax)
            fdm_range<N, T, NC>(
                sm, kmax, fS, fL, m, alpha, e0, min(kmax, ee - e0),
                [&](int e, int i, int j, long long flat, T* u) {
                    const NodeInfo ni = node_info<N>(m, e, i, j);
                    const bool own = ni_owner(ni);
                    const T wt = nn_weight<N, T>(m, ni, e);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const T r = rhs(ni, e, flat, c);
                        L[ir2][c * n + flat] = r;
                        W[iw1][c * n + flat] = T(0);
                        W[iw2][c * n + flat] = T(0);
                        u[c] = wt * r;
                        if (own) part = fma(r, r, part);
                    }
                },
                [&](int e, int i, int j, long long flat, const T* z) {
                    const T wt = nn_weight<N, T>(m, node_info<N>(m, e, i, j), e);
#pragma unroll
                    for (int c = 0; c < NC; ++c) Zl[c * n + flat] = wt * z[c];
                });
        if (!grid_barrier(gs, tmo)) return false;
        for (int e0 = eb; e0 < ee; e0 += kmax)
            apply_range<N, T, OP>(
                sm, kmax, nullptr, fac, pot, alpha, e0, min(kmax, ee - e0),
                [&](int e, int i, int j, long long flat, T* u) {
                    const NodeInfo ni = node_info<N>(m, e, i, j);
                    const bool own = ni_owner(ni);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const T z = dss_value<N, T, DSS_CONT>(m, Zl + c * n, ni, e, flat);
                        w.Z[0][c * n + flat] = z;
                        u[c] = z;
                        if (own) partz = fma(L[ir2][c * n + flat], z, partz);
                    }
                },
                store_y(w.Y[0]));
    } else {
        for (int e0 = eb; e0 < ee; e0 += kmax)
            apply_range<N, T, OP>(
                sm, kmax, nullptr, fac, pot, alpha, e0, min(kmax, ee - e0),
                [&](int e, int i, int j, long long flat, T* u) {
                    const NodeInfo ni = node_info<N>(m, e, i, j);
                    const bool own = ni_owner(ni);
                    const T pv = PRE == 1 ? pinv[flat] : T(1);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const T r = rhs(ni, e, flat, c);
                        L[ir2][c * n + flat] = r;
                        W[iw1][c * n + flat] = T(0);
                        W[iw2][c * n + flat] = T(0);
                        const T z = PRE == 1 ? pv * r : r;
                        u[c] = z;
                        if (own) {
                            part = fma(r, r, part);
                            partz = fma(r, z, partz);
                        }
                    }
                },
                store_y(w.Y[0]));
    }
    double bb = 0.0, bz = 0.0;
    grid_sum2_t<T>(part, partz, w.partials, slot, gs, tmo, red, ok, bb, bz);
    slot ^= 1;
    if (!ok) return false;
    if (threadIdx.x == 0) {
        // minres.hpp:28,31; preconditioned runs measure the stop relative to
        // the preconditioned norm sqrt(r.P^-1 r) their phibar estimates
        scal_init(sc, PRE ? sqrt(bz) : sqrt(bb), sqrt(bz));
        scal_publish(sc, 1, 0.0);
    }
    __syncthreads();
    int it = 1;
    if (maxit >= 1) {
        for (;;) {
            // ---- Phase B_it
            const T inv_b = sc.inv_b, c1 = sc.c1;
            const bool pending = sc.pending != 0;
            const T tpg = sc.tpg, tpeps = sc.tpeps, tpdelta = sc.tpdelta, tpphi = sc.tpphi, tpinvb = sc.tpinvb;
            const T* Ycur = w.Y[(it - 1) & 1];
            T s1 = T(0);
            const T* Zc = PRE == 2 ? w.Z[(it - 1) & 1] : L[ir2];
            const T* Zq = PRE == 2 ? w.Z[it & 1] : nullptr;
            T* const x1 = NC == 2 ? xp[1] : nullptr;
#pragma unroll 2
            for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x)
                phase_b_node<N, T, NC, PRE>(m, n, idx, it, pending, inv_b, c1, tpg, tpeps, tpdelta, tpphi, tpinvb,
                                            Ycur, L[ir1], Zc, Zq, W[iw1], W[iw2], pinv, L[iy], W[iw], xp[0], x1,
                                            s1);
            if (pending) {
                const int tmp = iw1;
                iw1 = iw2;
                iw2 = iw;
                iw = tmp;
            }
            if constexpr (PRE == 2) {
                // local solves of y itself, ahead of alpha: the preconditioner
                // is linear, so P^-1 y5 = P^-1 y - (alpha/beta) z_it is formed
                // in Phase A without a barrier of its own (y of this block's
                // elements is complete after the block barrier)
                __syncthreads();
                for (int e0 = eb; e0 < ee; e0 += kmax)
                    fdm_range<N, T, NC>(
                        sm, kmax, fS, fL, m, alpha, e0, min(kmax, ee - e0),
                        [&](int e, int i, int j, long long flat, T* u) {
                            const T wt = nn_weight<N, T>(m, node_info<N>(m, e, i, j), e);
#pragma unroll
                            for (int c = 0; c < NC; ++c) u[c] = wt * L[iy][c * n + flat];
                        },
                        [&](int e, int i, int j, long long flat, const T* z) {
                            const T wt = nn_weight<N, T>(m, node_info<N>(m, e, i, j), e);
#pragma unroll
                            for (int c = 0; c < NC; ++c) w.Y3[c * n + flat] = wt * z[c];
                        });
            }
            double S1 = 0.0, dummy = 0.0;
            grid_sum2_t<T>(s1, T(0), w.partials, slot, gs, tmo, red, ok, S1, dummy);
            slot ^= 1;
            if (!ok) return false;
            if (threadIdx.x == 0) {
                sc.pending = 0;
                sc.alpha_i = S1;
                sc.c2 = (T)(S1 / sc.beta);
            }
            __syncthreads();
            // ---- Phase A_it+1
            const T c2 = sc.c2;
            T ss = T(0);
            T* Ynext = w.Y[it & 1];
            if constexpr (PRE == 2) {
                // z_{it+1} = DSS(local solves of y) - c2 z_it, y5 = y - c2 r2
                const T* Zc = w.Z[(it - 1) & 1];
                T* Zn = w.Z[it & 1];
                for (int e0 = eb; e0 < ee; e0 += kmax)
                    apply_range_post<N, T, OP, true>(
                        sm, kmax, nullptr, fac, pot, alpha, e0, min(kmax, ee - e0),
                        [&](int e, int i, int j, long long flat, T* u, T* aux) {
                            const NodeInfo ni = node_info<N>(m, e, i, j);
#pragma unroll
                            for (int c = 0; c < NC; ++c) {
                                const long long q = c * n + flat;
                                u[c] = dss_value<N, T, DSS_CONT>(m, w.Y3 + c * n, ni, e, flat) - c2 * Zc[q];
                                aux[c] = L[iy][q] - c2 * L[ir2][q];
                            }
                        },
                        [&](int e, int i, int j, long long flat, const T* u, const T* aux) {
                            const bool own = ni_owner(node_info<N>(m, e, i, j));
#pragma unroll
                            for (int c = 0; c < NC; ++c) {
                                L[iy][c * n + flat] = aux[c];
                                Zn[c * n + flat] = u[c];
                                if (own) ss = fma(aux[c], u[c], ss);
                            }
                        },
                        store_y(Ynext));
            } else {
                for (int e0 = eb; e0 < ee; e0 += kmax)
                    apply_range_post<N, T, OP, true>(
                        sm, kmax, nullptr, fac, pot, alpha, e0, min(kmax, ee - e0),
                        [&](int, int, int, long long flat, T* u, T* aux) {
                            const T pv = PRE == 1 ? pinv[flat] : T(1);
#pragma unroll
                            for (int c = 0; c < NC; ++c) {
                                const long long q = c * n + flat;
                                const T y5 = L[iy][q] - c2 * L[ir2][q];
                                aux[c] = y5;
                                u[c] = PRE == 1 ? pv * y5 : y5;  // y = precond(r2), minres.hpp:60
                            }
                        },
                        [&](int e, int i, int j, long long flat, const T* u, const T* aux) {
                            const bool own = ni_owner(node_info<N>(m, e, i, j));
#pragma unroll
                            for (int c = 0; c < NC; ++c) {
                                L[iy][c * n + flat] = aux[c];
                                if (own) ss = fma(aux[c], u[c], ss);
                            }
                        },
                        store_y(Ynext));
            }
            double bnew2 = 0.0;
            grid_sum2_t<T>(ss, T(0), w.partials, slot, gs, tmo, red, ok, bnew2, dummy);
            slot ^= 1;
            if (!ok) return false;
            {
                const int tmp = ir1;
                ir1 = ir2;
                ir2 = iy;
                iy = tmp;
            }
            if (threadIdx.x == 0) {
                scal_step_rsqrt(sc, sc.alpha_i, bnew2, eps_mach, tol_rel, tol_abs);
                sc.stop = sc.conv || it == maxit;
            }
            __syncthreads();
            if (sc.stop) break;
            ++it;
        }
        // ---- Phase F: w/x update of the last iteration
        const T tpg = sc.tpg, tpeps = sc.tpeps, tpdelta = sc.tpdelta, tpphi = sc.tpphi, tpinvb = sc.tpinvb;
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const int e = (int)(idx / NN);
            const int node = (int)(idx - (long long)e * NN);
            const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
            if (!ni_owner(ni)) continue;
            const T pv = PRE == 1 ? pinv[idx] : T(1);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const long long q = c * n + idx;
                const T vprev = tpinvb * (PRE == 2 ? w.Z[(it - 1) & 1][q] : PRE == 1 ? pv * L[ir1][q] : L[ir1][q]);
                const T wn = tpg * ((vprev - tpeps * W[iw1][q]) - tpdelta * W[iw2][q]);
                xp[c][idx] += tpphi * wn;
            }
        }
    }
    res.it = it;
    res.phibar = sc.phibar;
    res.conv = sc.conv != 0;
    __syncthreads();
    return true;
}

// Single-barrier variant of minres_core (same recurrences, Givens rotations
// and stopping test) for the Res operator in the FP32 inner solve.  The
// element operator is linear, so the next operator product is carried as
//   A z_{i+1} = DSS(A_local(P^-1 y_i)) - (alpha_i/beta_i) A z_i,
// with A_local(P^-1 y_i) computed in the same pass that forms y_i, and
//   beta_{i+1}^2 = y_i . P^-1 y_i - alpha_i^2
// comes out of the same reduction as alpha_i = z_i . y_i / beta_i.  The
// subtraction is benign for Res = [M, aL; aL, -M], whose spectrum is
// symmetric about zero (Lanczos alpha_i stay small against beta_i); it
// would cancel for one-sided spectra, which therefore use minres_core.
// Rounding in the recurred A z is not re-anchored: the FP64 refinement
// around the inner solve judges the true residual.
template <int N, typename T, int OP, bool PRE, class Rhs>
__device__ __forceinline__ bool minres_core_fused(T* sm, int kmax, double* red, MinresScal<T>& sc,
                                                  const DevMesh& m, const T* pot, T alpha, int eb, int ee,
                                                  const KrylovWork<T>& w, GridSync* gs, long long tmo,
                                                  int& slot, Rhs&& rhs, T* const* xp, int maxit,
                                                  double tol_rel, double tol_abs, MinresOut& res,
                                                  const T* __restrict__ pinv)
{
    constexpr int NN = N * N;
    constexpr int NC = op_nc<OP>();
    const Fac<T> fac = fac_of<T>(m);
    const long long n = m.n;
    const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
    const double eps_mach = (double)std::numeric_limits<T>::epsilon();
    bool ok = true;
    T* Q[3] = {w.L[0], w.L[1], w.L[2]};  // q_i (= r2), q_{i-1} (= r1), free
    T* W[3] = {w.W[0], w.W[1], w.W[2]};
    T* TT[2] = {w.Y[0], w.Y[1]};         // element-local A_local(P^-1 y) ping-pong
    T* AZ = w.AZ;
    T* Y3 = w.Y3;
    int iq = 0, iq1 = 1, iqf = 2;
    int iw1 = 0, iw2 = 1, iw = 2;
    auto store_t = [&](T* Tb) {
        return [=](int, int, int, long long flat, const T* o) {
#pragma unroll
            for (int c = 0; c < NC; ++c) Tb[c * n + flat] = o[c];
        };
    };
    // P1: q_1 = r0, z_1 = P^-1 q_1; |r0|^2, q_1.z_1; W[0] = W[1] = 0; T[1] = A_local(z_1)
    T part = T(0), partz = T(0);
    for (int e0 = eb; e0 < ee; e0 += kmax)
        apply_range<N, T, OP>(
            sm, kmax, nullptr, fac, pot, alpha, e0, min(kmax, ee - e0),
            [&](int e, int i, int j, long long flat, T* u) {
                const NodeInfo ni = node_info<N>(m, e, i, j);
                const bool own = ni_owner(ni);
                const T pv = PRE ? pinv[flat] : T(1);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const T r = rhs(ni, e, flat, c);
                    Q[iq][c * n + flat] = r;
                    W[iw1][c * n + flat] = T(0);
                    W[iw2][c * n + flat] = T(0);
                    const T z = PRE ? pv * r : r;
                    u[c] = z;
                    if (own) {
                        part = fma(r, r, part);
                        partz = fma(r, z, partz);
                    }
                }
            },
            store_t(TT[1]));
    double bb = 0.0, bz = 0.0;
    grid_sum2_t<T>(part, partz, w.partials, slot, gs, tmo, red, ok, bb, bz);
    slot ^= 1;
    if (!ok) return false;
    if (threadIdx.x == 0) {
        scal_init(sc, PRE ? sqrt(bz) : sqrt(bb), sqrt(bz));  // as minres_core
        scal_publish(sc, 1, 0.0);
    }
    __syncthreads();
    int it = 1;
    if (maxit >= 1) {
        for (;;) {
            const T inv_b = sc.inv_b, c1 = sc.c1, cq = sc.cq;
            const bool pending = sc.pending != 0;
            const T tpg = sc.tpg, tpeps = sc.tpeps, tpdelta = sc.tpdelta, tpphi = sc.tpphi, tpinvb = sc.tpinvb;
            const bool first = (it == 1);
            const T* Tin = TT[it & 1];  // A_local of the previous pass
            T* Tout = TT[(it + 1) & 1];
            T s1 = T(0), s2 = T(0);
            for (int e0 = eb; e0 < ee; e0 += kmax)
                apply_range<N, T, OP>(
                    sm, kmax, nullptr, fac, pot, alpha, e0, min(kmax, ee - e0),
                    [&](int e, int i, int j, long long flat, T* u) {
                        const NodeInfo ni = node_info<N>(m, e, i, j);
                        const bool own = ni_owner(ni);
                        const T pv = PRE ? pinv[flat] : T(1);
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            const long long q = c * n + flat;
                            const T tsum = dss_value<N, T, DSS_CONT>(m, Tin + c * n, ni, e, flat);
                            T qi, az, r1v = T(0);
                            if (first) {
                                qi = Q[iq][q];
                                az = tsum;
                            } else {
                                r1v = Q[iq1][q];
                                qi = Y3[q] - cq * r1v;  // q_i = y_{i-1} - (alpha/beta) q_{i-1}
                                az = tsum - cq * AZ[q];
                                Q[iq][q] = qi;
                            }
                            AZ[q] = az;
                            const T y = az * inv_b - c1 * r1v;
                            Y3[q] = y;
                            const T zi = PRE ? pv * qi : qi;
                            const T py = PRE ? pv * y : y;
                            if (own) {
                                s1 = fma(zi, y, s1);
                                s2 = fma(y, py, s2);
                            }
                            if (pending) {
                                const T vprev = tpinvb * (PRE ? pv * r1v : r1v);
                                const T wn = tpg * ((vprev - tpeps * W[iw1][q]) - tpdelta * W[iw2][q]);
                                W[iw][q] = wn;
                                if (own) xp[c][flat] += tpphi * wn;
                            }
                            u[c] = py;
                        }
                    },
                    store_t(Tout));
            if (pending) {
                const int tmp = iw1;
                iw1 = iw2;
                iw2 = iw;
                iw = tmp;
            }
            double S1 = 0.0, S2 = 0.0;
            grid_sum2_t<T>(s1, s2, w.partials, slot, gs, tmo, red, ok, S1, S2);
            slot ^= 1;
            if (!ok) return false;
            {
                const int tmp = iqf;  // the next pass writes q_{i+1} into the free slot
                iqf = iq1;
                iq1 = iq;
                iq = tmp;
            }
            if (threadIdx.x == 0) {
                const double alpha_i = S1 / sc.beta;
                double bnew2 = S2 - alpha_i * alpha_i;
                if (bnew2 < 0.0) bnew2 = 0.0;
                const double cnext = alpha_i / sc.beta;
                scal_givens(sc, alpha_i, sqrt(bnew2), eps_mach, tol_rel, tol_abs);
                sc.stop = sc.conv || it == maxit || sc.beta == 0.0;
                scal_publish(sc, it + 1, cnext);
            }
            __syncthreads();
            if (sc.stop) break;
            ++it;
        }
        // ---- final w/x update of the last iteration (v = P^-1 q_it / beta_it; q_it is Q[iq1])
        const T tpg = sc.tpg, tpeps = sc.tpeps, tpdelta = sc.tpdelta, tpphi = sc.tpphi, tpinvb = sc.tpinvb;
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const int e = (int)(idx / NN);
            const int node = (int)(idx - (long long)e * NN);
            const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
            if (!ni_owner(ni)) continue;
            const T pv = PRE ? pinv[idx] : T(1);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const long long q = c * n + idx;
                const T vprev = tpinvb * (PRE ? pv * Q[iq1][q] : Q[iq1][q]);
                const T wn = tpg * ((vprev - tpeps * W[iw1][q]) - tpdelta * W[iw2][q]);
                xp[c][idx] += tpphi * wn;
            }
        }
    }
    res.it = it;
    res.phibar = sc.phibar;
    res.conv = sc.conv != 0;
    __syncthreads();
    return true;
}

// ------------------------------------------- mixed-precision refinement
// FP64 iterative refinement around an FP32 inner MINRES.  Each sweep:
// r = b - A x in FP64 (true residual, continuous format); stop when
// |r| < tol |r_0| + tol (for x_0 = 0 the reference's criterion minres.hpp:92
// with the true residual in place of the recursive estimate; with rel_to_b,
// |b| replaces |r_0|); else solve A d = r in FP32 to relative tolerance
// inner_tol and add d to x in FP64 on owner copies.
//
// The refinement itself is a device function over the element range
// [eb, ee): the cooperative kernel gives every block a slice of one mesh
// (grid barriers and grid reductions); the batched kernel gives one block a
// whole instance (a.sync == nullptr: block barriers and block reductions).
// Returns false when a wait timed out.  `leader` writes a.out.
//
// The element-preconditioned stage solves run on cg_refine (sem_cg.cuh); here
// their preconditioned MINRES takes over when that iteration gives up.
enum MixedKind : int {
    MIXED_PLAIN = 0,  // no or diagonal preconditioner
    MIXED_BATCH = 1,  // batched instances: no preconditioner or the element one
    MIXED_FDM = 2     // element preconditioner
};
template <int N, int OP, int KIND>
__device__ __forceinline__ bool mixed_solve(const DevMesh& m, const SolveArgs& a, const KrylovWork<float>& w,
                                            const MixedArgs& mx, int eb, int ee, bool leader,
                                            unsigned char* smraw, double* red, MinresScal<float>& sc,
                                            double* sweep_state, float* fdmS, float* fdmL,
                                            const EoD<N, double>& et)
{
    static_assert(KIND == MIXED_PLAIN || OP == OP_RES, "the element preconditioner is the stage operator's");
    constexpr int NN = N * N;
    constexpr int NC = op_nc<OP>();
    double* sm64 = (double*)smraw;
    float* sm32 = (float*)smraw;
    const Fac<double> fac64 = fac_of<double>(m);
    const double* pot64 = (const double*)a.pot;
    const double* bp[2] = {(const double*)a.b[0], (const double*)a.b[1]};
    double* xp[2] = {(double*)a.x[0], (double*)a.x[1]};
    const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
    const int kmax = a.kmax;
    int slot = 0;
    bool ok = true;
    int sweep = 0, inner_total = 0;
    bool conv = false;
    for (;;) {
        // ---- FP64 residual r = unmask(b) - DSS(A_local(unmask(x)))
        const bool applied = (sweep > 0) || !a.x_is_zero;
        if (applied) {
            __syncthreads();  // the staging area overlays the inner solve's
            load_dmat_raw<N, double>(sm64, m);
            __syncthreads();
            for (int e0 = eb; e0 < ee; e0 += a.kmax64)
                apply_range<N, double, OP>(
                    sm64, a.kmax64, &et, fac64, pot64, a.alpha, e0, min(a.kmax64, ee - e0),
                    [&](int e, int i, int j, long long flat, double* u) {
                        const long long src = ni_gather_src(m, node_info<N>(m, e, i, j), e, flat);
#pragma unroll
                        for (int c = 0; c < NC; ++c) u[c] = xp[c][src];
                    },
                    [&](int, int, int, long long flat, const double* o) {
#pragma unroll
                        for (int c = 0; c < NC; ++c) mx.Y64[c][flat] = o[c];
                    });
            if (!grid_barrier(a.sync, a.timeout_ns)) return false;
        }
        double part = 0.0, partb = 0.0;
        const bool want_b = (sweep == 0) && a.rel_to_b;
#pragma unroll 4
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const int e = (int)(idx / NN);
            const int node = (int)(idx - (long long)e * NN);
            const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
            const long long src = ni_gather_src(m, ni, e, idx);
            const bool own = ni_owner(ni);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const double bv = bp[c][src];
                double r = bv;
                if (applied) r = r - dss_value<N, double, DSS_CONT>(m, mx.Y64[c], ni, e, idx);
                mx.r64[c][idx] = r;
                mx.x32[c][idx] = 0.0f;
                if (own) {
                    part = fma(r, r, part);
                    if (want_b) partb = fma(bv, bv, partb);
                }
            }
        }
        double rr = 0.0, bbv = 0.0;
        grid_sum2_t<double>(part, partb, w.partials, slot, a.sync, a.timeout_ns, red, ok, rr, bbv);
        slot ^= 1;
        if (!ok) return false;
        if (threadIdx.x == 0) {
            const double rn = sqrt(rr);
            if (sweep == 0) sweep_state[0] = a.r0_given > 0.0 ? a.r0_given : want_b ? sqrt(bbv) : rn;
            sweep_state[1] = rn;
            const double r0 = sweep_state[0];
            const bool c = rn < mx.outer_scale * (a.tol * r0 + a.tol);
            sweep_state[2] = (c || sweep >= mx.max_sweeps || inner_total >= a.maxit) ? (c ? 2.0 : 1.0) : 0.0;
        }
        __syncthreads();
        if (sweep_state[2] != 0.0) {
            conv = sweep_state[2] == 2.0;
            break;
        }
        // ---- FP32 inner solve A d = r (relative tolerance inner_tol)
        const double* r64c[2] = {mx.r64[0], mx.r64[1]};
        const int budget = min(mx.inner_maxit, a.maxit - inner_total);
        // the inner solve reduces by inner_tol, or (last sweep) by no more
        // than the outer test still needs, with a margin for the FP32
        // estimate: a good initial guess then saves iterations, not sweeps
        double itol = mx.inner_tol;
        if (mx.adaptive) {
            const double need = mx.outer_scale * (a.tol * sweep_state[0] + a.tol) / sweep_state[1];
            itol = fmax(itol, fmin(0.3 * need, 0.5));
        }
        if (KIND != MIXED_PLAIN && mx.fdm) load_fdm_basis<N, float>(fdmS, fdmL, m);
        load_dmat_raw<N, float>(sm32, m);
        __syncthreads();
        auto rhs = [&](const NodeInfo&, int, long long flat, int c) -> float { return (float)r64c[c][flat]; };
        MinresOut ir{};
        bool okc = false;
        bool done_fdm = false;
        if constexpr (KIND != MIXED_PLAIN) {
            if (mx.fdm) {
                okc = minres_core<N, float, OP, 2>(sm32, kmax, red, sc, m, mx.pot32, (float)a.alpha, eb, ee, w,
                                                   a.sync, a.timeout_ns, slot, rhs, mx.x32, budget, itol,
                                                   0.0, ir, (const float*)nullptr, fdmS, fdmL);
                done_fdm = true;
            }
        }
        if (done_fdm || KIND == MIXED_FDM) {
        } else if constexpr (KIND != MIXED_PLAIN) {
            okc = minres_core<N, float, OP, 0>(sm32, kmax, red, sc, m, mx.pot32, (float)a.alpha, eb, ee, w, a.sync,
                                               a.timeout_ns, slot, rhs, mx.x32, budget, itol, 0.0, ir,
                                               (const float*)nullptr);
        } else if (OP == OP_RES && mx.fused)
            okc = mx.pinv32
                      ? minres_core_fused<N, float, OP, true>(sm32, kmax, red, sc, m, mx.pot32, (float)a.alpha, eb,
                                                              ee, w, a.sync, a.timeout_ns, slot, rhs, mx.x32,
                                                              budget, itol, 0.0, ir, mx.pinv32)
                      : minres_core_fused<N, float, OP, false>(sm32, kmax, red, sc, m, mx.pot32, (float)a.alpha,
                                                               eb, ee, w, a.sync, a.timeout_ns, slot, rhs, mx.x32,
                                                               budget, itol, 0.0, ir, (const float*)nullptr);
        else
            okc = mx.pinv32
                      ? minres_core<N, float, OP, 1>(sm32, kmax, red, sc, m, mx.pot32, (float)a.alpha, eb, ee,
                                                        w, a.sync, a.timeout_ns, slot, rhs, mx.x32, budget,
                                                        itol, 0.0, ir, mx.pinv32)
                      : minres_core<N, float, OP, 0>(sm32, kmax, red, sc, m, mx.pot32, (float)a.alpha, eb, ee,
                                                         w, a.sync, a.timeout_ns, slot, rhs, mx.x32, budget,
                                                         itol, 0.0, ir, (const float*)nullptr);
        if (!okc) return false;
        inner_total += ir.it;
        ++sweep;
        // ---- x += d (FP64, owner copies; d is zero on the others)
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
#pragma unroll
            for (int c = 0; c < NC; ++c) xp[c][idx] += (double)mx.x32[c][idx];
        }
        if (!grid_barrier(a.sync, a.timeout_ns)) return false;
    }
    if (leader && threadIdx.x == 0) {
        a.out->success = conv ? 1 : 0;
        a.out->n_iter = inner_total;
        a.out->residual = sweep_state[1];
        a.out->status = 0;
        a.out->inner_iters = inner_total;
        a.out->sweeps = sweep;
    }
    __syncthreads();
    return true;
}

template <int N, int OP>
__global__ void __launch_bounds__(SOLVER_TPB, 1)
    k_minres_mixed(DevMesh m, SolveArgs a, KrylovWork<float> w, MixedArgs mx,
                   const __grid_constant__ EoD<N, double> et)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[34];
    __shared__ MinresScal<float> sc;
    __shared__ double sweep_state[3];  // r0, |r|, done
    int eb, ee;
    block_range(m.E, eb, ee);
    mixed_solve<N, OP, MIXED_PLAIN>(m, a, w, mx, eb, ee, blockIdx.x == 0, smraw, red, sc, sweep_state, nullptr,
                                    nullptr, et);
}

// the element-preconditioned MINRES (after the conjugate gradients gave up)
template <int N>
__global__ void __launch_bounds__(SOLVER_TPB, 1)
    k_minres_fdm(DevMesh m, SolveArgs a, KrylovWork<float> w, MixedArgs mx, const __grid_constant__ EoD<N, double> et)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[34];
    __shared__ MinresScal<float> sc;
    __shared__ double sweep_state[3];  // r0, |r|, done
    __shared__ float fdmS[N * N], fdmL[N];  // element preconditioner basis
    int eb, ee;
    block_range(m.E, eb, ee);
    mixed_solve<N, OP_RES, MIXED_FDM>(m, a, w, mx, eb, ee, blockIdx.x == 0, smraw, red, sc, sweep_state, fdmS, fdmL,
                                      et);
}

// the element-preconditioned stage solve (streaming form)
// Threads and blocks per SM: measured per iteration at 192x192, 100x100 and
// 64x64, p = 8: 269, 83, 57 us; 128 x 5: 290, 102, 91; 256 x 3 (80 registers,
// spills): 247, 94, 67; before the vectors were interleaved as pairs and the
// factors packed in 16 bytes (then 209, 55, 38).  At 128 registers the line passes
// spill from N = 9 on (114 bytes of stores there, 302 at N = 10, 978 at N = 13,
// 1,250 at N = 17)
constexpr int CG_TPB = 256, CG_BLOCKS = 2;
template <int N>
__global__ void __launch_bounds__(CG_TPB, CG_BLOCKS)
    k_cg_mixed(DevMesh m, SolveArgs a, KrylovWork<float> w, MixedArgs mx, const __grid_constant__ EoD<N, double> et,
               const __grid_constant__ CgTab<N> tab)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ float lam[N];
    int eb, ee;
    block_range(m.E, eb, ee);
    Team tm{a.sync, a.timeout_ns, w.partials, 0, (int)blockIdx.x, (int)gridDim.x};
    CgRefine r{};
    if (!cg_refine<N, TEAM_GRID>(m, a, w, mx, eb, ee, smraw, lam, et, tab, tm, r)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->success = r.conv ? 1 : 0;
        a.out->n_iter = r.inner;
        a.out->residual = r.rn;
        a.out->status = 0;
        a.out->inner_iters = r.inner;
        a.out->sweeps = r.sweeps;
        a.out->fallback = r.fallback ? 1 : 0;
        a.out->r0 = r.r0;
    }
}

// ------------------------------------------------------------- launchers

// dynamic shared memory of a solver kernel for a given staging capacity
template <int N>
size_t solver_smem(int op, int kind, int kmax)
{
    if (kind == SOLVE_FP64 || kind == SOLVE_FP64_RES) {
        const bool r = kind == SOLVE_FP64_RES;
        return op == OP_RES    ? k64_smem_bytes<N, OP_RES>(kmax, r)
               : op == OP_HELM ? k64_smem_bytes<N, OP_HELM>(kmax, r)
                               : k64_smem_bytes<N, OP_LAPLACE>(kmax, r);
    }
    if (kind == SOLVE_MIXED_FDM) return cg_smem_bytes<N>(kmax);
    return op == OP_RES ? range_smem_bytes<N, double, OP_RES>(kmax) : range_smem_bytes<N, double, OP_HELM>(kmax);
}

template <int N>
static const void* solver_fn(int op, int kind)
{
    if (kind == SOLVE_MIXED_FDM) return (const void*)k_cg_mixed<N>;
    if (kind == SOLVE_MINRES_FDM) return (const void*)k_minres_fdm<N>;
    if (kind == SOLVE_MIXED)
        return op == OP_RES ? (const void*)k_minres_mixed<N, OP_RES> : (const void*)k_minres_mixed<N, OP_HELM>;
    if (kind == SOLVE_FP64_RES)
        return op == OP_RES    ? (const void*)k_minres64r<N, OP_RES>
               : op == OP_HELM ? (const void*)k_minres64r<N, OP_HELM>
                               : (const void*)k_pcg64r<N>;
    switch (op) {
        case OP_RES: return (const void*)k_minres64<N, OP_RES>;
        case OP_HELM: return (const void*)k_minres64<N, OP_HELM>;
        default: return (const void*)k_pcg64<N>;
    }
}

// threads of the FP64 solvers: one per value of a small share (the smaller the
// block, the cheaper its barriers), at most K64_TPB
inline int k64_threads(int N, int nc, int share)
{
    const int v = nc * share * N * N, top = K64_TPB;
    return v >= top ? top : v < 128 ? 128 : (v + 31) / 32 * 32;
}

// Opts a kernel in to all the dynamic shared memory that a block may have beside
// its static arrays (*limit, bytes).  The attribute belongs to the kernel and the
// device, not to a context, so it is never set to what one plan needs: another
// context's plan for the same kernel may come between a plan and its launch (from
// another thread, or before an ensemble's step is captured), and lowering it would
// have that launch refused.
inline bool smem_opt_in_all(const void* fn, size_t* limit)
{
    int dev = 0, optin = 0;
    cudaFuncAttributes at{};
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&at, fn) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)at.sharedSizeBytes) !=
            cudaSuccess) {
        cudaGetLastError();  // the caller reports the failure; later calls start clean
        return false;
    }
    *limit = (size_t)optin - at.sharedSizeBytes;
    return true;
}

// elements of one element-preconditioned pass: one line per thread
template <int N>
constexpr int cg_pass()
{
    return CG_TPB / N;
}

// Plan a cooperative launch: one block per SM (fewer for small meshes), for the
// element-preconditioned kernel as many of its small blocks per SM as the mesh
// fills with a pass each (a block alternates between loading a pass and the
// line contractions behind block barriers, so only other blocks of the SM hide
// its memory latency), and the largest staging capacities
// kmax <= the block's element count that fit smem_budget bytes per SM and,
// together with the kernel's own static arrays (4,224 bytes of k_pcg64, 2,176 of
// k_minres64), the device's limit per block.
// Returns the grid, or 0 on failure (for SOLVE_FP64_RES also when the block's
// elements do not fit in one pass).
template <int N>
int solver_plan(int op, int kind, int E, int sms, size_t smem_budget, int* kmax_out, int* kmax64_out,
                size_t* smem_out)
{
    const bool fdm = kind == SOLVE_MIXED_FDM;
    const bool f64 = kind == SOLVE_FP64 || kind == SOLVE_FP64_RES;
    const void* fn = solver_fn<N>(op, kind);
    size_t limit = 0;
    if (!smem_opt_in_all(fn, &limit)) return 0;
    int per = 1;
    if (fdm) {
        per = E / (sms * cg_pass<N>());
        per = per < 1 ? 1 : per > CG_BLOCKS ? CG_BLOCKS : per;
        smem_budget = smem_budget / CG_BLOCKS;
    }
    smem_budget = std::min(smem_budget, limit);
    if (f64 && sms > 32 * K64_MAXQ) sms = 32 * K64_MAXQ;
    int grid = E < per * sms ? E : per * sms;
    if (grid < 1) grid = 1;
    int kmax = (E + grid - 1) / grid;
    const int share = kmax;
    if (kind == SOLVE_FP64_RES && solver_smem<N>(op, kind, kmax) > smem_budget) return 0;  // does not fit
    if (fdm && kmax > cg_pass<N>()) kmax = cg_pass<N>();
    while (kmax > 1 && solver_smem<N>(op, kind, kmax) > smem_budget)
        kmax = fdm || f64 ? kmax - 1 : (kmax + 1) / 2;
    if (fdm || f64)  // even passes
        kmax = (share + (share + kmax - 1) / kmax - 1) / ((share + kmax - 1) / kmax);
    size_t smem = solver_smem<N>(op, kind, kmax);
    int kmax64 = kmax;
    if (fdm) {
        while (kmax64 > 1 && range_smem_bytes<N, double, OP_RES>(kmax64) > (smem > smem_budget ? smem : smem_budget))
            --kmax64;
        const size_t s64 = range_smem_bytes<N, double, OP_RES>(kmax64);
        if (s64 > smem) smem = s64;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, fdm ? CG_TPB : f64 ? K64_TPB : SOLVER_TPB,
                                                      smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (per_sm < 1) return 0;
    if (grid > per_sm * sms) {  // fewer blocks per SM: the passes cover the rest
        grid = per_sm * sms;
    }
    *kmax_out = kmax;
    *kmax64_out = kmax64;
    *smem_out = smem;
    return grid;
}

template <int N>
cudaError_t launch_cg_prep(const DevMesh& m, void* fac, float* wt, cudaStream_t st)
{
    const int grid = (int)std::min<long long>((m.n + 255) / 256, 152 * 32);
    k_cg_prep<N><<<grid, 256, 0, st>>>(m, (float4*)fac, wt);
    return cudaGetLastError();
}

template <int N>
cudaError_t launch_solver(const DevMesh& m, const SolveArgs& a, const void* work, const MixedArgs* mx,
                          int grid, size_t smem, cudaStream_t st)
{
    DevMesh mm = m;
    SolveArgs aa = a;
    const int kind = !mx          ? (a.resident ? SOLVE_FP64_RES : SOLVE_FP64)
                     : mx->minres ? SOLVE_MINRES_FDM
                     : mx->fdm    ? SOLVE_MIXED_FDM
                                  : SOLVE_MIXED;
    const void* fn = solver_fn<N>(a.op, kind);
    if (!m.Dh || !m.Sh) return cudaErrorInvalidValue;
    EoD<N, double> et = eo_d_table<N, double>(m.Dh);
    if (mx) {
        KrylovWork<float> ww = *(const KrylovWork<float>*)work;
        MixedArgs xx = *mx;
        if (kind == SOLVE_MIXED_FDM) {
            CgTab<N> tab = cg_table<N>(m);
            void* args[] = {&mm, &aa, &ww, &xx, &et, &tab};
            return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(CG_TPB), args, smem, st);
        }
        void* args[] = {&mm, &aa, &ww, &xx, &et};
        return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(SOLVER_TPB), args, smem, st);
    }
    KrylovWork<double> ww = *(const KrylovWork<double>*)work;
    void* args[] = {&mm, &aa, &ww, &et, &ww.slots, &ww.epoch0};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(k64_threads(N, a.nc, (m.E + grid - 1) / grid)), args,
                                       smem, st);
}

}  // namespace semgb

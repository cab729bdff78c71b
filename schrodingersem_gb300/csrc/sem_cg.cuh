// FP32 inner solver of the Schroedinger stage operator: conjugate gradients
// for complex symmetric matrices (H. A. van der Vorst and J. B. M. Melissen,
// "A Petrov-Galerkin type method for solving Ax = b, where A is symmetric
// complex", IEEE Trans. Magn. 26, 1990: the unconjugated inner product).
//
// The stage system [M, aL; aL, -M] (u, v) = (b0, b1) (schrodinger.hpp:344-366)
// is the real form of
//     (M + i a L) w = b0 + i b1,     w = u - i v,
// with M and L real symmetric.  MINRES on the real form sees a spectrum
// symmetric about zero; the complex one lies on the half line m + i a l, and
// the unconjugated recurrence needs about a fifth of the iterations at the
// same cost per iteration (CPU study on assembled stage systems, p = 6..12,
// element preconditioner: 45-65 against 240-530 for eight digits).
//
// The element preconditioner keeps its form (sum over elements of weighted
// local solves in the basis S x S) with the element's own complex symbol,
// d = 1 / (m_e + i a l_ij), instead of the real 1 / |m_e + i a l_ij|.
//
// Storage: residuals and right-hand sides hold (Re, Im); z, p and the solution
// hold (Re, -Im), i.e. the (u, v) of the real form, so the operator is the
// library's Res operator and no sign is moved.  Both inner products are sums
// over element-local values, p.Ap = sum_e p_e.(A_e p_e) and r.z = sum over
// element modes of d t^2 (t the weighted residual in the basis), so neither
// needs the assembled vector and the assembly gather and the reduction wait
// at one barrier: two barriers per iteration.
//   Phase A: z = DSS(Zl); x += a_{i-1} p; p = z + beta p; Y = A_local p; p.Ap
//   Phase B: a_i = r.z / p.Ap; r -= a_i DSS(Y); Zl = local solves of r; r.z, |r|^2
#pragma once
#include <cmath>

#include "sem_device.cuh"

namespace semgb {

// All-reduce of K per-thread FP32 partials over the team that solves one mesh:
// a cooperative grid (gs) behind one grid barrier, or one block (gs null).
// Warp sums in FP32, FP64 from there on, every sum in one fixed order.
// partials: [slot][K][grid], consecutive reductions alternate slots
template <int K>
__device__ __forceinline__ void team_sum(const float (&v)[K], double* partials, int slot, GridSync* gs, long long tmo,
                                         bool& ok, double (&out)[K])
{
    __shared__ double ts[K][33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    float a[K];
#pragma unroll
    for (int k = 0; k < K; ++k) a[k] = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < K; ++k) a[k] += __shfl_down_sync(0xffffffffu, a[k], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) ts[k][wid] = (double)a[k];
    __syncthreads();
    const int G = gridDim.x;
    double* p = partials + (size_t)slot * K * G;
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double s = lane < nw ? ts[k][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) {
                if (gs) p[(size_t)k * G + blockIdx.x] = s;
                else ts[k][32] = s;
            }
        }
    }
    ok = true;
    if (gs) {
        ok = grid_barrier(gs, tmo);
        if (wid == 0)
#pragma unroll
            for (int k = 0; k < K; ++k) {
                double s = 0.0;
                for (int q = lane; q < G; q += 32) s += __ldcg(p + (size_t)k * G + q);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
                if (lane == 0) ts[k][32] = s;
            }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) out[k] = ts[k][32];
}

// coefficient tables of the FP32 line passes (kernel parameter)
template <int N>
struct CgTab {
    EoD<N, f2_t> D;
    EoS<N, f2_t> S;
};
template <int N>
inline CgTab<N> cg_table(const DevMesh& m)
{
    CgTab<N> t;
    t.D = eo_d_table<N, f2_t>(m.Dh);
    t.S = eo_s_table<N, f2_t>(m.Sh);
    return t;
}

// shared memory of a pass over kmax elements: three planes of pairs, three of
// factors
template <int N>
__host__ __device__ constexpr size_t cg_smem_bytes(int kmax)
{
    return (size_t)kmax * line_es(N) * (3 * sizeof(f2_t) + 3 * sizeof(float));
}

// the three operator passes on staged elements (all threads; leading and
// trailing barriers are the caller's): su holds p; on return s1 holds
// D_xi^T f1 + D_eta^T f2 (the weak Laplacian) of both components
template <int N>
__device__ __forceinline__ void cg_laplace(const EoD<N, f2_t>& t, const f2_t* su, f2_t* s1, f2_t* s2,
                                           const float* sg, int gst, int ne)
{
    constexpr int ES = line_es(N);
    const LineNe nb = line_ne(ne);
    const int lines = ne * N;
    for (int L = threadIdx.x; L < lines; L += blockDim.x) {  // xi lines: u_xi
        int pos, le;
        line_of(L, nb, pos, le);
        const int o = le * ES + pos * N;
        f2_t u[N];
#pragma unroll
        for (int k = 0; k < N; ++k) u[k] = su[o + k];
        eo_d<N, false>(t, u, u);
#pragma unroll
        for (int k = 0; k < N; ++k) s1[o + k] = u[k];
    }
    __syncthreads();
    for (int L = threadIdx.x; L < lines; L += blockDim.x) {  // eta lines: u_eta, fluxes, D^T f2
        int pos, le;
        line_of(L, nb, pos, le);
        const int o = le * ES + pos;
        f2_t us[N];
#pragma unroll
        for (int k = 0; k < N; ++k) us[k] = su[o + k * N];
        eo_d<N, false>(t, us, us);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int q = o + k * N;
            const f2_t ur = s1[q];
            const f2_t g11 = f2dup(sg[q]), g12 = f2dup(-sg[gst + q]), g22 = f2dup(sg[2 * gst + q]);
            s1[q] = f2fma(g12, us[k], f2mul(g11, ur));
            us[k] = f2fma(g12, ur, f2mul(g22, us[k]));
        }
        eo_d<N, true>(t, us, us);
#pragma unroll
        for (int k = 0; k < N; ++k) s2[o + k * N] = us[k];
    }
    __syncthreads();
    for (int L = threadIdx.x; L < lines; L += blockDim.x) {  // xi lines: D^T f1 + (D^T f2)
        int pos, le;
        line_of(L, nb, pos, le);
        const int o = le * ES + pos * N;
        f2_t f[N];
#pragma unroll
        for (int k = 0; k < N; ++k) f[k] = s1[o + k];
        eo_d<N, true>(t, f, f);
#pragma unroll
        for (int k = 0; k < N; ++k) s1[o + k] = f2add(f[k], s2[o + k]);
    }
}

// complex product d t for one mode: (Re, Im) pair times dr - i di
__device__ __forceinline__ f2_t cg_cmul(f2_t t, float dr, float di)
{
    float a, b;
    f2unpack(t, a, b);
    return f2pack(fmaf(di, b, dr * a), fmaf(-di, a, dr * b));
}

// the three preconditioner passes, in place on s (pairs (Re, Im) of the
// weighted residual -> local solve); adds d t^2 over the block's lines to
// (rz0, rz1).  el(le) gives {m_e, rx, ry} of element le, lam the eigenvalues
template <int N, class El>
__device__ __forceinline__ void cg_fdm(const EoS<N, f2_t>& t, f2_t* s, const float* lam, float alpha, int ne, El&& el,
                                       float& rz0, float& rz1)
{
    constexpr int ES = line_es(N);
    const LineNe nb = line_ne(ne);
    const int lines = ne * N;
    for (int L = threadIdx.x; L < lines; L += blockDim.x) {
        int pos, le;
        line_of(L, nb, pos, le);
        const int o = le * ES + pos * N;
        f2_t u[N], m[N];
#pragma unroll
        for (int k = 0; k < N; ++k) u[k] = s[o + k];
        eo_st<N>(t, u, m);
#pragma unroll
        for (int k = 0; k < N; ++k) s[o + k] = m[k];
    }
    __syncthreads();
    for (int L = threadIdx.x; L < lines; L += blockDim.x) {
        int pos, le;
        line_of(L, nb, pos, le);
        const int o = le * ES + pos;
        const float4 g = el(le);
        const float mm = g.x * g.x, lx = alpha * g.y * lam[pos], ly = alpha * g.z;
        f2_t u[N], m[N];
#pragma unroll
        for (int k = 0; k < N; ++k) u[k] = s[o + k * N];
        eo_st<N>(t, u, m);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float al = fmaf(ly, lam[k], lx);
            const float inv = __fdividef(1.f, fmaf(al, al, mm));
            const f2_t d = cg_cmul(m[k], g.x * inv, al * inv);
            float a, b, c, e;
            f2unpack(m[k], a, b);
            f2unpack(d, c, e);
            rz0 = fmaf(a, c, fmaf(-b, e, rz0));
            rz1 = fmaf(a, e, fmaf(b, c, rz1));
            m[k] = d;
        }
        eo_s<N>(t, m, u);
#pragma unroll
        for (int k = 0; k < N; ++k) s[o + k * N] = u[k];
    }
    __syncthreads();
    for (int L = threadIdx.x; L < lines; L += blockDim.x) {
        int pos, le;
        line_of(L, nb, pos, le);
        const int o = le * ES + pos * N;
        f2_t u[N], m[N];
#pragma unroll
        for (int k = 0; k < N; ++k) m[k] = s[o + k];
        eo_s<N>(t, m, u);
#pragma unroll
        for (int k = 0; k < N; ++k) s[o + k] = u[k];
    }
}

// scalar state of the recurrence, identical on every thread (FP32; the
// right-hand side is scaled to unit norm)
struct CgScal {
    float rho0, rho1;  // r.z
    float a0, a1;      // step
    float b0, b1;      // beta
    float best;        // smallest |r|^2 so far and the iteration that gave it
    int best_it;
};
// a = rho / (p.Ap); false when it is not a finite number
__device__ __forceinline__ bool cg_step(CgScal& s, float d0, float d1)
{
    const float den = fmaf(d0, d0, d1 * d1);
    const float inv = 1.f / den;
    s.a0 = fmaf(s.rho0, d0, s.rho1 * d1) * inv;
    s.a1 = fmaf(s.rho1, d0, -s.rho0 * d1) * inv;
    return isfinite(s.a0) && isfinite(s.a1);
}
__device__ __forceinline__ bool cg_beta(CgScal& s, float r0, float r1)
{
    const float den = fmaf(s.rho0, s.rho0, s.rho1 * s.rho1);
    const float inv = 1.f / den;
    s.b0 = fmaf(r0, s.rho0, r1 * s.rho1) * inv;
    s.b1 = fmaf(r1, s.rho0, -r0 * s.rho1) * inv;
    s.rho0 = r0;
    s.rho1 = r1;
    return isfinite(s.b0) && isfinite(s.b1);
}
// the last sweep reduces to this share of what the outer test needs, so that
// the solutions end as far below its threshold as MINRES left them (at 0.3, the
// MINRES margin in the preconditioned norm, their errors were up to twice as
// large); about 2.5 of 35 iterations
constexpr double CG_MARGIN = 0.1;
constexpr int CG_STALL = 200;  // iterations without a smaller residual: give up (MINRES takes over)

struct CgOut {
    int it;
    bool conv;    // |r| fell below tol_rel |b|
    bool usable;  // the correction is finite
};

// Solves A d = b for the block's element range [eb, ee) (a team of blocks: a
// cooperative grid, gs != nullptr, or one block).  rhs(flat, c) is the
// right-hand side scaled to unit norm (continuous format).  The correction
// (continuous format, scaled like b) is left in xo.  w: L[0] r, L[1] p, Y[0]
// Y, Y[1] Zl.  Returns false when a wait timed out.
template <int N, class Rhs>
__device__ __forceinline__ bool cg_core(unsigned char* smraw, int kmax, const DevMesh& m,
                                        const CgTab<N>& tab, const float* __restrict__ pot, float alpha, int eb,
                                        int ee, const KrylovWork<float>& w, GridSync* gs, long long tmo, int& slot,
                                        Rhs&& rhs, float* const* xo, int maxit, float tol_rel, const float* lam,
                                        CgOut& res)
{
    constexpr int NN = N * N;
    constexpr int ES = line_es(N);
    const long long n = m.n;
    const int gst = kmax * ES;
    f2_t* su = (f2_t*)smraw;
    f2_t* s1 = su + gst;
    f2_t* s2 = s1 + gst;
    float* sg = (float*)(s2 + gst);
    float* R = w.L[0];
    float* Pv = w.L[1];
    float* Y = w.Y[0];
    float* Zl = w.Y[1];
    CgScal sc{};
    bool ok = true;
    res.it = 0;
    res.conv = false;
    res.usable = true;
    if (maxit < 1) return true;
    // Phase B of every iteration (first: r = b)
    auto phase_b = [&](bool first, double (&out)[3]) {
        float rz0 = 0.f, rz1 = 0.f, rr = 0.f;
        for (int e0 = eb; e0 < ee; e0 += kmax) {
            const int ne = min(kmax, ee - e0);
            const int total = ne * NN;
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += blockDim.x) {
                const int le = t / NN;
                const int node = t - le * NN;
                const int e = e0 + le;
                const long long flat = (long long)e * NN + node;
                const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
                float r0, r1;
                if (first) {
                    r0 = rhs(flat, 0);
                    r1 = rhs(flat, 1);
                } else {
                    const float q0 = dss_value<N, float, DSS_CONT>(m, Y, ni, e, flat);
                    const float q1 = dss_value<N, float, DSS_CONT>(m, Y + n, ni, e, flat);
                    r0 = R[flat] - fmaf(sc.a0, q0, -sc.a1 * q1);
                    r1 = R[n + flat] - fmaf(sc.a0, q1, sc.a1 * q0);
                }
                R[flat] = r0;
                R[n + flat] = r1;
                if (ni_owner(ni)) rr = fmaf(r0, r0, fmaf(r1, r1, rr));
                const float wt = nn_weight<N, float>(m, ni, e);
                su[le * ES + node] = f2pack(wt * r0, wt * r1);
            }
            __syncthreads();
            cg_fdm<N>(tab.S, su, lam, alpha, ne, [&](int le) { return __ldg(m.fdm_el + e0 + le); }, rz0, rz1);
            __syncthreads();
            for (int t = threadIdx.x; t < total; t += blockDim.x) {
                const int le = t / NN;
                const int node = t - le * NN;
                const int e = e0 + le;
                const long long flat = (long long)e * NN + node;
                const float wt = nn_weight<N, float>(m, node_info<N>(m, e, node % N, node / N), e);
                float a, b;
                f2unpack(su[le * ES + node], a, b);
                Zl[flat] = wt * a;
                Zl[n + flat] = -wt * b;
            }
            __syncthreads();
        }
        const float v[3] = {rz0, rz1, rr};
        team_sum<3>(v, w.partials, slot, gs, tmo, ok, out);
        slot ^= 1;
    };
    double o3[3], o2[2];
    phase_b(true, o3);
    if (!ok) return false;
    sc.rho0 = (float)o3[0];
    sc.rho1 = (float)o3[1];
    const float bb = (float)o3[2];
    sc.best = bb;
    if (!(bb > 0.f)) {  // nothing to solve (or a NaN right-hand side: the caller sees |b|)
        res.conv = bb == 0.f;
        res.usable = false;
        return true;
    }
    bool good = isfinite(sc.rho0) && isfinite(sc.rho1);
    int it = 0;
    while (good && it < maxit) {
        ++it;
        const bool first = it == 1;
        // ---- Phase A
        float d0 = 0.f, d1 = 0.f;
        for (int e0 = eb; e0 < ee; e0 += kmax) {
            const int ne = min(kmax, ee - e0);
            const int total = ne * NN;
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += blockDim.x) {
                const int le = t / NN;
                const int node = t - le * NN;
                const int e = e0 + le;
                const long long flat = (long long)e * NN + node;
                const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
                const int q = le * ES + node;
                sg[q] = __ldg(m.g11f + flat);
                sg[gst + q] = __ldg(m.g12f + flat);
                sg[2 * gst + q] = __ldg(m.g22f + flat);
                float p0 = dss_value<N, float, DSS_CONT>(m, Zl, ni, e, flat);
                float p1 = dss_value<N, float, DSS_CONT>(m, Zl + n, ni, e, flat);
                float x0 = 0.f, x1 = 0.f;
                if (!first) {
                    const float a = Pv[flat], b = Pv[n + flat];
                    x0 = fmaf(sc.a0, a, sc.a1 * b);
                    x1 = fmaf(sc.a0, b, -sc.a1 * a);
                    if (it > 2) {
                        x0 += xo[0][flat];
                        x1 += xo[1][flat];
                    }
                    p0 += fmaf(sc.b0, a, sc.b1 * b);
                    p1 += fmaf(sc.b0, b, -sc.b1 * a);
                    xo[0][flat] = x0;
                    xo[1][flat] = x1;
                }
                Pv[flat] = p0;
                Pv[n + flat] = p1;
                su[q] = f2pack(p0, p1);
            }
            __syncthreads();
            cg_laplace<N>(tab.D, su, s1, s2, sg, gst, ne);
            __syncthreads();
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += blockDim.x) {
                const int le = t / NN;
                const int node = t - le * NN;
                const long long flat = (long long)(e0 + le) * NN + node;
                const float ms = __ldg(m.massf + flat);
                const float mv = ms * __ldg(pot + flat);
                float u0, u1, l0, l1;
                f2unpack(su[le * ES + node], u0, u1);
                f2unpack(s1[le * ES + node], l0, l1);
                const float q0 = ms * u0 + alpha * (l1 + mv * u1);
                const float q1 = alpha * (l0 + mv * u0) - ms * u1;
                d0 = fmaf(u0, q0, fmaf(u1, q1, d0));
                d1 = fmaf(u0, q1, fmaf(-u1, q0, d1));
                Y[flat] = q0;
                Y[n + flat] = q1;
            }
            __syncthreads();
        }
        const float v2[2] = {d0, d1};
        team_sum<2>(v2, w.partials, slot, gs, tmo, ok, o2);
        slot ^= 1;
        if (!ok) return false;
        if (!cg_step(sc, (float)o2[0], (float)o2[1])) {
            --it;
            good = false;
            break;
        }
        // ---- Phase B
        phase_b(false, o3);
        if (!ok) return false;
        const float rr = (float)o3[2];
        if (!isfinite(rr)) {
            good = false;
            break;
        }
        if (rr < tol_rel * tol_rel * bb) {
            res.conv = true;
            break;
        }
        if (rr < sc.best) {
            sc.best = rr;
            sc.best_it = it;
        } else if (it - sc.best_it >= CG_STALL) {
            break;
        }
        if (it < maxit) good = cg_beta(sc, (float)o3[0], (float)o3[1]);
    }
    res.it = it;
    res.usable = good && it > 0;
    // x += a p of the last iteration
    if (res.usable) {
        const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const float a = Pv[idx], b = Pv[n + idx];
            float x0 = fmaf(sc.a0, a, sc.a1 * b), x1 = fmaf(sc.a0, b, -sc.a1 * a);
            if (it > 1) {
                x0 += xo[0][idx];
                x1 += xo[1][idx];
            }
            xo[0][idx] = x0;
            xo[1][idx] = x1;
        }
    }
    __syncthreads();
    return true;
}

}  // namespace semgb

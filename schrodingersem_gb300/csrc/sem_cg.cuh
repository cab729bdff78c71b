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

// ------------------------------------------------------------------- teams
// The blocks that solve one mesh together: a cooperative grid (one mesh), or a
// thread-block cluster (one instance of a batch; a cluster of one is a block).
enum TeamKind : int { TEAM_GRID = 0, TEAM_CLUSTER = 1 };
// words a block publishes in one reduction, at most: the slots lie this far apart
// for every reduction, whatever it publishes, so that the words of one slot are
// never those of the other (a fast block writes the next slot while a slow one
// still reads this one)
constexpr int TEAM_WORDS = 3;
struct Team {
    GridSync* gs;      // grid
    long long tmo;
    double* partials;  // grid: [slot][TEAM_WORDS][grid] partial sums
    int slot;          // alternates
    int rank, size;
};
__device__ __forceinline__ int cluster_rank()
{
    int r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ int cluster_size()
{
    int r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// every thread of every block of the cluster; orders their memory accesses
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_put(void* p, int rank, unsigned long long v)
{
    unsigned la = (unsigned)__cvta_generic_to_shared(p), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(la), "r"(rank));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(ra), "l"(v) : "memory");
}
template <int TEAM>
__device__ __forceinline__ bool team_barrier(Team& t)
{
    if (TEAM == TEAM_GRID) return grid_barrier(t.gs, t.tmo);
    if (t.size > 1) cluster_sync();
    else __syncthreads();
    return true;
}

// (hi, lo) += (h, l): hi + lo carries twice FP32's precision (TwoSum, D. E.
// Knuth, The Art of Computer Programming 2, 4.2.2).  FP64 additions and
// conversions take 64 cycles each on GB300 and would dominate a reduction.
__device__ __forceinline__ void two_add(float& hi, float& lo, float h, float l)
{
    const float s = __fadd_rn(hi, h), t = __fadd_rn(s, -hi);
    const float e = __fadd_rn(__fadd_rn(hi, -__fadd_rn(s, -t)), __fadd_rn(h, -t));
    hi = s;
    lo = __fadd_rn(lo, __fadd_rn(l, e));
}

// All-reduce of K per-thread FP32 partials over the team: warp sums in FP32,
// pairs (hi, lo) from there on, every sum in one fixed order.  Consecutive
// reductions alternate slots.
constexpr int TEAM_MAX_CLUSTER = 8;
template <int TEAM, int K>
__device__ __forceinline__ bool team_sum(const float (&v)[K], Team& tm, float (&out)[K])
{
    __shared__ float ts[K][33];
    __shared__ f2_t cs[2][K][TEAM_MAX_CLUSTER];
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
        for (int k = 0; k < K; ++k) ts[k][wid] = a[k];
    __syncthreads();
    float hi[K], lo[K];
    auto tree = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < K; ++k)
                two_add(hi[k], lo[k], __shfl_down_sync(0xffffffffu, hi[k], o), __shfl_down_sync(0xffffffffu, lo[k], o));
    };
    const int slot = tm.slot;
    tm.slot ^= 1;
    const int G = gridDim.x;
    static_assert(K <= TEAM_WORDS, "words per slot");
    f2_t* p = (f2_t*)tm.partials + (size_t)slot * TEAM_WORDS * G;
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            hi[k] = lane < nw ? ts[k][lane] : 0.f;
            lo[k] = 0.f;
        }
        tree();
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const f2_t w = f2pack(hi[k], lo[k]);
            if (TEAM == TEAM_GRID) {
                if (lane == 0) p[(size_t)k * G + blockIdx.x] = w;
            } else if (tm.size == 1) {
                if (lane == 0) ts[k][32] = hi[k] + lo[k];
            } else {
                const f2_t w0 = __shfl_sync(0xffffffffu, w, 0);
                if (lane < tm.size) cluster_put(&cs[slot][k][tm.rank], lane, w0);
            }
        }
    }
    bool ok = true;
    if (TEAM == TEAM_GRID || tm.size > 1) {
        ok = team_barrier<TEAM>(tm);
        if (wid == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                hi[k] = lo[k] = 0.f;
                if (TEAM == TEAM_GRID) {
                    for (int q = lane; q < G; q += 32) {
                        float h, l;
                        f2unpack(__ldcg(p + (size_t)k * G + q), h, l);
                        two_add(hi[k], lo[k], h, l);
                    }
                } else if (lane < tm.size) {
                    f2unpack(cs[slot][k][lane], hi[k], lo[k]);
                }
            }
            tree();
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < K; ++k) ts[k][32] = hi[k] + lo[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) out[k] = ts[k][32];
    return ok;
}
// the same of two FP64 values (the refinement's norms)
template <int TEAM>
__device__ __forceinline__ bool team_sum64(double v0, double v1, Team& tm, double& r0, double& r1)
{
    __shared__ double ts[2][33];
    __shared__ double cs[2][2][TEAM_MAX_CLUSTER];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    auto tree = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v0 += __shfl_down_sync(0xffffffffu, v0, o);
            v1 += __shfl_down_sync(0xffffffffu, v1, o);
        }
    };
    tree();
    __syncthreads();
    if (lane == 0) {
        ts[0][wid] = v0;
        ts[1][wid] = v1;
    }
    __syncthreads();
    const int slot = tm.slot;
    tm.slot ^= 1;
    const int G = gridDim.x;
    double* p = tm.partials + (size_t)slot * TEAM_WORDS * G;
    if (wid == 0) {
        v0 = lane < nw ? ts[0][lane] : 0.0;
        v1 = lane < nw ? ts[1][lane] : 0.0;
        tree();
        if (TEAM == TEAM_GRID) {
            if (lane == 0) {
                p[blockIdx.x] = v0;
                p[G + blockIdx.x] = v1;
            }
        } else {
            const double w0 = __shfl_sync(0xffffffffu, v0, 0), w1 = __shfl_sync(0xffffffffu, v1, 0);
            if (tm.size > 1) {
                if (lane < tm.size) {
                    cluster_put(&cs[slot][0][tm.rank], lane, (unsigned long long)__double_as_longlong(w0));
                    cluster_put(&cs[slot][1][tm.rank], lane, (unsigned long long)__double_as_longlong(w1));
                }
            } else if (lane == 0) {
                cs[slot][0][0] = w0;
                cs[slot][1][0] = w1;
            }
        }
    }
    const bool ok = team_barrier<TEAM>(tm);
    if (wid == 0) {
        v0 = v1 = 0.0;
        if (TEAM == TEAM_GRID) {
            for (int q = lane; q < G; q += 32) {
                v0 += __ldcg(p + q);
                v1 += __ldcg(p + G + q);
            }
        } else if (lane < tm.size) {
            v0 = cs[slot][0][lane];
            v1 = cs[slot][1][lane];
        }
        tree();
        if (lane == 0) {
            ts[0][32] = v0;
            ts[1][32] = v1;
        }
    }
    __syncthreads();
    r0 = ts[0][32];
    r1 = ts[1][32];
    return ok;
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

// shared memory of a pass over kmax elements: the factors {g11, -g12, g22, mass}
// and three planes of pairs
template <int N>
__host__ __device__ constexpr size_t cg_smem_bytes(int kmax)
{
    return (size_t)kmax * line_es(N) * (sizeof(float4) + 3 * sizeof(f2_t));
}

// Per-node data of the streaming iteration, built once per mesh: the factors in
// one 16-byte load, and the Neumann-Neumann weight (1 / copies, 0 on a Dirichlet
// boundary), negative on copies that are not the owner
template <int N>
__global__ void k_cg_prep(DevMesh m, float4* __restrict__ fac, float* __restrict__ wt)
{
    constexpr int NN = N * N;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < m.n;
         idx += (long long)gridDim.x * blockDim.x) {
        const int e = (int)(idx / NN);
        const int node = (int)(idx - (long long)e * NN);
        const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
        const float w = nn_weight<N, float>(m, ni, e);
        fac[idx] = make_float4(m.g11f[idx], -m.g12f[idx], m.g22f[idx], m.massf[idx]);
        wt[idx] = ni_owner(ni) ? w : -w;
    }
}

// the three operator passes on staged elements (all threads; leading and
// trailing barriers are the caller's): su holds p; on return s1 holds
// D_xi^T f1 + D_eta^T f2 (the weak Laplacian) of both components
template <int N>
__device__ __forceinline__ void cg_laplace(const EoD<N, f2_t>& t, const f2_t* su, f2_t* s1, f2_t* s2,
                                           const float4* sg, int ne)
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
            const float4 g = sg[q];
            const f2_t g11 = f2dup(g.x), g12 = f2dup(g.y), g22 = f2dup(g.z);
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
            // the symbol of a preconditioner (2 ulp; an exact division made no
            // difference to the solutions' errors and cost 3 % at 96 x 96, p = 12)
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

// Assembly of the ring copies (continuous format, dss_value's sums) of ne
// staged elements from e0 on, in place: s holds the block's own element values
// Y every block's.  One task per ring node, so that the
// dependent table and value loads of a pass are all in flight at once and the
// loops over all nodes stay free of branches.
template <int N>
__device__ __forceinline__ void cg_ring(const DevMesh& m, const f2_t* Y, f2_t* s, int e0, int ne)
{
    constexpr int R = 4 * (N - 1), ES = line_es(N);
#pragma unroll 2
    for (int t = threadIdx.x; t < ne * R; t += blockDim.x) {
        const int le = t / R, r = t - le * R;
        const int sc = r / (N - 1), h = r - sc * (N - 1);  // h = 0: the corner the side starts at
        const int i = sc == 0 ? h : sc == 1 ? N - 1 : sc == 2 ? N - 1 - h : 0;
        const int j = sc == 0 ? 0 : sc == 1 ? h : sc == 2 ? N - 1 : N - 1 - h;
        const int e = e0 + le;
        const int fl = __ldg(m.flags + e);
        f2_t* v = s + le * ES + j * N + i;
        if (h != 0) {
            const int sb = __ldg(m.side_base + 4 * e + sc), ss = __ldg(m.side_step + 4 * e + sc);
            if ((fl >> (4 + sc)) & 1) {  // Dirichlet boundary
                *v = 0ull;
            } else if (!((fl >> (16 + sc)) & 1)) {
                const long long q = (long long)sb + (long long)((sc & 1) ? j : i) * ss;
                *v = f2add(*v, __ldcg(Y + q));
            }
        } else {
            const int4* cl = reinterpret_cast<const int4*>(m.corner_nb + (size_t)(4 * e + sc) * CORNER_NB_MAX);
            const int4 qa = __ldg(cl), qb = __ldg(cl + 1);
            const int q[CORNER_NB_MAX] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
            f2_t sum = 0ull;  // csum = 0, then += in connected_elements order
            if ((fl >> (12 + sc)) & 1) {
            } else if (q[0] == -2) {  // more copies than the table holds
                const int node = __ldg(m.corner_node + 4 * e + sc);
                const int q0 = __ldg(m.node_ptr + node), q1 = __ldg(m.node_ptr + node + 1);
                for (int k = q0; k < q1; ++k) {
                    const int f = __ldg(m.node_flat + k);
                    sum = f2add(sum, __ldcg(Y + f));
                }
            } else {
                f2_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) w[k] = q[k] >= 0 ? __ldcg(Y + q[k]) : 0ull;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (q[k] >= 0) sum = f2add(sum, w[k]);
#pragma unroll
                for (int k = 4; k < CORNER_NB_MAX; ++k)
                    if (q[k] >= 0) sum = f2add(sum, __ldcg(Y + q[k]));
            }
            *v = sum;
        }
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
// the power of two that brings the larger of |a|, |b| to [1, 2).  The quotients
// below divide by |d|^2; the inner products carry the unit of length (an element's
// measure to the power -1) and |r|^2, and their squares left FP32's range for
// element sides above some 1e4 or below 1e-8.  Scaling by powers of two changes
// no bit of a quotient whose squares did stay in it.
__device__ __forceinline__ float cg_scale(float a, float b)
{
    const int e = (__float_as_int(fmaxf(fabsf(a), fabsf(b))) >> 23) & 255;
    return __int_as_float(max(254 - e, 1) << 23);
}
// a = rho / (p.Ap); false when it is not a finite number
__device__ __forceinline__ bool cg_step(CgScal& s, float d0, float d1)
{
    const float c = cg_scale(d0, d1);
    d0 *= c;
    d1 *= c;
    const float r0 = s.rho0 * c, r1 = s.rho1 * c;
    const float den = fmaf(d0, d0, d1 * d1);
    const float inv = 1.f / den;
    s.a0 = fmaf(r0, d0, r1 * d1) * inv;
    s.a1 = fmaf(r1, d0, -r0 * d1) * inv;
    return isfinite(s.a0) && isfinite(s.a1);
}
// beta = r.z / rho, rho = r.z
__device__ __forceinline__ bool cg_beta(CgScal& s, float r0, float r1)
{
    const float c = cg_scale(s.rho0, s.rho1);
    const float d0 = s.rho0 * c, d1 = s.rho1 * c, q0 = r0 * c, q1 = r1 * c;
    const float den = fmaf(d0, d0, d1 * d1);
    const float inv = 1.f / den;
    s.b0 = fmaf(q0, d0, q1 * d1) * inv;
    s.b1 = fmaf(q1, d0, -q0 * d1) * inv;
    s.rho0 = r0;
    s.rho1 = r1;
    return isfinite(s.b0) && isfinite(s.b1);
}
// the last sweep reduces to this share of what the outer test needs, so that
// the solutions end as far below its threshold as MINRES left them (at 0.3, the
// MINRES margin in the preconditioned norm, their errors were up to twice as
// large); about 2.5 of 35 iterations
constexpr double CG_MARGIN = 0.1;
// Iterations without a smaller residual before MINRES takes over.  Not monotone,
// the residual of a hard system (deep wells, strong refinement) may stay above its
// smallest value for thousands of iterations and converge all the same: at a limit
// of 200 a well of depth 1e4 on 32 x 32 elements of p = 8 took 8,594 iterations and
// 226 ms, nearly all in the streaming MINRES, against 6,844 and 61 ms (on-chip MINRES
// before the conjugate gradients: 82 ms).  Of 195 solves with potentials to 1e5,
// alpha to 0.1, graded, stretched and distorted meshes none that this limit or 4,000
// gave to MINRES was solved by it, and some that 1,000 gave away were solved without
constexpr int CG_STALL = 20000;
// Whether a sweep left so much of the true residual that MINRES should take over:
// more than halfway between its inner tolerance and one.  Once a sweep of the
// solve has reduced it tenfold the iteration is sound on this operator, and a
// later one that does not has met the rounding of the FP64 residual, which stops
// MINRES as well and costs it more (64 x 64, p = 8, tol = 1e-16, out of reach:
// 57 ms with MINRES taking over there)
__device__ __forceinline__ bool cg_sweep_failed(double rn, double last_rn, double last_itol, bool& sound)
{
    sound = sound || rn < 0.1 * last_rn;
    return !sound && !(rn < 0.5 * (1.0 + last_itol) * last_rn);
}

struct CgOut {
    int it;
    bool conv;    // |r| fell below tol_rel |b|
    bool usable;  // the correction is finite
};

// Solves A d = b for the block's element range [eb, ee) of its team's mesh.
// rhs(flat) is the right-hand side pair scaled to unit norm (continuous format).
// The correction (continuous format, scaled like b) is left in X.  Vectors are
// arrays of n pairs: r, p, Y (element output of A p), Zl (weighted local
// solves).  Returns false when a wait timed out.
template <int N, int TEAM, class Rhs>
__device__ __forceinline__ bool cg_core(unsigned char* smraw, int kmax, const DevMesh& m, const CgTab<N>& tab,
                                        const float4* __restrict__ fac, const float* __restrict__ nnw,
                                        const float* __restrict__ pot, float alpha, int eb, int ee,
                                        const KrylovWork<float>& w, Team& tm, Rhs&& rhs, f2_t* __restrict__ X,
                                        int maxit, float tol_rel, const float* lam, CgOut& res)
{
    constexpr int NN = N * N;
    constexpr int ES = line_es(N);
    constexpr int U = 4;  // nodes a thread has in flight
    float4* sg = (float4*)smraw;
    f2_t* su = (f2_t*)(sg + kmax * ES);
    f2_t* s1 = su + kmax * ES;
    f2_t* s2 = s1 + kmax * ES;
    float* sw = (float*)s2;  // Phase B: weights
    f2_t* __restrict__ const R = (f2_t*)w.L[0];
    f2_t* __restrict__ const P = (f2_t*)w.L[1];
    f2_t* const Y = (f2_t*)w.Y[0];
    f2_t* const Zl = (f2_t*)w.Y[1];
    CgScal sc{};
    res.it = 0;
    res.conv = false;
    res.usable = true;
    if (maxit < 1) return true;
    // Phase B of every iteration (first: r = b)
    auto phase_b = [&](bool first, float (&out)[3]) -> bool {
        float rz0 = 0.f, rz1 = 0.f, rr = 0.f;
        const f2_t na0 = f2dup(-sc.a0), cross = f2pack(sc.a1, -sc.a1);
        for (int e0 = eb; e0 < ee; e0 += kmax) {
            const int ne = min(kmax, ee - e0);
            const int total = ne * NN;
            const long long base = (long long)e0 * NN;
            if (!first) {  // the assembled A p
#pragma unroll 4
                for (int t = threadIdx.x; t < total; t += blockDim.x) su[t + t / NN * (ES - NN)] = __ldcg(Y + base + t);
                __syncthreads();
                cg_ring<N>(m, Y, su, e0, ne);
                __syncthreads();
            }
            for (int t0 = threadIdx.x; t0 < total; t0 += U * blockDim.x) {
                f2_t r[U];
                float wt[U];
#pragma unroll
                for (int h = 0; h < U; ++h) {  // every load of the group before its stores
                    const int t = t0 + h * blockDim.x;
                    if (t < total) {
                        r[h] = first ? rhs(base + t) : R[base + t];
                        wt[h] = __ldg(nnw + base + t);
                    }
                }
#pragma unroll
                for (int h = 0; h < U; ++h) {
                    const int t = t0 + h * blockDim.x;
                    if (t >= total) continue;
                    const int q = t + t / NN * (ES - NN);
                    if (!first) {  // r -= a A p
                        float q0, q1;
                        const f2_t qv = su[q];
                        f2unpack(qv, q0, q1);
                        r[h] = f2fma(cross, f2pack(q1, q0), f2fma(na0, qv, r[h]));
                    }
                    R[base + t] = r[h];
                    float r0, r1;
                    f2unpack(r[h], r0, r1);
                    if (wt[h] > 0.f) rr = fmaf(r0, r0, fmaf(r1, r1, rr));
                    const float wa = fabsf(wt[h]);
                    su[q] = f2mul(f2dup(wa), r[h]);
                    sw[q] = wa;
                }
            }
            __syncthreads();
            cg_fdm<N>(tab.S, su, lam, alpha, ne, [&](int le) { return __ldg(m.fdm_el + e0 + le); }, rz0, rz1);
            __syncthreads();
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += blockDim.x) {
                const int q = t + t / NN * (ES - NN);
                const float wa = sw[q];
                Zl[base + t] = f2mul(f2pack(wa, -wa), su[q]);
            }
            __syncthreads();
        }
        const float v[3] = {rz0, rz1, rr};
        return team_sum<TEAM, 3>(v, tm, out);
    };
    float o3[3], o2[2];
    if (!phase_b(true, o3)) return false;
    sc.rho0 = o3[0];
    sc.rho1 = o3[1];
    const float bb = o3[2];
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
        const f2_t b0 = f2dup(sc.b0), bx = f2pack(sc.b1, -sc.b1), a0 = f2dup(sc.a0), ax = f2pack(sc.a1, -sc.a1);
        for (int e0 = eb; e0 < ee; e0 += kmax) {
            const int ne = min(kmax, ee - e0);
            const int total = ne * NN;
            const long long base = (long long)e0 * NN;
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += blockDim.x) {  // the assembled z, the factors
                const int q = t + t / NN * (ES - NN);
                const f2_t z = __ldcg(Zl + base + t);
                const float4 g = __ldg(fac + base + t);
                su[q] = z;
                sg[q] = g;
            }
            __syncthreads();
            cg_ring<N>(m, Zl, su, e0, ne);
            __syncthreads();
            for (int t0 = threadIdx.x; t0 < total; t0 += U * blockDim.x) {
                f2_t pv[U], xv[U];
#pragma unroll
                for (int h = 0; h < U; ++h) {
                    const int t = t0 + h * blockDim.x;
                    if (t < total && !first) {
                        pv[h] = P[base + t];
                        xv[h] = it > 2 ? X[base + t] : 0ull;
                    }
                }
#pragma unroll
                for (int h = 0; h < U; ++h) {
                    const int t = t0 + h * blockDim.x;
                    if (t >= total) continue;
                    const int q = t + t / NN * (ES - NN);
                    f2_t z = su[q];
                    if (!first) {  // x += a p, p = z + beta p
                        float a, b;
                        f2unpack(pv[h], a, b);
                        const f2_t swp = f2pack(b, a);
                        X[base + t] = f2fma(ax, swp, f2fma(a0, pv[h], xv[h]));
                        z = f2fma(bx, swp, f2fma(b0, pv[h], z));
                    }
                    P[base + t] = z;
                    su[q] = z;
                }
            }
            __syncthreads();
            cg_laplace<N>(tab.D, su, s1, s2, sg, ne);
            __syncthreads();
#pragma unroll 4
            for (int t = threadIdx.x; t < total; t += blockDim.x) {
                const int q = t + t / NN * (ES - NN);
                const float ms = sg[q].w;
                const float mv = ms * __ldg(pot + base + t);
                float u0, u1, l0, l1;
                f2unpack(su[q], u0, u1);
                f2unpack(s1[q], l0, l1);
                const float q0 = ms * u0 + alpha * (l1 + mv * u1);
                const float q1 = alpha * (l0 + mv * u0) - ms * u1;
                d0 = fmaf(u0, q0, fmaf(u1, q1, d0));
                d1 = fmaf(u0, q1, fmaf(-u1, q0, d1));
                Y[base + t] = f2pack(q0, q1);
            }
            __syncthreads();
        }
        const float v2[2] = {d0, d1};
        if (!team_sum<TEAM, 2>(v2, tm, o2)) return false;
        if (!cg_step(sc, o2[0], o2[1])) {
            --it;
            good = false;
            break;
        }
        // ---- Phase B
        if (!phase_b(false, o3)) return false;
        const float rr = o3[2];
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
        if (it < maxit) good = cg_beta(sc, o3[0], o3[1]);
    }
    res.it = it;
    res.usable = good && it > 0;
    // x += a p of the last iteration
    if (res.usable) {
        const f2_t a0 = f2dup(sc.a0), ax = f2pack(sc.a1, -sc.a1);
        const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
#pragma unroll 2
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const f2_t pv = P[idx];
            const f2_t x = it > 1 ? X[idx] : 0ull;
            float a, b;
            f2unpack(pv, a, b);
            X[idx] = f2fma(ax, f2pack(b, a), f2fma(a0, pv, x));
        }
    }
    __syncthreads();
    return true;
}

// FP64 iterative refinement around cg_core for the block's range of its team's
// mesh: r = b - A x in FP64 (true residual, continuous format); stop when
// |r| < scale (tol |r0| + tol) (the reference's criterion, minres.hpp:92; with
// rel_to_b |b| in the place of |r0|); else solve A d = r to the inner tolerance
// and add d to x on owner copies.  res.fallback: the inner iteration broke
// down, stalled or hardly reduced the true residual, and MINRES should go on
// from x.  Returns false when a wait timed out.
struct CgRefine {
    int sweeps, inner;
    bool conv, fallback;
    double rn, r0;
};
template <int N, int TEAM>
__device__ __forceinline__ bool cg_refine(const DevMesh& m, const SolveArgs& a, const KrylovWork<float>& w,
                                          const MixedArgs& mx, int eb, int ee, unsigned char* smraw, float* lam,
                                          const EoD<N, double>& et, const CgTab<N>& tab, Team& tm, CgRefine& res)
{
    constexpr int NN = N * N;
    double* sm64 = (double*)smraw;
    const Fac<double> fac64 = fac_of<double>(m);
    const double* b0 = (const double*)a.b[0];
    const double* b1 = (const double*)a.b[1];
    double* x0 = (double*)a.x[0];
    double* x1 = (double*)a.x[1];
    double* const Y0 = mx.Y64[0];
    double* const Y1 = mx.Y64[1];
    const long long nb = (long long)eb * NN, ne = (long long)ee * NN;
    f2_t* const X = (f2_t*)mx.x32[0];
    res.sweeps = res.inner = 0;
    res.conv = res.fallback = false;
    double last_rn = 0.0, itol = 0.0;
    bool sound = false;
    for (int l = threadIdx.x; l < N; l += blockDim.x) lam[l] = m.fdmL32[l];
    for (;;) {
        const bool applied = res.sweeps > 0 || !a.x_is_zero;
        if (applied) {
            __syncthreads();  // the staging area overlays the inner solve's
            load_dmat_raw<N, double>(sm64, m);
            __syncthreads();
            for (int e0 = eb; e0 < ee; e0 += a.kmax64)
                apply_range<N, double, OP_RES>(
                    sm64, a.kmax64, &et, fac64, (const double*)a.pot, a.alpha, e0, min(a.kmax64, ee - e0),
                    [&](int e, int i, int j, long long flat, double* u) {
                        const long long src = ni_gather_src(m, node_info<N>(m, e, i, j), e, flat);
                        u[0] = x0[src];
                        u[1] = x1[src];
                    },
                    [&](int, int, int, long long flat, const double* o) {
                        Y0[flat] = o[0];
                        Y1[flat] = o[1];
                    });
            if (!team_barrier<TEAM>(tm)) return false;
        }
        double part = 0.0, partb = 0.0;
        const bool want_b = res.sweeps == 0 && a.rel_to_b;
#pragma unroll 2
        for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
            const int e = (int)(idx / NN);
            const int node = (int)(idx - (long long)e * NN);
            const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
            const long long src = ni_gather_src(m, ni, e, idx);
            const double bv0 = b0[src], bv1 = b1[src];
            double r0 = bv0, r1 = bv1;
            if (applied) {
                r0 -= dss_value<N, double, DSS_CONT>(m, Y0, ni, e, idx);
                r1 -= dss_value<N, double, DSS_CONT>(m, Y1, ni, e, idx);
            }
            mx.r64[0][idx] = r0;
            mx.r64[1][idx] = r1;
            if (ni_owner(ni)) {
                part = fma(r0, r0, fma(r1, r1, part));
                if (want_b) partb = fma(bv0, bv0, fma(bv1, bv1, partb));
            }
        }
        double rr = 0.0, bbv = 0.0;
        if (!team_sum64<TEAM>(part, partb, tm, rr, bbv)) return false;
        const double rn = sqrt(rr);
        if (res.sweeps == 0) res.r0 = a.r0_given > 0.0 ? a.r0_given : want_b ? sqrt(bbv) : rn;
        res.rn = rn;
        const double thr = mx.outer_scale * (a.tol * res.r0 + a.tol);
        res.conv = rn < thr;
        if (res.conv || res.sweeps >= mx.max_sweeps || res.inner >= a.maxit || !(rn == rn)) return true;
        if (res.sweeps > 0 && cg_sweep_failed(rn, last_rn, itol, sound)) {
            res.fallback = true;
            return true;
        }
        last_rn = rn;
        // the inner solve reduces by inner_tol, or (last sweep) by CG_MARGIN of
        // what the outer test still needs: a good initial guess then saves
        // iterations, not sweeps
        itol = mx.inner_tol;
        if (mx.adaptive) itol = fmax(itol, fmin(CG_MARGIN * thr / rn, 0.5));
        const double inv = 1.0 / rn;
        const double* r64a = mx.r64[0];
        const double* r64b = mx.r64[1];
        CgOut cr{};
        if (!cg_core<N, TEAM>(smraw, a.kmax, m, tab, mx.fac4, mx.nnw, mx.pot32, (float)a.alpha, eb, ee, w, tm,
                              [&](long long flat) {
                                  return f2pack((float)(r64a[flat] * inv), (float)(r64b[flat] * inv));
                              },
                              X, min(mx.inner_maxit, a.maxit - res.inner), (float)itol, lam, cr))
            return false;
        res.inner += cr.it;
        ++res.sweeps;
        if (cr.usable) {  // x += d
#pragma unroll 4
            for (long long idx = nb + threadIdx.x; idx < ne; idx += blockDim.x) {
                if (!(__ldg(mx.nnw + idx) > 0.f)) continue;
                float d0, d1;
                f2unpack(X[idx], d0, d1);
                x0[idx] += (double)d0 * rn;
                x1[idx] += (double)d1 * rn;
            }
        }
        if (!team_barrier<TEAM>(tm)) return false;
        if (!(cr.usable && cr.conv) && res.inner < a.maxit) {
            res.fallback = true;
            return true;
        }
    }
}

}  // namespace semgb

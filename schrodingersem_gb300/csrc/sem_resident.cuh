// On-chip resident FP32 inner solve of the Schroedinger stage operator with
// the element preconditioner (the complex-symmetric conjugate gradients of
// sem_cg.cuh), inside the same FP64 iterative refinement as mixed_solve.
//
// When a block's share of the mesh fits in shared memory and registers, every
// vector of the inner iteration stays on chip for the whole solve: the search
// direction p, the operator output q and the preconditioned residual z in
// shared memory as (Re, Im) pairs, the residual r and the correction x in
// registers of the thread that owns the element row.  Only the element-ring
// copies (sides and corners, 4(N-1) of N^2 nodes) leave the SM: each is
// published as two 64-bit words (FP32 value, epoch tag; one per component, one
// 16-byte access) and the neighbours assemble every shared node from those
// words in the library's fixed order (dss_value's sums), so every copy of a
// node holds the same bits.  Per iteration:
//   Phase A: x += a p, p = z + beta p, q = A_local p (ring words out)
//            -> exchange (p.q)
//   Phase B: r -= a q, z = local solves of r (ring words out)
//            -> exchange (r.z, |r|^2)
// An exchange is a grid all-reduce and the ring assembly at once
// (res_exchange).
//
// Each phase is three line passes: one thread takes one element line of both
// components (N packed FP32 pairs in registers) and forms the N results of a
// parity-split contraction (eo_d, eo_st, eo_s) with the coefficients as
// constant-bank operands.  The vector updates ride on the row passes, whose
// thread holds r and x of its row, and the second contraction of the column
// direction follows the first in the same thread, so an iteration has four
// block barriers beside the two exchanges.  Measured at 64 x 64 elements,
// p = 8 (27 elements per SM): 15.9 us per iteration all-in (residual checks and
// launches included), against 37.7 for the streaming form; two thirds are the
// latency of the two exchanges and the four barriers, the rest FP32 issue.
//
// All-reduce: each block publishes its partials as 64-bit words (FP32 value,
// 32-bit epoch tag) on its own 128-byte line; every block's first warp polls
// the grid's words (bounded by SEM_OPT_WAIT_TIMEOUT_MS through %globaltimer)
// and sums them in one fixed order, so every block obtains the same bits.  Two
// word sets alternate by epoch parity.  Epochs run on from launch to launch
// (ResArgs::epoch0; the host clears the words when it allocates them, after a
// failed wait and before the counter could wrap).
#pragma once
#include "sem_solvers.cuh"

namespace semgb {

// one row of both components per thread: 243 rows at 27 elements of p = 8.  With
// 512 threads half the warps had no row and 128 registers spilled the line
// contractions: 18.0 us per iteration at 64 x 64 elements of p = 8 against 15.9,
// 11.8 against 9.7 at 24 x 24, 12.0 against 10.9 at 48 x 48 of p = 4.  256 threads
// have up to 255 registers, which N <= 7 and one row of N = 9 (208) keep to; 2 and
// 4 rows of N = 9 spill 240 and 176 bytes, N = 11 between 764 and 1,300
constexpr int RES_TPB = 256;
constexpr int RES_MAXQ = 8;     // words polled per lane: grids up to 256 blocks
constexpr int RES_PAIRS = 4;    // planes of FP32 pairs: p, q, z, preconditioner symbol
constexpr int RES_PLANES = 6;   // FP32 planes: g11, -g12, g22, mass, mass V, weight
constexpr int RES_WSTRIDE = RESIDENT_SLOT_STRIDE;  // all-reduce words 128 bytes apart
// rows per thread held in registers: 1, 2 or 4, by the block's share
constexpr int RES_MAXROWS = 4;
inline int res_rows(int kres, int N)
{
    const int r = (kres * N + RES_TPB - 1) / RES_TPB;
    return r <= 1 ? 1 : r <= 2 ? 2 : r <= RES_MAXROWS ? RES_MAXROWS : 0;
}

struct ResArgs {
    int st;                     // shared-memory plane length (max elements per block * N^2)
    ulonglong2* xa;             // [n] tagged ring words of the operator output
    ulonglong2* xb;             // [n] tagged ring words of the preconditioner output
    unsigned long long* slots;  // [2][gridDim.x][RES_WSTRIDE] tagged partial sums
    unsigned epoch0;            // last epoch used on these words
};

// one 64-bit word: FP32 value in the low half, epoch in the high half
__device__ __forceinline__ unsigned long long res_word(float v, unsigned epoch)
{
    return ((unsigned long long)epoch << 32) | (unsigned long long)__float_as_uint(v);
}
__device__ __forceinline__ unsigned long long res_ld(const unsigned long long* p)
{
    return *(const volatile unsigned long long*)p;
}
// both components' words of a ring copy; each word carries its own tag, so a
// 16-byte access that were split in two would still be read correctly
__device__ __forceinline__ ulonglong2 res_ld2(const ulonglong2* p)
{
    ulonglong2 v;
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool res_ready(const ulonglong2& v, unsigned tag)
{
    return (unsigned)(v.x >> 32) == tag && (unsigned)(v.y >> 32) == tag;
}
__device__ __forceinline__ f2_t res_pair(const ulonglong2& v)
{
    return f2pack(__uint_as_float((unsigned)v.x), __uint_as_float((unsigned)v.y));
}
__device__ __forceinline__ void res_put(ulonglong2* X, long long flat, f2_t v, unsigned tag)
{
    float a, b;
    f2unpack(v, a, b);
    __stcg(X + flat, make_ulonglong2(res_word(a, tag), res_word(b, tag)));
}

// ------------------------------------------------------- shared-memory planes
// pairs first (16-byte aligned base): p, q, z, symbol; then the FP32 planes.
// The symbol and the FP32 planes hold for the whole launch; the FP64
// refinement's staging area overlays p, q, z (plane 3 of the pairs and the
// rest follow after it, ResPlanes::stage bytes in).
struct ResPlanes {
    f2_t *P, *Q, *Z;
    f2_t* Sy;
    float *G11, *G12, *G22, *MS, *MV, *WT;
};
__device__ __forceinline__ ResPlanes res_planes(unsigned char* sm, int st, size_t stage)
{
    ResPlanes r;
    r.P = (f2_t*)sm;
    r.Q = r.P + st;
    r.Z = r.Q + st;
    r.Sy = (f2_t*)(sm + stage);
    r.G11 = (float*)(r.Sy + st);
    r.G12 = r.G11 + st;
    r.G22 = r.G12 + st;
    r.MS = r.G22 + st;
    r.MV = r.MS + st;
    r.WT = r.MV + st;
    return r;
}

template <int N>
__device__ __forceinline__ void res_setup(const DevMesh& m, const ResPlanes& s, int eb, int ne, const float* pot32,
                                          float alpha)
{
    constexpr int NN = N * N;
    const float* lam = m.fdmL32;
    for (int l = threadIdx.x; l < ne * NN; l += RES_TPB) {
        const int le = l / NN;
        const int node = l - le * NN;
        const int i = node % N, j = node / N;
        const int e = eb + le;
        const long long flat = (long long)e * NN + node;
        const float ms = __ldg(m.massf + flat);
        s.G11[l] = __ldg(m.g11f + flat);
        s.G12[l] = -__ldg(m.g12f + flat);
        s.G22[l] = __ldg(m.g22f + flat);
        s.MS[l] = ms;
        s.MV[l] = ms * __ldg(pot32 + flat);
        const float4 g = __ldg(m.fdm_el + e);
        const float al = alpha * (g.y * __ldg(lam + i) + g.z * __ldg(lam + j));
        const float inv = 1.f / (g.x * g.x + al * al);
        s.Sy[l] = f2pack(g.x * inv, al * inv);
        s.WT[l] = nn_weight<N, float>(m, node_info<N>(m, e, i, j), e);
    }
}

// Assembly of the ring copies in place (continuous format, dss_value's
// sums), from tagged words.  The element-local plane P holds this block's
// partials; X holds every block's ring partials, so a load that returns the
// right tags is the data itself: no flag, fence or barrier stands between a
// neighbour's store and its use.  One task per element side (its N-2 side
// nodes: own + the neighbour's copy at side_base + k side_step) and one per
// element corner (the corner node's copies in CSR order); stale words are
// reloaded until their tags match (bounded: returns false after recording
// gs->err when tmo runs out).  Dirichlet boundary copies become zero; lone
// (Neumann) sides keep their own value.  Threads [t_first, RES_TPB) take the
// tasks.
template <int N>
__device__ __forceinline__ bool res_ring(const DevMesh& m, const ulonglong2* X, f2_t* P, int eb, int ne, unsigned tag,
                                         int t_first, GridSync* gs, long long tmo)
{
    constexpr int NN = N * N;
    const int nside = ne * 4;  // (element, side)
    const int ntask = ne * 8;
    bool ok = true;
    const unsigned long long t0 = global_ns();
    auto expired = [&](unsigned polls) {
        if ((polls & 31u) == 0 && (*(volatile int*)&gs->err || (long long)(global_ns() - t0) > tmo)) {
            atomicExch(&gs->err, 1);
            return true;
        }
        return false;
    };
    for (int t = threadIdx.x - t_first; t < ntask && ok; t += RES_TPB - t_first) {
        const bool corner = t >= nside;
        const int u = corner ? t - nside : t;
        const int sc = u & 3;
        const int le = u >> 2;
        const int e = eb + le;
        const int fl = __ldg(m.flags + e);
        f2_t* pe = P + le * NN;
        if (!corner) {
            const int l0 = sc == 0 ? 0 : sc == 1 ? N - 1 : sc == 2 ? (N - 1) * N : 0;
            const int lk = (sc == 0 || sc == 2) ? 1 : N;
            if ((fl >> (4 + sc)) & 1) {  // Dirichlet boundary side
#pragma unroll
                for (int k = 1; k < N - 1; ++k) pe[l0 + k * lk] = 0ull;
            } else if (!((fl >> (16 + sc)) & 1)) {  // interior side: own + other
                const long long sb = __ldg(m.side_base + 4 * e + sc), ss = __ldg(m.side_step + 4 * e + sc);
                ulonglong2 w[N];
#pragma unroll
                for (int k = 1; k < N - 1; ++k) w[k] = res_ld2(X + sb + k * ss);
                for (unsigned polls = 1;; ++polls) {
                    bool ready = true;
#pragma unroll
                    for (int k = 1; k < N - 1; ++k) ready &= res_ready(w[k], tag);
                    if (ready) break;
                    if (expired(polls)) {
                        ok = false;
                        break;
                    }
#pragma unroll
                    for (int k = 1; k < N - 1; ++k)
                        if (!res_ready(w[k], tag)) w[k] = res_ld2(X + sb + k * ss);
                }
#pragma unroll
                for (int k = 1; k < N - 1; ++k) pe[l0 + k * lk] = f2add(pe[l0 + k * lk], res_pair(w[k]));
            }
        } else {
            const int lc = sc == 0 ? 0 : sc == 1 ? N - 1 : sc == 2 ? NN - 1 : (N - 1) * N;
            if ((fl >> (12 + sc)) & 1) {  // Dirichlet boundary corner
                pe[lc] = 0ull;
                continue;
            }
            const int* cl = m.corner_nb + (size_t)(4 * e + sc) * CORNER_NB_MAX;
            int q[CORNER_NB_MAX];
#pragma unroll
            for (int k = 0; k < CORNER_NB_MAX; ++k) q[k] = __ldg(cl + k);
            f2_t sum = 0ull;  // csum = 0, then += in connected_elements order
            if (q[0] == -2) {  // more copies than the table holds: the CSR, one by one
                const int node = __ldg(m.corner_node + 4 * e + sc);
                const int q0 = __ldg(m.node_ptr + node), q1 = __ldg(m.node_ptr + node + 1);
                for (int k = q0; k < q1 && ok; ++k) {
                    const int f = __ldg(m.node_flat + k);
                    ulonglong2 v = res_ld2(X + f);
                    for (unsigned polls = 1; !res_ready(v, tag); ++polls) {
                        if (expired(polls)) {
                            ok = false;
                            break;
                        }
                        v = res_ld2(X + f);
                    }
                    sum = f2add(sum, res_pair(v));
                }
            } else {
                const unsigned long long none = res_word(0.f, tag);
                ulonglong2 w[CORNER_NB_MAX];
#pragma unroll
                for (int k = 0; k < CORNER_NB_MAX; ++k) w[k] = q[k] >= 0 ? res_ld2(X + q[k]) : make_ulonglong2(none, none);
                for (unsigned polls = 1;; ++polls) {
                    bool ready = true;
#pragma unroll
                    for (int k = 0; k < CORNER_NB_MAX; ++k) ready &= res_ready(w[k], tag);
                    if (ready) break;
                    if (expired(polls)) {
                        ok = false;
                        break;
                    }
#pragma unroll
                    for (int k = 0; k < CORNER_NB_MAX; ++k)
                        if (!res_ready(w[k], tag)) w[k] = res_ld2(X + q[k]);
                }
#pragma unroll
                for (int k = 0; k < CORNER_NB_MAX; ++k)
                    if (q[k] >= 0) sum = f2add(sum, res_pair(w[k]));
            }
            pe[lc] = sum;
        }
    }
    return ok;
}

// One phase boundary: the grid all-reduce of K values (first warp: publish
// this block's words, poll every block's) and, at the same time, the in-place
// ring assembly of P from the tagged words X (the other warps).  Both wait for
// the same stores of the other blocks, so the phase costs one round trip after
// the last of them.  The ring words and the all-reduce words carry the same
// epoch.  Returns false when a wait hit its limit.
template <int N, int K>
__device__ __forceinline__ bool res_exchange(const float (&v)[K], const DevMesh& m, const ulonglong2* X, f2_t* P,
                                             int eb, int ne, unsigned long long* slots, unsigned& epoch, GridSync* gs,
                                             long long tmo, float (*red)[RES_TPB / 32], float* tot, float (&out)[K])
{
    static_assert(K <= 3, "words per line");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float a[K];
#pragma unroll
    for (int k = 0; k < K; ++k) a[k] = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < K; ++k) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) red[k][wid] = a[k];
    ++epoch;
    __syncthreads();
    bool ok = true;
    if (wid == 0) {
        // the block's sum in FP32, as the word that carries it; pairs (two_add) made
        // no difference to the solutions' errors and cost 8 % at 48 x 48, p = 4
        // (12.2 to 13.1 us per iteration)
        constexpr int nw = RES_TPB / 32;
#pragma unroll
        for (int k = 0; k < K; ++k) a[k] = lane < nw ? red[k][lane] : 0.f;
#pragma unroll
        for (int o = nw / 2; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < K; ++k) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
        const int G = gridDim.x;
        unsigned long long* sl = slots + (size_t)(epoch & 1u) * G * RES_WSTRIDE;
        if (lane == 0) {
            unsigned long long* own = sl + blockIdx.x * RES_WSTRIDE;
            __stcg((ulonglong2*)own, make_ulonglong2(res_word(a[0], epoch), res_word(K > 1 ? a[K > 1] : 0.f, epoch)));
            if (K > 2) __stcg(own + 2, res_word(a[K - 1], epoch));
        }
        ulonglong2 u[RES_MAXQ];
        unsigned long long u2[RES_MAXQ];
        const unsigned long long none = res_word(0.f, epoch);
        const unsigned long long t0 = global_ns();
#pragma unroll
        for (int q = 0; q < RES_MAXQ; ++q) {
            const int blk = lane + 32 * q;
            u[q] = blk < G ? res_ld2((const ulonglong2*)(sl + blk * RES_WSTRIDE)) : make_ulonglong2(none, none);
            u2[q] = K > 2 && blk < G ? res_ld(sl + blk * RES_WSTRIDE + 2) : none;
        }
        for (unsigned polls = 1;; ++polls) {
            bool ready = true;
#pragma unroll
            for (int q = 0; q < RES_MAXQ; ++q) ready &= res_ready(u[q], epoch) && (K < 3 || (unsigned)(u2[q] >> 32) == epoch);
            if (ready) break;
            if ((polls & 31u) == 0 && (*(volatile int*)&gs->err || (long long)(global_ns() - t0) > tmo)) {
                atomicExch(&gs->err, 1);
                ok = false;
                break;
            }
#pragma unroll
            for (int q = 0; q < RES_MAXQ; ++q) {
                const int blk = lane + 32 * q;
                if (blk >= G) continue;
                if (!res_ready(u[q], epoch)) u[q] = res_ld2((const ulonglong2*)(sl + blk * RES_WSTRIDE));
                if (K > 2 && (unsigned)(u2[q] >> 32) != epoch) u2[q] = res_ld(sl + blk * RES_WSTRIDE + 2);
            }
        }
        // sums of the words in twice FP32 precision (two_add): FP64 additions
        // and conversions, 64 cycles each on GB300, took 2.7 us per iteration
        float hi[K], lo[K];
#pragma unroll
        for (int k = 0; k < K; ++k) hi[k] = lo[k] = 0.f;
#pragma unroll
        for (int q = 0; q < RES_MAXQ; ++q) {
            two_add(hi[0], lo[0], __uint_as_float((unsigned)u[q].x), 0.f);
            if (K > 1) two_add(hi[K > 1], lo[K > 1], __uint_as_float((unsigned)u[q].y), 0.f);
            if (K > 2) two_add(hi[K - 1], lo[K - 1], __uint_as_float((unsigned)u2[q]), 0.f);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < K; ++k)
                two_add(hi[k], lo[k], __shfl_down_sync(0xffffffffu, hi[k], o),
                        __shfl_down_sync(0xffffffffu, lo[k], o));
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < K; ++k) tot[k] = hi[k] + lo[k];
    } else {
        ok = res_ring<N>(m, X, P, eb, ne, epoch, 32, gs, tmo);
    }
    const bool fail = __syncthreads_or(!ok) != 0;
#pragma unroll
    for (int k = 0; k < K; ++k) out[k] = tot[k];
    return !fail;
}

// The inner solve A d = r (r64: FP64 residual planes, continuous format,
// |r| = rn > 0) to |r_it| < tol_rel |r|, at most maxit iterations; adds d to
// the FP64 solution on owner copies when it is finite.  Returns false when a
// wait hit its limit.
template <int N, int RW>
__device__ __forceinline__ bool res_inner(const DevMesh& m, const CgTab<N>& tab, const ResPlanes& s, int eb, int ne,
                                          const double* const* r64, double rn, float alpha, const ResArgs& ra,
                                          unsigned& epoch, GridSync* gs, long long tmo, float (*red)[RES_TPB / 32],
                                          float* tot, int maxit, float tol_rel, double* const* xp, CgOut& res)
{
    constexpr int NN = N * N;
    const int lines = ne * N;
    const LineNe nb = line_ne(ne);
    res.it = 0;
    res.conv = false;
    res.usable = false;
    if (maxit < 1) return true;
    const double inv_rn = 1.0 / rn;
    f2_t r[RW][N], x[RW][N];  // this thread's rows
    unsigned own[RW];         // owner copies of the row
    CgScal sc{};
    // Phase B: r -= a q (first: r = b), local solves into Z, exchange
    auto phase_b = [&](bool first, float (&out)[3]) -> bool {
        float rz0 = 0.f, rz1 = 0.f, rr = 0.f;
        const f2_t na0 = f2dup(-sc.a0), cross = f2pack(sc.a1, -sc.a1);
#pragma unroll
        for (int q = 0; q < RW; ++q) {
            const int L = threadIdx.x + q * RES_TPB;
            if (L >= lines) continue;
            int pos, le;
            line_of(L, nb, pos, le);
            const int o = le * NN + pos * N;
            f2_t u[N], md[N];
            if (first) {
                const long long flat = (long long)eb * NN + o;
                own[q] = 0u;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    r[q][i] = f2pack((float)(__ldcg(r64[0] + flat + i) * inv_rn), (float)(__ldcg(r64[1] + flat + i) * inv_rn));
                    x[q][i] = 0ull;
                    if (ni_owner(node_info<N>(m, eb + le, i, pos))) own[q] |= 1u << i;
                }
            } else {
#pragma unroll
                for (int i = 0; i < N; ++i) {  // r -= (a0 + i a1)(q0 + i q1)
                    float q0, q1;
                    const f2_t qv = s.Q[o + i];
                    f2unpack(qv, q0, q1);
                    r[q][i] = f2fma(cross, f2pack(q1, q0), f2fma(na0, qv, r[q][i]));
                }
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                float a, b;
                f2unpack(r[q][i], a, b);
                if ((own[q] >> i) & 1u) rr = fmaf(a, a, fmaf(b, b, rr));
                u[i] = f2mul(f2dup(s.WT[o + i]), r[q][i]);
            }
            eo_st<N>(tab.S, u, md);
#pragma unroll
            for (int i = 0; i < N; ++i) s.Z[o + i] = md[i];
        }
        __syncthreads();
        for (int L = threadIdx.x; L < lines; L += RES_TPB) {  // columns
            int pos, le;
            line_of(L, nb, pos, le);
            const int o = le * NN + pos;
            f2_t u[N], md[N];
#pragma unroll
            for (int k = 0; k < N; ++k) u[k] = s.Z[o + k * N];
            eo_st<N>(tab.S, u, md);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                float dr, di, a, b, c, e;
                f2unpack(s.Sy[o + k * N], dr, di);
                const f2_t d = cg_cmul(md[k], dr, di);
                f2unpack(md[k], a, b);
                f2unpack(d, c, e);
                rz0 = fmaf(a, c, fmaf(-b, e, rz0));
                rz1 = fmaf(a, e, fmaf(b, c, rz1));
                md[k] = d;
            }
            eo_s<N>(tab.S, md, u);
#pragma unroll
            for (int k = 0; k < N; ++k) s.Z[o + k * N] = u[k];
        }
        __syncthreads();
        for (int L = threadIdx.x; L < lines; L += RES_TPB) {  // rows
            int pos, le;
            line_of(L, nb, pos, le);
            const int o = le * NN + pos * N;
            const long long flat = (long long)eb * NN + o;
            f2_t u[N], md[N];
#pragma unroll
            for (int k = 0; k < N; ++k) md[k] = s.Z[o + k];
            eo_s<N>(tab.S, md, u);
            const bool side = pos == 0 || pos == N - 1;
#pragma unroll
            for (int k = 0; k < N; ++k) {  // stored as (Re, -Im)
                const float wt = s.WT[o + k];
                const f2_t z = f2mul(f2pack(wt, -wt), u[k]);
                s.Z[o + k] = z;
                if (side || k == 0 || k == N - 1) res_put(ra.xb, flat + k, z, epoch + 1);
            }
        }
        const float v[3] = {rz0, rz1, rr};
        return res_exchange<N, 3>(v, m, ra.xb, s.Z, eb, ne, ra.slots, epoch, gs, tmo, red, tot, out);
    };
    float o3[3], o2[2];
    __syncthreads();
    if (!phase_b(true, o3)) return false;
    sc.rho0 = o3[0];
    sc.rho1 = o3[1];
    const float bb = o3[2];
    sc.best = bb;
    bool good = isfinite(sc.rho0) && isfinite(sc.rho1) && bb > 0.f;
    int it = 0;
    while (good && it < maxit) {
        ++it;
        // ---- Phase A (Z holds the assembled z)
        float d0 = 0.f, d1 = 0.f;
        {
            const f2_t b0 = f2dup(sc.b0), bx = f2pack(sc.b1, -sc.b1);
            const f2_t a0 = f2dup(sc.a0), ax = f2pack(sc.a1, -sc.a1);
#pragma unroll
            for (int q = 0; q < RW; ++q) {
                const int L = threadIdx.x + q * RES_TPB;
                if (L >= lines) continue;
                int pos, le;
                line_of(L, nb, pos, le);
                const int o = le * NN + pos * N;
                f2_t u[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    u[i] = s.Z[o + i];
                    if (it > 1) {
                        const f2_t pv = s.P[o + i];
                        float a, b;
                        f2unpack(pv, a, b);
                        const f2_t sw = f2pack(b, a);
                        x[q][i] = f2fma(ax, sw, f2fma(a0, pv, x[q][i]));
                        u[i] = f2fma(bx, sw, f2fma(b0, pv, u[i]));
                    }
                    s.P[o + i] = u[i];
                }
                eo_d<N, false>(tab.D, u, u);
#pragma unroll
                for (int i = 0; i < N; ++i) s.Q[o + i] = u[i];
            }
        }
        __syncthreads();
        for (int L = threadIdx.x; L < lines; L += RES_TPB) {  // columns: u_eta, fluxes, D^T f2 (into Z)
            int pos, le;
            line_of(L, nb, pos, le);
            const int o = le * NN + pos;
            f2_t us[N];
#pragma unroll
            for (int k = 0; k < N; ++k) us[k] = s.P[o + k * N];
            eo_d<N, false>(tab.D, us, us);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const int q = o + k * N;
                const f2_t ur = s.Q[q];
                const f2_t g11 = f2dup(s.G11[q]), g12 = f2dup(s.G12[q]), g22 = f2dup(s.G22[q]);
                s.Q[q] = f2fma(g12, us[k], f2mul(g11, ur));
                us[k] = f2fma(g12, ur, f2mul(g22, us[k]));
            }
            eo_d<N, true>(tab.D, us, us);
#pragma unroll
            for (int k = 0; k < N; ++k) s.Z[o + k * N] = us[k];
        }
        __syncthreads();
        for (int L = threadIdx.x; L < lines; L += RES_TPB) {  // rows: D^T f1 + D^T f2, the Res combination
            int pos, le;
            line_of(L, nb, pos, le);
            const int o = le * NN + pos * N;
            const long long flat = (long long)eb * NN + o;
            f2_t f[N];
#pragma unroll
            for (int k = 0; k < N; ++k) f[k] = s.Q[o + k];
            eo_d<N, true>(tab.D, f, f);
            const bool side = pos == 0 || pos == N - 1;
#pragma unroll
            for (int k = 0; k < N; ++k) {
                float u0, u1, l0, l1;
                f2unpack(s.P[o + k], u0, u1);
                f2unpack(f2add(f[k], s.Z[o + k]), l0, l1);
                const float ms = s.MS[o + k], mv = s.MV[o + k];
                const float q0 = ms * u0 + alpha * (l1 + mv * u1);
                const float q1 = alpha * (l0 + mv * u0) - ms * u1;
                d0 = fmaf(u0, q0, fmaf(u1, q1, d0));
                d1 = fmaf(u0, q1, fmaf(-u1, q0, d1));
                const f2_t qv = f2pack(q0, q1);
                s.Q[o + k] = qv;
                if (side || k == 0 || k == N - 1) res_put(ra.xa, flat + k, qv, epoch + 1);
            }
        }
        const float v2[2] = {d0, d1};
        if (!res_exchange<N, 2>(v2, m, ra.xa, s.Q, eb, ne, ra.slots, epoch, gs, tmo, red, tot, o2)) return false;
        if (!cg_step(sc, o2[0], o2[1])) {
            --it;
            good = false;
            break;
        }
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
    if (res.usable) {  // x += d (FP64, owner copies): d = |r| (x + a p of the last iteration)
        const f2_t a0 = f2dup(sc.a0), ax = f2pack(sc.a1, -sc.a1);
#pragma unroll
        for (int q = 0; q < RW; ++q) {
            const int L = threadIdx.x + q * RES_TPB;
            if (L >= lines) continue;
            int pos, le;
            line_of(L, nb, pos, le);
            const int o = le * NN + pos * N;
            const long long flat = (long long)eb * NN + o;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const f2_t pv = s.P[o + i];
                float a, b;
                f2unpack(pv, a, b);
                f2unpack(f2fma(ax, f2pack(b, a), f2fma(a0, pv, x[q][i])), a, b);
                if ((own[q] >> i) & 1u) {
                    xp[0][flat + i] += (double)a * rn;
                    xp[1][flat + i] += (double)b * rn;
                }
            }
        }
    }
    return true;
}

// ------------------------------------------------------------------ kernel
// FP64 iterative refinement (the sweep of mixed_solve: true residual
// r = b - A x, the reference's stopping test on |r|) around res_inner.  When
// the inner iteration breaks down, stalls or hardly reduces the true residual
// the kernel ends with SolveOut::fallback set and the host continues on the
// staged kernel with MINRES.
// bytes of the FP64 staging area and, at least, of p, q and z (a multiple of 16)
template <int N>
__host__ __device__ constexpr size_t res_stage_bytes(int st, int k64)
{
    const size_t pairs = (size_t)(RES_PAIRS - 1) * st * sizeof(f2_t);
    const size_t f64 = range_smem_bytes<N, double, OP_RES>(k64);
    return ((pairs > f64 ? pairs : f64) + 15) & ~(size_t)15;
}
enum ResEnd : int { RES_GO = 0, RES_STOP = 1, RES_CONVERGED = 2, RES_FALLBACK = 3 };
template <int N, int RW>
__global__ void __launch_bounds__(RES_TPB, 1)
    k_resident(DevMesh m, SolveArgs a, KrylovWork<float> w, MixedArgs mx, const __grid_constant__ EoD<N, double> et,
               const __grid_constant__ CgTab<N> tab, ResArgs ra)
{
    constexpr int NN = N * N;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[34];
    __shared__ float redf[3][RES_TPB / 32], tot[3];
    // r0, |r|, end of the refinement (ResEnd), last |r|, inner tolerance, sound
    // (cg_sweep_failed): thread 0's, so that no register holds them across the
    // inner solve (kept by every thread: 18.7 us per iteration at 64 x 64, p = 8, and 11.7 at
    // 24 x 24, against 17.8 and 10.6)
    __shared__ double sweep_state[6];
    const ResPlanes s = res_planes(smraw, ra.st, res_stage_bytes<N>(ra.st, a.kmax));
    int eb, ee;
    block_range(m.E, eb, ee);
    const int ne = ee - eb;
    const float alpha32 = (float)a.alpha;
    res_setup<N>(m, s, eb, ne, mx.pot32, alpha32);
    double* sm64 = (double*)smraw;  // FP64 staging of the refinement
    const Fac<double> fac64 = fac_of<double>(m);
    const double* pot64 = (const double*)a.pot;
    const double* bp[2] = {(const double*)a.b[0], (const double*)a.b[1]};
    double* xp[2] = {(double*)a.x[0], (double*)a.x[1]};
    const long long nb = (long long)eb * NN, nend = (long long)ee * NN;
    const int kmax = a.kmax;
    int slot = 0;
    unsigned epoch = ra.epoch0;
    bool ok = true;
    int sweep = 0, inner_total = 0;
    bool conv = false, fallback = false;
    for (;;) {
        // ---- FP64 residual r = unmask(b) - DSS(A_local(unmask(x)))
        const bool applied = (sweep > 0) || !a.x_is_zero;
        if (applied) {
            __syncthreads();  // the staging area overlays the inner solve's planes
            load_dmat_raw<N, double>(sm64, m);
            __syncthreads();
            for (int e0 = eb; e0 < ee; e0 += kmax)
                apply_range<N, double, OP_RES>(
                    sm64, kmax, &et, fac64, pot64, a.alpha, e0, min(kmax, ee - e0),
                    [&](int e, int i, int j, long long flat, double* u) {
                        const long long src = ni_gather_src(m, node_info<N>(m, e, i, j), e, flat);
                        u[0] = xp[0][src];
                        u[1] = xp[1][src];
                    },
                    [&](int, int, int, long long flat, const double* o) {
                        mx.Y64[0][flat] = o[0];
                        mx.Y64[1][flat] = o[1];
                    });
            if (!grid_barrier(a.sync, a.timeout_ns)) return;
        }
        double part = 0.0, partb = 0.0;
        const bool want_b = (sweep == 0) && a.rel_to_b;
#pragma unroll 4
        for (long long idx = nb + threadIdx.x; idx < nend; idx += blockDim.x) {
            const int e = (int)(idx / NN);
            const int node = (int)(idx - (long long)e * NN);
            const NodeInfo ni = node_info<N>(m, e, node % N, node / N);
            const long long src = ni_gather_src(m, ni, e, idx);
            const bool own = ni_owner(ni);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const double bv = bp[c][src];
                double r = bv;
                if (applied) r = r - dss_value<N, double, DSS_CONT>(m, mx.Y64[c], ni, e, idx);
                mx.r64[c][idx] = r;
                if (own) {
                    part = fma(r, r, part);
                    if (want_b) partb = fma(bv, bv, partb);
                }
            }
        }
        double rr = 0.0, bbv = 0.0;
        grid_sum2_t<double>(part, partb, w.partials, slot, a.sync, a.timeout_ns, red, ok, rr, bbv);
        slot ^= 1;
        if (!ok) return;
        if (threadIdx.x == 0) {
            const double rn = sqrt(rr);
            if (sweep == 0) {
                sweep_state[0] = want_b ? sqrt(bbv) : rn;
                sweep_state[5] = 0.0;
            }
            const double need = mx.outer_scale * (a.tol * sweep_state[0] + a.tol);
            double end = RES_GO;
            if (rn < need || rn == 0.0) {
                end = RES_CONVERGED;
            } else if (sweep >= mx.max_sweeps || inner_total >= a.maxit || !(rn == rn)) {
                end = RES_STOP;
            } else if (sweep > 0) {
                bool sound = sweep_state[5] != 0.0;
                if (cg_sweep_failed(rn, sweep_state[3], sweep_state[4], sound)) end = RES_FALLBACK;
                sweep_state[5] = sound ? 1.0 : 0.0;
            }
            sweep_state[1] = sweep_state[3] = rn;
            sweep_state[2] = end;
            sweep_state[4] = mx.adaptive ? fmax(mx.inner_tol, fmin(CG_MARGIN * (need / rn), 0.5)) : mx.inner_tol;
        }
        __syncthreads();
        if (sweep_state[2] != RES_GO) {
            conv = sweep_state[2] == RES_CONVERGED;
            fallback = sweep_state[2] == RES_FALLBACK;
            break;
        }
        // ---- FP32 inner solve A d = r on chip; x += d
        const int budget = min(mx.inner_maxit, a.maxit - inner_total);
        const double rn = sweep_state[1], itol = sweep_state[4];
        const double* r64c[2] = {mx.r64[0], mx.r64[1]};
        CgOut ir{};
        if (!res_inner<N, RW>(m, tab, s, eb, ne, r64c, rn, alpha32, ra, epoch, a.sync, a.timeout_ns, redf, tot, budget,
                          (float)itol, xp, ir))
            return;
        inner_total += ir.it;
        ++sweep;
        if (!grid_barrier(a.sync, a.timeout_ns)) return;
        if (!(ir.usable && ir.conv) && inner_total < a.maxit) {
            fallback = true;
            break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->success = conv ? 1 : 0;
        a.out->n_iter = inner_total;
        a.out->residual = sweep_state[1];
        a.out->status = 0;
        a.out->inner_iters = inner_total;
        a.out->sweeps = sweep;
        a.out->fallback = fallback ? 1 : 0;
        a.out->r0 = sweep_state[0];
        a.out->epoch = epoch;
    }
}

// ---------------------------------------------------------------- launcher
// Plan: one block per SM (fewer for small meshes); fits when a block's rows
// fit its threads' registers and the planes fit smem_budget.  kmax64: elements
// per pass of the FP64 refinement's staged apply, which overlays p, q and z
// (extended when a pass of one element needs more).
template <int N>
bool resident_plan(int E, int sms, size_t smem_budget, int* grid_out, int* st_out, int* kmax64_out,
                   size_t* smem_out)
{
    constexpr int NN = N * N;
    int grid = E < sms ? E : sms;
    if (grid < 1 || grid > 32 * RES_MAXQ) return false;
    const int kres = (E + grid - 1) / grid;
    const int st = kres * NN;
    if (res_rows(kres, N) == 0) return false;
    const size_t fixed = (size_t)st * (sizeof(f2_t) + RES_PLANES * sizeof(float));
    int k64 = kres;
    auto need = [&](int k) { return fixed + res_stage_bytes<N>(st, k); };
    while (k64 > 1 && need(k64) > smem_budget) --k64;
    const size_t smem = need(k64);
    if (smem > smem_budget) return false;
    *grid_out = grid;
    *st_out = st;
    *kmax64_out = k64;
    *smem_out = smem;
    return true;
}

template <int N>
cudaError_t launch_resident(const DevMesh& m, const SolveArgs& a, const KrylovWork<float>& w, const MixedArgs& mx,
                            int st, unsigned long long* slots, void* xa, void* xb, unsigned epoch0, int grid,
                            size_t smem, cudaStream_t stream)
{
    const int rows = res_rows((m.E + grid - 1) / grid, N);
    const void* fn = rows == 1   ? (const void*)k_resident<N, 1>
                     : rows == 2 ? (const void*)k_resident<N, 2>
                                 : (const void*)k_resident<N, RES_MAXROWS>;
    if (!m.Dh || !m.Sh) return cudaErrorInvalidValue;
    // a per-device function attribute: set on every launch (cheap), so a
    // context on any device of the process gets the opt-in
    size_t limit = 0;
    if (!smem_opt_in_all(fn, &limit) || smem > limit) return cudaErrorInvalidConfiguration;
    DevMesh mm = m;
    SolveArgs aa = a;
    KrylovWork<float> ww = w;
    MixedArgs xx = mx;
    EoD<N, double> et = eo_d_table<N, double>(m.Dh);
    CgTab<N> tab = cg_table<N>(m);
    ResArgs ra{st, (ulonglong2*)xa, (ulonglong2*)xb, slots, epoch0};
    void* args[] = {&mm, &aa, &ww, &xx, &et, &tab, &ra};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(RES_TPB), args, smem, stream);
}

#define SEM_INSTANTIATE_RESIDENT(NV)                                                                           \
    template bool resident_plan<NV>(int, int, size_t, int*, int*, int*, size_t*);                             \
    template cudaError_t launch_resident<NV>(const DevMesh&, const SolveArgs&, const KrylovWork<float>&,      \
                                             const MixedArgs&, int, unsigned long long*, void*, void*, unsigned, \
                                             int, size_t, cudaStream_t);

}  // namespace semgb

// Line contractions of one element direction, split by parity.
//
// The LGL nodes are symmetric about 0, so the derivative matrix is
// centro-antisymmetric, D(N-1-i, N-1-k) = -D(i, k), and the eigenvectors of
// the 1-D preconditioner basis are even or odd.  With the even and odd parts
// of a line, s_k = u_k + u_{N-1-k} and d_k = u_k - u_{N-1-k} (s_m = u_m in the
// middle of an odd N), a contraction needs half the products:
//   D u:    a_i = sum_k P(i,k) s_k,  b_i = sum_k Q(i,k) d_k,
//           (D u)_i = b_i + a_i,  (D u)_{N-1-i} = b_i - a_i
//   D^T u:  the same with P and Q transposed and exchanged
// (P, Q: H x C and C x H, H = N/2, C = (N+1)/2).  For N = 9 that is 40
// products and 16 additions instead of 81 products.  The tables are passed to
// the kernels by value: the unrolled code reads them as constant-bank
// operands.
#pragma once
#include <cstdint>
#include <cstring>
#include <type_traits>

namespace semgb {

// ------------------------------------------------ packed FP32 pair arithmetic
// (each lane an IEEE FP32 operation)
typedef unsigned long long f2_t;
__device__ __forceinline__ unsigned long long f2pack(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2unpack(unsigned long long v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long f2fma(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2_t f2add(f2_t a, f2_t b)
{
    f2_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2sub(f2_t a, f2_t b)
{
    f2_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2mul(f2_t a, f2_t b)
{
    f2_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2dup(float a) { return f2pack(a, a); }
__device__ __forceinline__ float f2x(f2_t v)
{
    float a, b;
    f2unpack(v, a, b);
    return a;
}
__device__ __forceinline__ float f2y(f2_t v)
{
    float a, b;
    f2unpack(v, a, b);
    return b;
}

// values a line pass works on: an FP32 pair (both components) or a double
__device__ __forceinline__ f2_t lv_add(f2_t a, f2_t b) { return f2add(a, b); }
__device__ __forceinline__ f2_t lv_sub(f2_t a, f2_t b) { return f2sub(a, b); }
__device__ __forceinline__ double lv_add(double a, double b) { return a + b; }
__device__ __forceinline__ double lv_sub(double a, double b) { return a - b; }

// Table entries of FP32 pairs: both lanes' coefficient, (c, c), for packed FMAs, or
// one FP32 value for two scalar FMAs.  A packed FMA issues half as often, but its
// coefficient occupies a register pair that has to be loaded, so the form follows
// the degree.  Measured per iteration of the stage solver, packed against scalar:
//   N = 9   64 x 64 elements on chip 15.9 us against 18.5, 192 x 192 streaming 209 against 206
//   N = 11  30 x 30 on chip 17.5 against 14.6
//   N = 13  96 x 96 streaming 123 against 96
//   N = 5   48 x 48 on chip 12.6 against 12.0; N = 6 40 x 40 18.7 against 18.9
// (the same rounding either way: each lane is one IEEE FP32 FMA)
template <int N>
__host__ __device__ constexpr bool eo_packed() { return N >= 8 && N <= 10; }
template <int N, class V>
struct EoCoef {
    using type = double;
};
template <int N>
struct EoCoef<N, f2_t> {
    using type = typename std::conditional<eo_packed<N>(), f2_t, float>::type;
};
__host__ inline void eo_set(double& t, double v) { t = v; }
__host__ inline void eo_set(float& t, double v) { t = (float)v; }
__host__ inline void eo_set(f2_t& t, double v)
{
    const float f = (float)v;
    uint32_t u;
    memcpy(&u, &f, sizeof(u));
    t = ((f2_t)u << 32) | u;
}
__device__ __forceinline__ f2_t lv_cmul(f2_t c, f2_t b) { return f2mul(c, b); }
__device__ __forceinline__ f2_t lv_cfma(f2_t c, f2_t b, f2_t a) { return f2fma(c, b, a); }
__device__ __forceinline__ f2_t lv_cmul(float c, f2_t b)
{
    float x, y;
    f2unpack(b, x, y);
    return f2pack(c * x, c * y);
}
__device__ __forceinline__ f2_t lv_cfma(float c, f2_t b, f2_t a)
{
    float x, y, u, v;
    f2unpack(b, x, y);
    f2unpack(a, u, v);
    return f2pack(fmaf(c, x, u), fmaf(c, y, v));
}
__device__ __forceinline__ double lv_cmul(double c, double b) { return c * b; }
__device__ __forceinline__ double lv_cfma(double c, double b, double a) { return fma(c, b, a); }

template <int N, class V>
struct EoD {
    static constexpr int H = N / 2, C = (N + 1) / 2;
    using K = typename EoCoef<N, V>::type;
    K P[H * C];  // P(i,k) at [i*C+k]
    K Q[C * H];  // Q(i,k) at [i*H+k]
};
// preconditioner basis, even modes first (fdm_basis orders them so)
template <int N, class V>
struct EoS {
    static constexpr int H = N / 2, C = (N + 1) / 2;
    using K = typename EoCoef<N, V>::type;
    K E[C * C];  // S(i,k), k even mode, at [i*C+k]
    K O[H * H];  // S(i,C+k) at [i*H+k]
};

// host: tables from D and S, row-major
template <int N, class V>
inline EoD<N, V> eo_d_table(const double* D)
{
    EoD<N, V> t;
    constexpr int H = N / 2, C = (N + 1) / 2;
    for (int i = 0; i < H; ++i)
        for (int k = 0; k < C; ++k)
            eo_set(t.P[i * C + k], k == H ? D[i * N + k] : 0.5 * (D[i * N + k] + D[i * N + N - 1 - k]));
    for (int i = 0; i < C; ++i)
        for (int k = 0; k < H; ++k) eo_set(t.Q[i * H + k], 0.5 * (D[i * N + k] - D[i * N + N - 1 - k]));
    return t;
}
template <int N, class V>
inline EoS<N, V> eo_s_table(const double* S)
{
    EoS<N, V> t;
    constexpr int H = N / 2, C = (N + 1) / 2;
    for (int i = 0; i < C; ++i)
        for (int k = 0; k < C; ++k) eo_set(t.E[i * C + k], S[i * N + k]);
    for (int i = 0; i < H; ++i)
        for (int k = 0; k < H; ++k) eo_set(t.O[i * H + k], S[i * N + C + k]);
    return t;
}

// o = D u (TR false) or D^T u (TR true) of one line; o may be u
template <int N, bool TR, class V>
__device__ __forceinline__ void eo_d(const EoD<N, V>& t, const V* u, V* o)
{
    constexpr int H = N / 2, C = (N + 1) / 2;
    V s[C], d[H], a[H], b[C];
#pragma unroll
    for (int k = 0; k < H; ++k) {
        s[k] = lv_add(u[k], u[N - 1 - k]);
        d[k] = lv_sub(u[k], u[N - 1 - k]);
    }
    if (C > H) s[C - 1] = u[H];
#pragma unroll
    for (int k = 0; k < C; ++k)
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const typename EoCoef<N, V>::type c = TR ? t.Q[k * H + i] : t.P[i * C + k];
            a[i] = k == 0 ? lv_cmul(c, s[k]) : lv_cfma(c, s[k], a[i]);
        }
#pragma unroll
    for (int k = 0; k < H; ++k)
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const typename EoCoef<N, V>::type c = TR ? t.P[k * C + i] : t.Q[i * H + k];
            b[i] = k == 0 ? lv_cmul(c, d[k]) : lv_cfma(c, d[k], b[i]);
        }
#pragma unroll
    for (int i = 0; i < H; ++i) {
        o[i] = lv_add(b[i], a[i]);
        o[N - 1 - i] = lv_sub(b[i], a[i]);
    }
    if (C > H) o[H] = b[C - 1];
}

// t = S^T u (modes, even first); o may be u
template <int N, class V>
__device__ __forceinline__ void eo_st(const EoS<N, V>& t, const V* u, V* o)
{
    constexpr int H = N / 2, C = (N + 1) / 2;
    V s[C], d[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
        s[k] = lv_add(u[k], u[N - 1 - k]);
        d[k] = lv_sub(u[k], u[N - 1 - k]);
    }
    if (C > H) s[C - 1] = u[H];
#pragma unroll
    for (int i = 0; i < C; ++i)
#pragma unroll
        for (int k = 0; k < C; ++k) o[k] = i == 0 ? lv_cmul(t.E[k], s[0]) : lv_cfma(t.E[i * C + k], s[i], o[k]);
#pragma unroll
    for (int i = 0; i < H; ++i)
#pragma unroll
        for (int k = 0; k < H; ++k)
            o[C + k] = i == 0 ? lv_cmul(t.O[k], d[0]) : lv_cfma(t.O[i * H + k], d[i], o[C + k]);
}

// u = S t; o may be t
template <int N, class V>
__device__ __forceinline__ void eo_s(const EoS<N, V>& t, const V* m, V* o)
{
    constexpr int H = N / 2, C = (N + 1) / 2;
    V a[C], b[H];
#pragma unroll
    for (int k = 0; k < C; ++k)
#pragma unroll
        for (int i = 0; i < C; ++i)
            a[i] = k == 0 ? lv_cmul(t.E[i * C], m[0]) : lv_cfma(t.E[i * C + k], m[k], a[i]);
#pragma unroll
    for (int k = 0; k < H; ++k)
#pragma unroll
        for (int i = 0; i < H; ++i)
            b[i] = k == 0 ? lv_cmul(t.O[i * H], m[C]) : lv_cfma(t.O[i * H + k], m[C + k], b[i]);
#pragma unroll
    for (int i = 0; i < H; ++i) {
        o[i] = lv_add(a[i], b[i]);
        o[N - 1 - i] = lv_sub(a[i], b[i]);
    }
    if (C > H) o[H] = a[C - 1];
}

// ------------------------------------------------------------- line indexing
// Elements of a block's pass sit in shared memory ES words apart (odd, so that
// a warp whose lanes take the same line of consecutive elements touches all
// banks); line L of ne elements is (pos, le) with the element fastest.
__host__ __device__ constexpr int line_es(int N) { return (N * N) | 1; }
// ne and its FP32 reciprocal: (L + 0.5) * (1/ne) in FP32 is at least 0.5 / ne
// from an integer and within a few ulp of the exact quotient, so its
// truncation is L / ne (checked exhaustively for ne <= 1024, L < 34 ne)
struct LineNe {
    int n;
    float inv;
};
__device__ __forceinline__ LineNe line_ne(int ne) { return LineNe{ne, 1.f / (float)ne}; }
__device__ __forceinline__ void line_of(int L, LineNe ne, int& pos, int& le)
{
    pos = (int)(((float)L + 0.5f) * ne.inv);
    le = L - pos * ne.n;
}

}  // namespace semgb

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
__device__ __forceinline__ f2_t lv_mul(f2_t a, f2_t b) { return f2mul(a, b); }
__device__ __forceinline__ f2_t lv_fma(f2_t a, f2_t b, f2_t c) { return f2fma(a, b, c); }
__device__ __forceinline__ double lv_add(double a, double b) { return a + b; }
__device__ __forceinline__ double lv_sub(double a, double b) { return a - b; }
__device__ __forceinline__ double lv_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double lv_fma(double a, double b, double c) { return fma(a, b, c); }

template <int N, class V>
struct EoD {
    static constexpr int H = N / 2, C = (N + 1) / 2;
    V P[H * C];  // P(i,k) at [i*C+k]
    V Q[C * H];  // Q(i,k) at [i*H+k]
};
// preconditioner basis, even modes first (fdm_basis orders them so)
template <int N, class V>
struct EoS {
    static constexpr int H = N / 2, C = (N + 1) / 2;
    V E[C * C];  // S(i,k), k even mode, at [i*C+k]
    V O[H * H];  // S(i,C+k) at [i*H+k]
};

// host: a table entry of type V
template <class V>
inline V eo_entry(double v);
template <>
inline double eo_entry<double>(double v) { return v; }
template <>
inline f2_t eo_entry<f2_t>(double v)
{
    const float f = (float)v;
    uint32_t u;
    memcpy(&u, &f, sizeof(u));
    return ((f2_t)u << 32) | u;
}

// host: tables from D and S, row-major
template <int N, class V>
inline EoD<N, V> eo_d_table(const double* D)
{
    EoD<N, V> t;
    constexpr int H = N / 2, C = (N + 1) / 2;
    for (int i = 0; i < H; ++i)
        for (int k = 0; k < C; ++k)
            t.P[i * C + k] = eo_entry<V>(k == H ? D[i * N + k] : 0.5 * (D[i * N + k] + D[i * N + N - 1 - k]));
    for (int i = 0; i < C; ++i)
        for (int k = 0; k < H; ++k) t.Q[i * H + k] = eo_entry<V>(0.5 * (D[i * N + k] - D[i * N + N - 1 - k]));
    return t;
}
template <int N, class V>
inline EoS<N, V> eo_s_table(const double* S)
{
    EoS<N, V> t;
    constexpr int H = N / 2, C = (N + 1) / 2;
    for (int i = 0; i < C; ++i)
        for (int k = 0; k < C; ++k) t.E[i * C + k] = eo_entry<V>(S[i * N + k]);
    for (int i = 0; i < H; ++i)
        for (int k = 0; k < H; ++k) t.O[i * H + k] = eo_entry<V>(S[i * N + C + k]);
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
            const V c = TR ? t.Q[k * H + i] : t.P[i * C + k];
            a[i] = k == 0 ? lv_mul(c, s[k]) : lv_fma(c, s[k], a[i]);
        }
#pragma unroll
    for (int k = 0; k < H; ++k)
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const V c = TR ? t.P[k * C + i] : t.Q[i * H + k];
            b[i] = k == 0 ? lv_mul(c, d[k]) : lv_fma(c, d[k], b[i]);
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
        for (int k = 0; k < C; ++k) o[k] = i == 0 ? lv_mul(t.E[k], s[0]) : lv_fma(t.E[i * C + k], s[i], o[k]);
#pragma unroll
    for (int i = 0; i < H; ++i)
#pragma unroll
        for (int k = 0; k < H; ++k)
            o[C + k] = i == 0 ? lv_mul(t.O[k], d[0]) : lv_fma(t.O[i * H + k], d[i], o[C + k]);
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
            a[i] = k == 0 ? lv_mul(t.E[i * C], m[0]) : lv_fma(t.E[i * C + k], m[k], a[i]);
#pragma unroll
    for (int k = 0; k < H; ++k)
#pragma unroll
        for (int i = 0; i < H; ++i)
            b[i] = k == 0 ? lv_mul(t.O[i * H], m[C]) : lv_fma(t.O[i * H + k], m[C + k], b[i]);
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

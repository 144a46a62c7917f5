// Arithmetic and operand loads shared by the transform-sweep kernels (kernels_lagr.cu, kernels_plan.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace amdg {

// ---- double-float arithmetic (float2 = hi + lo, |lo| <= ulp(hi)/2, about 48 bits) -------------
// The error-free transformations two-sum (Knuth) and the FMA-based exact product, combined as in
// the double-double algorithms of Hida, Li and Bailey ("accurate" addition): the point-value
// sweeps of the mixed mode run on the FP32 pipe with near-FP64 accuracy.  Products whose rounding is taken
// apart are __fmul_rn: the compiler must not contract them into the additions that follow.
__device__ __forceinline__ float2 df_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return make_float2(s, (a - (s - bb)) + (b - bb));
}
__device__ __forceinline__ float2 df_quick_two_sum(float a, float b) {
    const float s = a + b;
    return make_float2(s, b - (s - a));
}
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
    float2 s = df_two_sum(a.x, b.x);
    const float2 t = df_two_sum(a.y, b.y);
    s.y += t.x;
    s = df_quick_two_sum(s.x, s.y);
    s.y += t.y;
    return df_quick_two_sum(s.x, s.y);
}
__device__ __forceinline__ float2 df_mul(float2 a, float2 b) {
    const float p = __fmul_rn(a.x, b.x);
    float e = fmaf(a.x, b.x, -p);
    e = fmaf(a.x, b.y, e);
    e = fmaf(a.y, b.x, e);
    return df_quick_two_sum(p, e);
}

// the sweep's arithmetic for T = double, float or float2 (double-float)
__device__ __forceinline__ double madd(double x, double m, double acc) { return fma(x, m, acc); }
__device__ __forceinline__ float madd(float x, float m, float acc) { return fmaf(x, m, acc); }
__device__ __forceinline__ float2 madd(float2 x, float2 m, float2 acc) { return df_add(df_mul(x, m), acc); }
__device__ __forceinline__ double scale(double a, double c) { return a * c; }
__device__ __forceinline__ float scale(float a, float c) { return a * c; }
__device__ __forceinline__ float2 scale(float2 a, float2 c) { return df_mul(a, c); }
template <typename T>
__device__ __forceinline__ T from_double(double v) { return T(v); }
template <>
__device__ __forceinline__ float2 from_double<float2>(double v) {
    const float hi = float(v);
    return make_float2(hi, float(v - double(hi)));
}
__device__ __forceinline__ double to_double(double v) { return v; }
__device__ __forceinline__ double to_double(float v) { return double(v); }
__device__ __forceinline__ double to_double(float2 v) { return double(v.x) + double(v.y); }

// entries between the blocks of a table: FP32 blocks are padded to whole 16-byte loads
template <typename T>
__host__ __device__ constexpr int table_stride(int n) {
    return sizeof(T) == 4 ? (n + 3) / 4 * 4 : n;
}

// acc + sum over four neighbours j (in order) and k < NF of x[j][k*stride] * m[j][k*ncols],
// all operands loaded before the first multiply-add.  (The inputs x by plain loads: a kernel launched
// ahead of its predecessor's end must not read what that one writes through the read-only path.)
template <int NF, typename T>
__device__ __forceinline__ T fibre_quad(const T* const* x, const T* const* m, int stride, int ncols, T acc) {
    T xv[4][NF], mv[4][NF];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            xv[j][k] = x[j][k * stride];
            mv[j][k] = __ldg(m[j] + size_t(k) * ncols);
        }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < NF; ++k) acc = madd(xv[j][k], mv[j][k], acc);
    return acc;
}

// the N entries of a table block: 16-byte loads where its stride in the table is a multiple of 16 bytes
template <typename T, int N>
__device__ __forceinline__ void load_block(const T* p, T (&v)[N]) {
    constexpr int S = table_stride<T>(N);
    if constexpr ((S * sizeof(T)) % 16 == 0) {
        constexpr int V = S * sizeof(T) / 16;
        const float4* p4 = reinterpret_cast<const float4*>(p);
        float4 w[V];
#pragma unroll
        for (int i = 0; i < V; ++i) w[i] = __ldg(p4 + i);
        const T* wt = reinterpret_cast<const T*>(w);
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = wt[i];
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = __ldg(p + i);
    }
}

__device__ __forceinline__ double shfl_from(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float shfl_from(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float2 shfl_from(float2 v, int src) {
    return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ double add_t(double a, double b) { return a + b; }
__device__ __forceinline__ float add_t(float a, float b) { return a + b; }
__device__ __forceinline__ float2 add_t(float2 a, float2 b) { return df_add(a, b); }

// one lane's share of a column: neighbours i = first, first + P, ... < end, two per pass
template <typename T, int NF, int NT>
__device__ __forceinline__ void warp_column(const int2* __restrict__ nbr, int first, int end, int P, const T* in,
                                            int64_t in_block, int in_off, int stride, const T* M, size_t mrow, int oe,
                                            T (&acc)[NT]) {
    constexpr int BS = NF * NT;
    int i = first;
    for (; i + P < end; i += 2 * P) {
        const int2 n0 = __ldg(nbr + i), n1 = __ldg(nbr + i + P);
        const T* x0 = in + int64_t(n0.x) * in_block + in_off;
        const T* x1 = in + int64_t(n1.x) * in_block + in_off;
        T xa[NF], xb[NF], ma[BS], mb[BS];
#pragma unroll
        for (int p = 0; p < NF; ++p) {
            xa[p] = __ldg(x0 + p * stride);
            xb[p] = __ldg(x1 + p * stride);
        }
        load_block<T, BS>(M + (size_t(n0.y) * mrow + oe) * table_stride<T>(BS), ma);
        load_block<T, BS>(M + (size_t(n1.y) * mrow + oe) * table_stride<T>(BS), mb);
#pragma unroll
        for (int p = 0; p < NF; ++p)
#pragma unroll
            for (int q = 0; q < NT; ++q) acc[q] = madd(xa[p], ma[p * NT + q], acc[q]);
#pragma unroll
        for (int p = 0; p < NF; ++p)
#pragma unroll
            for (int q = 0; q < NT; ++q) acc[q] = madd(xb[p], mb[p * NT + q], acc[q]);
    }
    if (i < end) {
        const int2 n0 = __ldg(nbr + i);
        const T* x0 = in + int64_t(n0.x) * in_block + in_off;
        T xa[NF], ma[BS];
#pragma unroll
        for (int p = 0; p < NF; ++p) xa[p] = __ldg(x0 + p * stride);
        load_block<T, BS>(M + (size_t(n0.y) * mrow + oe) * table_stride<T>(BS), ma);
#pragma unroll
        for (int p = 0; p < NF; ++p)
#pragma unroll
            for (int q = 0; q < NT; ++q) acc[q] = madd(xa[p], ma[p * NT + q], acc[q]);
    }
}

}  // namespace amdg

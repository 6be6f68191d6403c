// Device helpers of the flat-layer kernels (logic.cu, logic_bwd.cu).
#pragma once

#include "clb_common.cuh"

namespace clb {

// Each half-warp reduces the 16 values of one neuron (the two halves' neurons are unrelated): v is value (lane & 15) of the lane's.
// Returns that neuron's gate in every lane of the half-warp, plus the lane's mixture value p.
template <typename T> __device__ __forceinline__ Gate<T> half_warp_gate_of(T v, int wmode, int lane, T &p)
{
    const int i = lane & 15;
    if (wmode == CLB_W_SOFTMAX) {
        T m = v;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const T u = __shfl_xor_sync(0xffffffffu, m, o);
            m = u > m ? u : m;
        }
        v = exp(v - m);
        T s = v;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        v = v / s;
    } else if (wmode == CLB_W_ARGMAX) {
        // first maximum: compare (value, -index) pairs
        T m = v;
        int bi = i;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const T um = __shfl_xor_sync(0xffffffffu, m, o);
            const int ui = __shfl_xor_sync(0xffffffffu, bi, o);
            if (um > m || (um == m && ui < bi)) {
                m = um;
                bi = ui;
            }
        }
        v = (i == bi) ? T(1) : T(0);
    }
    p = v;
    Gate<T> g;
    g.kab = T(kcoef(0, i)) * v;
    g.ka = T(kcoef(1, i)) * v;
    g.kb = T(kcoef(2, i)) * v;
    g.k1 = T(kcoef(3, i)) * v;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        g.kab += __shfl_xor_sync(0xffffffffu, g.kab, o);
        g.ka += __shfl_xor_sync(0xffffffffu, g.ka, o);
        g.kb += __shfl_xor_sync(0xffffffffu, g.kb, o);
        g.k1 += __shfl_xor_sync(0xffffffffu, g.k1, o);
    }
    return g;
}

template <typename T, int V> struct Vec;
template <> struct Vec<float, 4> { using type = float4; };
template <> struct Vec<float, 2> { using type = float2; };
template <> struct Vec<float, 1> { using type = float; };
template <> struct Vec<double, 1> { using type = double; };

template <typename T, int V> __device__ __forceinline__ void vload(const T *p, T (&r)[V])
{
    using VT = typename Vec<T, V>::type;
    const VT v = __ldg(reinterpret_cast<const VT *>(p));
    const T *e = reinterpret_cast<const T *>(&v);
#pragma unroll
    for (int k = 0; k < V; ++k) r[k] = e[k];
}
template <typename T, int V> __device__ __forceinline__ void vstore(T *p, const T (&r)[V])
{
    using VT = typename Vec<T, V>::type;
    VT v;
    T *e = reinterpret_cast<T *>(&v);
#pragma unroll
    for (int k = 0; k < V; ++k) e[k] = r[k];
    *reinterpret_cast<VT *>(p) = v;
}

// the same for what does not fit the L2 until it is read again
template <typename T, int V> __device__ __forceinline__ void vstore_once(T *p, const T (&r)[V])
{
    using VT = typename Vec<T, V>::type;
    VT v;
    T *e = reinterpret_cast<T *>(&v);
#pragma unroll
    for (int k = 0; k < V; ++k) e[k] = r[k];
    __stcs(reinterpret_cast<VT *>(p), v);
}

template <typename T, int V> __device__ __forceinline__ void vload_once(const T *p, T (&r)[V])
{
    using VT = typename Vec<T, V>::type;
    const VT v = __ldcs(reinterpret_cast<const VT *>(p));
    const T *e = reinterpret_cast<const T *>(&v);
#pragma unroll
    for (int k = 0; k < V; ++k) r[k] = e[k];
}

// a gate's 16 values as four vectors
__device__ __forceinline__ void load16(const float *__restrict__ w, float (&v)[16])
{
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(w) + q);
        v[4 * q] = t.x, v[4 * q + 1] = t.y, v[4 * q + 2] = t.z, v[4 * q + 3] = t.w;
    }
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float sum2(f32x2 v)
{
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a + b;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// R vectors of V floats at stride LPR * V, as R * V / 2 packed pairs; zeros beyond the row
template <int LPR, int V, int R> struct Row {
    static constexpr int P = R * V / 2;
    f32x2 p[P];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int i = 0; i < P; ++i) p[i] = 0ull;
    }
    __device__ __forceinline__ void load(const float *__restrict__ row, int left) // row: the lane's first element, left: how many follow
    {
        if constexpr (V == 4) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                ulonglong2 q = make_ulonglong2(0ull, 0ull);
                if (r * LPR * 4 < left) q = __ldg(reinterpret_cast<const ulonglong2 *>(row + r * LPR * 4));
                p[2 * r] = q.x, p[2 * r + 1] = q.y;
            }
        } else if constexpr (V == 2) {
#pragma unroll
            for (int r = 0; r < R; ++r) p[r] = r * LPR * 2 < left ? __ldg(reinterpret_cast<const f32x2 *>(row + r * LPR * 2)) : 0ull;
        } else {
            float t[R];
#pragma unroll
            for (int r = 0; r < R; ++r) t[r] = r * LPR < left ? __ldg(row + r * LPR) : 0.f;
#pragma unroll
            for (int r = 0; r < P; ++r) p[r] = pack2(t[2 * r], t[2 * r + 1]);
        }
    }
    __device__ __forceinline__ void store(float *__restrict__ row, int left) const
    {
        if constexpr (V == 4) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r * LPR * 4 < left) __stcs(reinterpret_cast<float4 *>(row + r * LPR * 4), *reinterpret_cast<const float4 *>(&p[2 * r]));
        } else if constexpr (V == 2) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r * LPR * 2 < left) __stcs(reinterpret_cast<float2 *>(row + r * LPR * 2), *reinterpret_cast<const float2 *>(&p[r]));
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r * LPR < left) row[r * LPR] = __uint_as_float((unsigned)(r & 1 ? p[r / 2] >> 32 : p[r / 2]));
        }
    }
};

} // namespace clb

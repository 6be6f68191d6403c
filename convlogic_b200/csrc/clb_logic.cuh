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

} // namespace clb

// Compiled network, small calls: the whole stack in ONE launch.
//
// A small network on a small batch is bound by launches: run layer by layer, a mnist-sized stack at batch 1 to 256 was 12 to
// 15 launches of 2 to 5 us (72-76 us per call, of which no kernel was busy for more than a few).  But a slab of samples of
// packed activations goes through the network on its own -- no layer mixes samples -- so a slab can be given to one
// thread-block cluster, which packs its input, runs layer after layer with a cluster barrier in between (about 0.5 us instead
// of a launch) and counts the class sums.  Activations stay in global memory in units of 4, 8 or 16 bytes (32, 64 or 128 samples of
// one feature): a few hundred KB, L2 and L1 resident.  Every storage is written once and read after a barrier, each slab has its
// own, and conv inputs are stored with their padding as a halo of zeros, so that a tap is one unconditional load.
//
// The size of a unit: what a thread waits for is the eight taps of a window on their way from the L2 and the barrier behind a layer, so that
// small units pay twice, in bytes per tap and in slabs, hence SMs, per call (clb_net_cluster_launch; us with units of 4 / 8 / 16
// bytes: mnist k = 16 batch 1 10.4 / 11.6 / 13.7, batch 256 13.5 / 12.9 / 15.2; cifar k = 32 batch 1000 40.0 / 39.1 / 42.2).
//
// Work split: a thread owns one unit of one feature.  Warps are dealt to the blocks of the cluster round robin (32
// consecutive features per warp), so that a layer with few features still uses every SM of the cluster.  Gates are the
// three-lop3 multiplexer, since the features of a warp belong to several channels.
#include "clb_common.cuh"
#include "clb_net.cuh"

#include <atomic>

namespace clb {

namespace {

constexpr int kNetThreads = 512;

// 32 * N samples of one feature
template <int N> struct __align__(4 * N) Unit {
    unsigned w[N];
    static __device__ __forceinline__ Unit zero()
    {
        Unit u;
#pragma unroll
        for (int i = 0; i < N; ++i) u.w[i] = 0u;
        return u;
    }
    __device__ __forceinline__ void operator|=(const Unit &o)
    {
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] |= o.w[i];
    }
};

// not the read-only path: the units were written earlier in this kernel by other blocks
__device__ __forceinline__ Unit<4> ld_unit(const Unit<4> *p)
{
    Unit<4> v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ Unit<2> ld_unit(const Unit<2> *p)
{
    Unit<2> v;
    asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.w[0]), "=r"(v.w[1]) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ Unit<1> ld_unit(const Unit<1> *p)
{
    Unit<1> v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v.w[0]) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// gate `op` (truth-table bits 3..0 = f(0,0), f(0,1), f(1,0), f(1,1)) on a unit
template <int N> __device__ __forceinline__ Unit<N> gate(int op, const Unit<N> &a, const Unit<N> &b)
{
    const unsigned m11 = (op & 1) ? ~0u : 0u, m10 = (op & 2) ? ~0u : 0u, m01 = (op & 4) ? ~0u : 0u, m00 = (op & 8) ? ~0u : 0u;
    Unit<N> r;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const unsigned x = a.w[i], y = b.w[i], r1 = (y & m11) | (~y & m10), r0 = (y & m01) | (~y & m00);
        r.w[i] = (x & r1) | (~x & r0);
    }
    return r;
}

// lane s gets, in bit t, bit s of lane t's word
__device__ __forceinline__ unsigned transpose32(unsigned x, int lane)
{
    unsigned m = 0x0000ffffu;
#pragma unroll
    for (int j = 16; j >= 1; j >>= 1) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
        m ^= m << (j >> 1);
    }
    return x;
}

// bit 0 of byte k of the result: byte k of v is not zero
__device__ __forceinline__ unsigned nonzero_bytes(unsigned v) { return ((((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) >> 7) & 0x01010101u; }

// One pooled window of a conv block: its channel's gates and the units its taps read at the window's first position.
struct ConvWindow {
    int c, py, px;
    int op[7], tap[8];
    __device__ __forceinline__ void load(const NetLayer &L, const unsigned char *__restrict__ params, const NetStorage &in, int o)
    {
        c = L.by_windows.div(o);
        const int win = o - c * (int)L.by_windows.d;
        py = L.by_Wp.div(win), px = win - py * L.Wp;
        const int4 *sel = reinterpret_cast<const int4 *>(params + L.off_a) + 2 * c;
        const int4 wa = __ldg(sel), wb = __ldg(sel + 1);
#pragma unroll
        for (int g = 0; g < 7; ++g) op[g] = __ldg(params + L.off_ops + c * 7 + g);
        const int word[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
        const int first = 2 * py * L.stride * in.pitch + 2 * px * L.stride;
#pragma unroll
        for (int k = 0; k < 8; ++k) tap[k] = first + ((word[k] >> 16) & 0xFFFF) * in.per_channel + ((word[k] >> 8) & 0xFF) * in.pitch + (word[k] & 0xFF);
    }
    template <int N> __device__ __forceinline__ Unit<N> position(const Unit<N> *x) const
    {
        Unit<N> a[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = ld_unit(x + tap[k]);
        const Unit<N> g0 = gate(op[0], a[0], a[1]), g1 = gate(op[1], a[2], a[3]);
        const Unit<N> g2 = gate(op[2], a[4], a[5]), g3 = gate(op[3], a[6], a[7]);
        return gate(op[6], gate(op[4], g0, g1), gate(op[5], g2, g3));
    }
};

} // namespace

template <int N>
__global__ void __launch_bounds__(kNetThreads, 1) net_cluster_kernel(const __grid_constant__ NetPlan net, const void *__restrict__ input,
                                                                     const float *__restrict__ thresholds, const unsigned char *__restrict__ params,
                                                                     Unit<N> *work, int *counts, long long batch)
{
    using U = Unit<N>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned rank, csize;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    const int slab = blockIdx.x / csize;
    const int gwarp = warp * (int)csize + (int)rank, nwarps = (kNetThreads / 32) * (int)csize;
    U *const base = work + (size_t)slab * net.slab_units;
    __shared__ int cutoff[kNetMaxLevels]; // byte pixels: the first value above the threshold, by the comparison u / 255 > t itself
    if (net.input_kind == 2) {
        for (int i = threadIdx.x; i < net.levels; i += kNetThreads) {
            const float t = __ldg(thresholds + i);
            int lo = 0, hi = 256; // first u in [0, 256] with u / 255 > t (u / 255 does not fall with u)
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__fdiv_rn((float)mid, 255.0f) > t)
                    hi = mid;
                else
                    lo = mid + 1;
            }
            cutoff[i] = lo;
        }
        __syncthreads();
    }
    const long long s0 = (long long)slab * (32 * N);
    const int live = (int)min(32LL * N, batch - s0); // samples of this slab

    // ---- input: one 32-sample word of every feature per (feature group, word) task; class sums cleared
    for (int i = gwarp * 32 + lane; i < live * net.classes; i += nwarps * 32) counts[s0 * net.classes + i] = 0;
    {
        const NetStorage st = net.store[0];
        unsigned *words = reinterpret_cast<unsigned *>(base + st.base);
        for (int i = gwarp * 32 + lane; i < st.halo_units; i += nwarps * 32) // zeros of the halo (the interior follows)
            if (st.halo(i)) base[st.base + i] = U::zero();
        if (net.input_kind == 0) { // bytes [batch][features]
            const unsigned char *x = static_cast<const unsigned char *>(input);
            const long long F = net.in_features;
            const bool quad = (F & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 3) == 0; // four features per lane and load
            const int per = quad ? 128 : 32, groups = (int)((F + per - 1) / per);
            for (int task = gwarp; task < groups * N; task += nwarps) {
                const int w = task % N;
                const long long f = (long long)(task / N) * per + (quad ? 4 * lane : lane);
                const int n0 = w * 32, n = min(32, live - n0);
                if (f >= F) continue;
                const unsigned char *src = x + (s0 + n0) * F + f;
                if (quad) {
                    unsigned g[4] = {0u, 0u, 0u, 0u}; // byte k of g[q]: samples 8q..8q+7 of feature f + k
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        unsigned v[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = 8 * q + j < n ? __ldg(reinterpret_cast<const unsigned *>(src + (8 * q + j) * F)) : 0u;
#pragma unroll
                        for (int j = 0; j < 8; ++j) g[q] |= nonzero_bytes(v[j]) << j;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const unsigned lo = __byte_perm(g[0], g[1], 0x40 + 0x11 * k), hi = __byte_perm(g[2], g[3], 0x40 + 0x11 * k);
                        words[N * st.unit((int)f + k) + w] = (lo & 0xffffu) | (hi << 16);
                    }
                } else {
                    unsigned v = 0u;
                    for (int j = 0; j < n; ++j) v |= (__ldg(src + j * F) != 0 ? 1u : 0u) << j;
                    words[N * st.unit((int)f) + w] = v;
                }
            }
        } else { // pixels [batch][P], features threshold-major: feature i * P + p is pixel p > threshold i
            const int P = (int)(net.in_features / net.levels);
            const int level_step = st.halo_units ? P / st.image * st.per_channel : P; // units from a feature to its next threshold's
            const int groups = (P + 31) / 32;
            for (int task = gwarp; task < groups * N; task += nwarps) {
                const int w = task % N, p = task / N * 32 + lane;
                const int n0 = w * 32, n = min(32, live - n0);
                if (p >= P) continue;
                const unsigned mask = n >= 32 ? ~0u : n > 0 ? (1u << n) - 1u : 0u; // a negative threshold must not set pad bits
                if (net.input_kind == 1) {
                    const float *src = static_cast<const float *>(input) + (s0 + n0) * P + p;
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = j < n ? __ldg(src + (long long)j * P) : 0.f;
                    unsigned *dst = words + N * st.unit(p) + w;
                    for (int i = 0; i < net.levels; ++i, dst += N * level_step) {
                        const float t = __ldg(thresholds + i);
                        unsigned m = 0u;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (v[j] > t) m |= 1u << j;
                        *dst = m & mask;
                    }
                } else {
                    const unsigned char *src = static_cast<const unsigned char *>(input) + (s0 + n0) * P + p;
                    int v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = j < n ? (int)__ldg(src + (long long)j * P) : 0;
                    unsigned *dst = words + N * st.unit(p) + w;
                    for (int i = 0; i < net.levels; ++i, dst += N * level_step) {
                        const int t = cutoff[i];
                        unsigned m = 0u;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (v[j] >= t) m |= 1u << j;
                        *dst = m & mask;
                    }
                }
            }
        }
    }

    // ---- layers
    for (int li = 0; li < net.n_layers; ++li) {
        const NetLayer &L = net.layer[li];
        const NetStorage in = net.store[li], out = net.store[li + 1];
        const bool conv = L.kind == 1;
        // A window's four positions go to four lanes while that takes at most two rounds of the cluster's threads: small layers are
        // bound by the latency of a thread's loads (4000 -> 2200 cycles for one of a mnist-sized stack); otherwise one thread takes all four.
        const int windows = conv ? L.C * L.Hp * L.Wp : 0;
        const bool split = 2 * windows <= nwarps * 32;
        const int items = split ? 4 * windows : windows;
        int item = gwarp * 32 + lane;
        ConvWindow cw;
        cluster_arrive();
        // between arrive and wait: what does not depend on the other blocks' results
        if (conv) {
            for (int i = gwarp * 32 + lane; i < out.halo_units; i += nwarps * 32) // the next layer's padding
                if (out.halo(i)) base[out.base + i] = U::zero();
            if (item < items) cw.load(L, params, in, split ? item >> 2 : item);
        }
        cluster_wait();
        if (conv) {
            const U *x = base + in.base;
            U *y = base + out.base;
            while (item < items) {
                U acc;
                if (split) {
                    const int d = item & 3;
                    acc = cw.position(x + (d >> 1) * L.stride * in.pitch + (d & 1) * L.stride);
                    // the four lanes of a window are all in range or all out
                    const unsigned quad = 0xfu << (lane & 28);
#pragma unroll
                    for (int o = 1; o <= 2; o <<= 1) {
#pragma unroll
                        for (int i = 0; i < N; ++i) acc.w[i] |= __shfl_xor_sync(quad, acc.w[i], o);
                    }
                } else {
                    acc = U::zero();
#pragma unroll
                    for (int d = 0; d < 4; ++d) acc |= cw.position(x + (d >> 1) * L.stride * in.pitch + (d & 1) * L.stride);
                }
                if (!split || (item & 3) == 0) y[cw.c * out.per_channel + (cw.py + out.ph) * out.pitch + cw.px + out.pw] = acc;
                item += nwarps * 32;
                if (item < items) cw.load(L, params, in, split ? item >> 2 : item);
            }
            continue;
        }
        // flat layer (kind 2: one gate on two rows; kind 3: a gate tree on 4 or 8 rows)
        const bool last = li + 1 == net.n_layers;
        const int S = last ? L.out_dim / net.classes : L.out_dim;  // features per class
        const int chunks = (S + 31) / 32, total = chunks * (last ? net.classes : 1);
        const U *x = base + in.base;
        // (flat) a warp takes consecutive chunks of 32 features, so that its class changes rarely
        const int lo = (int)((long long)total * gwarp / nwarps), hi = (int)((long long)total * (gwarp + 1) / nwarps);
        int cls = -1, sum[N];
#pragma unroll
        for (int w = 0; w < N; ++w) sum[w] = 0;
        auto flush = [&]() {
            if (cls < 0) return;
#pragma unroll
            for (int w = 0; w < N; ++w)
                if (w * 32 + lane < live && sum[w]) atomicAdd(counts + (s0 + w * 32 + lane) * net.classes + cls, sum[w]);
#pragma unroll
            for (int w = 0; w < N; ++w) sum[w] = 0;
        };
        for (int ch = lo; ch < hi; ++ch) {
            const int c = ch / chunks, i = (ch - c * chunks) * 32 + lane; // feature i of class c
            const int t = c * S + i;
            U r = U::zero();
            if (i < S) {
                if (L.kind == 2) {
                    const long long a = __ldg(reinterpret_cast<const long long *>(params + L.off_a) + t), b = __ldg(reinterpret_cast<const long long *>(params + L.off_b) + t);
                    r = gate(__ldg(params + L.off_ops + t), ld_unit(x + a), ld_unit(x + b));
                } else if (L.levels == 3) {
                    const int4 *leaf = reinterpret_cast<const int4 *>(params + L.off_a) + 2 * t;
                    const int4 la = __ldg(leaf), lb = __ldg(leaf + 1);
                    int op[7];
#pragma unroll
                    for (int g = 0; g < 7; ++g) op[g] = __ldg(params + L.off_ops + (long long)t * 7 + g);
                    const U v0 = ld_unit(x + la.x), v1 = ld_unit(x + la.y), v2 = ld_unit(x + la.z), v3 = ld_unit(x + la.w);
                    const U v4 = ld_unit(x + lb.x), v5 = ld_unit(x + lb.y), v6 = ld_unit(x + lb.z), v7 = ld_unit(x + lb.w);
                    r = gate(op[6], gate(op[4], gate(op[0], v0, v1), gate(op[1], v2, v3)),
                                gate(op[5], gate(op[2], v4, v5), gate(op[3], v6, v7)));
                } else {
                    const int4 la = __ldg(reinterpret_cast<const int4 *>(params + L.off_a) + t);
                    int op[3];
#pragma unroll
                    for (int g = 0; g < 3; ++g) op[g] = __ldg(params + L.off_ops + (long long)t * 3 + g);
                    const U v0 = ld_unit(x + la.x), v1 = ld_unit(x + la.y), v2 = ld_unit(x + la.z), v3 = ld_unit(x + la.w);
                    r = gate(op[2], gate(op[0], v0, v1), gate(op[1], v2, v3));
                }
                if (!last) base[out.base + t] = r;
            }
            if (last) {
                if (c != cls) flush();
                cls = c;
#pragma unroll
                for (int w = 0; w < N; ++w) sum[w] += __popc(transpose32(r.w[w], lane));
            }
        }
        if (last) flush();
    }
}

} // namespace clb

using namespace clb;
using namespace clb_host;

// Blocks per cluster: the largest cluster with which all slabs are resident at once, so that a call is
// one wave (a second wave doubled a call: 16.7 -> 31 us at 8 slabs of a mnist-sized stack on clusters of 16, of which this
// GPU holds 7).  One block per SM: with two smaller ones some clusters share SMs and the slowest sets the time (47 -> 60 us at 8
// slabs of a cifar-sized stack).
static constexpr int kSizes[] = {16, 9, 6, 5, 4, 3, 2, 1};
static constexpr int kNSizes = sizeof(kSizes) / sizeof(kSizes[0]);

// The largest cluster of N-word units with which so many slabs are resident at once; 0: with none.
template <int N> static int cluster_size(int slabs)
{
    static std::atomic<int> resident[64][kNSizes]; // clusters resident at once + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    for (int i = 0; i < kNSizes; ++i) {
        int have = resident[dev][i].load(std::memory_order_relaxed);
        if (!have) {
            if (i == 0 && cudaFuncSetAttribute(net_cluster_kernel<N>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return 0;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)kSizes[i]), cfg.blockDim = dim3(kNetThreads);
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)kSizes[i], attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr, cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, net_cluster_kernel<N>, &cfg) != cudaSuccess) cudaGetLastError(), n = 0;
            have = n + 1;
            resident[dev][i].store(have, std::memory_order_relaxed);
        }
        if (slabs <= have - 1) return kSizes[i];
    }
    return 0;
}

template <int N>
static int launch(const NetPlan &net, int slabs, int csize, const void *input, const float *thresholds, const unsigned char *params, void *work, int32_t *counts,
                  int64_t batch, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(slabs * csize)), cfg.blockDim = dim3(kNetThreads), cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)csize, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    CLB_TRACED("net_cluster_kernel", st,
               cudaLaunchKernelEx(&cfg, net_cluster_kernel<N>, net, input, thresholds, params, static_cast<Unit<N> *>(work), counts, (long long)batch));
    return check_launch();
}

int clb_net_cluster_launch(const NetPlan &net, const void *input, const float *thresholds, const unsigned char *params, void *work, int32_t *counts,
                           int64_t batch, cudaStream_t st)
{
    const int s1 = (int)((batch + 31) / 32), s2 = (int)((batch + 63) / 64), s4 = (int)((batch + 127) / 128);
    // a thread's time goes as 1.5 + the words of a unit, and with the features that the blocks of a cluster share
    const int c1 = cluster_size<1>(s1), c2 = cluster_size<2>(s2), c4 = cluster_size<4>(s4);
    const double t1 = c1 ? 2.5 / c1 : 1e9, t2 = c2 ? 3.5 / c2 : 1e9, t4 = 5.5 / (c4 ? c4 : 1);
    if (t1 < t2 && t1 < t4) return launch<1>(net, s1, c1, input, thresholds, params, work, counts, batch, st);
    if (t2 < t4) return launch<2>(net, s2, c2, input, thresholds, params, work, counts, batch, st);
    return launch<4>(net, s4, c4 ? c4 : 1, input, thresholds, params, work, counts, batch, st); // (the last shape: in several waves)
}

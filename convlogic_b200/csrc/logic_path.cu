// Flat LogicLayer on paths (fp32, feature-major activations).
//
// A layer is a graph: features are vertices, neurons are edges between their two inputs.  Walked as trails -- the next neuron reads
// what the last one read second -- a forward pass loads ONE row per neuron instead of two, and where a feature has exactly two
// readers (every feature of a layer whose connections are randperm(2 * out) % in with out = in) a backward pass loads one row of x
// and one of gy per neuron and has the feature's input gradient complete in registers when it leaves it: every row of x, gy and
// gx crosses the memory system once, in order of use, whatever the caches hold.
//
// Plan (once per layer).  Each list of readers is paired up two by two (`link`: half-edge 2 * j + side -> the half-edge it is paired
// with), some pairs are left apart so that trails stay short enough to be walked by one thread (every kCut-th by a hash: a thread per
// trail end, a few hundred dependent loads), and trails are laid one behind the other in `rec`.  Neurons on closed trails without a
// cut (a few dozen) stand alone.  The order of trails in `rec` may differ between runs; no sum depends on it.
// A feature whose gradient the walk completes is `closed`; the others (cuts, features with other than two readers) are
// in the `open` list, and their gradient is taken from the consumer lists (logic_bwd.cu).
//
// What bounds both passes is DRAM: 256000 -> 256000, 1024 samples, kernels alone (a profiler's times): forward 2.1 GB in 344 us and 9.5 for the records and
// coefficients (436 and 6 as a walk of the neurons in their own order, stretch by stretch), backward 3.3 GB with the sums in 494 + 16 us (951 + 20 for
// the walk of the features), open features 13.
// Eight lanes own a range of positions and a stretch of 64 samples, the stretches of a row lying side by side in a block. Two
// neurons' rows in flight per group and four (forward) or two (backward: 100 registers) blocks per SM; of a backward that took 564 us,
// its sums not merged yet, three blocks spill (624), four neurons at two blocks wait longer for the first (650), stretches of 32 samples read pieces too
// small for a DRAM page (654); the forward with one neuron and six blocks 378, eight neurons and two blocks 620.
#include "clb_common.cuh"
#include "clb_logic.cuh"

#include <initializer_list>

namespace clb {

constexpr unsigned kCut = 128; // pairs left apart: one in kCut
constexpr int kLongest = 64 * kCut; // no trail is longer ((1 - 1 / kCut)^kLongest = 1e-28), unless lists contradict the connections
constexpr int kFwdBlocks = 4, kBwdBlocks = 2; // resident per SM
enum { kLinked = 1, kCloses = 2 };

__device__ __forceinline__ bool cut_here(unsigned e)
{
    e *= 0x9E3779B1u, e ^= e >> 15, e *= 0x85EBCA77u, e ^= e >> 13;
    return e % kCut == 0;
}

// (lists of any values: what lies outside the tables is not followed, and what is listed twice gives a count that tells)
__global__ void __launch_bounds__(256) path_link_kernel(const int32_t *__restrict__ start, const int2 *__restrict__ entry, int32_t *__restrict__ link, int in_dim,
                                                        int out_dim)
{
    const int f = blockIdx.x * 256 + threadIdx.x;
    if (f >= in_dim) return;
    const int hi = min(start[f + 1], 2 * out_dim);
    for (int e = max(start[f], 0); e + 1 < hi; e += 2) { // (the last of an odd number stays apart)
        const int h0 = entry[e].x, h1 = entry[e + 1].x;
        if ((unsigned)h0 >= 2u * (unsigned)out_dim || (unsigned)h1 >= 2u * (unsigned)out_dim) continue;
        if ((h0 >> 1) != (h1 >> 1) && !cut_here((unsigned)e)) link[h0] = h1, link[h1] = h0; // a neuron fed twice by f is no link
    }
}

// A thread per half-edge that is the end of a trail; of a trail's two ends the one with the smaller number lays it out.
__global__ void __launch_bounds__(128) path_walk_kernel(const int32_t *__restrict__ link, int32_t *__restrict__ order, uint8_t *__restrict__ placed,
                                                        unsigned long long *__restrict__ laid, int out_dim)
{
    const int h = blockIdx.x * 128 + threadIdx.x;
    if (h >= 2 * out_dim || link[h] >= 0) return;
    int n = 1, cur = h;
    for (int next; n <= kLongest && (next = __ldg(link + (cur ^ 1))) >= 0; ++n) cur = next;
    if (n <= kLongest && h > (cur ^ 1)) return;
    const unsigned long long p = atomicAdd(laid, n <= kLongest ? (unsigned long long)n : out_dim + 1ull);
    if (p + n > (unsigned long long)out_dim) return; // a neuron is listed twice, or there is no end: the count tells
    cur = h;
    for (int i = 0; i < n; ++i) {
        order[p + i] = cur, placed[cur >> 1] = i > 0 ? 2 : 1;
        cur = __ldg(link + (cur ^ 1));
    }
}

// neurons that no trail end reaches stand alone
__global__ void __launch_bounds__(256) path_rest_kernel(int32_t *__restrict__ order, uint8_t *__restrict__ placed, unsigned long long *__restrict__ laid, int out_dim)
{
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= out_dim || placed[j]) return;
    const unsigned long long p = atomicAdd(laid, 1ull);
    if (p < (unsigned long long)out_dim) order[p] = 2 * j;
    placed[j] = 1;
}

// rec[p] = {2 * j + (1: entered through the second input), feature entered from, feature left through, flags}
__global__ void __launch_bounds__(256) path_record_kernel(const int64_t *__restrict__ ia, const int64_t *__restrict__ ib, const int32_t *__restrict__ start,
                                                          const int32_t *__restrict__ order, const uint8_t *__restrict__ placed, int4 *__restrict__ rec,
                                                          uint8_t *__restrict__ closed, int out_dim)
{
    const int p = blockIdx.x * 256 + threadIdx.x;
    if (p >= out_dim) return;
    const int code = max(order[p], 0), j = code >> 1;
    const int a = (int)ia[j], b = (int)ib[j], u = code & 1 ? b : a, v = code & 1 ? a : b;
    bool linked = placed[j] == 2 && p > 0;
    if (linked) { // entered through the feature that the neuron before is left through
        const int before = max(order[p - 1], 0);
        linked = (int)(before & 1 ? ia[before >> 1] : ib[before >> 1]) == u;
    }
    const bool closes = linked && start[u + 1] - start[u] == 2;
    if (closes) closed[u] = 1;
    rec[p] = make_int4(code, u, v, (linked ? kLinked : 0) | (closes ? kCloses : 0));
}

__global__ void __launch_bounds__(256) path_open_kernel(const uint8_t *__restrict__ closed, int32_t *__restrict__ open, int32_t *__restrict__ count,
                                                       const unsigned long long *__restrict__ laid, int in_dim)
{
    const int f = blockIdx.x * 256 + threadIdx.x;
    if (f == 0) count[0] = (int)min(*laid, 0x7fffffffull);
    if (f < in_dim && !closed[f]) open[atomicAdd(count + 1, 1)] = f;
}

// What a forward pass walks: the plan's order of the neurons, with the connections as they are now (they may have been written since the
// plan was laid out, in a way that nothing tells), and the coefficients of the gates.  A thread per position and neuron, in the launch that
// the coefficients take anyway.
__global__ void __launch_bounds__(256) logic_path_live_kernel(const int64_t *__restrict__ ia, const int64_t *__restrict__ ib, const int4 *__restrict__ rec,
                                                              int4 *__restrict__ live, const float *__restrict__ w, float4 *__restrict__ coef, int out_dim, int wmode)
{
    const int p = blockIdx.x * 256 + threadIdx.x;
    if (p >= out_dim) return;
    const int code = __ldg(&rec[p].x), j = code >> 1, prev = p > 0 ? __ldg(&rec[p - 1].x) : -1;
    const int a = (int)__ldg(ia + j), b = (int)__ldg(ib + j), u = code & 1 ? b : a;
    const int before = prev < 0 ? -1 : (int)__ldg((prev & 1 ? ia : ib) + (prev >> 1));
    live[p] = make_int4(code, u, code & 1 ? a : b, before == u ? kLinked : 0);
    float v[16], mix[16];
    load16(w + (size_t)p * 16, v);
    gate_mixture<float>(v, wmode, mix);
    const Gate<float> g = gate_from_mixture<float>(mix);
    coef[p] = make_float4(g.k1, g.ka, g.kb, g.kab);
}

// Eight lanes own a range of positions and 8 * V * R samples; the ranges of neighbouring groups are the same one, a stretch of samples
// further on, so that a block reads whole rows.  Every group makes the same number of turns: warps stay whole.
struct PathUnit {
    int l, col, p0, p1, turns;
    __device__ __forceinline__ PathUnit(int n, int cols, int ranges)
    {
        const int unit = (int)((blockIdx.x * 256u + threadIdx.x) >> 3), r = unit / cols;
        l = threadIdx.x & 7, col = unit - r * cols;
        turns = (n + ranges - 1) / ranges;
        p0 = r * turns, p1 = min(n, p0 + turns);
        if (p0 > p1) p0 = p1;
    }
};

template <int V, int R, int U>
__global__ void __launch_bounds__(256, kFwdBlocks) logic_path_fwd_kernel(const float *__restrict__ x, const int4 *__restrict__ rec, const float4 *__restrict__ coef,
                                                             float *__restrict__ y, int n, int B, int cols, int ranges)
{
    using RowT = Row<8, V, R>;
    const PathUnit t(n, cols, ranges);
    const int s0 = t.col * 8 * V * R + t.l * V, left = B - s0;
    if (t.p0 >= t.p1 || left <= 0) return;
    x += s0, y += s0;
    const int4 none = make_int4(-1, 0, 0, kLinked);
    int4 r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) r[u] = t.p0 + u < t.p1 ? __ldg(rec + t.p0 + u) : none;
    RowT a;
    a.load(x + (size_t)r[0].y * B, left); // the row of the neuron before, where the first is linked to it
    r[0].w |= kLinked;
    for (int p = t.p0; p < t.p1; p += U) {
        RowT b[U];
        float4 c[U];
        int4 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (r[u].x >= 0) {
                c[u] = __ldg(coef + (r[u].x >> 1));
                b[u].load(x + (size_t)r[u].z * B, left);
            }
#pragma unroll
        for (int u = 0; u < U; ++u) q[u] = r[u], r[u] = p + U + u < t.p1 ? __ldg(rec + p + U + u) : none;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (q[u].x >= 0) {
                if (!(q[u].w & kLinked)) a.load(x + (size_t)q[u].y * B, left);
                const bool second = q[u].x & 1;
                const float ka = second ? c[u].z : c[u].y, kb = second ? c[u].y : c[u].z;
                const f32x2 k1 = pack2(c[u].x, c[u].x), ka2 = pack2(ka, ka), kb2 = pack2(kb, kb), kab = pack2(c[u].w, c[u].w);
                RowT o;
#pragma unroll
                for (int i = 0; i < RowT::P; ++i) o.p[i] = fma2(a.p[i], fma2(kab, b[u].p[i], ka2), fma2(kb2, b[u].p[i], k1));
                o.store(y + (size_t)(q[u].x >> 1) * B, left);
                a = b[u];
            }
    }
}

// Input gradient of the closed features and the four basis sums of every neuron, partial [stretch, or four of them][position][4].
// MERGED: a warp's four groups are neighbouring stretches of the same neurons, and their sums are added (as a branch it cost the rest 7 to 19 %).
template <int V, int R, int U, bool MERGED>
__global__ void __launch_bounds__(256, kBwdBlocks) logic_path_bwd_kernel(const float *__restrict__ x, const float *__restrict__ gy, const int4 *__restrict__ rec,
                                                             const float4 *__restrict__ coef, float *__restrict__ gx, float *__restrict__ partial, int n,
                                                             int B, int cols, int ranges)
{
    using RowT = Row<8, V, R>;
    static_assert(U % 2 == 0, "the sums of two neurons are reduced at a time");
    const PathUnit t(n, cols, ranges);
    const int s0 = t.col * 8 * V * R + t.l * V, left = B - s0;
    x += s0, gy += s0, gx += s0;
    partial += ((size_t)(MERGED ? t.col >> 2 : t.col) * n + t.p0) * 4 + t.l;
    const bool writes = !MERGED || (threadIdx.x & 24) == 0;
    const bool up4 = t.l & 4, up2 = t.l & 2, up1 = t.l & 1;
    const int4 none = make_int4(-1, 0, 0, kLinked);
    int4 r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) r[u] = t.p0 + u < t.p1 ? __ldg(rec + t.p0 + u) : none;
    RowT a, carry;
    a.zero(), carry.zero();
    if (t.p0 < t.p1) {
        a.load(x + (size_t)r[0].y * B, left);
        if (r[0].w & kCloses) { // the last neuron of the range before reads that feature too
            const int4 q = __ldg(rec + t.p0 - 1);
            const float4 c = __ldg(coef + (q.x >> 1));
            const float kb = q.x & 1 ? c.y : c.z;
            RowT g, o;
            g.load(gy + (size_t)(q.x >> 1) * B, left);
            o.load(x + (size_t)q.y * B, left);
#pragma unroll
            for (int i = 0; i < RowT::P; ++i) carry.p[i] = mul2(g.p[i], fma2(pack2(c.w, c.w), o.p[i], pack2(kb, kb)));
        }
    }
    r[0].w |= kLinked;
    for (int d = 0; d < t.turns; d += U) {
        RowT g[U], b[U];
        float4 c[U];
        int4 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (r[u].x >= 0) {
                g[u].load(gy + (size_t)(r[u].x >> 1) * B, left);
                b[u].load(x + (size_t)r[u].z * B, left);
                c[u] = __ldg(coef + (r[u].x >> 1));
            } else {
                g[u].zero(), b[u].zero(), c[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) q[u] = r[u], r[u] = t.p0 + d + U + u < t.p1 ? __ldg(rec + t.p0 + d + U + u) : none;
#pragma unroll
        for (int u0 = 0; u0 < U; u0 += 2) {
            float v[8];
#pragma unroll
            for (int u = u0; u < u0 + 2; ++u) {
                if (!(q[u].w & kLinked)) a.load(x + (size_t)q[u].y * B, left);
                const bool second = q[u].x & 1;
                const float ka = second ? c[u].z : c[u].y, kb = second ? c[u].y : c[u].z;
                const f32x2 ka2 = pack2(ka, ka), kb2 = pack2(kb, kb), kab = pack2(c[u].w, c[u].w);
                RowT o;
#pragma unroll
                for (int i = 0; i < RowT::P; ++i) {
                    o.p[i] = fma2(g[u].p[i], fma2(kab, b[u].p[i], ka2), carry.p[i]);
                    carry.p[i] = mul2(g[u].p[i], fma2(kab, a.p[i], kb2));
                }
                if (q[u].w & kCloses) o.store(gx + (size_t)q[u].y * B, left);
                f32x2 t0 = 0ull, t1 = 0ull, t2 = 0ull, t3 = 0ull;
#pragma unroll
                for (int i = 0; i < RowT::P; ++i) {
                    const f32x2 ga = mul2(g[u].p[i], a.p[i]);
                    t0 = fma2(ga, b[u].p[i], t0), t1 = add2(t1, ga), t2 = fma2(g[u].p[i], b[u].p[i], t2), t3 = add2(t3, g[u].p[i]);
                }
                v[4 * (u - u0)] = sum2(t0), v[4 * (u - u0) + 1] = sum2(t1), v[4 * (u - u0) + 2] = sum2(t2), v[4 * (u - u0) + 3] = sum2(t3);
                a = b[u];
            }
            float a4[4], a2[2], s;
#pragma unroll
            for (int i = 0; i < 4; ++i) a4[i] = (up4 ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, up4 ? v[i] : v[4 + i], 4);
#pragma unroll
            for (int i = 0; i < 2; ++i) a2[i] = (up2 ? a4[2 + i] : a4[i]) + __shfl_xor_sync(0xffffffffu, up2 ? a4[i] : a4[2 + i], 2);
            s = (up1 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, up1 ? a2[0] : a2[1], 1);
            if (MERGED) s += __shfl_xor_sync(0xffffffffu, s, 8), s += __shfl_xor_sync(0xffffffffu, s, 16);
            if (writes && t.p0 + d + u0 + (t.l >> 2) < t.p1) partial[(size_t)(d + u0) * 4] = s; // lane i: sum i & 3 of neuron i >> 2
        }
    }
}

// Adds the stretches' basis sums of a neuron in stretch order and turns them into its 16 gradients: a thread per position.
__global__ void __launch_bounds__(128) logic_path_finish_kernel(const float4 *__restrict__ partial, const int4 *__restrict__ rec, const float *__restrict__ w,
                                                                float *__restrict__ gw, int n, int parts, int wmode)
{
    const int p = blockIdx.x * 128 + threadIdx.x;
    if (p >= n) return;
    const int code = __ldg(&rec[p].x), j = code >> 1;
    float v[16], s[4] = {0.f, 0.f, 0.f, 0.f}, out[16];
    load16(w + (size_t)j * 16, v);
#pragma unroll 8
    for (int c = 0; c < parts; ++c) {
        const float4 q = __ldg(partial + (size_t)c * n + p);
        s[0] += q.x, s[1] += q.y, s[2] += q.z, s[3] += q.w;
    }
    if (code & 1) {
        const float t = s[1];
        s[1] = s[2], s[2] = t;
    }
    gate_grad_store<float>(s, v, wmode, out);
#pragma unroll
    for (int q = 0; q < 4; ++q) reinterpret_cast<float4 *>(gw + (size_t)j * 16)[q] = make_float4(out[4 * q], out[4 * q + 1], out[4 * q + 2], out[4 * q + 3]);
}

} // namespace clb

using namespace clb;
using namespace clb_host;

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static size_t up16(size_t n) { return (n + 15) & ~(size_t)15; }

int clb_logic_bwd_open(const float *x, const float *gy, const float *coef, const int32_t *start32, const void *entry, const int32_t *open, int64_t n_open,
                       float *gx, int64_t B, int vec, int wide, cudaStream_t st); // logic_bwd.cu

// A group's stretch is 64 samples, or 32 where that leaves a quarter fewer lanes idle (equally full, stretches of 32 are a quarter slower);
// as many ranges as the resident blocks have groups for, of eight positions at least.  Partial sums beyond 24 MB are added over four
// stretches first (us of a whole backward without / with: 256000 x 1024 560 / 532, 250000 x 511 357 / 349; 64000 x 256 60 / 64, 24000 x 1020 83 / 91).
struct PathCut {
    bool wide;
    int cols, ranges, sums; // sums: partial sums per neuron
    unsigned blocks;
};
static PathCut path_cut(int64_t n, int64_t B, int resident)
{
    PathCut c;
    const int64_t c64 = (B + 63) / 64, c32 = (B + 31) / 32;
    c.wide = 3 * c64 < 2 * c32;
    c.cols = (int)(c.wide ? c64 : c32);
    c.sums = c.cols % 4 || !c.wide || n * c.cols * 16 < (24LL << 20) ? c.cols : c.cols / 4;
    int64_t r = (int64_t)sm_count() * resident * 32 / c.cols;
    if (r > n / 8) r = n / 8;
    if (r < 1) r = 1;
    c.ranges = (int)r;
    c.blocks = (unsigned)((r * c.cols + 31) / 32);
    return c;
}
// floats an access may have: rows of x, y, gx, gy start at multiples of B floats
static int path_vec(int64_t B, std::initializer_list<const void *> rows)
{
    uintptr_t bits = (uintptr_t)(B * 4);
    for (const void *p : rows) bits |= reinterpret_cast<uintptr_t>(p);
    return bits % 16 == 0 ? 4 : bits % 8 == 0 ? 2 : 1;
}

// Where each feature has two readers, so that nearly all gradients are completed on the way, from these sizes of x on (us of the whole pass, the
// L2 flushed before it, without / with).  Forward, beyond the L2's useful half: 128000 x 300 84 / 75, 250000 x 128 68 / 64, 64000 x 1000 120 / 116; 250000 x
// 101 66 / 69, 100000 x 250 53 / 54, 64000 x 256 35 / 38; not where a batch of more than 48 samples leaves much of its stretches empty: 458000 x 72 84 /
// 87, 347000 x 95 84 / 102, 243000 x 136 76 / 85 (444000 x 136 134 / 154), but 687000 x 48 105 / 97, 344000 x 96 78 / 75, 206000 x 160 74 / 73, 187500 x 176 72 /
// 73, 166000 x 360 140 / 110.  Backward, where three launches have something to do: 65536 x 128 42 / 42, 16000 x 512 42 / 38, 20000 x 420 46 / 40, 260000 x 32
// 70 / 60, 100000 x 97 71 / 56, 250000 x 66 138 / 95, 250000 x 511 783 / 349; 64000 x 64 28 / 32, 8000 x 100 19 / 24.  Elsewhere the input is in the L2, or
// is read once either way (4096 -> 40960 x 500 forward 29 / 32, backward 71 / 89; 300000 -> 200000 x 256 103 / 110, 265 / 267).
extern "C" int clb_logic_path_pays(int64_t in_dim, int64_t out_dim, int64_t B, int64_t n_open, int what)
{
    const int64_t bytes = in_dim * B * 4;
    if (in_dim != out_dim || 16 * n_open > in_dim) return 0;
    if (what == 0) return bytes >= 120LL << 20 && (B >= 160 || B % 32 == 0 || B <= 48);
    return bytes >= 32LL << 20;
}

extern "C" size_t clb_logic_path_scratch_bytes(int64_t in_dim, int64_t out_dim)
{
    if (in_dim <= 0 || out_dim <= 0 || in_dim > 0x3fffffff || out_dim > 0x3fffffff) return 0;
    return 16 + 12 * (size_t)out_dim + up16((size_t)out_dim) + (size_t)in_dim;
}

extern "C" int clb_logic_path(const int64_t *a, const int64_t *b, const int32_t *start32, const void *entry, void *rec, int32_t *open, int32_t *count,
                              void *scratch, size_t scratch_bytes, int64_t in_dim, int64_t out_dim, void *stream)
{
    if (!a || !b || !start32 || !entry || !rec || !open || !count || !scratch || in_dim <= 0 || out_dim <= 0) return CLB_ERR_ARG;
    if (in_dim > 0x3fffffff || out_dim > 0x3fffffff || !aligned16(rec)) return CLB_ERR_SHAPE;
    if (scratch_bytes < clb_logic_path_scratch_bytes(in_dim, out_dim) || (reinterpret_cast<uintptr_t>(scratch) & 7)) return CLB_ERR_SCRATCH;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long *laid = (unsigned long long *)scratch; // neurons laid out; more than there are where one is listed twice
    int32_t *link = (int32_t *)scratch + 4, *order = link + 2 * out_dim;
    uint8_t *placed = (uint8_t *)(order + out_dim), *closed = placed + up16((size_t)out_dim);
    const int in = (int)in_dim, out = (int)out_dim;
    const unsigned fin = (unsigned)((in_dim + 255) / 256), fout = (unsigned)((out_dim + 255) / 256);
    cudaError_t e = cudaMemsetAsync(placed, 0, up16((size_t)out_dim) + (size_t)in_dim, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(laid, 0, 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(link, 0xff, 12 * (size_t)out_dim, st); // order too: 2 * j + side of no neuron
    if (e != cudaSuccess) {
        set_last_cuda_error((int)e);
        return CLB_ERR_LAUNCH;
    }
    CLB_TRACED("path_link_kernel", st, path_link_kernel<<<fin, 256, 0, st>>>(start32, (const int2 *)entry, link, in, out));
    CLB_TRACED("path_walk_kernel", st, path_walk_kernel<<<(unsigned)((2 * out_dim + 127) / 128), 128, 0, st>>>(link, order, placed, laid, out));
    CLB_TRACED("path_rest_kernel", st, path_rest_kernel<<<fout, 256, 0, st>>>(order, placed, laid, out));
    CLB_TRACED("path_record_kernel", st, path_record_kernel<<<fout, 256, 0, st>>>(a, b, start32, order, placed, (int4 *)rec, closed, out));
    CLB_TRACED("path_open_kernel", st, path_open_kernel<<<fin, 256, 0, st>>>(closed, open, count, laid, in));
    return check_launch(5);
}

int clb_logic_coef(const float *w, float *coef, int64_t out_dim, int wmode, cudaStream_t st); // logic_bwd.cu

// live: room for the records of this call, or null: those of the plan as they are
static int path_fwd(const float *x, const int64_t *a, const int64_t *b, const void *rec, void *live, const float *w, float *y, float *coef, int64_t in_dim,
                    int64_t out_dim, int64_t B, int wmode, void *stream)
{
    if (!x || !rec || !w || !y || !coef || (live && (!a || !b)) || in_dim <= 0 || out_dim < 0 || B < 0 || wmode < 0 || wmode > 2) return CLB_ERR_ARG;
    if (out_dim == 0 || B == 0) return CLB_OK;
    if (in_dim > 0x3fffffff || out_dim > 0x3fffffff || B > 0x3fffffff || !aligned16(coef) || !aligned16(w) || !aligned16(rec) || !aligned16(live))
        return CLB_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    int rc = CLB_OK;
    if (live) {
        CLB_TRACED("logic_path_live_kernel", st,
                   logic_path_live_kernel<<<(unsigned)((out_dim + 255) / 256), 256, 0, st>>>(a, b, (const int4 *)rec, (int4 *)live, w, (float4 *)coef,
                                                                                             (int)out_dim, wmode));
        rc = check_launch();
        rec = live;
    } else {
        rc = clb_logic_coef(w, coef, out_dim, wmode, st);
    }
    if (rc != CLB_OK) return rc;
    const PathCut c = path_cut(out_dim, B, kFwdBlocks);
    auto go = [&](auto kern) {
        CLB_TRACED("logic_path_fwd_kernel", st,
                   kern<<<c.blocks, 256, 0, st>>>(x, (const int4 *)rec, (const float4 *)coef, y, (int)out_dim, (int)B, c.cols, c.ranges));
    };
    switch (path_vec(B, {x, y})) {
    case 4: c.wide ? go(logic_path_fwd_kernel<4, 2, 2>) : go(logic_path_fwd_kernel<4, 1, 2>); break;
    case 2: c.wide ? go(logic_path_fwd_kernel<2, 4, 2>) : go(logic_path_fwd_kernel<2, 2, 2>); break;
    default: c.wide ? go(logic_path_fwd_kernel<1, 8, 2>) : go(logic_path_fwd_kernel<1, 4, 2>); break;
    }
    return check_launch();
}

extern "C" int clb_logic_path_fwd(const float *x, const void *rec, const float *w, float *y, float *coef, int64_t in_dim, int64_t out_dim, int64_t B, int wmode,
                                  void *stream)
{
    return path_fwd(x, nullptr, nullptr, rec, nullptr, w, y, coef, in_dim, out_dim, B, wmode, stream);
}

extern "C" int clb_logic_path_fwd_live(const float *x, const int64_t *a, const int64_t *b, const void *rec, void *live, const float *w, float *y, float *coef,
                                       int64_t in_dim, int64_t out_dim, int64_t B, int wmode, void *stream)
{
    if (!live) return CLB_ERR_ARG;
    return path_fwd(x, a, b, rec, live, w, y, coef, in_dim, out_dim, B, wmode, stream);
}

extern "C" size_t clb_logic_path_bwd_scratch_bytes(int64_t out_dim, int64_t B)
{
    return out_dim > 0 && B > 0 ? (size_t)path_cut(out_dim, B, kBwdBlocks).sums * (size_t)out_dim * 16 : 0;
}

extern "C" int clb_logic_path_bwd(const float *x, const float *w, const float *coef, const float *gy, float *gx, float *gw, const int32_t *start32,
                                  const void *entry, const void *rec, const int32_t *open, int64_t n_open, void *scratch, size_t scratch_bytes, int64_t in_dim,
                                  int64_t out_dim, int64_t B, int wmode, void *stream)
{
    if (!x || !w || !coef || !gy || !gx || !gw || !start32 || !entry || !rec || !open || n_open < 0 || in_dim <= 0 || out_dim < 0 || B < 0 || wmode < 0 ||
        wmode > 2)
        return CLB_ERR_ARG;
    if (B == 0 || out_dim == 0) return CLB_OK;
    if (in_dim > 0x3fffffff || out_dim > 0x3fffffff || B > 0x3fffffff || !aligned16(coef) || !aligned16(w) || !aligned16(rec) || !aligned16(gw))
        return CLB_ERR_SHAPE;
    if (!scratch || !aligned16(scratch) || scratch_bytes < clb_logic_path_bwd_scratch_bytes(out_dim, B)) return CLB_ERR_SCRATCH;
    cudaStream_t st = (cudaStream_t)stream;
    const PathCut c = path_cut(out_dim, B, kBwdBlocks);
    const int vec = path_vec(B, {x, gy, gx});
    auto go = [&](auto kern) {
        CLB_TRACED("logic_path_bwd_kernel", st,
                   kern<<<c.blocks, 256, 0, st>>>(x, gy, (const int4 *)rec, (const float4 *)coef, gx, (float *)scratch, (int)out_dim, (int)B, c.cols, c.ranges));
    };
    // (stretches of 32 samples are few: their sums are never merged)
    const bool merged = c.sums != c.cols;
    switch (vec) {
    case 4: merged ? go(logic_path_bwd_kernel<4, 2, 2, true>) : c.wide ? go(logic_path_bwd_kernel<4, 2, 2, false>) : go(logic_path_bwd_kernel<4, 1, 4, false>); break;
    case 2: merged ? go(logic_path_bwd_kernel<2, 4, 2, true>) : c.wide ? go(logic_path_bwd_kernel<2, 4, 2, false>) : go(logic_path_bwd_kernel<2, 2, 4, false>); break;
    default: merged ? go(logic_path_bwd_kernel<1, 8, 2, true>) : c.wide ? go(logic_path_bwd_kernel<1, 8, 2, false>) : go(logic_path_bwd_kernel<1, 4, 4, false>); break;
    }
    int rc = check_launch();
    if (rc == CLB_OK && n_open) rc = clb_logic_bwd_open(x, gy, coef, start32, entry, open, n_open, gx, B, vec, c.wide, st);
    if (rc != CLB_OK) return rc;
    CLB_TRACED("logic_path_finish_kernel", st,
               logic_path_finish_kernel<<<(unsigned)((out_dim + 127) / 128), 128, 0, st>>>((const float4 *)scratch, (const int4 *)rec, w, gw, (int)out_dim,
                                                                                           c.sums, wmode));
    return check_launch();
}

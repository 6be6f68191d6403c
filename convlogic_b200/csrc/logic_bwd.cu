// Flat LogicLayer, backward of both gradients in one pass (fp32, feature-major activations).
//
// The two gradients read the same rows: the input gradient of feature f needs, for every neuron j that reads f, the rows gy[j]
// and x[other input of j]; the gate gradient of j needs gy[j] and both input rows.  Walking the features' consumer lists once
// gives both -- when the list of f names j by its FIRST input, x[f] (read once per feature) and the two rows at hand are all
// that j's four basis sums need -- so a layer reads 1 + 2 * 2 rows per feature instead of 2 * 2 + 3, and one kernel instead of two
// (of which the input gradient took the soft-max of every consumer again) is launched.
//
// A group of LPR lanes owns one feature and one stretch of LPR * V * R samples: R vectors of V floats per lane (V = 4 where the
// rows are 16-byte aligned).  One wave of blocks walks the features stretch by stretch, so that all work on the same columns of x
// and gy: with 64 samples (256 bytes of a row) the columns of a layer whose activation is ten times the L2 are about a cache's
// worth, and a row fetched for one consumer is often still there for the next (256000 neurons, batch 1024: 3.8 GB read from DRAM
// instead of 5.2; layers with as many neurons as features no longer come here at such sizes, logic_path.cu).  Shorter stretches make DRAM pages short of work, longer ones fall out of the cache.
// What binds is the bytes in flight per SM (the rows of 24 warps; 61 % of the DRAM rate): eight lanes with two vectors each at
// three blocks per SM beat 16 lanes with one vector (0.95 against 1.00 to 1.2 ms for 256000 x 1024), four entries at a time (1.57),
// two blocks (1.23) and fetching the tables a feature ahead (1.03: it costs registers, hence rows).  No division anywhere, sums
// in packed two-float FMAs and without a branch on the entry's side, which would split nearly every warp.
// What varies by neuron is prepared: `coef` (k1, ka, kb, kab of every gate, written by the forward pass) and the entry table
// (consumer and other input of every list entry, laid out once per layer).
// The basis sums of a stretch go to `partial` [stretch][out] and are finished by logic_bwd_finish_kernel; every sum has a fixed
// order.
#include "clb_common.cuh"
#include "clb_logic.cuh"

namespace clb {

// entry e of the consumer lists: {2 * j + (1: f is j's second input), other input of j}
__global__ void __launch_bounds__(256) logic_entries_kernel(const int64_t *__restrict__ ia, const int64_t *__restrict__ ib, const int64_t *__restrict__ start,
                                                            const int64_t *__restrict__ cons, int32_t *__restrict__ start32, int2 *__restrict__ entry,
                                                            long long in_dim)
{
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f <= in_dim; f += (long long)gridDim.x * blockDim.x) {
        const long long lo = start[f];
        start32[f] = (int32_t)lo;
        if (f == in_dim) continue;
        const long long hi = start[f + 1];
        long long prev = -1;
        for (long long e = lo; e < hi; ++e) {
            const long long j = cons[e], a = ia[j], b = ib[j];
            // a neuron fed twice by f is listed twice in a row: the first entry is w.r.t. a, the second w.r.t. b
            const bool second = a != f || (b == f && prev == j);
            entry[e] = make_int2((int)(2 * j + (second ? 1 : 0)), (int)(second ? a : b));
            prev = j;
        }
    }
}

// What the forward pass leaves for the backward where it does not run logic_fwd_kernel: a thread per neuron.
__global__ void __launch_bounds__(256) logic_coef_kernel(const float *__restrict__ w, float4 *__restrict__ coef, long long out_dim, int wmode)
{
    const long long j = (long long)blockIdx.x * 256 + threadIdx.x;
    if (j >= out_dim) return;
    float v[16], p[16];
    load16(w + j * 16, v);
    gate_mixture<float>(v, wmode, p);
    const Gate<float> g = gate_from_mixture<float>(p);
    coef[j] = make_float4(g.k1, g.ka, g.kb, g.kab);
}

// Forward of a layer whose activation exceeds the L2: the same walk, stretch by stretch, a group of LPR lanes per neuron.  One wave
// of resident blocks: a block per 16 neurons and stretch instead cost more in block launches than the walk takes (0.48 ms).
template <int LPR>
__global__ void __launch_bounds__(256) logic_fwd_cols_kernel(const float *__restrict__ x, const int64_t *__restrict__ ia, const int64_t *__restrict__ ib,
                                                             const float4 *__restrict__ coef, float *__restrict__ y, int out_dim, int B)
{
    const int l = threadIdx.x & (LPR - 1), step = (int)gridDim.x * (256 / LPR);
    int j = (int)(((unsigned)blockIdx.x * 256 + threadIdx.x) / LPR), b0 = l * 4;
    for (;; j += step) {
        while (j >= out_dim) j -= out_dim, b0 += LPR * 4;
        if (b0 - l * 4 >= B) return;
        if (b0 >= B) continue;
        const long long ja = __ldg(ia + j), jb = __ldg(ib + j);
        const float4 k = __ldg(coef + j);
        const float4 a = __ldg(reinterpret_cast<const float4 *>(x + ja * B + b0)), b = __ldg(reinterpret_cast<const float4 *>(x + jb * B + b0));
        const Gate<float> g{k.x, k.y, k.z, k.w};
        __stcs(reinterpret_cast<float4 *>(y + (long long)j * B + b0), make_float4(gate_eval<float>(g, a.x, b.x), gate_eval<float>(g, a.y, b.y),
                                                                                     gate_eval<float>(g, a.z, b.z), gate_eval<float>(g, a.w, b.w)));
    }
}

template <int LPR, int V, int R, int U, bool GW>
__global__ void __launch_bounds__(256, 3) logic_bwd_kernel(const float *__restrict__ x, const float *__restrict__ gy, const float4 *__restrict__ coef,
                                                        const int32_t *__restrict__ start, const int2 *__restrict__ entry, float *__restrict__ gx,
                                                        float *__restrict__ partial, int in_dim, int out_dim, int B,
                                                        const int32_t *__restrict__ list /* !GW: the features, or null for all of them */)
{
    using RowT = Row<LPR, V, R>;
    constexpr int GPW = 32 / LPR; // features a warp works on at a time
    static_assert(U % 2 == 0 && LPR == 8, "eight lanes reduce the sums of two entries at a time");
    const int l = threadIdx.x & (LPR - 1), grp = (threadIdx.x & 31) / LPR;
    const int warps = (in_dim + GPW - 1) / GPW, step = (int)gridDim.x * 8; // warps' worth of features; all of a warp stays in one stretch
    int wf = (int)((blockIdx.x * 256u + threadIdx.x) >> 5), left = B - l * V;
    x += l * V, gy += l * V, gx += l * V;
    // reduction of an entry pair: lane i ends up with sum i & 3 of entry i >> 2
    const bool up4 = l & 4, up2 = l & 2, up1 = l & 1;
    partial += l & 3;
    for (;; wf += step) {
        while (wf >= warps) { // the next stretch
            wf -= warps, left -= LPR * V * R;
            x += LPR * V * R, gy += LPR * V * R, gx += LPR * V * R, partial += (size_t)out_dim * 4;
        }
        if (left + l * V <= 0) return; // the whole warp
        int f = wf * GPW + grp;
        const bool mine = f < in_dim;
        if (!GW && list != nullptr && mine) f = __ldg(list + f);
        int lo = 0, hi = 0;
        if (mine) lo = __ldg(start + f), hi = __ldg(start + f + 1);
        RowT xf, acc;
        acc.zero(), xf.zero();
        if (GW && mine) xf.load(x + (size_t)f * B, left);
        for (int e0 = lo; __any_sync(0xffffffffu, e0 < hi); e0 += U) { // U entries' rows in flight
            int2 t[U];
            float4 c[U];
            RowT g[U], o[U];
#pragma unroll
            for (int u = 0; u < U; ++u) t[u] = e0 + u < hi ? __ldg(entry + e0 + u) : make_int2(-1, 0);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                c[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (t[u].x >= 0) {
                    c[u] = __ldg(coef + (t[u].x >> 1));
                    g[u].load(gy + (size_t)(t[u].x >> 1) * B, left);
                    o[u].load(x + (size_t)t[u].y * B, left);
                } else {
                    g[u].zero(), o[u].zero();
                }
            }
#pragma unroll
            for (int u0 = 0; u0 < U; u0 += 2) {
                float v[8];
#pragma unroll
                for (int u = u0; u < u0 + 2; ++u) {
                    const float k0 = (t[u].x & 1) ? c[u].z : c[u].y;
                    const f32x2 k2 = pack2(k0, k0), kab2 = pack2(c[u].w, c[u].w);
#pragma unroll
                    for (int i = 0; i < RowT::P; ++i) acc.p[i] = fma2(g[u].p[i], fma2(kab2, o[u].p[i], k2), acc.p[i]);
                    if (GW) { // also for second inputs, whose sums nobody stores: a branch would split the warp nearly every time
                        f32x2 s0 = 0ull, s1 = 0ull, s2 = 0ull, s3 = 0ull;
#pragma unroll
                        for (int i = 0; i < RowT::P; ++i) {
                            const f32x2 gx2 = mul2(g[u].p[i], xf.p[i]);
                            s0 = fma2(gx2, o[u].p[i], s0), s1 = add2(s1, gx2), s2 = fma2(g[u].p[i], o[u].p[i], s2), s3 = add2(s3, g[u].p[i]);
                        }
                        v[4 * (u - u0)] = sum2(s0), v[4 * (u - u0) + 1] = sum2(s1), v[4 * (u - u0) + 2] = sum2(s2), v[4 * (u - u0) + 3] = sum2(s3);
                    }
                }
                if (GW) {
                    float a4[4], a2[2], r;
#pragma unroll
                    for (int i = 0; i < 4; ++i) a4[i] = (up4 ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, up4 ? v[i] : v[4 + i], 4);
#pragma unroll
                    for (int i = 0; i < 2; ++i) a2[i] = (up2 ? a4[2 + i] : a4[i]) + __shfl_xor_sync(0xffffffffu, up2 ? a4[i] : a4[2 + i], 2);
                    r = (up1 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, up1 ? a2[0] : a2[1], 1);
                    const int code = up4 ? t[u0 + 1].x : t[u0].x; // the entry of this lane's sum
                    if (code >= 0 && !(code & 1)) partial[(size_t)(code >> 1) * 4] = r;
                }
            }
        }
        if (mine) acc.store(gx + (size_t)f * B, left);
    }
}

// Adds the stretches' basis sums of a neuron in stretch order and turns them into its 16 gradients: a thread per neuron.
__global__ void __launch_bounds__(128) logic_bwd_finish_kernel(const float4 *__restrict__ partial, const float *__restrict__ w, float *__restrict__ gw,
                                                               long long out_dim, int cols, int wmode)
{
    const long long j = (long long)blockIdx.x * 128 + threadIdx.x;
    if (j >= out_dim) return;
    float v[16], s[4] = {0.f, 0.f, 0.f, 0.f}, out[16];
    load16(w + j * 16, v);
#pragma unroll 8
    for (int c = 0; c < cols; ++c) {
        const float4 q = __ldg(partial + (long long)c * out_dim + j);
        s[0] += q.x, s[1] += q.y, s[2] += q.z, s[3] += q.w;
    }
    gate_grad_store<float>(s, v, wmode, out);
#pragma unroll
    for (int q = 0; q < 4; ++q) reinterpret_cast<float4 *>(gw + j * 16)[q] = make_float4(out[4 * q], out[4 * q + 1], out[4 * q + 2], out[4 * q + 3]);
}

} // namespace clb

using namespace clb;
using namespace clb_host;

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// How a layer's rows are cut.  wide: 64 samples per group (16 bytes twice per lane), two list entries in flight; otherwise 32
// samples and four entries: where features have long lists or 64-sample groups would be too few to fill the GPU.
struct BwdCut {
    bool wide;
    int cols;
};
static BwdCut bwd_cut(int64_t in_dim, int64_t out_dim, int64_t B)
{
    const int64_t c64 = (B + 63) / 64;
    BwdCut c;
    c.wide = 2 * out_dim < 8 * in_dim && in_dim * c64 >= (int64_t)sm_count() * 32 * 4;
    c.cols = (int)(c.wide ? c64 : (B + 31) / 32);
    return c;
}

// Is the combined pass the faster way?  us with it / with the two separate kernels, fp32.
// Both gradients: yes (64000 x 1024 199 / 329, 8000 x 100 10 / 29, 64000 -> 512000 x 256 377 / 523), but for inputs of a few MB in 32-sample
// stretches, where the separate kernels' second reading costs nothing and the stretches' sums do (1000 x 1024 15 / 11, 1000 -> 256000
// x 512 473 / 419, 2000 x 512 12 / 10; 4000 x 512 24 / 27, 300 -> 76800 x 1024 249 / 364), and for neurons that read a feature once
// each, far beyond the L2, in rows that are not whole stretches (200000 -> 100000, 1000 samples 677 / 605, 300 228 / 218; 1024 544 / 580,
// 64000 -> 32000 x 1000 173 / 203).
// The input gradient alone (no rows are saved by combining): while the input is in the L2 or little beyond and lists are short, where the soft-max of
// every consumer that it saves is most of the work (64000 x 128 17 / 72, 8000 -> 64000 x 256 32 / 39; 8000 -> 256000 x 512 253 / 227, 64000
// -> 256000 x 1024 870 / 636); beyond, where features have one to four readers and rows are whole sectors (200000 x 512 314 / 334, 64000
// x 1024 167 / 214; 200000 x 1000 781 / 683, 200000 -> 100000 x 512 236 / 202); unaligned rows, which the separate kernel reads a float at
// a time (64000 x 511 121 / 172; 200000 -> 100000 368 / 321).
static bool combined_pays(int64_t in_dim, int64_t out_dim, int64_t B, bool gates)
{
    const int64_t bytes = in_dim * B * 4, reads = 2 * out_dim;
    const bool wide = bwd_cut(in_dim, out_dim, B).wide, few = 4 * out_dim < 3 * in_dim && in_dim >= 131072;
    if (B % 4 == 0 && !wide && B >= 512 && bytes > (3LL << 19) && bytes <= (4LL << 20)) return false;
    if (gates) return !(few && B >= 256 && B % 32 && bytes > (192LL << 20));
    if (B % 4) return !few;
    if (!wide) return reads < 64 * in_dim ? bytes <= (100LL << 20) : B <= 128 || bytes <= (3LL << 19);
    if (4 * out_dim < 3 * in_dim && bytes > (160LL << 20) && B > 128) return false;
    return in_dim < 131072 || B % 32 == 0 || B <= 128;
}

extern "C" int clb_logic_entries(const int64_t *a, const int64_t *b, const int64_t *start, const int64_t *consumers, int32_t *start32, void *entry,
                                 int64_t in_dim, int64_t out_dim, void *stream)
{
    if (!a || !b || !start || !consumers || !start32 || !entry || in_dim <= 0 || out_dim < 0) return CLB_ERR_ARG;
    if (in_dim > 0x3fffffff || out_dim > 0x3fffffff) return CLB_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    const int grid = (int)((in_dim + 256) / 256);
    CLB_TRACED("logic_entries_kernel", st, logic_entries_kernel<<<grid, 256, 0, st>>>(a, b, start, consumers, start32, (int2 *)entry, in_dim));
    return check_launch();
}

extern "C" size_t clb_logic_bwd_scratch_bytes(int64_t in_dim, int64_t out_dim, int64_t B)
{
    if (in_dim <= 0 || out_dim <= 0 || B <= 0 || !combined_pays(in_dim, out_dim, B, true)) return 0;
    return (size_t)bwd_cut(in_dim, out_dim, B).cols * (size_t)out_dim * 16;
}

extern "C" int clb_logic_bwd(const float *x, const float *w, const float *coef, const float *gy, float *gx, float *gw, const int32_t *start32,
                             const void *entry, void *scratch, size_t scratch_bytes, int64_t in_dim, int64_t out_dim, int64_t B, int wmode, void *stream)
{
    if (!x || !w || !coef || !gy || !gx || !start32 || !entry || in_dim <= 0 || out_dim < 0 || B < 0 || wmode < 0 || wmode > 2) return CLB_ERR_ARG;
    if (B == 0) return CLB_OK;
    if (in_dim > 0x3fffffff || out_dim > 0x3fffffff || B > 0x3fffffff || !aligned16(coef)) return CLB_ERR_SHAPE;
    const bool vec = B % 4 == 0;
    if ((vec && !(aligned16(x) && aligned16(gy) && aligned16(gx))) || !aligned16(w) || (gw && !aligned16(gw))) return CLB_ERR_SHAPE;
    if (in_dim * 16 > 0x7fffffffLL * 256 || !combined_pays(in_dim, out_dim, B, gw != nullptr)) return CLB_ERR_SHAPE;
    if (gw && (!scratch || !aligned16(scratch) || scratch_bytes < clb_logic_bwd_scratch_bytes(in_dim, out_dim, B))) return CLB_ERR_SCRATCH;
    cudaStream_t st = (cudaStream_t)stream;
    const BwdCut cut = bwd_cut(in_dim, out_dim, B);
    if (cut.cols > 65535) return CLB_ERR_SHAPE;
    const bool pairs = B % 2 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gy) | reinterpret_cast<uintptr_t>(gx)) & 7) == 0;
    auto go = [&](auto kern, int lanes) {
        long long blocks = (in_dim * cut.cols * lanes + 255) / 256;
        const long long wave = (long long)sm_count() * 3; // resident at once; a second wave would walk all stretches again
        if (blocks > wave) blocks = wave;
        CLB_TRACED("logic_bwd_kernel", st,
                   kern<<<(unsigned)blocks, 256, 0, st>>>(x, gy, (const float4 *)coef, start32, (const int2 *)entry, gx, (float *)scratch, (int)in_dim, (int)out_dim, (int)B, nullptr));
    };
    if (vec && cut.wide)
        gw ? go(logic_bwd_kernel<8, 4, 2, 2, true>, 8) : go(logic_bwd_kernel<8, 4, 2, 2, false>, 8);
    else if (vec)
        gw ? go(logic_bwd_kernel<8, 4, 1, 4, true>, 8) : go(logic_bwd_kernel<8, 4, 1, 4, false>, 8);
    else if (pairs && cut.wide)
        gw ? go(logic_bwd_kernel<8, 2, 4, 2, true>, 8) : go(logic_bwd_kernel<8, 2, 4, 2, false>, 8);
    else if (pairs)
        gw ? go(logic_bwd_kernel<8, 2, 2, 4, true>, 8) : go(logic_bwd_kernel<8, 2, 2, 4, false>, 8);
    else if (cut.wide)
        gw ? go(logic_bwd_kernel<8, 1, 8, 2, true>, 8) : go(logic_bwd_kernel<8, 1, 8, 2, false>, 8);
    else
        gw ? go(logic_bwd_kernel<8, 1, 4, 4, true>, 8) : go(logic_bwd_kernel<8, 1, 4, 4, false>, 8);
    if (!gw || out_dim == 0) return check_launch(1);
    CLB_TRACED("logic_bwd_finish_kernel", st,
               logic_bwd_finish_kernel<<<(unsigned)((out_dim + 127) / 128), 128, 0, st>>>((const float4 *)scratch, w, gw, out_dim, cut.cols, wmode));
    return check_launch(2);
}

// Input gradient of the features in a list alone (logic_path.cu).  vec: floats per access.
int clb_logic_bwd_open(const float *x, const float *gy, const float *coef, const int32_t *start32, const void *entry, const int32_t *open, int64_t n_open,
                       float *gx, int64_t B, int vec, int wide, cudaStream_t st)
{
    const int64_t cols = wide ? (B + 63) / 64 : (B + 31) / 32;
    long long blocks = (n_open * cols * 8 + 255) / 256;
    if (blocks > (long long)sm_count() * 3) blocks = (long long)sm_count() * 3;
    auto go = [&](auto kern) {
        CLB_TRACED("logic_bwd_kernel", st,
                   kern<<<(unsigned)blocks, 256, 0, st>>>(x, gy, (const float4 *)coef, start32, (const int2 *)entry, gx, nullptr, (int)n_open, 0, (int)B, open));
    };
    switch (vec) {
    case 4: wide ? go(logic_bwd_kernel<8, 4, 2, 2, false>) : go(logic_bwd_kernel<8, 4, 1, 4, false>); break;
    case 2: wide ? go(logic_bwd_kernel<8, 2, 4, 2, false>) : go(logic_bwd_kernel<8, 2, 2, 4, false>); break;
    default: wide ? go(logic_bwd_kernel<8, 1, 8, 2, false>) : go(logic_bwd_kernel<8, 1, 4, 4, false>); break;
    }
    return check_launch();
}

int clb_logic_coef(const float *w, float *coef, int64_t out_dim, int wmode, cudaStream_t st)
{
    CLB_TRACED("logic_coef_kernel", st, logic_coef_kernel<<<(unsigned)((out_dim + 255) / 256), 256, 0, st>>>(w, (float4 *)coef, out_dim, wmode));
    return check_launch();
}

// Forward of a layer too large for the L2 (V = 4 rows): the gates' coefficients, then the rows stretch by stretch.
int clb_logic_fwd_cols(const float *x, const int64_t *a, const int64_t *b, const float *w, float *y, float *coef, int64_t out_dim, int64_t B, int wmode,
                       cudaStream_t st)
{
    constexpr int LPR = 16;
    CLB_TRACED("logic_coef_kernel", st, logic_coef_kernel<<<(unsigned)((out_dim + 255) / 256), 256, 0, st>>>(w, (float4 *)coef, out_dim, wmode));
    CLB_TRACED("logic_fwd_cols_kernel", st, logic_fwd_cols_kernel<LPR><<<(unsigned)(sm_count() * 8), 256, 0, st>>>(x, a, b, (const float4 *)coef, y, (int)out_dim, (int)B));
    return check_launch(2);
}

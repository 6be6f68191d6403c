// Packed (discretised) inference kernels: every bit of a word is one sample.
//
// A packed tensor is [rows, words] of `bits`-wide integers, sample bits*word + i in bit i.  On a
// little-endian machine that is the same as a row of ceil(B/bits)*bits/8 BYTES with sample s in bit
// (s & 7) of byte (s >> 3), whatever `bits` is; bitwise gates do not care about the word width either.
// The kernels therefore see rows of bytes and move them in the widest unit the row length and the
// pointers allow (16, 8 or 4 bytes; rows of any other length as 4-byte words shifted into place);
// `bits` only fixes how many pad samples a row ends with.
//
// A 2-input gate with truth table (f00, f01, f10, f11), given as four all-ones/all-zero masks, is the
// two-level multiplexer  y = a ? (b ? m11 : m10) : (b ? m01 : m00): three 3-input logic operations per
// 32 bits, branch-free, with the masks uniform over the thread block.
#include "clb_common.cuh"
#include "clb_slab.cuh"

#include <algorithm>
#include <type_traits>

namespace clb {

template <typename U> struct OpMasks {
    U m00, m01, m10, m11;
};
template <typename U> __device__ __forceinline__ OpMasks<U> op_masks(int op)
{
    OpMasks<U> m;
    const U ones = ~U(0);
    m.m00 = (op & 8) ? ones : U(0);
    m.m01 = (op & 4) ? ones : U(0);
    m.m10 = (op & 2) ? ones : U(0);
    m.m11 = (op & 1) ? ones : U(0);
    return m;
}
template <typename U> __device__ __forceinline__ U op_apply(const OpMasks<U> &m, U a, U b)
{
    const U r1 = (b & m.m11) | (~b & m.m10);
    const U r0 = (b & m.m01) | (~b & m.m00);
    return (a & r1) | (~a & r0);
}

// ------------------------------------------------------------------------------------- pack bits
// feature-major source t [F,B]; one thread builds one output byte from 8 consecutive samples.
__global__ void pack_bits_kernel(const uint8_t *__restrict__ t, uint8_t *__restrict__ out, long long F, long long B, long long rowbytes)
{
    const long long total = F * rowbytes;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long f = i / rowbytes, q = i % rowbytes;
        const uint8_t *src = t + f * B + q * 8;
        unsigned v = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (q * 8 + k < B) v |= (src[k] != 0 ? 1u : 0u) << k;
        out[i] = (uint8_t)v;
    }
}

// sample-major source t [N, F]: the transpose and the packing in one pass.  Block: 128 features x 256 samples, warp w the
// samples 32w..32w+31, lane l the features 4l..4l+3 of the block: a load is four features of one sample (one 32-bit word when F
// and t allow it), and eight samples' words, each byte 0 or 1, shifted by the sample's number and OR-ed are the eight-sample
// bytes of four features at once.  The words leave through shared memory, so that every row receives 32 contiguous bytes
// (rows layout, words beyond the row cut off) or every (channel, slab) 16 bytes per position (slab layout).
// Bound by the bytes read (a feature per thread, one byte per load, took 68 us for 30.7 MB; this takes 9).
__device__ __forceinline__ unsigned nonzero_bytes(unsigned v) { return ((((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) >> 7) & 0x01010101u; }

template <bool QUAD>
__global__ void __launch_bounds__(256) pack_bits_nmajor_kernel(const uint8_t *__restrict__ t, uint8_t *__restrict__ out, long long N, long long F,
                                                               long long rowbytes, int word_stores, int HW, int side, long long U)
{
    __shared__ unsigned sm[128 * 9];
    const int lane = threadIdx.x & 31, wv = threadIdx.x >> 5;
    const long long f0 = (long long)blockIdx.x * 128, f = f0 + 4 * lane;
    for (long long n0 = (long long)blockIdx.y * 256; n0 < rowbytes * 8; n0 += (long long)gridDim.y * 256) {
        const long long nb = n0 + wv * 32;
        const int live = (int)max(0LL, min(32LL, N - nb));
        const uint8_t *src = t + nb * F + f;
        unsigned g[4] = {0u, 0u, 0u, 0u}; // byte k of g[q]: samples 8q..8q+7 of feature f + k
        if (f < F) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                unsigned v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[j] = 0u;
                    if (8 * q + j < live) {
                        const uint8_t *p = src + (8 * q + j) * F;
                        if (QUAD) {
                            v[j] = __ldg(reinterpret_cast<const unsigned *>(p));
                        } else {
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                if (f + k < F) v[j] |= (unsigned)__ldg(p + k) << (8 * k);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) g[q] |= nonzero_bytes(v[j]) << j;
            }
        }
        __syncthreads(); // the previous pass has been written out
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned lo = __byte_perm(g[0], g[1], 0x40 + 0x11 * k), hi = __byte_perm(g[2], g[3], 0x40 + 0x11 * k);
            sm[(4 * lane + k) * 9 + wv] = (lo & 0xffffu) | (hi << 16);
        }
        __syncthreads();
        if (HW > 0) { // slab layout [channel][U][HW] of 16-byte units, in split order if a side is given
            for (int e = threadIdx.x; e < 1024; e += 256) {
                const int q = e & 3, i = (e >> 2) & 127, h = e >> 9;
                const long long u = n0 / 128 + h, ff = f0 + i;
                if (ff < F && u < U) {
                    const long long c = ff / HW;
                    int yx = (int)(ff - c * HW);
                    if (side) yx = split_position(yx, side);
                    reinterpret_cast<unsigned *>(out)[((c * U + u) * HW + yx) * 4 + q] = sm[i * 9 + 4 * h + q];
                }
            }
        } else if (word_stores) {
            for (int e = threadIdx.x; e < 1024; e += 256) {
                const int w = e & 7, i = e >> 3;
                const long long at = n0 / 8 + 4 * w;
                if (f0 + i < F && at < rowbytes) *reinterpret_cast<unsigned *>(out + (f0 + i) * rowbytes + at) = sm[i * 9 + w];
            }
        } else {
            for (int e = threadIdx.x; e < 4096; e += 256) {
                const int y = e & 31, i = e >> 5;
                const long long at = n0 / 8 + y;
                if (f0 + i < F && at < rowbytes) out[(f0 + i) * rowbytes + at] = (uint8_t)(sm[i * 9 + (y >> 2)] >> (8 * (y & 3)));
            }
        }
    }
}

// ---------------------------------------------------------------------------- thermometer + pack
// Fused input stage of packed inference: pixels [N][P] (P = channels * H * W, fp32 in [0,1] or uint8 that is
// divided by 255 as torchvision's ToTensor does) -> the L*P thermometer features "pixel > threshold[i]",
// threshold-major (feature i*P + p), bit-packed along the batch, without the [N, L*P] byte tensor in between.
// A block has 256 samples, 32 to a warp, and 32 pixel positions at a time, one to a lane: a thread builds, for its position, the 32-sample
// word of every level in registers; the words go through shared memory so that each feature row receives 32 contiguous bytes
// (rows layout) or each (feature, slab) 512 contiguous bytes (slab layout, one 16-byte unit per position).  Levels are taken 8 G at a
// time, G = 1 .. 4 by their number.
struct ThermoOut {
    unsigned *out;
    int P, HW;
    long long words32;
    int to_slab, side; // side: split column order
};

// nl levels from l0 of positions p0 .. p0 + 31: thread = (position, word), so only the level walks -- one shared load, one store and
// two additions per level
__device__ __forceinline__ void thermo_write(const unsigned *sm, const ThermoOut &o, int l0, int nl, int p0, long long n0)
{
    const long long w0 = n0 / 32; // first 32-bit word of this block in a row
    if (!o.to_slab) {
        // (level, position, word): 8 consecutive lanes write the 32 bytes of one row
        const int w = threadIdx.x & 7, pos = (threadIdx.x >> 3) & 31;
        const int pp = p0 + pos;
        if (pp < o.P && w0 + w < o.words32) {
            unsigned *dst = o.out + ((long long)l0 * o.P + pp) * o.words32 + w0 + w;
            const unsigned *srcw = sm + pos * 9 + w;
            const long long dstep = (long long)o.P * o.words32;
            for (int i = 0; i < nl; ++i) dst[i * dstep] = srcw[i * 32 * 9];
        }
    } else {
        // slab layout [feature channel][U][HW] of 16-byte units: 4 consecutive lanes write one unit
        const long long U = o.words32 / 4;
        const int q = threadIdx.x & 3, pos = (threadIdx.x >> 2) & 31, u2 = (threadIdx.x >> 7) & 1;
        const int pp = p0 + pos;
        const long long u = w0 / 4 + u2;
        if (pp < o.P && u < U) {
            const int c = pp / o.HW;
            int yx = pp - c * o.HW;
            if (o.side) yx = split_position(yx, o.side);
            unsigned *dst = o.out + ((((long long)l0 * (o.P / o.HW) + c) * U + u) * o.HW + yx) * 4 + q;
            const unsigned *srcw = sm + pos * 9 + u2 * 4 + q;
            const long long dstep = (long long)(o.P / o.HW) * U * o.HW * 4;
            for (int i = 0; i < nl; ++i) dst[i * dstep] = srcw[i * 32 * 9];
        }
    }
}

// word |= bit where v > t: a comparison and a predicated OR (the compiler makes five instructions of the expression)
__device__ __forceinline__ void set_if_above(unsigned &word, float v, float t, unsigned bit)
{
    asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %1, %2;\n\t@p or.b32 %0, %0, %3;\n\t}" : "+r"(word) : "f"(v), "f"(t), "r"(bit));
}

// Bound by the comparisons, two instructions per level and sample.  The passes over the levels are gridDim.z blocks' work where the grid is
// small (100 images, 64 levels: 25 us in one block after the other, 17 side by side), and samples that a batch does not have are skipped.
template <int G>
__global__ void __launch_bounds__(256) thermometer_pack_kernel(const float *__restrict__ pix, const float *__restrict__ thr, int L, long long N, ThermoOut o)
{
    constexpr int NL = 8 * G;
    __shared__ unsigned sm[NL * 32 * 9];
    const int lane = threadIdx.x & 31, wv = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    const long long n0 = (long long)blockIdx.y * 256, nb = n0 + wv * 32;
    const int live = p < o.P ? (int)max(0LL, min(32LL, N - nb)) : 0;
    for (int l0 = blockIdx.z * NL; l0 < L; l0 += gridDim.z * NL) {
        const int nl = min(NL, L - l0);
        float th[NL];
        unsigned word[NL];
#pragma unroll
        for (int i = 0; i < NL; ++i) th[i] = i < nl ? __ldg(thr + l0 + i) : 0.f, word[i] = 0u;
        const float *src = pix + nb * o.P + p;
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 16) { // sixteen samples in flight
            if (j0 >= live) break;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = j0 + j < live ? __ldg(src + (long long)(j0 + j) * o.P) : __int_as_float(0x7fc00000); // a NaN is above nothing
#pragma unroll
            for (int j = 0; j < 16; ++j)
#pragma unroll
                for (int i = 0; i < NL; ++i) set_if_above(word[i], v[j], th[i], 1u << (j0 + j));
        }
        __syncthreads(); // the previous pass has been written out
#pragma unroll
        for (int i = 0; i < NL; ++i) sm[(i * 32 + lane) * 9 + wv] = word[i];
        __syncthreads();
        thermo_write(sm, o, l0, nl, blockIdx.x * 32, n0);
    }
}

// uint8 pixels take 256 values: thread t builds the level mask of value t once per block (the float expression of the other kernel,
// so the bits are the same), a sample is then one byte and one table look-up, and 8x8 bit transposes in registers turn the
// masks of 32 samples into sample words, eight levels at a time.  The bytes come through a tile of 256 samples x 128 positions, read in
// 16-byte pieces where the rows allow it: read position by position, a warp fetched 32 bytes from each of 32 rows at a time, and
// 20000 images of 3 levels took 132 us, now 59.
// CH: positions of a block / 32, fewer where the larger blocks would not fill the GPU twice.
template <int G, int CH>
__global__ void __launch_bounds__(256) thermometer_pack_bytes_kernel(const uint8_t *__restrict__ pix, const float *__restrict__ thr, int L, long long N, int vec, ThermoOut o)
{
    constexpr int NL = 8 * G;
    using Mask = std::conditional_t<G == 1, uint8_t, std::conditional_t<G == 2, uint16_t, unsigned>>;
    constexpr int W = 32 * CH;
    __shared__ __align__(16) uint8_t tile[256 * W];
    __shared__ Mask lut[256];
    extern __shared__ unsigned sm[]; // [NL][32][9]
    const int tid = threadIdx.x, lane = tid & 31, wv = tid >> 5;
    const int p0 = blockIdx.x * W;
    const long long n0 = (long long)blockIdx.y * 256;
    if (vec) {
#pragma unroll
        for (int i = 0; i < 2 * CH; ++i) {
            const int u = tid + 256 * i, row = u / (2 * CH), q = u % (2 * CH) * 16;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (n0 + row < N && p0 + q < o.P) v = __ldg(reinterpret_cast<const uint4 *>(pix + (n0 + row) * o.P + p0 + q));
            *reinterpret_cast<uint4 *>(tile + row * W + q) = v;
        }
    } else {
        for (int i = tid; i < 256 * W; i += 256) {
            const int row = i / W, q = i % W;
            tile[i] = n0 + row < N && p0 + q < o.P ? __ldg(pix + (n0 + row) * o.P + p0 + q) : 0;
        }
    }
    const int live = (int)max(0LL, min(32LL, N - (n0 + wv * 32)));
    for (int l0 = 0; l0 < L; l0 += NL) {
        const int nl = min(NL, L - l0);
        __syncthreads(); // the previous pass no longer reads the table
        {
            const float v = __fdiv_rn((float)tid, 255.0f);
            unsigned m = 0u;
#pragma unroll
            for (int i = 0; i < NL; ++i) m |= ((i < nl && v > __ldg(thr + l0 + min(i, nl - 1))) ? 1u : 0u) << i;
            lut[tid] = (Mask)m;
        }
        __syncthreads();
#pragma unroll 1
        for (int chunk = 0; chunk < CH && p0 + chunk * 32 < o.P; ++chunk) {
            unsigned m[32];
            const uint8_t *src = tile + wv * 32 * W + chunk * 32 + lane;
#pragma unroll
            for (int j = 0; j < 32; ++j) m[j] = j < live ? (unsigned)lut[src[j * W]] : 0u;
            if (chunk) __syncthreads(); // the previous chunk has been written out
#pragma unroll
            for (int g = 0; g < G; ++g) {
                unsigned w[8]; // byte b of w[q]: sample 8 b + q
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const unsigned lo = __byte_perm(m[q], m[8 + q], 0x0040 + 0x0011 * g), hi = __byte_perm(m[16 + q], m[24 + q], 0x0040 + 0x0011 * g);
                    w[q] = __byte_perm(lo, hi, 0x5410);
                }
#pragma unroll
                for (int s = 4; s >= 1; s >>= 1) {
                    const unsigned keep = s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (!(q & s)) {
                            const unsigned t = ((w[q] >> s) ^ w[q + s]) & keep;
                            w[q + s] ^= t, w[q] ^= t << s;
                        }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) sm[((8 * g + i) * 32 + lane) * 9 + wv] = w[i];
            }
            __syncthreads();
            thermo_write(sm, o, l0, nl, p0 + chunk * 32, n0);
        }
    }
}

// ----------------------------------------------------------------------------------- flat layer
template <typename V> struct Words { // a transfer unit as 32-bit words
    static constexpr int N = sizeof(V) / 4;
    unsigned w[N];
};
template <typename V> __device__ __forceinline__ Words<V> load_words(const V *p)
{
    const V v = __ldg(p);
    Words<V> r;
    const unsigned *q = reinterpret_cast<const unsigned *>(&v);
#pragma unroll
    for (int i = 0; i < Words<V>::N; ++i) r.w[i] = q[i];
    return r;
}

// Rows of `units` units of type V (4, 8 or 16 bytes).  A group of 2^lg lanes (the power of two that covers a row, at most a
// warp) owns a neuron at a time: its indices and gate are read once, the next neuron's one neuron ahead, and its row is walked
// with R units per lane in flight.  Bound by L2: two gathered rows in, one out.
template <typename V, int R>
__global__ void __launch_bounds__(256) packed_logic_kernel(const V *__restrict__ x, const int64_t *__restrict__ ia, const int64_t *__restrict__ ib,
                                                           const uint8_t *__restrict__ ops, V *__restrict__ y, long long out_dim, int units, int lg)
{
    const long long first = ((long long)blockIdx.x * 256 + threadIdx.x) >> lg, step = ((long long)gridDim.x * 256) >> lg;
    const int g = 1 << lg, l = threadIdx.x & (g - 1);
    long long a = 0, b = 0;
    int op = 0;
    if (first < out_dim) a = __ldg(ia + first), b = __ldg(ib + first), op = __ldg(ops + first);
    for (long long j = first; j < out_dim; j += step) {
        const V *xa = x + a * units, *xb = x + b * units;
        V *yo = y + j * units;
        const OpMasks<unsigned> m = op_masks<unsigned>(op);
        const long long jn = j + step;
        if (jn < out_dim) a = __ldg(ia + jn), b = __ldg(ib + jn), op = __ldg(ops + jn);
        for (int u0 = l; u0 < units; u0 += g * R) {
            Words<V> va[R], vb[R];
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (u0 + r * g < units) va[r] = load_words(xa + u0 + r * g), vb[r] = load_words(xb + u0 + r * g);
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (u0 + r * g < units) {
                    V o;
                    unsigned *q = reinterpret_cast<unsigned *>(&o);
#pragma unroll
                    for (int i = 0; i < Words<V>::N; ++i) q[i] = op_apply<unsigned>(m, va[r].w[i], vb[r].w[i]);
                    yo[u0 + r * g] = o;
                }
        }
    }
}

constexpr int kPathBlocks = 6; // packed_path_kernel: resident per SM

// An order of the neurons in which the next one reads what the last one read second.  The half-edges of a feature (2 * j + side of
// neuron j) are paired up as they come, one waiting in `slot` for the next; one pair in 128 is left apart, so that trails stay short
// enough to be walked by one thread.  Each half-edge has at most one partner, and that is mutual, so that every neuron is laid out once,
// whatever the connections.  The order may differ between runs; the outputs are bits.
__global__ void __launch_bounds__(256) packed_pair_kernel(const int64_t *__restrict__ ia, const int64_t *__restrict__ ib, int32_t *slot, int32_t *link,
                                                          int in_dim, int out_dim)
{
    const int h = blockIdx.x * 256 + threadIdx.x;
    if (h >= 2 * out_dim) return;
    const int64_t f = (h & 1 ? ib : ia)[h >> 1];
    if (f < 0 || f >= in_dim) return;
    for (int tries = 0; tries < 256; ++tries) { // (one that never gets through stays alone)
        const int waiting = atomicCAS(slot + f, -1, h);
        if (waiting < 0) return;
        if (atomicCAS(slot + f, waiting, -1) != waiting) continue;
        unsigned e = (unsigned)min(h, waiting);
        e *= 0x9E3779B1u, e ^= e >> 15, e *= 0x85EBCA77u, e ^= e >> 13;
        if ((waiting >> 1) != (h >> 1) && e % 128 != 0) link[waiting] = h, link[h] = waiting; // (a neuron fed twice by f is no link)
        return;
    }
}

// A thread per half-edge that is the end of a trail; of a trail's two ends the one with the smaller number lays it out.
__global__ void __launch_bounds__(128) packed_walk_kernel(const int32_t *__restrict__ link, int32_t *__restrict__ order, uint8_t *__restrict__ placed,
                                                          int32_t *__restrict__ count, int out_dim)
{
    const int h = blockIdx.x * 128 + threadIdx.x;
    if (h >= 2 * out_dim || link[h] >= 0) return;
    int n = 1, cur = h;
    for (int next; n < out_dim && (next = __ldg(link + (cur ^ 1))) >= 0; ++n) cur = next;
    if (h > (cur ^ 1)) return;
    const int p = atomicAdd(count, n);
    cur = h;
    for (int i = 0; i < n; ++i) {
        order[p + i] = cur, placed[cur >> 1] = 1;
        cur = __ldg(link + (cur ^ 1));
    }
}

// neurons that no trail end reaches (closed trails) stand alone
__global__ void __launch_bounds__(256) packed_rest_kernel(int32_t *__restrict__ order, const uint8_t *__restrict__ placed, int32_t *__restrict__ count, int out_dim)
{
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j < out_dim && !placed[j]) order[atomicAdd(count, 1)] = 2 * j;
}

// The same layer walked in such an order (or in that of logic_path.cu's records): one gathered row per neuron instead of two.
// A group of 2^LG lanes owns a range of positions and a stretch of R units per lane.  What bound it first was the issue
// of integer instructions (171 per neuron and stretch of five words): offsets within a row are constants now, which lanes are inside
// it is found once, and a gate's four masks come from a table; then the bytes in flight, for which many warps with one row each beat
// fewer with two to four (128000 neurons, rows of 2500 bytes: four blocks and two rows 141 us, six and one 128).  us for one layer, x in the L2 as the layer
// before leaves it, two rows per neuron / this: 3072 -> 64000 neurons, 1252 bytes 37.6 / 22.9, 64000 -> 64000 45.3 / 34.3, 128000 x 2500 171 / 126.
// step 1: an order, the connections from ia and ib as they are now (a lane each for as many positions as there are lanes, fetched as many
// positions ahead, then through shared memory); step 4: records, with their own.
template <typename V, int R, int LG>
__global__ void __launch_bounds__(256, kPathBlocks) packed_path_kernel(const V *__restrict__ x, const int32_t *__restrict__ order, int step,
                                                             const int64_t *__restrict__ ia, const int64_t *__restrict__ ib, const uint8_t *__restrict__ ops,
                                                             V *__restrict__ y, int n, int units, int cols, int ranges)
{
    constexpr int N = Words<V>::N, G = 1 << LG;
    __shared__ uint4 masks[32]; // of gate op, and from 16 on of the gate with its inputs swapped
    __shared__ int4 table[256];
    if (threadIdx.x < 32) {
        const int op = threadIdx.x & 15, o = threadIdx.x < 16 ? op : (op & 9) | (op & 2) << 1 | (op & 4) >> 1;
        masks[threadIdx.x] = make_uint4(o & 1 ? ~0u : 0u, o & 2 ? ~0u : 0u, o & 4 ? ~0u : 0u, o & 8 ? ~0u : 0u);
    }
    __syncthreads();
    const int unit = (int)((blockIdx.x * 256u + threadIdx.x) >> LG), range = unit / cols, col = unit - range * cols, lane = threadIdx.x & (G - 1);
    const unsigned group = LG == 5 ? ~0u : ((1u << G % 32) - 1) << (threadIdx.x & 31 & ~(G - 1)); // its lanes make the same turns
    const int turns = (n + ranges - 1) / ranges, p0 = range * turns, p1 = min(n, p0 + turns), u0 = col * G * R + lane;
    if (p0 >= p1) return;
    x += u0, y += u0;
    bool in[R];
#pragma unroll
    for (int r = 0; r < R; ++r) in[r] = u0 + r * G < units;
    Words<V> a[R];
    auto load = [&](Words<V>(&row)[R], int f) {
        const V *p = x + (size_t)f * units;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (in[r]) row[r] = load_words(p + r * G);
    };
    auto code_at = [&](int p) { return p < p1 ? __ldg(order + (size_t)p * step) : -1; };
    // features entered from and left through
    auto features = [&](int code, int p, int &u, int &v) {
        u = v = 0;
        if (code < 0) return;
        if (step == 1) {
            const int fa = (int)__ldg(ia + (code >> 1)), fb = (int)__ldg(ib + (code >> 1));
            u = code & 1 ? fb : fa, v = code & 1 ? fa : fb;
        } else {
            u = __ldg(order + (size_t)p * 4 + 1), v = __ldg(order + (size_t)p * 4 + 2);
        }
    };
    int code = code_at(p0 + lane), next = code_at(p0 + G + lane), u, v;
    features(code, p0 + lane, u, v);
    for (int base = p0; base < p1; base += G) {
        int before = __shfl_up_sync(group, v, 1, G);
        if (lane == 0) before = base > p0 ? table[threadIdx.x + G - 1].z : -1;
        __syncwarp(group); // the positions before are done with
        table[threadIdx.x] = make_int4(code, u == before ? -1 : u, v, 0); // (-1: the row entered through is there)
        __syncwarp(group);
        code = next;
        features(code, base + G + lane, u, v);
        next = code_at(base + 2 * G + lane);
        for (int i = 0; i < min(G, p1 - base); ++i) {
            const int4 t = table[(threadIdx.x & ~(G - 1)) + i];
            Words<V> b[R];
            load(b, t.z);
            const int op = __ldg(ops + (t.x >> 1)) & 15;
            if (t.y >= 0) load(a, t.y);
            const uint4 k = masks[op | (t.x & 1) << 4];
            V *row = y + (size_t)(t.x >> 1) * units;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                V o;
                unsigned *w = reinterpret_cast<unsigned *>(&o);
#pragma unroll
                for (int q = 0; q < N; ++q) {
                    const unsigned va = a[r].w[q], vb = b[r].w[q], r1 = (vb & k.x) | (~vb & k.y), r0 = (vb & k.z) | (~vb & k.w);
                    w[q] = (va & r1) | (~va & r0);
                }
                if (in[r]) row[r * G] = o;
                a[r] = b[r];
            }
        }
    }
}

// bytes 4 w .. 4 w + 3 from p on, of which `valid` (more than 4: all) belong to the row: only words that hold one of those are read
__device__ __forceinline__ unsigned word_at(const uint8_t *p, long long w, long long valid = 4)
{
    const unsigned *q = reinterpret_cast<const unsigned *>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3) + w;
    const unsigned at = (unsigned)(reinterpret_cast<uintptr_t>(p) & 3), lo = __ldg(q);
    return at ? __funnelshift_r(lo, at + min(4LL, valid) > 4 ? __ldg(q + 1) : 0u, 8 * at) : lo;
}

// Rows whose length is no multiple of four bytes, so that a neuron's two input rows and its output row start anywhere: the
// output is written in aligned 32-bit words, each input word put together from the two aligned words it straddles; up to three
// bytes at either end of a row go one by one.  The same split as above.
__global__ void __launch_bounds__(256) packed_logic_bytes_kernel(const uint8_t *__restrict__ x, const int64_t *__restrict__ ia, const int64_t *__restrict__ ib,
                                                                 const uint8_t *__restrict__ ops, uint8_t *__restrict__ y, long long out_dim, int rowbytes,
                                                                 int lg)
{
    const long long first = ((long long)blockIdx.x * 256 + threadIdx.x) >> lg, step = ((long long)gridDim.x * 256) >> lg;
    const int g = 1 << lg, l = threadIdx.x & (g - 1);
    for (long long j = first; j < out_dim; j += step) {
        const uint8_t *xa = x + __ldg(ia + j) * rowbytes, *xb = x + __ldg(ib + j) * rowbytes;
        uint8_t *yo = y + j * rowbytes;
        const OpMasks<unsigned> m = op_masks<unsigned>(__ldg(ops + j));
        const int head = min(rowbytes, (int)(-reinterpret_cast<uintptr_t>(yo) & 3)), words = (rowbytes - head) >> 2, tail = rowbytes - head - 4 * words;
        for (int w0 = l; w0 < words; w0 += 4 * g) {
            unsigned va[4], vb[4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (w0 + r * g < words) va[r] = word_at(xa + head, w0 + r * g), vb[r] = word_at(xb + head, w0 + r * g);
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (w0 + r * g < words) reinterpret_cast<unsigned *>(yo + head)[w0 + r * g] = op_apply<unsigned>(m, va[r], vb[r]);
        }
        for (int e = l; e < head + tail; e += g) {
            const int at = e < head ? e : 4 * words + e;
            yo[at] = (uint8_t)op_apply<unsigned>(m, __ldg(xa + at), __ldg(xb + at));
        }
    }
}

// Two or three consecutive flat layers as one pass.  When a layer's outputs are each read about once by the next
// layer (the stacks halve their width from layer to layer, and `randperm(2*out) % in` then uses every output
// exactly once), a neuron of the last layer is a gate tree over 2^M rows of the FIRST layer's input: the
// intermediate activations (the largest tensors of the stack) are never written or read.  leaf [out][2^M] are the
// input rows in tree order (gate p of the first level reads leaves 2p and 2p+1), ops [out][2^M - 1] the gate ids
// level by level (first level, ..., root).  Rows move in 8- or 16-byte units like the single layer.
template <typename V4, int M, typename IDX>
__global__ void __launch_bounds__(256) packed_tree_kernel(const V4 *__restrict__ x, const int32_t *__restrict__ leaf,
                                                          const uint8_t *__restrict__ ops, V4 *__restrict__ y, long long out_dim,
                                                          long long units, long long u_lo, long long u_n)
{
    // one launch covers units [u_lo, u_lo + u_n) of every row
    constexpr int L = 1 << M, G = L - 1;
    constexpr int W = sizeof(V4) / 4;
    // (tree, unit) of the thread's items by carried additions: one 64-bit division per thread instead of two per item
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    const long long dj = stride / u_n, du = stride - dj * u_n;
    long long j = t0 / u_n, ur = t0 - j * u_n;
    for (; j < out_dim; j += dj, ur += du) {
        if (ur >= u_n) ur -= u_n, ++j;
        if (j >= out_dim) break;
        const long long u = u_lo + ur, i = j * units + u;
        unsigned v[L][W];
#pragma unroll
        for (int k = 0; k < L; ++k) {
            const V4 q = __ldg(x + ((IDX)__ldg(leaf + j * L + k) * (IDX)units + (IDX)u)); // IDX: 32 bits when the input has < 2^32 units
            const unsigned *qw = reinterpret_cast<const unsigned *>(&q);
#pragma unroll
            for (int w = 0; w < W; ++w) v[k][w] = qw[w];
        }
        int g = 0;
#pragma unroll
        for (int n = L / 2; n >= 1; n /= 2) { // n gates on this level
#pragma unroll
            for (int p = 0; p < n; ++p) {
                const OpMasks<unsigned> m = op_masks<unsigned>(__ldg(ops + j * G + g + p));
#pragma unroll
                for (int w = 0; w < W; ++w) v[p][w] = op_apply<unsigned>(m, v[2 * p][w], v[2 * p + 1][w]);
            }
            g += n;
        }
        V4 r;
        unsigned *rw = reinterpret_cast<unsigned *>(&r);
#pragma unroll
        for (int w = 0; w < W; ++w) rw[w] = v[0][w];
        y[i] = r;
    }
}

// ----------------------------------------------------------------------------------- group sum
// x rows as 32-bit units (32 samples each).  Block (32 units, part of a class's rows, class): lane <-> unit, the eight warps
// share the rows of the part.  Rows are added 16 at a time into bit-sliced counters (carry-save adders: ones, twos, fours,
// eights + ripple counter for the sixteens), so a row costs a handful of logic operations per 32 samples; the eight warps' counters
// are added in bit-sliced form through shared memory, and only then are the per-sample integers extracted, four of a unit's 32
// by each warp.  With more than one part they are combined with integer atomics (exact, order-independent) into a zeroed
// output: per part, not per thread (a thread's 32 atomics were most of the kernel: 50 us for 80 MB).
__device__ __forceinline__ void csa(unsigned &hi, unsigned &lo, unsigned a, unsigned b, unsigned c)
{
    const unsigned u = a ^ b;
    hi = (a & b) | (u & c);
    lo = u ^ c;
}

// PLANES bit planes above the sixteens: a warp can count 16 * 2^PLANES rows, and so can the sum of the eight warps.
// ANY: rows of any number of bytes, whose words are put together from the two aligned ones that they straddle.
template <int PLANES, bool ANY>
__global__ void __launch_bounds__(256, 3) group_popcount_kernel(const uint8_t *__restrict__ xb, int *__restrict__ counts, long long S, long long rowbytes, long long B,
                                                             int k)
{
    constexpr int P = PLANES + 4;
    __shared__ unsigned sm[4][P][32];
    const int lane = threadIdx.x & 31, wv = threadIdx.x >> 5;
    const long long units = ANY ? (rowbytes + 3) / 4 : rowbytes / 4;
    const long long u = (long long)blockIdx.x * 32 + lane;
    const int cls = blockIdx.z, parts = gridDim.y, sp = blockIdx.y * 8 + wv;
    const long long r_lo = S * sp / (8LL * parts), r_hi = S * (sp + 1) / (8LL * parts);
    unsigned n[P]; // plane p: bit p of the counts
#pragma unroll
    for (int p = 0; p < P; ++p) n[p] = 0;
    if (u < units) {
        const uint8_t *row = xb + ((long long)cls * S + r_lo) * rowbytes; // walks down the rows: one addition per load, no multiplication
        const unsigned *pr = ANY ? nullptr : reinterpret_cast<const unsigned *>(row) + u;
        unsigned next[16]; // sixteen rows ahead
        auto one = [&] {
            unsigned v;
            if constexpr (ANY)
                v = word_at(row, u, rowbytes - 4 * u), row += rowbytes;
            else
                v = __ldg(pr), pr += units;
            return v;
        };
        auto load = [&](long long r) {
            if (r + 16 <= r_hi) {
#pragma unroll
                for (int q = 0; q < 16; ++q) next[q] = one();
            } else {
#pragma unroll
                for (int q = 0; q < 16; ++q) next[q] = r + q < r_hi ? one() : 0u;
            }
        };
        load(r_lo);
        for (long long r = r_lo; r < r_hi; r += 16) {
            unsigned v[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = next[q];
            load(r + 16);
            unsigned t2a, t2b, t4a, t4b, t8a, t8b, carry;
            csa(t2a, n[0], n[0], v[0], v[1]);
            csa(t2b, n[0], n[0], v[2], v[3]);
            csa(t4a, n[1], n[1], t2a, t2b);
            csa(t2a, n[0], n[0], v[4], v[5]);
            csa(t2b, n[0], n[0], v[6], v[7]);
            csa(t4b, n[1], n[1], t2a, t2b);
            csa(t8a, n[2], n[2], t4a, t4b);
            csa(t2a, n[0], n[0], v[8], v[9]);
            csa(t2b, n[0], n[0], v[10], v[11]);
            csa(t4a, n[1], n[1], t2a, t2b);
            csa(t2a, n[0], n[0], v[12], v[13]);
            csa(t2b, n[0], n[0], v[14], v[15]);
            csa(t4b, n[1], n[1], t2a, t2b);
            csa(t8b, n[2], n[2], t4a, t4b);
            csa(carry, n[3], n[3], t8a, t8b);
#pragma unroll
            for (int p = 4; p < P; ++p) { // ripple the sixteens into the upper planes
                const unsigned c = n[p] & carry;
                n[p] ^= carry;
                carry = c;
            }
        }
    }
#pragma unroll
    for (int half = 4; half >= 1; half >>= 1) { // warps [half, 2 half) hand their counters to warps [0, half)
        if (wv >= half && wv < 2 * half)
#pragma unroll
            for (int p = 0; p < P; ++p) sm[wv - half][p][lane] = n[p];
        __syncthreads();
        if (wv < half) {
            unsigned carry = 0u;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                unsigned c;
                csa(c, n[p], n[p], sm[wv][p][lane], carry);
                carry = c;
            }
        }
        __syncthreads();
    }
    if (wv == 0)
#pragma unroll
        for (int p = 0; p < P; ++p) sm[0][p][lane] = n[p];
    __syncthreads();
    if (u >= units) return;
#pragma unroll
    for (int p = 0; p < P; ++p) n[p] = sm[0][p][lane] >> (4 * wv);
#pragma unroll
    for (int bit = 0; bit < 4; ++bit) {
        const long long s = u * 32 + 4 * wv + bit;
        int c = 0;
#pragma unroll
        for (int p = 0; p < P; ++p) c += (int)((n[p] >> bit) & 1u) << p;
        if (s >= B) continue;
        if (parts == 1)
            counts[s * k + cls] = c;
        else if (c)
            atomicAdd(counts + s * k + cls, c);
    }
}

constexpr int kTreeCountBlocks = 2; // per SM (655360 trees, 8192 samples: 481 us; three 500, four, which spill, 539)

// The last fused layers and the class sums in one pass: the trees' outputs go into bit-sliced counters as they are produced and are
// neither written nor read again.  Block (2^LG units, part of a class, class): 256 / 2^LG walkers of 2^LG lanes, a unit of 128
// samples each, take every 256 / 2^LG-th tree of the part.  The lowest four planes are in registers and the rest, into which sixteen
// trees carry at most once, in shared memory; then the walkers' counters are added plane by plane.
// Bound by the L2, which the gathered rows come from: 655360 trees of eight rows, 8192 samples 481 us, where the trees alone took 503 and
// the class sums another 117 for the 671 MB of outputs.  The next tree's row numbers are fetched a tree ahead; its rows as well: 564.
template <int M, int LG>
__global__ void __launch_bounds__(256, kTreeCountBlocks) packed_tree_count_kernel(const uint4 *__restrict__ x, const int32_t *__restrict__ leaf,
                                                                                  const uint8_t *__restrict__ ops, int *__restrict__ counts, long long S,
                                                                                  unsigned units, unsigned u_lo, unsigned u_n, long long B, int k, int planes)
{
    constexpr int L = 1 << M, G = L - 1, WALK = 256 >> LG;
    extern __shared__ uint4 plane[]; // [planes][256]
    const int lane = threadIdx.x & ((1 << LG) - 1), walker = threadIdx.x >> LG;
    const int cls = blockIdx.z, part = blockIdx.y, parts = gridDim.y;
    const int hi = (int)(cls * S + S * (part + 1) / parts);
    int t = (int)(cls * S + S * part / parts) + walker;
    const unsigned first = blockIdx.x << LG;
    const uint4 *xu = x + (u_lo + min(first + lane, u_n - 1)); // lanes behind the last unit count it, too, and keep it to themselves
    unsigned n[4][4] = {};
    for (int p = 4; p < planes; ++p) plane[p * 256 + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    int next[L]; // the rows of the next tree
    auto fetch = [&](int j) {
        if (j < hi)
#pragma unroll
            for (int q = 0; q < L / 4; ++q) {
                const int4 r = __ldg(reinterpret_cast<const int4 *>(leaf) + (long long)j * (L / 4) + q);
                next[4 * q] = r.x, next[4 * q + 1] = r.y, next[4 * q + 2] = r.z, next[4 * q + 3] = r.w;
            }
    };
    fetch(t);
    auto tree = [&](unsigned (&out)[4]) { // of tree t, none behind the last
        unsigned v[L][4];
        const int j = t;
        t += WALK;
        if (j < hi) {
#pragma unroll
            for (int q = 0; q < L; ++q) {
                const uint4 r = __ldg(xu + (unsigned)next[q] * units);
                v[q][0] = r.x, v[q][1] = r.y, v[q][2] = r.z, v[q][3] = r.w;
            }
            fetch(t);
            int g = 0;
#pragma unroll
            for (int m = L / 2; m >= 1; m /= 2) {
#pragma unroll
                for (int p = 0; p < m; ++p) {
                    const OpMasks<unsigned> o = op_masks<unsigned>(__ldg(ops + (long long)j * G + g + p));
#pragma unroll
                    for (int w = 0; w < 4; ++w) v[p][w] = op_apply<unsigned>(o, v[2 * p][w], v[2 * p + 1][w]);
                }
                g += m;
            }
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) out[w] = j < hi ? v[0][w] : 0u;
    };
    while (t < hi) {
        unsigned carry[4] = {};
#pragma unroll 1
        for (int q = 0; q < 4 && t < hi; ++q) {
            unsigned a[4], b[4], two[4];
            tree(a), tree(b);
#pragma unroll
            for (int w = 0; w < 4; ++w) csa(two[w], n[0][w], n[0][w], a[w], b[w]);
            tree(a), tree(b);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                unsigned also, four;
                csa(also, n[0][w], n[0][w], a[w], b[w]);
                csa(four, n[1][w], n[1][w], two[w], also);
                const unsigned eight = n[2][w] & four;
                n[2][w] ^= four;
                carry[w] |= n[3][w] & eight;
                n[3][w] ^= eight;
            }
        }
        for (int p = 4; p < planes && (carry[0] | carry[1] | carry[2] | carry[3]); ++p) {
            const uint4 h = plane[p * 256 + threadIdx.x];
            plane[p * 256 + threadIdx.x] = make_uint4(h.x ^ carry[0], h.y ^ carry[1], h.z ^ carry[2], h.w ^ carry[3]);
            carry[0] &= h.x, carry[1] &= h.y, carry[2] &= h.z, carry[3] &= h.w;
        }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
        if (p < planes) plane[p * 256 + threadIdx.x] = make_uint4(n[p][0], n[p][1], n[p][2], n[p][3]);
    __syncthreads();
    // a thread per word of 32 samples and EACH of these: bit p of their sums is the parity of what plane p and the carries hold
    constexpr int WORDS = 4 << LG, EACH = 32 * WORDS / 256, BITS = 9 - LG; // carries stay below WALK = 2^(BITS - 1)
    const int word = threadIdx.x & (WORDS - 1), s0 = threadIdx.x / WORDS * EACH;
    if (first + (word >> 2) >= u_n) return;
    const unsigned *pw = reinterpret_cast<const unsigned *>(plane) + word;
    int count[EACH] = {};
    unsigned sum[BITS] = {};
    for (int p = 0; p < planes + BITS - 1; ++p) {
        if (p < planes)
#pragma unroll 8
            for (int w = 0; w < WALK; ++w) {
                unsigned carry = pw[p * 1024 + w * WORDS];
#pragma unroll
                for (int i = 0; i < BITS; ++i) {
                    const unsigned c = sum[i] & carry;
                    sum[i] ^= carry, carry = c;
                }
            }
#pragma unroll
        for (int i = 0; i < EACH; ++i) count[i] += (int)(sum[0] >> (s0 + i) & 1u) << p;
#pragma unroll
        for (int i = 0; i + 1 < BITS; ++i) sum[i] = sum[i + 1];
        sum[BITS - 1] = 0u;
    }
    const long long s = ((long long)(u_lo + first) * 4 + word) * 32 + s0;
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        if (s + i >= B) break;
        if (parts == 1)
            counts[(s + i) * k + cls] = count[i];
        else if (count[i])
            atomicAdd(counts + (s + i) * k + cls, count[i]);
    }
}

// --------------------------------------------------------------------------- packed ConvLogic block
struct PackedShape {
    int Ci, H, W, C, Ho, Wo, sh, sw, ph, pw;
};

// grid (chunks over (py, px, unit), C); thread <-> (py, px, unit) with unit fastest.
template <typename U>
__global__ void __launch_bounds__(256) packed_convtree_kernel(const U *__restrict__ x, const uint8_t *__restrict__ ops,
                                                              const int32_t *__restrict__ sel, U *__restrict__ y, PackedShape s,
                                                              long long units)
{
    __shared__ OpMasks<U> sm[7];
    __shared__ Tap stap[8];
    const int c = blockIdx.y;
    if (threadIdx.x < 7) sm[threadIdx.x] = op_masks<U>(ops[c * 7 + threadIdx.x]);
    if (threadIdx.x >= 32 && threadIdx.x < 40) stap[threadIdx.x - 32] = unpack_tap(sel[c * 8 + threadIdx.x - 32], s.ph, s.pw);
    __syncthreads();
    const int Hp = s.Ho / 2, Wp = s.Wo / 2;
    const long long total = (long long)Hp * Wp * units;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long u = i % units;
        const int win = (int)(i / units);
        const int py = win / Wp, px = win % Wp;
        U acc = U(0);
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const int oy = 2 * py + (d >> 1), ox = 2 * px + (d & 1);
            U a[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int iy = oy * s.sh + stap[t].dy, ix = ox * s.sw + stap[t].dx;
                a[t] = ((unsigned)iy < (unsigned)s.H && (unsigned)ix < (unsigned)s.W)
                           ? __ldg(x + (((long long)stap[t].ch * s.H + iy) * s.W + ix) * units + u)
                           : U(0);
            }
            const U g0 = op_apply<U>(sm[0], a[0], a[1]), g1 = op_apply<U>(sm[1], a[2], a[3]);
            const U g2 = op_apply<U>(sm[2], a[4], a[5]), g3 = op_apply<U>(sm[3], a[6], a[7]);
            const U t0 = op_apply<U>(sm[4], g0, g1), t1 = op_apply<U>(sm[5], g2, g3);
            acc |= op_apply<U>(sm[6], t0, t1);
        }
        y[((long long)c * Hp * Wp + win) * units + u] = acc;
    }
}

// 16-byte variant for rows that are a multiple of 16 bytes (the usual case: 64-bit words, batches that
// are a multiple of 128).  One thread produces one uint4 (128 samples) of one pooled output.  Everything
// block-uniform (the 7 gates as 32-bit multiplexer masks, the 8 tap offsets) sits in registers; a window
// whose 4 x 8 taps all fall inside the image takes a path without bounds tests; indices are 32-bit.
struct Masks32 {
    unsigned m00, m01, m10, m11;
};
__device__ __forceinline__ unsigned mux32(const Masks32 &m, unsigned a, unsigned b)
{
    const unsigned r1 = (b & m.m11) | (~b & m.m10);
    const unsigned r0 = (b & m.m01) | (~b & m.m00);
    return (a & r1) | (~a & r0);
}
__device__ __forceinline__ uint4 mux128(const Masks32 &m, const uint4 &a, const uint4 &b)
{
    return make_uint4(mux32(m, a.x, b.x), mux32(m, a.y, b.y), mux32(m, a.z, b.z), mux32(m, a.w, b.w));
}

__global__ void __launch_bounds__(256) packed_convtree_v4_kernel(const uint4 *__restrict__ x, const uint8_t *__restrict__ ops,
                                                                 const int32_t *__restrict__ sel, uint4 *__restrict__ y, PackedShape s,
                                                                 int units)
{
    const int c = blockIdx.y;
    Masks32 gm[7];
#pragma unroll
    for (int g = 0; g < 7; ++g) {
        const int op = ops[c * 7 + g];
        gm[g].m00 = (op & 8) ? ~0u : 0u, gm[g].m01 = (op & 4) ? ~0u : 0u, gm[g].m10 = (op & 2) ? ~0u : 0u, gm[g].m11 = (op & 1) ? ~0u : 0u;
    }
    int tb[8], tdy[8], tdx[8]; // tap: element offset (in units) relative to the position, row / col displacement
    int ymin = 0, ymax = 0, xmin = 0, xmax = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const Tap t = unpack_tap(sel[c * 8 + k], s.ph, s.pw);
        tdy[k] = t.dy, tdx[k] = t.dx;
        tb[k] = ((t.ch * s.H + t.dy) * s.W + t.dx) * units;
        ymin = min(ymin, t.dy), ymax = max(ymax, t.dy), xmin = min(xmin, t.dx), xmax = max(xmax, t.dx);
    }
    const int Hp = s.Ho / 2, Wp = s.Wo / 2;
    const int total = Hp * Wp * units;
    const int rowstep = s.sh * s.W * units, colstep = s.sw * units;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int win = i / units, u = i - win * units;
        const int py = win / Wp, px = win - py * Wp;
        const int oy0 = 2 * py * s.sh, ox0 = 2 * px * s.sw;
        const int p0 = (oy0 * s.W + ox0) * units + u; // first position of the window
        const bool interior = oy0 + ymin >= 0 && oy0 + s.sh + ymax < s.H && ox0 + xmin >= 0 && ox0 + s.sw + xmax < s.W;
        uint4 acc = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const int pd = p0 + ((d >> 1) ? rowstep : 0) + ((d & 1) ? colstep : 0);
            uint4 a[8];
            if (interior) {
#pragma unroll
                for (int k = 0; k < 8; ++k) a[k] = __ldg(x + (pd + tb[k]));
            } else {
                const int oy = oy0 + (d >> 1) * s.sh, ox = ox0 + (d & 1) * s.sw;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    a[k] = ((unsigned)(oy + tdy[k]) < (unsigned)s.H && (unsigned)(ox + tdx[k]) < (unsigned)s.W) ? __ldg(x + (pd + tb[k]))
                                                                                                              : make_uint4(0u, 0u, 0u, 0u);
            }
            const uint4 g0 = mux128(gm[0], a[0], a[1]), g1 = mux128(gm[1], a[2], a[3]);
            const uint4 g2 = mux128(gm[2], a[4], a[5]), g3 = mux128(gm[3], a[6], a[7]);
            const uint4 t0 = mux128(gm[4], g0, g1), t1 = mux128(gm[5], g2, g3);
            const uint4 z = mux128(gm[6], t0, t1);
            acc.x |= z.x, acc.y |= z.y, acc.z |= z.z, acc.w |= z.w;
        }
        y[(c * Hp * Wp + win) * units + u] = acc;
    }
}

// ---- slab layout --------------------------------------------------------------------------------
// The [C][H][W][words] layout makes a pixel's words contiguous, which suits the flat layers but forces the
// conv block to gather 32 scattered 16-byte pieces per output piece through L1/L2.  In the slab layout
// [C][U][H][W] of uint4 (U = words/2; one uint4 = 128 samples) the image of one (channel, sample slab) is
// contiguous.  A persistent block walks (output channel, group of UB slabs) items; for each it copies the two
// channel planes the output channel reads into a shared tile (halo zeroed once, columns de-interleaved as in
// the float forward so that window columns are consecutive 16-byte slots) with cp.async into the buffer the
// previous item is not using, so the copy of item i+1 runs under the gate tree of item i.  Every tap is then a
// conflict-free 128-bit shared-memory load.  The per-item bookkeeping (tap offsets, gate ids, the two
// channels) is parsed two items ahead by eight threads into a small shared record, and a gate is applied by a
// block-uniform switch over its id to eight words at a time: one LOP3 per word instead of the three a
// multiplexer with run-time masks needs.  UB * windows-per-image <= 256 threads.  An output channel with a tap
// on a third channel or outside the kernel window (hand-made selections only) takes a global-memory path.
struct SlabShape {
    int Ci, H, W, C, Ho, Wo, ph, pw, kh, kw;
    int U, UB;       // slabs in total / per block
    int PH, pwh;     // padded rows, uint4 slots per column-parity plane of a padded row
    int CS, SS;      // plane stride (one channel slot) and slab stride in the tile, in uint4
    int n_ug, items; // slab groups per channel, items = C * n_ug
    int per_thread;  // copies per thread and channel plane group: ceil(UB*H*W / threads)
};

struct __align__(16) SlabRec {
    int tb0[8], tb1[8]; // tile offsets (bytes) of tap k for the left / right conv column of a window
    int op[8];          // gate ids (7 used)
    int ch[2], nst, all_in_tile;
    int word[8];        // the raw selection words (global path)
};

__device__ __forceinline__ void cp_async16(uint4 *dst_shared, const uint4 *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_shared);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// a[w] = gate(a[w], b[w]) for eight words; `op` is uniform over the block.  Every case is ONE lop3 per word written IN PLACE
// (the "+r" constraint): with plain C expressions the sixteen cases end in different registers and the compiler reconciles
// them with moves at the join -- more moves than logic operations.  Truth-table immediates for (A, B) = (0xF0, 0xCC); the
// third operand is unused (every table is symmetric in it).
// The sixteen cases sit behind ONE indexed branch (brx.idx over a table of the sixteen case labels) instead of the
// compare-and-branch tree a C switch compiles to (13 control instructions per gate, more than its 8 lop3).  `op` is uniform
// over the block, so the branch is declared uniform.  Eight words, in place.
__device__ __forceinline__ void gate_words_brx(int op, unsigned (&a)[8], const unsigned (&b)[8])
{
    asm(
        "{\n\t.reg .u32 gi;\n\tand.b32 gi, %16, 15;\n\t"
        "gtab: .branchtargets G0, G1, G2, G3, G4, G5, G6, G7, G8, G9, G10, G11, G12, G13, G14, G15;\n\t"
        "brx.idx.uni gi, gtab;\n"
        "G0: lop3.b32 %0, %0, %8, %8, 0x00; lop3.b32 %1, %1, %9, %9, 0x00; lop3.b32 %2, %2, %10, %10, 0x00; lop3.b32 %3, %3, %11, %11, 0x00; lop3.b32 %4, %4, %12, %12, 0x00; lop3.b32 %5, %5, %13, %13, 0x00; lop3.b32 %6, %6, %14, %14, 0x00; lop3.b32 %7, %7, %15, %15, 0x00; bra.uni GDONE;\n"
        "G1: lop3.b32 %0, %0, %8, %8, 0xC0; lop3.b32 %1, %1, %9, %9, 0xC0; lop3.b32 %2, %2, %10, %10, 0xC0; lop3.b32 %3, %3, %11, %11, 0xC0; lop3.b32 %4, %4, %12, %12, 0xC0; lop3.b32 %5, %5, %13, %13, 0xC0; lop3.b32 %6, %6, %14, %14, 0xC0; lop3.b32 %7, %7, %15, %15, 0xC0; bra.uni GDONE;\n"
        "G2: lop3.b32 %0, %0, %8, %8, 0x30; lop3.b32 %1, %1, %9, %9, 0x30; lop3.b32 %2, %2, %10, %10, 0x30; lop3.b32 %3, %3, %11, %11, 0x30; lop3.b32 %4, %4, %12, %12, 0x30; lop3.b32 %5, %5, %13, %13, 0x30; lop3.b32 %6, %6, %14, %14, 0x30; lop3.b32 %7, %7, %15, %15, 0x30; bra.uni GDONE;\n"
        "G3: lop3.b32 %0, %0, %8, %8, 0xF0; lop3.b32 %1, %1, %9, %9, 0xF0; lop3.b32 %2, %2, %10, %10, 0xF0; lop3.b32 %3, %3, %11, %11, 0xF0; lop3.b32 %4, %4, %12, %12, 0xF0; lop3.b32 %5, %5, %13, %13, 0xF0; lop3.b32 %6, %6, %14, %14, 0xF0; lop3.b32 %7, %7, %15, %15, 0xF0; bra.uni GDONE;\n"
        "G4: lop3.b32 %0, %0, %8, %8, 0x0C; lop3.b32 %1, %1, %9, %9, 0x0C; lop3.b32 %2, %2, %10, %10, 0x0C; lop3.b32 %3, %3, %11, %11, 0x0C; lop3.b32 %4, %4, %12, %12, 0x0C; lop3.b32 %5, %5, %13, %13, 0x0C; lop3.b32 %6, %6, %14, %14, 0x0C; lop3.b32 %7, %7, %15, %15, 0x0C; bra.uni GDONE;\n"
        "G5: lop3.b32 %0, %0, %8, %8, 0xCC; lop3.b32 %1, %1, %9, %9, 0xCC; lop3.b32 %2, %2, %10, %10, 0xCC; lop3.b32 %3, %3, %11, %11, 0xCC; lop3.b32 %4, %4, %12, %12, 0xCC; lop3.b32 %5, %5, %13, %13, 0xCC; lop3.b32 %6, %6, %14, %14, 0xCC; lop3.b32 %7, %7, %15, %15, 0xCC; bra.uni GDONE;\n"
        "G6: lop3.b32 %0, %0, %8, %8, 0x3C; lop3.b32 %1, %1, %9, %9, 0x3C; lop3.b32 %2, %2, %10, %10, 0x3C; lop3.b32 %3, %3, %11, %11, 0x3C; lop3.b32 %4, %4, %12, %12, 0x3C; lop3.b32 %5, %5, %13, %13, 0x3C; lop3.b32 %6, %6, %14, %14, 0x3C; lop3.b32 %7, %7, %15, %15, 0x3C; bra.uni GDONE;\n"
        "G7: lop3.b32 %0, %0, %8, %8, 0xFC; lop3.b32 %1, %1, %9, %9, 0xFC; lop3.b32 %2, %2, %10, %10, 0xFC; lop3.b32 %3, %3, %11, %11, 0xFC; lop3.b32 %4, %4, %12, %12, 0xFC; lop3.b32 %5, %5, %13, %13, 0xFC; lop3.b32 %6, %6, %14, %14, 0xFC; lop3.b32 %7, %7, %15, %15, 0xFC; bra.uni GDONE;\n"
        "G8: lop3.b32 %0, %0, %8, %8, 0x03; lop3.b32 %1, %1, %9, %9, 0x03; lop3.b32 %2, %2, %10, %10, 0x03; lop3.b32 %3, %3, %11, %11, 0x03; lop3.b32 %4, %4, %12, %12, 0x03; lop3.b32 %5, %5, %13, %13, 0x03; lop3.b32 %6, %6, %14, %14, 0x03; lop3.b32 %7, %7, %15, %15, 0x03; bra.uni GDONE;\n"
        "G9: lop3.b32 %0, %0, %8, %8, 0xC3; lop3.b32 %1, %1, %9, %9, 0xC3; lop3.b32 %2, %2, %10, %10, 0xC3; lop3.b32 %3, %3, %11, %11, 0xC3; lop3.b32 %4, %4, %12, %12, 0xC3; lop3.b32 %5, %5, %13, %13, 0xC3; lop3.b32 %6, %6, %14, %14, 0xC3; lop3.b32 %7, %7, %15, %15, 0xC3; bra.uni GDONE;\n"
        "G10: lop3.b32 %0, %0, %8, %8, 0x33; lop3.b32 %1, %1, %9, %9, 0x33; lop3.b32 %2, %2, %10, %10, 0x33; lop3.b32 %3, %3, %11, %11, 0x33; lop3.b32 %4, %4, %12, %12, 0x33; lop3.b32 %5, %5, %13, %13, 0x33; lop3.b32 %6, %6, %14, %14, 0x33; lop3.b32 %7, %7, %15, %15, 0x33; bra.uni GDONE;\n"
        "G11: lop3.b32 %0, %0, %8, %8, 0xF3; lop3.b32 %1, %1, %9, %9, 0xF3; lop3.b32 %2, %2, %10, %10, 0xF3; lop3.b32 %3, %3, %11, %11, 0xF3; lop3.b32 %4, %4, %12, %12, 0xF3; lop3.b32 %5, %5, %13, %13, 0xF3; lop3.b32 %6, %6, %14, %14, 0xF3; lop3.b32 %7, %7, %15, %15, 0xF3; bra.uni GDONE;\n"
        "G12: lop3.b32 %0, %0, %8, %8, 0x0F; lop3.b32 %1, %1, %9, %9, 0x0F; lop3.b32 %2, %2, %10, %10, 0x0F; lop3.b32 %3, %3, %11, %11, 0x0F; lop3.b32 %4, %4, %12, %12, 0x0F; lop3.b32 %5, %5, %13, %13, 0x0F; lop3.b32 %6, %6, %14, %14, 0x0F; lop3.b32 %7, %7, %15, %15, 0x0F; bra.uni GDONE;\n"
        "G13: lop3.b32 %0, %0, %8, %8, 0xCF; lop3.b32 %1, %1, %9, %9, 0xCF; lop3.b32 %2, %2, %10, %10, 0xCF; lop3.b32 %3, %3, %11, %11, 0xCF; lop3.b32 %4, %4, %12, %12, 0xCF; lop3.b32 %5, %5, %13, %13, 0xCF; lop3.b32 %6, %6, %14, %14, 0xCF; lop3.b32 %7, %7, %15, %15, 0xCF; bra.uni GDONE;\n"
        "G14: lop3.b32 %0, %0, %8, %8, 0x3F; lop3.b32 %1, %1, %9, %9, 0x3F; lop3.b32 %2, %2, %10, %10, 0x3F; lop3.b32 %3, %3, %11, %11, 0x3F; lop3.b32 %4, %4, %12, %12, 0x3F; lop3.b32 %5, %5, %13, %13, 0x3F; lop3.b32 %6, %6, %14, %14, 0x3F; lop3.b32 %7, %7, %15, %15, 0x3F; bra.uni GDONE;\n"
        "G15: lop3.b32 %0, %0, %8, %8, 0xFF; lop3.b32 %1, %1, %9, %9, 0xFF; lop3.b32 %2, %2, %10, %10, 0xFF; lop3.b32 %3, %3, %11, %11, 0xFF; lop3.b32 %4, %4, %12, %12, 0xFF; lop3.b32 %5, %5, %13, %13, 0xFF; lop3.b32 %6, %6, %14, %14, 0xFF; lop3.b32 %7, %7, %15, %15, 0xFF; bra.uni GDONE;\n"
        "GDONE:\n\t}"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7])
        : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(op));
}

// Branch-free form of the same: the gate as a two-level multiplexer over four block-uniform masks, three lop3 per word
// (0xCA = a ? b : c) and no switch.  MUX selects it at compile time.
template <int N>
__device__ __forceinline__ void gate_words_mux(int op, unsigned (&a)[N], const unsigned (&b)[N])
{
    const unsigned m00 = (op & 8) ? ~0u : 0u, m01 = (op & 4) ? ~0u : 0u, m10 = (op & 2) ? ~0u : 0u, m11 = (op & 1) ? ~0u : 0u;
#pragma unroll
    for (int w = 0; w < N; ++w) {
        unsigned r1, r0;
        asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(r1) : "r"(b[w]), "r"(m11), "r"(m10));
        asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(r0) : "r"(b[w]), "r"(m01), "r"(m00));
        asm("lop3.b32 %0, %0, %1, %2, 0xCA;" : "+r"(a[w]) : "r"(r1), "r"(r0));
    }
}
template <bool MUX, int N> __device__ __forceinline__ void gate_apply(int op, unsigned (&a)[N], const unsigned (&b)[N])
{
    if (MUX)
        gate_words_mux<N>(op, a, b);
    else
        gate_words_brx(op, a, b);
}

// two 16-byte shared-memory loads (left and right conv column of a tap) into eight words
__device__ __forceinline__ void lds_pair(unsigned (&d)[8], unsigned addr0, unsigned addr1)
{
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(addr0));
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]) : "r"(addr1));
}

// one pooled output piece straight from global memory, for selections the tile does not cover
__device__ __noinline__ uint4 slab_window_global(const uint4 *__restrict__ xg, const SlabRec &R, const SlabShape &s, int py, int px)
{
    const int HW = s.H * s.W;
    Masks32 gm[7];
    for (int g = 0; g < 7; ++g) {
        const int op = R.op[g];
        gm[g].m00 = (op & 8) ? ~0u : 0u, gm[g].m01 = (op & 4) ? ~0u : 0u, gm[g].m10 = (op & 2) ? ~0u : 0u, gm[g].m11 = (op & 1) ? ~0u : 0u;
    }
    uint4 acc = make_uint4(0u, 0u, 0u, 0u);
    for (int d = 0; d < 4; ++d) {
        uint4 a[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int word = R.word[k];
            const int ch = min((word >> 16) & 0xFFFF, s.Ci - 1);
            const int iy = 2 * py + (d >> 1) + ((word >> 8) & 0xFF) - s.ph, ix = 2 * px + (d & 1) + (word & 0xFF) - s.pw;
            a[k] = ((unsigned)iy < (unsigned)s.H && (unsigned)ix < (unsigned)s.W) ? __ldg(xg + (size_t)ch * s.U * HW + iy * s.W + ix)
                                                                                : make_uint4(0u, 0u, 0u, 0u);
        }
        const uint4 g0 = mux128(gm[0], a[0], a[1]), g1 = mux128(gm[1], a[2], a[3]);
        const uint4 g2 = mux128(gm[2], a[4], a[5]), g3 = mux128(gm[3], a[6], a[7]);
        const uint4 t0 = mux128(gm[4], g0, g1), t1 = mux128(gm[5], g2, g3);
        const uint4 z = mux128(gm[6], t0, t1);
        acc.x |= z.x, acc.y |= z.y, acc.z |= z.z, acc.w |= z.w;
    }
    return acc;
}

// one record per output channel
__global__ void packed_slab_records_kernel(const uint8_t *__restrict__ ops, const int32_t *__restrict__ sel, SlabRec *__restrict__ recs,
                                           SlabShape s)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= s.C) return;
    SlabRec R;
    int ch0 = 0, ch1 = -1;
    bool all = true;
    for (int k = 0; k < 8; ++k) {
        const int w = sel[c * 8 + k];
        const int ch = min((w >> 16) & 0xFFFF, s.Ci - 1), r = (w >> 8) & 0xFF, sx = w & 0xFF;
        if (k == 0) ch0 = ch;
        if (ch1 < 0 && ch != ch0) ch1 = ch;
        all = all && (ch == ch0 || ch == ch1) && r < s.kh && sx < s.kw;
        const int rr = min(r, s.kh - 1), sc = min(sx, s.kw - 1);
        const int base = (ch == ch0 ? 0 : s.CS) + rr * 2 * s.pwh;
        R.tb0[k] = 16 * (base + (sc & 1) * s.pwh + (sc >> 1));
        R.tb1[k] = 16 * (base + ((sc + 1) & 1) * s.pwh + ((sc + 1) >> 1));
        R.word[k] = w;
        R.op[k] = k < 7 ? ops[c * 7 + k] : 0;
    }
    R.ch[0] = ch0, R.ch[1] = ch1 < 0 ? ch0 : ch1, R.nst = ch1 < 0 ? 1 : 2, R.all_in_tile = all;
    recs[c] = R;
}

template <bool MUX>
__global__ void __launch_bounds__(256, 2) packed_convtree_slab_kernel(const uint4 *__restrict__ x,
                                                                      const SlabRec *__restrict__ recs, uint4 *__restrict__ y,
                                                                      SlabShape s)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) SlabRec rec[3];
    uint4 *tile = reinterpret_cast<uint4 *>(smem_raw);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int HW = s.H * s.W;
    const int buf_elems = s.UB * s.SS;
    int *copy_off = reinterpret_cast<int *>(tile + 2 * buf_elems); // [per_thread][nt] tile offsets of a thread's copies
    for (int i = tid; i < 2 * buf_elems; i += nt) tile[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int q = tid; q < s.per_thread * nt; q += nt) {
        const int ub = q / HW, p = q - ub * HW, row = p / s.W, xp = p - row * s.W + s.pw;
        copy_off[q] = ub * s.SS + (row + s.ph) * 2 * s.pwh + (xp & 1) * s.pwh + (xp >> 1);
    }

    // the record of an item's output channel: 9 x 16 bytes from the table the record kernel wrote
    auto fetch_rec = [&](int c, SlabRec &R) {
        for (int j = tid; j < (int)(sizeof(SlabRec) / 16); j += nt) // a block may have fewer threads than pieces
            cp_async16(reinterpret_cast<uint4 *>(&R) + j, reinterpret_cast<const uint4 *>(recs + c) + j);
    };
    // copies of the planes of an item whose record is already visible
    auto stage = [&](int ug, const SlabRec &R, uint4 *dst) {
        const int u0 = ug * s.UB;
        const int n = min(s.UB, s.U - u0) * HW;
        if (!R.all_in_tile) return;
        for (int slot = 0; slot < R.nst; ++slot) {
            const uint4 *src = x + ((size_t)R.ch[slot] * s.U + u0) * HW;
            uint4 *d = dst + slot * s.CS;
            for (int j = 0, q = tid; j < s.per_thread && q < n; ++j, q += nt) cp_async16(d + copy_off[q], src + q);
        }
    };

    const int Hp = s.Ho / 2, Wp = s.Wo / 2, I = Hp * Wp;
    const int ub = tid / I, win = tid - ub * I;
    const int py = win / Wp, px = win - py * Wp;
    const int toff = ub * s.SS + 2 * py * 2 * s.pwh + px;
    const int RS = 2 * s.pwh;

    // items are (slab group ug, output channel c), c fastest: the blocks that run at the same time work on the same
    // few slabs of ALL input channels (a few MB, L2-resident) instead of all slabs of a few channels, so the planes are
    // fetched from DRAM once although every input channel is read by several output channels.  A block takes every
    // gridDim.x-th item and keeps the (c, ug) of its current and next two items by carrying additions instead of dividing.
    const int first = blockIdx.x, stride = gridDim.x;
    const int dug = stride / s.C, dc = stride - dug * s.C;
    auto advance = [&](int &c, int &ug) {
        c += dc, ug += dug;
        if (c >= s.C) c -= s.C, ++ug;
    };
    int ug0 = first / s.C, c0 = first - ug0 * s.C, c1 = c0, ug1 = ug0;
    advance(c1, ug1);
    int c2 = c1, ug2 = ug1;
    advance(c2, ug2);
    if (ug0 < s.n_ug) fetch_rec(c0, rec[0]);
    if (ug1 < s.n_ug) fetch_rec(c1, rec[1]);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads(); // records, copy offsets and halo zeros in place
    if (ug0 < s.n_ug) stage(ug0, rec[0], tile);
    cp_async_commit();
    int cur = 0, r0 = 0; // tile buffer and record slot of the current item
    for (; ug0 < s.n_ug; cur ^= 1, r0 = r0 == 2 ? 0 : r0 + 1) {
        const int r1 = r0 == 2 ? 0 : r0 + 1, r2 = r1 == 2 ? 0 : r1 + 1;
        // one barrier per item: this item's planes and the next item's record have landed, and every thread is
        // done with the previous item, whose tile buffer and whose predecessor's record slot are refilled now
        cp_async_wait<0>();
        __syncthreads();
        if (ug2 < s.n_ug) fetch_rec(c2, rec[r2]);
        if (ug1 < s.n_ug) stage(ug1, rec[r1], tile + (cur ^ 1) * buf_elems);
        cp_async_commit();
        const int c = c0, u0 = ug0 * s.UB;
        c0 = c1, ug0 = ug1, c1 = c2, ug1 = ug2;
        advance(c2, ug2);

        const SlabRec &R = rec[r0];
        if (ub < min(s.UB, s.U - u0)) {
            uint4 out;
            if (R.all_in_tile) {
                // tile offsets in the record are in bytes; a tap's two columns for the two conv rows of the window
                const unsigned t0 = (unsigned)__cvta_generic_to_shared(tile + cur * buf_elems + toff);
                const int4 o0a = *reinterpret_cast<const int4 *>(&R.tb0[0]), o0b = *reinterpret_cast<const int4 *>(&R.tb0[4]);
                const int4 o1a = *reinterpret_cast<const int4 *>(&R.tb1[0]), o1b = *reinterpret_cast<const int4 *>(&R.tb1[4]);
                const int4 opa = *reinterpret_cast<const int4 *>(&R.op[0]), opb = *reinterpret_cast<const int4 *>(&R.op[4]);
                const int o0[8] = {o0a.x, o0a.y, o0a.z, o0a.w, o0b.x, o0b.y, o0b.z, o0b.w};
                const int o1[8] = {o1a.x, o1a.y, o1a.z, o1a.w, o1b.x, o1b.y, o1b.z, o1b.w};
                const int op[7] = {opa.x, opa.y, opa.z, opa.w, opb.x, opb.y, opb.z};
                unsigned acc[4] = {0u, 0u, 0u, 0u};
                // The two conv rows of the window run through ONE copy of the code (the loop is not unrolled): the seven
                // 16-way gate switches are about 150 instructions each, and with fourteen of them the kernel did not fit
                // the instruction cache (stall reason "no instruction").  Inside a row the taps of the next gate are
                // fetched before the current gate's switch, so that the shared-memory latency runs under it (fetching all
                // sixteen loads of a row up front instead was measured slower: 2.49 -> 2.79 ms over the four c4 blocks).
#pragma unroll 1
                for (int dy = 0; dy < 2; ++dy) {
                    const unsigned tn = t0 + dy * RS * 16;
                    unsigned g[4][8], b[4][8];
                    lds_pair(g[0], tn + o0[0], tn + o1[0]);
                    lds_pair(b[0], tn + o0[1], tn + o1[1]);
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        if (p < 3) {
                            lds_pair(g[p + 1], tn + o0[2 * p + 2], tn + o1[2 * p + 2]);
                            lds_pair(b[p + 1], tn + o0[2 * p + 3], tn + o1[2 * p + 3]);
                        }
                        gate_apply<MUX, 8>(op[p], g[p], b[p]);
                    }
                    gate_apply<MUX, 8>(op[4], g[0], g[1]);
                    gate_apply<MUX, 8>(op[5], g[2], g[3]);
                    gate_apply<MUX, 8>(op[6], g[0], g[2]);
#pragma unroll
                    for (int w = 0; w < 4; ++w) acc[w] |= g[0][w] | g[0][w + 4];
                }
                out = make_uint4(acc[0], acc[1], acc[2], acc[3]);
            } else {
                out = slab_window_global(x + (size_t)(u0 + ub) * HW, R, s, py, px);
            }
            y[((size_t)c * s.U + u0 + ub) * I + win] = out;
        }
    }
    cp_async_wait<0>();
}

// rows [F][2U] of 64-bit words  <->  slab [C][U][HW] of uint4, F = C*HW (pure data movement)
__global__ void packed_rows_to_slab_kernel(const uint4 *__restrict__ rows, uint4 *__restrict__ slab, int C, int HW, int U, int to_slab, int side)
{
    const long long total = (long long)C * HW * U;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        // i enumerates the rows layout: ((c*HW + p)*U + u)
        const int u = (int)(i % U);
        const long long cp = i / U;
        int p = (int)(cp % HW);
        const long long c = cp / HW;
        if (side) p = split_position(p, side);
        const long long j = (c * U + u) * HW + p;
        if (to_slab)
            slab[j] = rows[i];
        else
            slab[i] = rows[j]; // here `rows` is the slab tensor and `slab` the rows tensor
    }
}

} // namespace clb

using namespace clb;
using namespace clb_host;

static bool bits_ok(int bits) { return bits == 8 || bits == 16 || bits == 32 || bits == 64; }
static bool aligned_to(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }
static int flat_grid(long long items, int threads)
{
    long long blocks = (items + threads - 1) / threads;
    const long long cap = (long long)sm_count() * 32;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

extern "C" int clb_pack_bits(const uint8_t *t, void *packed, int64_t F, int64_t B, int bits, void *stream)
{
    if (!t || !packed || F < 0 || B < 0 || !bits_ok(bits)) return CLB_ERR_ARG;
    const long long words = (B + bits - 1) / bits, rowbytes = words * (bits / 8);
    if (F == 0 || rowbytes == 0) return CLB_OK;
    CLB_TRACED("pack_bits_kernel", (cudaStream_t)stream, pack_bits_kernel<<<flat_grid(F * rowbytes, 256), 256, 0, (cudaStream_t)stream>>>(t, (uint8_t *)packed, F, B, rowbytes));
    return check_launch();
}

// rows of `rowbytes` bytes (HW == 0) or the slab layout [F / HW][U][HW] of 16-byte units
static int pack_nmajor(const uint8_t *t, void *packed, int64_t N, int64_t F, int64_t rowbytes, int64_t HW, int side, int64_t U, cudaStream_t st)
{
    long long gy = (rowbytes + 31) / 32;
    if (gy > 4096) gy = 4096;
    const dim3 grid((unsigned)((F + 127) / 128), (unsigned)gy);
    const int words = rowbytes % 4 == 0 && aligned_to(packed, 4);
    if (F % 4 == 0 && aligned_to(t, 4))
        CLB_TRACED("pack_bits_nmajor_kernel", st, pack_bits_nmajor_kernel<true><<<grid, 256, 0, st>>>(t, (uint8_t *)packed, N, F, rowbytes, words, (int)HW, side, U));
    else
        CLB_TRACED("pack_bits_nmajor_kernel", st, pack_bits_nmajor_kernel<false><<<grid, 256, 0, st>>>(t, (uint8_t *)packed, N, F, rowbytes, words, (int)HW, side, U));
    return check_launch();
}

extern "C" int clb_pack_bits_nmajor(const uint8_t *t, void *packed, int64_t N, int64_t F, int bits, void *stream)
{
    if (!t || !packed || F < 0 || N < 0 || !bits_ok(bits)) return CLB_ERR_ARG;
    const long long words = (N + bits - 1) / bits, rowbytes = words * (bits / 8);
    if (F == 0 || rowbytes == 0) return CLB_OK;
    return pack_nmajor(t, packed, N, F, rowbytes, 0, 0, 0, (cudaStream_t)stream);
}

int clb_pack_bits_units(const uint8_t *t, void *packed, int64_t N, int64_t F, int64_t U, int64_t HW, int side, Order order, cudaStream_t st)
{
    return pack_nmajor(t, packed, N, F, U * 16, order == kRows ? 0 : HW, order == kSplitSlabs ? side : 0, U, st);
}

int clb_thermometer_pack_units(const void *pixels, int pixels_u8, const float *thresholds, int levels, void *packed, int64_t N, int64_t channels, int64_t HW,
                               int64_t words, int side, Order order, cudaStream_t st)
{
    if (!pixels || !thresholds || !packed || levels <= 0 || N < 0 || channels <= 0 || HW <= 0 || words < 0) return CLB_ERR_ARG;
    const long long P = channels * HW;
    if (P > 0x7fffffff || (long long)levels * P > 0x7fffffffLL * 16) return CLB_ERR_SHAPE;
    const long long need = (N + 63) / 64;
    if (words == 0) words = need;
    if (words < need || words > need + 1) return CLB_ERR_SHAPE; // rows of ceil(N/64) words, or one more to reach an even count
    if (words == 0) return CLB_OK;
    const long long words32 = words * 2;
    const int to_slab = order != kRows;
    if (to_slab && (words32 % 4)) return CLB_ERR_SHAPE; // a slab unit is 128 samples
    if (order != kSplitSlabs) side = 0;
    if (!aligned_to(packed, 16)) return CLB_ERR_ARG;
    const long long gy = (words32 + 7) / 8; // a block writes 8 half-words of every row: all of them are written, bits beyond N as zeros
    if (gy > 65535) return CLB_ERR_SHAPE;
    const ThermoOut o{(unsigned *)packed, (int)P, (int)HW, words32, to_slab, side};
    const int groups = levels > 24 ? 4 : (levels + 7) / 8;
    auto go = [&](auto G) {
        constexpr int g = decltype(G)::value;
        if (pixels_u8) {
            const int vec = P % 16 == 0 && aligned_to(pixels, 16), bytes = 8 * g * 32 * 9 * 4;
            auto launch = [&](auto k, int width) {
                if (ensure_dynamic_smem(k, bytes) != cudaSuccess) return;
                CLB_TRACED("thermometer_pack_kernel", st,
                           k<<<dim3((unsigned)((P + width - 1) / width), (unsigned)gy), 256, bytes, st>>>((const uint8_t *)pixels, thresholds, levels, N, vec, o));
            };
            if ((P + 127) / 128 * gy >= 2LL * sm_count())
                launch(thermometer_pack_bytes_kernel<g, 4>, 128);
            else
                launch(thermometer_pack_bytes_kernel<g, 1>, 32);
        } else {
            const long long blocks = (P + 31) / 32 * gy, passes = (levels + 8 * g - 1) / (8 * g);
            CLB_TRACED("thermometer_pack_kernel", st,
                       thermometer_pack_kernel<g><<<dim3((unsigned)((P + 31) / 32), (unsigned)gy, (unsigned)(blocks < 2LL * sm_count() && passes < 65536 ? passes : 1)), 256, 0, st>>>(
                           (const float *)pixels, thresholds, levels, N, o));
        }
    };
    if (groups == 1)
        go(std::integral_constant<int, 1>{});
    else if (groups == 2)
        go(std::integral_constant<int, 2>{});
    else if (groups == 3)
        go(std::integral_constant<int, 3>{});
    else
        go(std::integral_constant<int, 4>{});
    return check_launch();
}

extern "C" int clb_thermometer_pack(const void *pixels, int pixels_u8, const float *thresholds, int levels, void *packed, int64_t N,
                                    int64_t channels, int64_t HW, int64_t words, int to_slab, void *stream)
{
    return clb_thermometer_pack_units(pixels, pixels_u8, thresholds, levels, packed, N, channels, HW, words, 0, to_slab ? kSlabs : kRows, (cudaStream_t)stream);
}

extern "C" int clb_packed_logic(const void *x, const int64_t *a, const int64_t *b, const uint8_t *ops, void *y, int64_t in_dim,
                                int64_t out_dim, int64_t words, int bits, void *stream)
{
    if (!x || !a || !b || !ops || !y || in_dim <= 0 || out_dim < 0 || words < 0 || !bits_ok(bits)) return CLB_ERR_ARG;
    const long long rowbytes = words * (bits / 8);
    if (out_dim == 0 || rowbytes == 0) return CLB_OK;
    if (rowbytes > 0x7fffffffLL) return CLB_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    auto group = [](long long units) { // log2 of the lanes per neuron
        int lg = 0;
        while (lg < 5 && (1LL << lg) < units) ++lg;
        return lg;
    };
    auto blocks = [&](int lg) { // eight resident blocks per SM walk the neurons
        const long long want = ((out_dim << lg) + 255) / 256, cap = (long long)sm_count() * 8;
        return (unsigned)(want < cap ? want : cap);
    };
    auto go = [&](auto unit, auto rounds) {
        using V = decltype(unit);
        const long long units = rowbytes / (long long)sizeof(V);
        const int lg = group(units);
        CLB_TRACED("packed_logic_kernel", st,
                   packed_logic_kernel<V, decltype(rounds)::value><<<blocks(lg), 256, 0, st>>>((const V *)x, a, b, ops, (V *)y, out_dim, (int)units, lg));
    };
    if (rowbytes % 16 == 0 && aligned_to(x, 16) && aligned_to(y, 16)) {
        go(uint4{}, std::integral_constant<int, 2>{});
    } else if (rowbytes % 8 == 0 && aligned_to(x, 8) && aligned_to(y, 8)) {
        go(uint2{}, std::integral_constant<int, 4>{});
    } else if (rowbytes % 4 == 0 && aligned_to(x, 4) && aligned_to(y, 4)) {
        go(0u, std::integral_constant<int, 5>{});
    } else {
        const int lg = group((rowbytes + 3) / 4);
        CLB_TRACED("packed_logic_bytes_kernel", st,
                   packed_logic_bytes_kernel<<<blocks(lg), 256, 0, st>>>((const uint8_t *)x, a, b, ops, (uint8_t *)y, out_dim, (int)rowbytes, lg));
    }
    return check_launch();
}

// Where no input is left unread, by bytes of output and by how the plain kernel reads a row: in units of 16, 8 or 4 bytes, by as many lanes, up to
// 32, as the power of two that covers it.  us per layer with it / on this walk, layer after layer in one graph:
//   rows of four units or fewer: never (32 bytes, 8 MB 5.7 / 12.4, 40 MB 30 / 54; 64 bytes, 20 MB 10.4 / 14.2; 24 bytes, 12 MB 13.8 / 17.1)
//   4-byte units, fewer than 64                     6 MB  36 bytes 18.1 / 8.6, 100 bytes 14.0 / 6.5, 252 bytes 7.5 / 6.1; at 4 MB 5.7 / 6.0
//   longer rows                                     8.5   500 bytes, 8 MB 6.4 / 6.0, 1252 bytes 6.0 / 6.6; at 12 MB 8.7 / 6.5, 7.8 / 6.5
//   8-byte units, fewer than 32                     6     40 bytes 9.3 / 7.3, 120 bytes 7.0 / 6.5, 248 bytes 6.9 / 7.2; at 4 MB 6.9 / 6.5, 5.2 / 7.0, 5.2 / 6.8
//   longer rows                                     12    504 bytes, 12 MB 7.6 / 6.6, 1256 bytes 6.9 / 6.6, 2008 bytes 6.0 / 6.5; at 8 MB 5.3 / 6.3
//   16-byte units, fewer than 32, no power of two   10    80 bytes, 8 MB 7.2 / 7.5, 12 MB 9.9 / 8.5, 400 bytes 6.3 / 6.7, 8.2 / 6.8
//   other rows                                      18    256 bytes, 12 MB 7.1 / 8.0, 20 MB 10.1 / 8.2, 1024 bytes 5.4 / 6.6, 7.5 / 7.1
extern "C" int clb_packed_path_pays(int64_t in_dim, int64_t out_dim, int64_t words, int bits)
{
    if (in_dim <= 0 || out_dim < in_dim || words <= 0 || !bits_ok(bits)) return 0;
    const int64_t rowbytes = words * (bits / 8), unit = rowbytes % 16 == 0 ? 16 : rowbytes % 8 == 0 ? 8 : 4, units = rowbytes / unit;
    if (rowbytes % 4 || units < 5) return 0;
    const bool idle = unit == 4 ? units < 64 : units < 32 && (units & (units - 1)) != 0;
    const int64_t line = unit == 4 ? (idle ? 6000000 : 8500000) : unit == 8 ? (idle ? 6000000 : 12000000) : (idle ? 10000000 : 18000000);
    return out_dim * rowbytes >= line;
}

extern "C" size_t clb_packed_order_scratch_bytes(int64_t in_dim, int64_t out_dim)
{
    if (in_dim <= 0 || out_dim <= 0 || in_dim > 0x3fffffff || out_dim > 0x3fffffff) return 0;
    return 4 * (size_t)in_dim + 9 * (size_t)out_dim + 4;
}

extern "C" int clb_packed_order(const int64_t *a, const int64_t *b, int32_t *order, void *scratch, size_t scratch_bytes, int64_t in_dim, int64_t out_dim,
                                void *stream)
{
    if (!a || !b || !order || !scratch || in_dim <= 0 || out_dim <= 0) return CLB_ERR_ARG;
    if (in_dim > 0x3fffffff || out_dim > 0x3fffffff) return CLB_ERR_SHAPE;
    if (scratch_bytes < clb_packed_order_scratch_bytes(in_dim, out_dim) || !aligned_to(scratch, 4)) return CLB_ERR_SCRATCH;
    cudaStream_t st = (cudaStream_t)stream;
    int32_t *slot = (int32_t *)scratch, *link = slot + in_dim, *count = link + 2 * out_dim;
    uint8_t *placed = (uint8_t *)(count + 1);
    const int in = (int)in_dim, out = (int)out_dim;
    if (cudaMemsetAsync(slot, 0xff, 4 * (size_t)in_dim + 8 * (size_t)out_dim, st) != cudaSuccess ||
        cudaMemsetAsync(count, 0, 4 + (size_t)out_dim, st) != cudaSuccess)
        return check_launch(0);
    CLB_TRACED("packed_pair_kernel", st, packed_pair_kernel<<<(unsigned)((2 * out_dim + 255) / 256), 256, 0, st>>>(a, b, slot, link, in, out));
    CLB_TRACED("packed_walk_kernel", st, packed_walk_kernel<<<(unsigned)((2 * out_dim + 127) / 128), 128, 0, st>>>(link, order, placed, count, out));
    CLB_TRACED("packed_rest_kernel", st, packed_rest_kernel<<<(unsigned)((out_dim + 255) / 256), 256, 0, st>>>(order, placed, count, out));
    return check_launch(3);
}

// order: step 1 an order (with a and b), 4 records
static int packed_path(const void *x, const void *rec, int step, const int64_t *a, const int64_t *b, const uint8_t *ops, void *y, int64_t in_dim,
                       int64_t out_dim, int64_t words, int bits, void *stream)
{
    if (!x || !rec || (step == 1 && (!a || !b)) || !ops || !y || in_dim <= 0 || out_dim < 0 || words < 0 || !bits_ok(bits)) return CLB_ERR_ARG;
    const long long rowbytes = words * (bits / 8);
    if (out_dim == 0 || rowbytes == 0) return CLB_OK;
    if (rowbytes % 4 || rowbytes > 0x7fffffffLL || in_dim > 0x3fffffff || out_dim > 0x3fffffff || !aligned_to(rec, 4 * (size_t)step) || !aligned_to(x, 4) || !aligned_to(y, 4))
        return CLB_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    auto go = [&](auto unit, auto per, auto lanes) {
        using V = decltype(unit);
        constexpr int R = decltype(per)::value, LG = decltype(lanes)::value;
        const long long units = rowbytes / (long long)sizeof(V), cols = (units + (R << LG) - 1) / (R << LG), groups = (long long)sm_count() * kPathBlocks * 256 >> LG;
        long long ranges = groups / cols; // one wave of resident blocks, eight positions per group at least
        if (ranges > out_dim / 8) ranges = out_dim / 8;
        if (ranges < 1) ranges = 1;
        if (((ranges * cols) << LG) + 255 > 0x7fffffffLL) return (int)CLB_ERR_SHAPE;
        CLB_TRACED("packed_path_kernel", st,
                   packed_path_kernel<V, R, LG><<<(unsigned)(((ranges * cols << LG) + 255) / 256), 256, 0, st>>>((const V *)x, (const int32_t *)rec, step, a, b, ops, (V *)y,
                                                                                                              (int)out_dim, (int)units, (int)cols, (int)ranges));
        return check_launch();
    };
    // a warp takes 2 to 5 (of 8 bytes 4, of 16 bytes 2) units per lane, whichever leaves the fewest lanes idle; short rows a quarter of a warp and two
    auto rows = [&](auto unit) {
        using V = decltype(unit);
        const long long units = rowbytes / (long long)sizeof(V);
        constexpr int most = sizeof(V) == 16 ? 2 : sizeof(V) == 8 ? 4 : 5;
        if (units <= 32) return go(unit, std::integral_constant<int, 2>{}, std::integral_constant<int, 3>{});
        int best = 2;
        long long idle = -1;
        for (int r = most; r >= 2; --r) {
            const long long over = (units + 32 * r - 1) / (32 * r) * (32 * r);
            if (idle < 0 || over < idle) best = r, idle = over;
        }
        const auto warp = std::integral_constant<int, 5>{};
        if constexpr (most >= 5)
            if (best == 5) return go(unit, std::integral_constant<int, 5>{}, warp);
        if constexpr (most >= 4) {
            if (best == 4) return go(unit, std::integral_constant<int, 4>{}, warp);
            if (best == 3) return go(unit, std::integral_constant<int, 3>{}, warp);
        }
        return go(unit, std::integral_constant<int, 2>{}, warp);
    };
    if (rowbytes % 16 == 0 && aligned_to(x, 16) && aligned_to(y, 16)) return rows(uint4{});
    if (rowbytes % 8 == 0 && aligned_to(x, 8) && aligned_to(y, 8)) return rows(uint2{});
    return rows(0u);
}

extern "C" int clb_packed_path(const void *x, const void *rec, const uint8_t *ops, void *y, int64_t in_dim, int64_t out_dim, int64_t words, int bits,
                               void *stream)
{
    return packed_path(x, rec, 4, nullptr, nullptr, ops, y, in_dim, out_dim, words, bits, stream);
}

extern "C" int clb_packed_walk(const void *x, const int64_t *a, const int64_t *b, const int32_t *order, const uint8_t *ops, void *y, int64_t in_dim,
                               int64_t out_dim, int64_t words, int bits, void *stream)
{
    return packed_path(x, order, 1, a, b, ops, y, in_dim, out_dim, words, bits, stream);
}

// The leaves are gathered from all over the input: when it is larger than about three quarters of the 126 MB L2, the
// rows are walked in pieces (a range of 16-byte units = a range of samples at a time), so that the piece of the input in
// use stays cached.  Measured on a 134 MB input: 0.64 ms in one piece, 0.50 in two or four, 0.56 in eight.
static long long tree_pieces(long long in_dim, long long units)
{
    long long pieces = 1;
    while (in_dim * units * 16 / pieces > (96LL << 20) && units % (pieces * 2) == 0 && units / (pieces * 2) >= 8) pieces *= 2;
    return pieces;
}

extern "C" int clb_packed_tree(const void *x, const int32_t *leaf, const uint8_t *ops, void *y, int64_t in_dim, int64_t out_dim, int levels,
                               int64_t words, int bits, void *stream)
{
    if (!x || !leaf || !ops || !y || in_dim <= 0 || out_dim < 0 || words < 0 || !bits_ok(bits) || (levels != 2 && levels != 3))
        return CLB_ERR_ARG;
    if (in_dim > 0x7fffffffLL) return CLB_ERR_SHAPE;
    const long long rowbytes = words * (bits / 8);
    if (out_dim == 0 || rowbytes == 0) return CLB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (rowbytes % 16 == 0 && aligned_to(x, 16) && aligned_to(y, 16)) {
        const long long units = rowbytes / 16;
        const long long pieces = tree_pieces(in_dim, units);
        const long long u_n = units / pieces;
        const int grid = flat_grid(out_dim * u_n, 256);
        for (long long pc = 0; pc < pieces; ++pc) {
            if (levels == 2)
                CLB_TRACED("packed_tree_kernel", st,
                           packed_tree_kernel<uint4, 2, long long><<<grid, 256, 0, st>>>((const uint4 *)x, leaf, ops, (uint4 *)y, out_dim, units, pc * u_n, u_n));
            else
                if (in_dim * units < 0xffffffffLL)
                    CLB_TRACED("packed_tree_kernel", st,
                               packed_tree_kernel<uint4, 3, unsigned><<<grid, 256, 0, st>>>((const uint4 *)x, leaf, ops, (uint4 *)y, out_dim, units, pc * u_n, u_n));
                else
                    CLB_TRACED("packed_tree_kernel", st,
                               packed_tree_kernel<uint4, 3, long long><<<grid, 256, 0, st>>>((const uint4 *)x, leaf, ops, (uint4 *)y, out_dim, units, pc * u_n, u_n));
        }
        return check_launch((int)pieces);
    } else if (rowbytes % 8 == 0 && aligned_to(x, 8) && aligned_to(y, 8)) {
        const long long units = rowbytes / 8;
        const int grid = flat_grid(out_dim * units, 256);
        if (levels == 2)
            CLB_TRACED("packed_tree_kernel", st, packed_tree_kernel<uint2, 2, long long><<<grid, 256, 0, st>>>((const uint2 *)x, leaf, ops, (uint2 *)y, out_dim, units, 0, units));
        else
            CLB_TRACED("packed_tree_kernel", st, packed_tree_kernel<uint2, 3, long long><<<grid, 256, 0, st>>>((const uint2 *)x, leaf, ops, (uint2 *)y, out_dim, units, 0, units));
    } else {
        return CLB_ERR_SHAPE; // rows of 64-bit words only
    }
    return check_launch();
}

int clb_packed_tree_count(const void *x, const int32_t *leaf, const uint8_t *ops, int32_t *counts, int64_t in_dim, int64_t out_dim, int levels, int64_t U,
                          int64_t B, int k, cudaStream_t st)
{
    if (k <= 0 || k > 65535 || out_dim % k || out_dim > 0x7fffff00LL || out_dim <= 0 || B <= 0 || in_dim * U >= 0xffffffffLL) return CLB_ERR_SHAPE;
    if ((levels != 2 && levels != 3) || !aligned_to(x, 16) || !aligned_to(leaf, 16)) return CLB_ERR_SHAPE;
    const long long pieces = tree_pieces(in_dim, U), u_n = U / pieces, S = out_dim / k;
    // lanes of a walker: as many as leave fewest idle, of two the more
    int lg = 5;
    for (int g = 4; g >= 3; --g)
        if (((u_n + (1 << g) - 1) >> g << g) < ((u_n + (1 << lg) - 1) >> lg << lg)) lg = g;
    const long long chunks = (u_n + (1 << lg) - 1) >> lg, walkers = 256 >> lg;
    // Adding up the walkers' counters takes 10 us or so and idle lanes read rows, too; the outputs of small layers stay in the L2 anyway.
    // us in one pass / apart: 10.5 MB of outputs 22 / 20, 21 MB 28 / 30 and 27 / 33, 42 MB 43 / 46, 84 MB 72 / 84, 671 MB 483 / 622;
    // 34 units on 40 lanes 36 / 33, 11 on 16 (115 MB) 127 / 122.
    if (out_dim * U * 16 < (20LL << 20) || 16 * u_n < 15 * (chunks << lg)) return CLB_ERR_SHAPE;
    // Parts of a class, of at least 16 trees per walker and no more than 2^12 - 1: those of the least time, in trees of a walker, when a wave of blocks
    // takes a part's trees and the adding up, and one with a block per SM at most 0.6 of that; one wave more for a twentieth at least.  (As many as fit one wave:
    // 150 classes of 2000 trees, 4096 samples have 150 blocks for 296 places, 147 us apart, 201 so, 138 in five parts; 10 of 2000, 30720 81 / 106 / 82.)
    const long long slots = (long long)kTreeCountBlocks * sm_count();
    const double adding = 3.0 + 0.4 * (double)walkers;
    const long long least = S / (walkers * 4000) + 1, limit = std::max(least, std::min(S / (16 * walkers), 1024LL));
    long long parts = least, full = -1;
    double cost = -1.0;
    for (long long p = least; p <= limit; ++p) {
        const long long blocks = chunks * k * p, rest = blocks % slots, waves = (blocks + slots - 1) / slots;
        const double c = ((double)(blocks / slots) + (rest == 0 ? 0.0 : 2 * rest <= slots ? 0.6 : 1.0)) * ((double)S / (double)(p * walkers) + adding);
        if (cost < 0.0 || c < (waves == full ? 1.0 : 0.95) * cost) cost = c, parts = p, full = waves;
    }
    // Many classes leave no choice of parts: apart where more than a third of that time is idle (50 classes of 500 trees, 12288 samples 48 / 63 us, 200 of
    // 500, 3000 samples 48 / 56; 100 of 500, 16384 samples, which fill it, 111 / 93).
    if (k >= 32 && (double)(chunks * k) / (double)slots * (double)S / (double)walkers < 0.62 * cost) return CLB_ERR_SHAPE;
    if (parts > 65535 || chunks > 0x7fffffffLL) return CLB_ERR_SHAPE;
    const long long most = (S / parts + 1 + walkers - 1) / walkers;
    int planes = 4;
    while (most >> planes) ++planes;
    if (parts > 1 && cudaMemsetAsync(counts, 0, (size_t)B * k * sizeof(int32_t), st) != cudaSuccess) return check_launch(0);
    const dim3 grid((unsigned)chunks, (unsigned)parts, (unsigned)k);
    auto go = [&](auto kern) {
        for (long long pc = 0; pc < pieces; ++pc)
            CLB_TRACED("packed_tree_count_kernel", st,
                       kern<<<grid, 256, planes * 4096, st>>>((const uint4 *)x, leaf, ops, counts, S, (unsigned)U, (unsigned)(pc * u_n), (unsigned)u_n, B, k, planes));
    };
    if (levels == 2)
        lg == 5 ? go(packed_tree_count_kernel<2, 5>) : lg == 4 ? go(packed_tree_count_kernel<2, 4>) : go(packed_tree_count_kernel<2, 3>);
    else
        lg == 5 ? go(packed_tree_count_kernel<3, 5>) : lg == 4 ? go(packed_tree_count_kernel<3, 4>) : go(packed_tree_count_kernel<3, 3>);
    return check_launch((int)pieces);
}

// Rows of rowbytes bytes of which B samples count (whatever the bits behind them).
static int group_popcount(const void *x, int32_t *counts, int64_t F, long long rowbytes, long long B, int k, cudaStream_t st)
{
    if (B <= 0) return CLB_OK;
    const long long S = F / k;
    const bool any = rowbytes % 4 != 0 || !aligned_to(x, 4);
    const long long ublocks = (rowbytes + 127) / 128;
    // parts of a class: three blocks per SM in all, at least 16 rows per warp.  All of them run at once (a second, short wave
    // cost 30 of 150 us for 335 MB), and no more parts than that, as each adds its counts with atomics.
    long long parts = 3LL * sm_count() / (ublocks * k);
    if (parts > S / 128) parts = S / 128;
    if (parts < 1) parts = 1;
    if (ublocks > 0x7fffffffLL || k > 65535) return CLB_ERR_SHAPE;
    if (parts > 1 && cudaMemsetAsync(counts, 0, (size_t)B * k * sizeof(int32_t), st) != cudaSuccess) return check_launch(0);
    const dim3 grid((unsigned)ublocks, (unsigned)parts, (unsigned)k);
    const long long rows = S / parts + 1; // of a block: what its counters have to hold
    auto launch = [&](auto kernel) {
        CLB_TRACED("group_popcount_kernel", st, kernel<<<grid, 256, 0, st>>>((const uint8_t *)x, counts, S, rowbytes, B, k));
    };
    auto go = [&](auto planes) {
        constexpr int P = decltype(planes)::value;
        any ? launch(group_popcount_kernel<P, true>) : launch(group_popcount_kernel<P, false>);
    };
    if (rows < (1LL << 14))
        go(std::integral_constant<int, 10>{});
    else if (rows < (1LL << 20))
        go(std::integral_constant<int, 16>{});
    else
        go(std::integral_constant<int, 27>{});
    return check_launch();
}

extern "C" int clb_group_popcount(const void *x, int32_t *counts, int64_t F, int64_t words, int bits, int pad_len, int k, void *stream)
{
    if (!x || !counts || F < 0 || words < 0 || !bits_ok(bits) || k <= 0 || pad_len < 0 || pad_len >= bits) return CLB_ERR_ARG;
    if (F % k) return CLB_ERR_SHAPE;
    return group_popcount(x, counts, F, words * (bits / 8), words * bits - pad_len, k, (cudaStream_t)stream);
}
int clb_group_popcount_units(const void *x, int32_t *counts, int64_t F, int64_t U, int64_t B, int k, cudaStream_t st)
{
    return group_popcount(x, counts, F, U * 16, B, k, st);
}

extern "C" int clb_packed_convtree(const void *x, const uint8_t *ops, const int32_t *sel, void *y, int Ci, int H, int W, int C,
                                   int sh, int sw, int ph, int pw, int kh, int kw, int64_t words, int bits, void *stream)
{
    if (!conv_args_ok(1, Ci, H, W, C, sh, sw, ph, pw, kh, kw) || !x || !ops || !sel || !y || words < 0 || !bits_ok(bits))
        return CLB_ERR_ARG;
    PackedShape s{Ci, H, W, C, conv_out(H, ph, kh, sh), conv_out(W, pw, kw, sw), sh, sw, ph, pw};
    if (s.Ho <= 0 || s.Wo <= 0) return CLB_ERR_SHAPE;
    if ((s.Ho & 1) || (s.Wo & 1)) return CLB_ERR_ODD_OUTPUT;
    if (C > 65535) return CLB_ERR_SHAPE;
    const long long rowbytes = words * (bits / 8);
    if (C == 0 || rowbytes == 0) return CLB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const long long wins = (long long)(s.Ho / 2) * (s.Wo / 2);
    const long long in_units16 = (long long)Ci * H * W * (rowbytes / 16), out_units16 = (long long)C * wins * (rowbytes / 16);
    if (rowbytes % 16 == 0 && aligned_to(x, 16) && aligned_to(y, 16) && in_units16 < (1LL << 30) && out_units16 < (1LL << 30)) {
        const int units = (int)(rowbytes / 16);
        long long gx = (wins * units + 255) / 256;
        const long long cap = ((long long)sm_count() * 32 + C - 1) / C;
        if (gx > cap) gx = cap;
        dim3 grid((unsigned)(gx < 1 ? 1 : gx), C);
        CLB_TRACED("packed_convtree_v4_kernel", st, packed_convtree_v4_kernel<<<grid, 256, 0, st>>>((const uint4 *)x, ops, sel, (uint4 *)y, s, units));
    } else if (rowbytes % 8 == 0 && aligned_to(x, 8) && aligned_to(y, 8)) {
        const long long units = rowbytes / 8;
        long long gx = (wins * units + 255) / 256;
        const long long cap = ((long long)sm_count() * 32 + C - 1) / C;
        if (gx > cap) gx = cap;
        dim3 grid((unsigned)(gx < 1 ? 1 : gx), C);
        CLB_TRACED("packed_convtree_kernel", st, packed_convtree_kernel<unsigned long long><<<grid, 256, 0, st>>>((const unsigned long long *)x, ops, sel,
                                                                         (unsigned long long *)y, s, units));
    } else {
        long long gx = (wins * rowbytes + 255) / 256;
        const long long cap = ((long long)sm_count() * 32 + C - 1) / C;
        if (gx > cap) gx = cap;
        dim3 grid((unsigned)(gx < 1 ? 1 : gx), C);
        CLB_TRACED("packed_convtree_kernel", st, packed_convtree_kernel<uint8_t><<<grid, 256, 0, st>>>((const uint8_t *)x, ops, sel, (uint8_t *)y, s, rowbytes));
    }
    return check_launch();
}

static int packed_layout(const void *src, void *dst, int64_t C, int64_t HW, int64_t U, int to_slab, int side, cudaStream_t st)
{
    if (!src || !dst || C < 0 || HW < 0 || U < 0) return CLB_ERR_ARG;
    if (!aligned_to(src, 16) || !aligned_to(dst, 16)) return CLB_ERR_ARG;
    if (C > 0x7fffffff || HW > 0x7fffffff || U > 0x7fffffff) return CLB_ERR_SHAPE;
    const long long total = C * HW * U;
    if (total == 0) return CLB_OK;
    CLB_TRACED("packed_rows_to_slab_kernel", st, packed_rows_to_slab_kernel<<<flat_grid(total, 256), 256, 0, st>>>((const uint4 *)src, (uint4 *)dst, (int)C, (int)HW,
                                                                                        (int)U, to_slab, side));
    return check_launch();
}
extern "C" int clb_packed_layout(const void *src, void *dst, int64_t C, int64_t HW, int64_t U, int to_slab, void *stream)
{
    return packed_layout(src, dst, C, HW, U, to_slab, 0, (cudaStream_t)stream);
}
int clb_packed_rows_to_slabs(const void *rows, void *slabs, int64_t C, int64_t HW, int64_t U, int side, Order order, cudaStream_t st)
{
    return packed_layout(rows, slabs, C, HW, U, 1, order == kSplitSlabs ? side : 0, st);
}

extern "C" int64_t clb_packed_convtree_slab_scratch_bytes(int C)
{
    if (C < 0) return 0;
    const int64_t a = (int64_t)C * (int64_t)sizeof(SlabRec), b = (int64_t)clb_slab3_record_bytes(C);
    return a > b ? a : b;
}

extern "C" int clb_packed_convtree_slab(const void *x, const uint8_t *ops, const int32_t *sel, void *y, void *scratch, int Ci, int H,
                                        int W, int C, int sh, int sw, int ph, int pw, int kh, int kw, int64_t U, void *stream)
{
    if (!conv_args_ok(1, Ci, H, W, C, sh, sw, ph, pw, kh, kw) || !x || !ops || !sel || !y || U < 0) return CLB_ERR_ARG;
    if (!aligned_to(x, 16) || !aligned_to(y, 16) || (C > 0 && (!scratch || !aligned_to(scratch, 16)))) return CLB_ERR_ARG;
    if (sh != 1 || sw != 1) return CLB_ERR_SHAPE; // the rows layout serves other strides
    SlabShape s;
    s.Ci = Ci, s.H = H, s.W = W, s.C = C, s.ph = ph, s.pw = pw, s.kh = kh, s.kw = kw;
    s.Ho = conv_out(H, ph, kh, 1), s.Wo = conv_out(W, pw, kw, 1);
    if (s.Ho <= 0 || s.Wo <= 0) return CLB_ERR_SHAPE;
    if ((s.Ho & 1) || (s.Wo & 1)) return CLB_ERR_ODD_OUTPUT;
    const int I = (s.Ho / 2) * (s.Wo / 2);
    if (C > 65535 || I > 256 || U > 0x7fffffff) return CLB_ERR_SHAPE;
    if ((long long)Ci * U * H * W >= (1LL << 31) || (long long)C * U * I >= (1LL << 31)) return CLB_ERR_SHAPE;
    if (C == 0 || U == 0) return CLB_OK;
    if (clb_slab3_covers(H, W, sh, sw, ph, pw, kh, kw)) { // the stacks' own geometry
        const int rc = clb_slab3_records(ops, sel, nullptr, scratch, Ci, H, C, (cudaStream_t)stream);
        return rc != CLB_OK ? rc : clb_slab3_block(x, scratch, y, Ci, H, C, U, kSlabs, kSlabs, (cudaStream_t)stream);
    }
    s.U = (int)U;
    s.UB = 256 / I;
    if (s.UB > s.U) s.UB = s.U;
    s.PH = H + 2 * ph;
    s.pwh = (W + 2 * pw + 1) / 2;
    s.CS = s.PH * 2 * s.pwh;
    s.SS = 2 * s.CS;
    auto smem_of = [&](int ub) { // two buffers + copy offsets
        const int th = ub * I;
        return 2 * (size_t)ub * s.SS * 16 + (size_t)((ub * H * W + th - 1) / th) * th * 4;
    };
    while (s.UB > 1 && smem_of(s.UB) > 110 * 1024) s.UB = (s.UB + 1) / 2; // small images: the halo doubles the tile; keep two blocks per SM
    const int threads = s.UB * I;
    s.per_thread = (s.UB * H * W + threads - 1) / threads;
    const size_t smem = smem_of(s.UB);
    if (smem > 200 * 1024) return CLB_ERR_SHAPE;
    s.n_ug = (s.U + s.UB - 1) / s.UB;
    s.items = C * s.n_ug;
    const bool mux = tune_get(CLB_TUNE_SLAB_MUX) != 0;
    auto k = mux ? packed_convtree_slab_kernel<true> : packed_convtree_slab_kernel<false>;
    if (clb_host::ensure_dynamic_smem(k, (int)smem) != cudaSuccess) return check_launch(0);
    int bps = (int)((227 * 1024) / (smem + 1024));
    const int by_regs = 512 / threads < 2 ? 2 : (512 / threads > 8 ? 8 : 512 / threads); // 112 registers per thread
    if (bps > by_regs) bps = by_regs;
    if (bps < 1) bps = 1;
    int grid = sm_count() * bps;
    if (grid > s.items) grid = s.items;
    CLB_TRACED("packed_slab_records_kernel", (cudaStream_t)stream, packed_slab_records_kernel<<<(C + 127) / 128, 128, 0, (cudaStream_t)stream>>>(ops, sel, (SlabRec *)scratch, s));
    CLB_TRACED("packed_convtree_slab_kernel", (cudaStream_t)stream, k<<<grid, threads, smem, (cudaStream_t)stream>>>((const uint4 *)x, (const SlabRec *)scratch, (uint4 *)y, s));
    return check_launch();
}

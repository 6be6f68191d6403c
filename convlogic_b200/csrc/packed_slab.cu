// Packed ConvLogic block on the slab layout for the stacks' own geometry: 3x3 window, padding 1, stride 1, square images of 32,
// 16, 8 or 4 pixels (other shapes: packed.cu).
//
// An item is (output channel, group of UB slabs); a persistent block copies the two channel planes that the output channel reads
// of the group's slabs into shared memory with cp.async and evaluates the gates from there.  What bounds it is the shared-memory
// pipe: per window and 128 samples 32 taps of 16 bytes are read and 8 units written, 200 of its cycles per warp when everything
// is conflict-free, twice that when the copies are not.  Hence
//   * the activations travel between the blocks with a row's even columns before its odd ones, as the tile holds them: a
//     copy from row-major pixels scatters neighbouring lanes' units, and then every lane of a cp.async takes a pass of its own
//     (k = 1024, 8192 samples, 32x32 images: 702 us with such copies, 445 without; a block with run-time geometry and
//     four words per gate took 665);
//   * a gate is one lop3 per word whose third operand is the output inversion, so that the sixteen gates are EIGHT cases behind one
//     indexed branch that a warp takes together;
//   * eight warps per scheduler at 64 registers a thread, one buffer per block, the copies of one block
//     running while the SM's others compute (two buffers and half the blocks measured 5 to 30 % slower), and blocks as small as a
//     slab or, for small images, a warp, so that few threads wait at an item's two barriers (k = 1024, 8192 samples, us with
//     blocks of 256, 256, 128 threads / of 64, 32, 32: 16x16 images 448 / 378, 8x8 479 / 430, 4x4 252 / 237; two warps for 8x8: 420, but
//     with 100 samples, a block's only slab, 24 against 17);
//   * the tap records (offsets, gate codes) are laid out once per network and arrive two items ahead, in an order in which
//     neighbours share an input channel (clb_slab3_order), whose plane then stays in the tile: half of the copies, 443, 464, 521, 275 us for
//     the four blocks in the channels' own order, 411, 452, 483, 254 in that one.
//
// Tile of one slab and channel: (S + 1) rows of units of 16 bytes (128 samples of a pixel).  A padded row holds its odd columns,
// one zero unit, and its even columns: the zero unit is the right halo of the odd columns and the left halo of the even ones,
// and a zero row is both the lower halo of one slab and the upper halo of the next.  The columns a conv position reads are then
// consecutive units over the lanes of a row, and the pitches of the small images are such that the lanes of each quarter-warp
// hit eight different 16-byte bank groups.
#include "clb_common.cuh"
#include "clb_slab.cuh"

#include <vector>

namespace clb {
namespace slab {

template <int S> struct Geo {
    static constexpr int H2 = S / 2, I = H2 * H2;                // pooled side, outputs (threads) per slab
    static constexpr int THREADS = S == 32 ? 256 : S == 16 ? 64 : 32;
    static constexpr int UB = THREADS / I;                       // slabs of a block
    static constexpr int PITCH = S == 8 ? 10 : S + 1;            // units of a padded row
    static constexpr int SLAB = S == 4 ? 28 : (S + 1) * PITCH;   // units from one slab to the next
    static constexpr int HW = S * S;
    static constexpr int ROW_BYTES = PITCH * 16;
    static constexpr int PLANE_BYTES = (UB * SLAB + PITCH) * 16; // the last slab's lower halo row follows it
};
template <int S> __host__ __device__ constexpr int column(int c) { return (c & 1) ? (c - 1) / 2 : S / 2 + c / 2; } // unit of padded column c

// tile bytes from unit p of the first slab to unit p + i * THREADS of the group
template <int S, typename G> __host__ __device__ constexpr int unit_step(int i)
{
    return 16 * (i * G::THREADS / G::HW * G::SLAB + i * G::THREADS % G::HW / S * G::PITCH);
}

__device__ __forceinline__ void cp_async16(unsigned dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int DST, int SRC> __device__ __forceinline__ void cp_async16_at(unsigned dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0+%2], [%1+%3], 16;" ::"r"(dst), "l"(src), "n"(DST), "n"(SRC) : "memory");
}

// a[w] = gate(a[w], b[w]) ^ inv for eight words.  code: gate ids 0..7 (a gate and its complement share a case), uniform over the
// block; inv: all ones for the complement.  Truth tables for (A, B, C) = (0xF0, 0xCC, 0xAA), the gate XOR C.
__device__ __forceinline__ void gate8(int code, unsigned inv, unsigned (&a)[8], const unsigned (&b)[8])
{
#define CLB_L(W, B, T) "lop3.b32 %" #W ", %" #W ", %" #B ", %16, " #T "; "
#define CLB_CASE(N, T)                                                                                                                      \
    "G" #N ": " CLB_L(0, 8, T) CLB_L(1, 9, T) CLB_L(2, 10, T) CLB_L(3, 11, T) CLB_L(4, 12, T) CLB_L(5, 13, T) CLB_L(6, 14, T) CLB_L(7, 15, T) \
    "bra.uni GDONE;\n"
    asm("{\n\tgtab: .branchtargets G0, G1, G2, G3, G4, G5, G6, G7;\n\tbrx.idx.uni %17, gtab;\n" CLB_CASE(0, 0xAA) CLB_CASE(1, 0x6A) CLB_CASE(2, 0x9A)
            CLB_CASE(3, 0x5A) CLB_CASE(4, 0xA6) CLB_CASE(5, 0x66) CLB_CASE(6, 0x96) CLB_CASE(7, 0x56) "GDONE:\n\t}"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7])
        : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(inv), "r"(code));
#undef CLB_CASE
#undef CLB_L
}

__device__ __forceinline__ void lds128(unsigned *d, unsigned addr)
{
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(addr));
}
// taps 2i and 2i + 1 of one conv row: words 0-3 / 4-7 left / right column of the window
__device__ __forceinline__ void taps(unsigned (&a)[8], unsigned (&b)[8], const Rec &R, int i, unsigned at)
{
    const int4 o = R.off[i];
    lds128(a, at + o.x), lds128(a + 4, at + o.y), lds128(b, at + o.z), lds128(b + 4, at + o.w);
}

struct Shape {
    int Ci, C, U, n_ug;
    int in, out;               // Order
    int runs, per_run, longer; // runs of items, items of a run, runs that have one more
};

// one pooled output straight from global memory, for selections the tile does not cover
template <int S> __device__ __noinline__ uint4 window_global(const uint4 *__restrict__ xg, const Rec &R, const Shape &s, int py, int px)
{
    uint4 acc = make_uint4(0u, 0u, 0u, 0u);
    for (int d = 0; d < 4; ++d) {
        unsigned v[8][4];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int word = R.word[k], ch = min((word >> 16) & 0xFFFF, s.Ci - 1);
            const int iy = 2 * py + (d >> 1) + ((word >> 8) & 0xFF) - 1, ix = 2 * px + (d & 1) + (word & 0xFF) - 1;
            uint4 q = make_uint4(0u, 0u, 0u, 0u);
            if ((unsigned)iy < (unsigned)S && (unsigned)ix < (unsigned)S)
                q = __ldg(xg + (size_t)ch * s.U * (S * S) + (s.in == kSplitSlabs ? split_position(iy * S + ix, S) : iy * S + ix));
            v[k][0] = q.x, v[k][1] = q.y, v[k][2] = q.z, v[k][3] = q.w;
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            auto g = [&](int i, unsigned a, unsigned b) {
                const int c = R.code[i];
                const unsigned m11 = (c & 1) ? ~0u : 0u, m10 = (c & 2) ? ~0u : 0u, m01 = (c & 4) ? ~0u : 0u; // code < 8: f(0, 0) = 0
                return ((a & ((b & m11) | (~b & m10))) | (~a & b & m01)) ^ R.inv[i];
            };
            const unsigned z = g(6, g(4, g(0, v[0][w], v[1][w]), g(1, v[2][w], v[3][w])), g(5, g(2, v[4][w], v[5][w]), g(3, v[6][w], v[7][w])));
            (w == 0 ? acc.x : w == 1 ? acc.y : w == 2 ? acc.z : acc.w) |= z;
        }
    }
    return acc;
}

// ONE: a block per item.  What lets a block go on from item to item (two more places of the fetches and copies, the items ahead) then only holds
// up the first: one slab, us for 32x32, 16x16, 8x8 images with it / without, k = 128 4.9, 4.5, 5.6 / 4.5, 4.1, 4.9, k = 256 5.7, 5.2, 7.9 / 5.3, 4.6, 7.4.
template <int S, bool ONE>
__global__ void __launch_bounds__(Geo<S>::THREADS, 1024 / Geo<S>::THREADS)
    packed_convtree_slab3_kernel(const uint4 *__restrict__ x, const Rec *__restrict__ recs, uint4 *__restrict__ y, Shape s)
{
    using G = Geo<S>;
    constexpr int NT = G::THREADS;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(16) Rec rec[3];
    const int tid = threadIdx.x;
    const unsigned base = (unsigned)__cvta_generic_to_shared(smem);
    for (int i = tid * 16; i < 2 * G::PLANE_BYTES; i += NT * 16) *reinterpret_cast<uint4 *>(smem + i) = make_uint4(0u, 0u, 0u, 0u); // halos stay zero

    auto fetch_rec = [&](int c, Rec &R) {
        if (tid < (int)(sizeof(Rec) / 16))
            cp_async16((unsigned)__cvta_generic_to_shared(&R) + 16u * tid, reinterpret_cast<const uint4 *>(recs + c) + tid);
    };
    // the planes of an item: four units a thread and channel, NT apart; NT is a whole number of rows, so that only the first
    // destination is computed and the others are constants away
    const unsigned sdst = base + 16u * (unsigned)((tid / G::HW) * G::SLAB + (tid % G::HW / S + 1) * G::PITCH +
                                          (s.in == kSplitSlabs ? tid % S + (tid % S >= G::H2) : column<S>(tid % S + 1)));
    auto stage = [&](int ug, const Rec &R, bool fresh) {
        if (!R.all_in_tile) return;
        const int u0 = ug * G::UB, n = (s.U - u0) * G::HW - tid; // units from this thread's first to the end
        const int which = fresh ? R.planes : (int)R.fresh;
#pragma unroll
        for (int slot = 0; slot < 2; ++slot) {
            if (!(which >> slot & 1)) continue;
            const uint4 *src = x + ((size_t)R.ch[slot] * s.U + u0) * G::HW + tid;
            const unsigned d = sdst + slot * G::PLANE_BYTES;
            constexpr int D1 = unit_step<S, G>(1), D2 = unit_step<S, G>(2), D3 = unit_step<S, G>(3);
            if (n > 3 * NT) {
                cp_async16_at<0, 0>(d, src), cp_async16_at<D1, NT * 16>(d, src);
                cp_async16_at<D2, 2 * NT * 16>(d, src), cp_async16_at<D3, 3 * NT * 16>(d, src);
            } else {
                if (n > 0) cp_async16_at<0, 0>(d, src);
                if (n > NT) cp_async16_at<D1, NT * 16>(d, src);
                if (n > 2 * NT) cp_async16_at<D2, 2 * NT * 16>(d, src);
            }
        }
    };

    const int ub = tid / G::I, t = tid % G::I, py = t / G::H2, px = t % G::H2; // window (py, px) of slab ub
    const unsigned at0 = base + 16u * (unsigned)(ub * G::SLAB + 2 * py * G::PITCH + px);

    // Items are (slab group ug, record), records fastest: the blocks that run together work on the same few slabs of all input
    // channels (L2-resident).  A block takes every gridDim.x-th run of consecutive items, within which a record copies
    // the planes only that the one before did not leave in the tile; the items of three are known ahead.
    struct Item {
        int left, run, ug, r; // items left of its run, the run; its slab group and record
        bool fresh;           // nothing in the tile
    };
    auto advance = [&](Item &t) {
        t.fresh = true;
        if (t.left > 0) {
            --t.left;
            t.fresh = ++t.r == s.C;
            if (t.fresh) t.r = 0, ++t.ug;
        } else if ((t.run += gridDim.x) < s.runs) {
            const int i = t.run * s.per_run + min(t.run, s.longer);
            t.left = s.per_run - (t.run < s.longer ? 0 : 1), t.ug = i / s.C, t.r = i - t.ug * s.C;
        } else {
            t.ug = s.n_ug;
        }
    };
    Item n0, n1, n2;
    if constexpr (ONE) {
        n0.ug = blockIdx.x / s.C, n0.r = blockIdx.x - n0.ug * s.C;
        n1.ug = n2.ug = s.n_ug;
        fetch_rec(n0.r, rec[0]);
    } else {
        n0.run = (int)blockIdx.x - (int)gridDim.x, n0.left = 0;
        advance(n0);
        n1 = n0;
        advance(n1);
        n2 = n1;
        if (n2.ug < s.n_ug) advance(n2);
        fetch_rec(n0.r, rec[0]);
        if (n1.ug < s.n_ug) fetch_rec(n1.r, rec[1]);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads(); // records and halo zeros in place
    stage(n0.ug, rec[0], true);
    cp_async_commit();
    for (int r0 = 0; ONE ? r0 == 0 : n0.ug < s.n_ug; r0 = r0 == 2 ? 0 : r0 + 1) {
        const int r1 = r0 == 2 ? 0 : r0 + 1, r2 = r1 == 2 ? 0 : r1 + 1;
        cp_async_wait_all();
        __syncthreads(); // this item's planes and the next item's record have landed
        if (!ONE && n2.ug < s.n_ug) fetch_rec(n2.r, rec[r2]);
        const Rec &R = rec[r0];
        const int u0 = n0.ug * G::UB;
        const bool live = ub < s.U - u0;
        uint4 out = make_uint4(0u, 0u, 0u, 0u);
        if (live) {
            if (R.all_in_tile) {
                // one copy of the gate code for both conv rows of the window (the instruction cache)
#pragma unroll 1
                for (int dy = 0; dy < 2; ++dy) {
                    const unsigned at = at0 + dy * G::ROW_BYTES;
                    unsigned g0[8], g1[8], t0[8], t1[8];
                    taps(g0, t0, R, 0, at);
                    taps(g1, t1, R, 1, at);
                    gate8(R.code[0], R.inv[0], g0, t0);
                    gate8(R.code[1], R.inv[1], g1, t1);
                    taps(t0, t1, R, 2, at);
                    gate8(R.code[4], R.inv[4], g0, g1);
                    gate8(R.code[2], R.inv[2], t0, t1);
                    taps(g1, t1, R, 3, at);
                    gate8(R.code[3], R.inv[3], g1, t1);
                    gate8(R.code[5], R.inv[5], t0, g1);
                    gate8(R.code[6], R.inv[6], g0, t0);
                    out.x |= g0[0] | g0[4], out.y |= g0[1] | g0[5], out.z |= g0[2] | g0[6], out.w |= g0[3] | g0[7];
                }
            } else {
                out = window_global<S>(x + (size_t)(u0 + ub) * G::HW, R, s, py, px);
            }
        }
        if constexpr (!ONE) {
            __syncthreads(); // every thread is done with the tile: the next item's planes go there while the SM's other blocks compute
            if (n1.ug < s.n_ug) stage(n1.ug, rec[r1], n1.fresh);
            cp_async_commit();
        }
        if (live) {
            const int c0 = R.c;
            if (s.out == kRows) y[((size_t)c0 * G::I + t) * s.U + u0 + ub] = out;
            else y[((size_t)c0 * s.U + u0 + ub) * G::I + (s.out == kSplitSlabs ? split_position(t, G::H2) : t)] = out;
        }
        if constexpr (!ONE) {
            n0 = n1, n1 = n2;
            if (n2.ug < s.n_ug) advance(n2);
        }
    }
    cp_async_wait_all();
}

// Record i: of output channel i, or as the order tells; offsets are bytes from a window's unit of the first plane.
template <int S>
__device__ __forceinline__ void lay_out_record(const uint8_t *__restrict__ ops, const int32_t *__restrict__ sel, const int32_t *__restrict__ order,
                                               Rec *__restrict__ recs, int i, int Ci)
{
    using G = Geo<S>;
    Rec R;
    int ch0 = -1, ch1 = -1, c = i;
    if (order) c = order[3 * i], ch0 = order[3 * i + 1], ch1 = order[3 * i + 2] & 0xFFFF;
    bool all = true;
    for (int k = 0; k < 8; ++k) {
        const int w = sel[c * 8 + k];
        const int ch = min((w >> 16) & 0xFFFF, Ci - 1), r = (w >> 8) & 0xFF, sx = w & 0xFF;
        if (ch0 < 0) ch0 = ch;
        if (ch1 < 0 && ch != ch0) ch1 = ch;
        all = all && (ch == ch0 || ch == ch1) && r < 3 && sx < 3;
        const int row = min(r, 2) * G::PITCH, col = min(sx, 2), second = ch == ch0 ? 0 : 1;
        const int l = second * G::PLANE_BYTES + 16 * (row + column<S>(col)), q = l + 16 * (column<S>(col + 1) - column<S>(col));
        if (k & 1) R.off[k / 2].z = l, R.off[k / 2].w = q;
        else R.off[k / 2].x = l, R.off[k / 2].y = q;
        R.word[k] = w;
        if (k < 7) {
            const int op = ops[c * 7 + k] & 15;
            R.code[k] = op < 8 ? op : 15 - op, R.inv[k] = op < 8 ? 0u : ~0u;
        }
    }
    R.c = c, R.ch[0] = ch0, R.ch[1] = ch1 < 0 ? ch0 : ch1, R.planes = ch1 < 0 ? 1 : 3, R.all_in_tile = all;
    R.fresh = order ? (unsigned)order[3 * i + 2] >> 16 : (unsigned)R.planes;
    recs[i] = R;
}

template <int S> __global__ void packed_slab3_records_kernel(const uint8_t *__restrict__ ops, const int32_t *__restrict__ sel,
                                                                    const int32_t *__restrict__ order, Rec *__restrict__ recs, int C, int Ci)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < C) lay_out_record<S>(ops, sel, order, recs, i, Ci);
}

template <int S> static int launch(const void *x, const void *recs, void *y, int Ci, int C, int64_t U, Order in, Order out, cudaStream_t st)
{
    using G = Geo<S>;
    using namespace clb_host;
    Shape s{Ci, C, (int)U, (int)((U + G::UB - 1) / G::UB), in, out, 0, 0, 0};
    constexpr int bytes = 2 * G::PLANE_BYTES;
    constexpr int by_smem = 227 * 1024 / (bytes + 2048), by_threads = 1024 / G::THREADS; // 64 registers a thread
    const long long items = (long long)C * s.n_ug, all = (long long)sm_count() * (by_smem < by_threads ? by_smem : by_threads);
    // runs of about 16 items, as many for one block as for another (k = 1024, 8192 samples, four blocks: 1610 us with 4, 1590 with 16 and 32)
    const long long grid = items < all ? items : all, rounds = (items + 8 * grid) / (16 * grid), runs = grid * (rounds > 0 ? rounds : 1);
    s.runs = (int)runs, s.per_run = (int)(items / runs), s.longer = (int)(items % runs);
    // A block per item up to a quarter more than are resident at once (4x4 images, 4096 items on 3552 places: 7.9 us with blocks that go on, 7.5; 8192:
    // 10.7 either way; 32x32, 1024 on 592: 11.2 / 12.3).
    const bool one = 4 * items <= 5 * all;
    auto k = one ? packed_convtree_slab3_kernel<S, true> : packed_convtree_slab3_kernel<S, false>;
    if (ensure_dynamic_smem(k, bytes) != cudaSuccess) return check_launch(0);
    CLB_TRACED("packed_convtree_slab3_kernel", st,
               k<<<(unsigned)(one ? items : grid), G::THREADS, bytes, st>>>((const uint4 *)x, (const Rec *)recs, (uint4 *)y, s));
    return check_launch();
}
template <int S> static int records(const uint8_t *ops, const int32_t *sel, const int32_t *order, Rec *recs, int Ci, int C, cudaStream_t st)
{
    CLB_TRACED("packed_slab3_records_kernel", st, packed_slab3_records_kernel<S><<<(C + 127) / 128, 128, 0, st>>>(ops, sel, order, recs, C, Ci));
    return clb_host::check_launch();
}

} // namespace slab
} // namespace clb

using namespace clb;
using namespace clb_host;

bool clb_slab3_covers(int H, int W, int sh, int sw, int ph, int pw, int kh, int kw)
{
    return H == W && (H == 32 || H == 16 || H == 8 || H == 4) && sh == 1 && sw == 1 && ph == 1 && pw == 1 && kh == 3 && kw == 3;
}
// Channels are vertices, output channels edges between the two that they read; the order follows trails: next comes an edge between
// both channels in the tile, else one that shares the channel with more edges left, whose other plane is then replaced.
bool clb_slab3_order(const int32_t *sel, int Ci, int C, int32_t *order)
{
    std::vector<int> a((size_t)C), b((size_t)C), start((size_t)Ci + 1, 0), edges;
    for (int c = 0; c < C; ++c) {
        int ch0 = -1, ch1 = -1;
        for (int k = 0; k < 8; ++k) {
            const int w = sel[c * 8 + k], ch = (w >> 16) & 0xFFFF;
            if (w < 0 || ch >= Ci || ((w >> 8) & 0xFF) > 2 || (w & 0xFF) > 2) return false;
            if (ch0 < 0) ch0 = ch;
            else if (ch != ch0 && ch1 < 0) ch1 = ch;
            else if (ch != ch0 && ch != ch1) return false;
        }
        a[c] = ch0, b[c] = ch1 < 0 ? ch0 : ch1;
        ++start[a[c] + 1];
        if (b[c] != a[c]) ++start[b[c] + 1];
    }
    for (int v = 0; v < Ci; ++v) start[v + 1] += start[v];
    edges.resize((size_t)start[Ci]);
    std::vector<int> end(start.begin(), start.end() - 1), left((size_t)Ci, 0);
    for (int c = 0; c < C; ++c) {
        edges[end[a[c]]++] = c, ++left[a[c]];
        if (b[c] != a[c]) edges[end[b[c]]++] = c, ++left[b[c]];
    }
    std::vector<char> used((size_t)C, 0);
    // an unused edge at v, one to `other` if there is one; used ones are dropped from the list's front
    auto pick = [&](int v, int other, bool &both) {
        int found = -1;
        both = false;
        for (int e = start[v], keep = e; e < end[v]; ++e) {
            const int c = edges[e];
            if (used[c]) {
                if (e == keep) start[v] = ++keep;
                continue;
            }
            if (found < 0) found = c;
            if (a[c] + b[c] - v == other || a[c] == b[c]) {
                both = true;
                return c;
            }
            if (e - start[v] >= 64) break;
        }
        return found;
    };
    int slot[2] = {-1, -1}, next = 0;
    for (int i = 0; i < C; ++i) {
        int c = -1;
        bool both = false;
        if (slot[0] >= 0) {
            const int k = left[slot[0]] >= left[slot[1]] ? 0 : 1;
            c = pick(slot[k], slot[1 - k], both);
            if (c < 0) c = pick(slot[1 - k], slot[k], both);
        }
        if (c < 0) {
            while (used[next]) ++next;
            c = next;
        }
        int fresh = 0;
        if (slot[0] < 0 || (a[c] != slot[0] && a[c] != slot[1] && b[c] != slot[0] && b[c] != slot[1])) {
            slot[0] = a[c], slot[1] = b[c], fresh = 3;
        } else {
            const bool has_a = a[c] == slot[0] || a[c] == slot[1], has_b = b[c] == slot[0] || b[c] == slot[1];
            if (!has_a || !has_b) {
                const int kept = has_a ? a[c] : b[c], k = kept == slot[0] ? 1 : 0; // the other plane goes
                slot[k] = has_a ? b[c] : a[c], fresh = 1 << k;
            }
        }
        used[c] = 1, --left[a[c]];
        if (b[c] != a[c]) --left[b[c]];
        order[3 * i] = c, order[3 * i + 1] = slot[0], order[3 * i + 2] = slot[1] | fresh << 16;
    }
    return true;
}

size_t clb_slab3_record_bytes(int C) { return (size_t)C * sizeof(slab::Rec); }

int clb_slab3_records(const uint8_t *ops, const int32_t *sel, const int32_t *order, void *recs, int Ci, int side, int C, cudaStream_t st)
{
    slab::Rec *r = (slab::Rec *)recs;
    if (side == 32) return slab::records<32>(ops, sel, order, r, Ci, C, st);
    if (side == 16) return slab::records<16>(ops, sel, order, r, Ci, C, st);
    if (side == 8) return slab::records<8>(ops, sel, order, r, Ci, C, st);
    return slab::records<4>(ops, sel, order, r, Ci, C, st);
}

int clb_slab3_block(const void *x, const void *recs, void *y, int Ci, int side, int C, int64_t U, Order in, Order out, cudaStream_t st)
{
    if (side == 32) return slab::launch<32>(x, recs, y, Ci, C, U, in, out, st);
    if (side == 16) return slab::launch<16>(x, recs, y, Ci, C, U, in, out, st);
    if (side == 8) return slab::launch<8>(x, recs, y, Ci, C, U, in, out, st);
    return slab::launch<4>(x, recs, y, Ci, C, U, in, out, st);
}

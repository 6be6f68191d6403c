// Backward, pass 1, of a fused ConvLogic block whose output channels each read (at most) two input channels: fp32, stride 1, 3x3
// window, padding 1, square images of 32, 28, 16, 12 or 6 pixels.
//
// A group of threads (a warp; four warps for 32 and 28 pixels) owns one output channel and a part of the batch.  It keeps the two
// channel planes of NIMG images in shared memory, recomputes the gate chain of every pooled window at its saved arg-max, keeps the
// 28 basis sums of the gate gradients in registers until the end, and adds the gradients w.r.t. the eight taps into a second
// tile of the same shape, one tap after the other (within one tap the map window -> pixel is injective, so that nothing is
// atomic and the order of additions is fixed).  The gradient planes of (image, output channel) are then written out;
// plane_sum_kernel adds them up per input channel.
//
// What bounds it is the shared-memory pipe: 24 accesses per window at positions that depend on its arg-max.  In a row-major tile
// the 32 windows of a warp step by two columns and two rows, and an access takes 2.95 passes on average.  The tile is therefore
// split by the parity of the padded row and column: the cells that the lanes hit then lie side by side in one of four planes
// whose distance is a multiple of 32 banks, and the pitch and the choice of a warp's rows keep those apart: 2.0 passes (the even
// columns sit one bank lower, so that four neighbouring pixels of an image row are two aligned pairs; without that it would
// be 1.66, and the copies in and out would cost more than the difference).  The planes arrive through registers, one iteration
// ahead, because no copy engine can split columns.
// 256 images, 256 -> 1024 channels of 16x16: 298 us with row-major tiles fetched by TMA, 241 with these.  (8x8 and 4x4 images keep the
// row-major tiles of convtree_plane.cu: the many small copies cost these kernels more than the passes they save, 291 against 279 us
// for 1024 -> 4096 channels of 8x8, 220 against 186 for 4096 -> 8192 of 4x4.)
#include "clb_plane.cuh"
#include "clb_tma.cuh"

namespace clb {
namespace plane {

template <int S> struct Tile {
    static constexpr int H2 = S / 2, I = H2 * H2;
    static constexpr int WARPS = S >= 28 ? 4 : 1, GROUPS = 4 / WARPS, GSIZE = 32 * WARPS;
    static constexpr int BLOCKS = S == 28 || S == 12 ? 3 : 4; // resident per SM: 128 registers a thread where the kernel fits them, else 168
    static constexpr int NIMG = S == 6 ? 3 : S == 12 ? 2 : 1;  // images per iteration
    // a warp's 32 lanes are RW window rows, PASSES apart, of H2 windows; a thread has its place in WPT of the PASSES such sets
    static constexpr int RW = S == 6 ? 9 : S == 12 ? 4 : 32 / H2, PASSES = NIMG * H2 / RW, WPT = (PASSES + WARPS - 1) / WARPS;
    static constexpr bool FULL = RW * H2 == 32;
    // floats: pitch of a parity plane's rows, distance of images in it, size of a plane, of a channel slot, of the tile
    static constexpr int P = S == 32 ? 22 : S == 28 ? 16 : S == 16 ? 12 : S == 6 ? 4 : 8;
    static constexpr int IMG = S == 12 ? 80 : S == 6 ? 21 : 0;
    static constexpr int PL = ((NIMG - 1) * IMG + H2 * P + H2 + 2 + 31) / 32 * 32, SLOT = 4 * PL, LEAD = 2;
    static constexpr int BYTES = (LEAD + 2 * SLOT + 2) * 4, GRAD = (BYTES + 15) / 16 * 16; // the gradient tile, GRAD bytes behind
    static constexpr int SMEM = GROUPS * 2 * GRAD;
    // a unit is QUAD neighbouring pixels of a row: u = (channel slot, row parity, image, row of that parity, column / QUAD), column fastest
    static constexpr int QUAD = S % 4 == 0 ? 4 : 2, W4 = S / QUAD, UNITS = 2 * NIMG * S * W4, UPT = (UNITS + GSIZE - 1) / GSIZE;
    static constexpr bool REGULAR = NIMG * H2 * W4 == GSIZE; // then unit q of a thread is its pixel quad in row parity q & 1 of channel slot q >> 1
    static_assert(NIMG * H2 == RW * PASSES && (NIMG == 1 || IMG >= H2 * P + H2 + 2) && P > H2 && (QUAD == 2 || P % 2 == 0), "tile geometry");
};

template <int OFF> __device__ __forceinline__ float lds1(uint32_t a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF> __device__ __forceinline__ void sts1(uint32_t a, float v) { asm volatile("st.shared.f32 [%0+%1], %2;" ::"r"(a), "n"(OFF), "f"(v) : "memory"); }
template <int OFF> __device__ __forceinline__ float2 lds2(uint32_t a)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF> __device__ __forceinline__ void sts2(uint32_t a, float x, float y)
{
    asm volatile("st.shared.v2.f32 [%0+%1], {%2, %3};" ::"r"(a), "n"(OFF), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ Gate<float> lds_gate(uint32_t a)
{
    Gate<float> g;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(g.k1), "=f"(g.ka), "=f"(g.kb), "=f"(g.kab) : "r"(a));
    return g;
}
// 16 bits of {hi, lo}, zero-extended (they are below 2^15: bit 3 of a selector nibble replicates the byte's sign)
__device__ __forceinline__ uint32_t pick16(uint32_t lo, uint32_t hi, uint32_t selector)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(lo), "r"(hi), "r"(selector));
    return d;
}

template <int S, bool FM>
__global__ void __launch_bounds__(kThreads, Tile<S>::BLOCKS) convtree_bwd_plane_kernel(ClbTileBwd s)
{
    using T = Tile<S>;
    constexpr int WPT = T::WPT, UPT = T::UPT, I = T::I, H2 = T::H2, HW = S * S, NIMG = T::NIMG, GT = T::GRAD, QUAD = T::QUAD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) Gate<float> sgs[T::GROUPS][7];
    __shared__ SlotInfo sis[T::GROUPS];
    __shared__ float red[4][28];

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0); // (what depends on it is then kept per warp, not per lane)
    const int gid = T::WARPS == 1 ? warp : 0, gt = T::WARPS == 1 ? lane : tid, gwarp = T::WARPS == 1 ? 0 : warp;
    const long long task = (long long)blockIdx.x * T::GROUPS + gid;
    if (task >= (long long)s.C * s.parts) return; // a whole group leaves together
    const int c = (int)(task % s.C), part = (int)(task / s.C);
    auto group_sync = [] {
        if (T::WARPS == 1)
            __syncwarp();
        else
            __syncthreads();
    };
    const int taps = gwarp == 0 ? __ldg(s.sel + (size_t)c * 8 + (lane & 7)) : 0;
    if (gt < 7) sgs[gid][gt] = gate_load<float>(s.w + ((size_t)c * 7 + gt) * 16, s.wmode);
    if (gwarp == 0) fill_slots(sis[gid], taps, s.Ci, lane);
    const uint32_t tile = clb_tma::smem_addr(smem_raw) + gid * 2 * T::GRAD;
    for (int i = gt; i < 2 * T::GRAD / 4; i += T::GSIZE) sts1<0>(tile + 4 * i, 0.f); // halos stay zero, the gradient tile starts as zeros
    group_sync();
    const SlotInfo &si = sis[gid];
    const uint32_t gates = clb_tma::smem_addr(&sgs[gid][0]);
    float acc[28];
#pragma unroll
    for (int i = 0; i < 28; ++i) acc[i] = 0.f;

    const int n_lo = (int)((long long)s.N * part / s.parts), n_hi = (int)((long long)s.N * (part + 1) / s.parts);
    const int iters = si.nslot <= 2 ? (n_hi - n_lo + NIMG - 1) / NIMG : 0; // the host only routes selections here that fit two planes

    // byte offsets of a tap from its window's cell, for the four positions of the window: 16 bits each
    uint32_t off_lo[8], off_hi[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int word = s.sel[c * 8 + k], ty = (word >> 8) & 0xFF, tx = word & 0xFF;
        auto at = [&](int by, int bx) {
            return 4u * (uint32_t)(si.slot[k] * T::SLOT + ((by + ty) & 1) * 2 * T::PL + ((bx + tx) & 1) * (T::PL + 1) + ((by + ty) >> 1) * T::P + ((bx + tx) >> 1));
        };
        off_lo[k] = at(0, 0) | at(0, 1) << 16, off_hi[k] = at(1, 0) | at(1, 1) << 16;
    }
    // the thread's windows
    uint32_t base[WPT];
    int a_win[WPT], o_win[WPT]; // element of amax and of gy for the part's first images
    int img_of[WPT];            // -1: no window
#pragma unroll
    for (int j = 0; j < WPT; ++j) {
        const int pass = gwarp + T::WARPS * j;
        const bool has = (T::FULL || lane < T::RW * H2) && pass < T::PASSES;
        const int row = has ? lane / H2 * T::PASSES + pass : 0, px = has ? lane % H2 : 0, img = row / H2, py = row - img * H2, win = py * H2 + px;
        base[j] = tile + 4u * (uint32_t)(T::LEAD - 1 + img * T::IMG + py * T::P + px);
        a_win[j] = img * s.C * I + win;
        o_win[j] = FM ? win * s.n_stride + img : a_win[j];
        img_of[j] = has ? img : -1;
    }
    // the thread's units of the planes
    const float *xb = s.x + (size_t)n_lo * s.Ci * HW;
    float *pb = s.planes + ((size_t)c * 2 * s.N + n_lo) * HW;
    constexpr int UR = T::REGULAR ? 1 : UPT; // places kept in registers; those of the others of a regular thread are constants away
    int xoff[UR], poff[UR], uimg[UR];
    uint32_t ucell[UR];
#pragma unroll
    for (int q = 0; q < UR; ++q) {
        const int u = gt + T::GSIZE * q;
        const int col4 = u % T::W4, k = u / T::W4 % H2, img = u / (T::W4 * H2) % NIMG, even = u / (T::W4 * H2 * NIMG) & 1, slot = u / (T::W4 * H2 * NIMG * 2);
        const int r = S == 16 ? (k % 4) * 2 + k / 4 : S == 32 ? (k % 2) * 8 + k / 2 : k; // rows of a half-warp's pairs in different banks
        const int y = 2 * r + even;                                                      // padded row y + 1
        xoff[q] = (img * s.Ci + (slot ? si.ch[1] : si.ch[0])) * HW + y * S + QUAD * col4;
        poff[q] = (slot * s.N + img) * HW + y * S + QUAD * col4;
        ucell[q] = tile + 4u * (uint32_t)(T::LEAD + slot * T::SLOT + (even ? 0 : 2 * T::PL) + img * T::IMG + (r + even) * T::P + QUAD / 2 * col4);
        uimg[q] = u < T::UNITS ? img : 1 << 20;
    }
    const int second = T::REGULAR ? (si.ch[1] - si.ch[0]) * HW : 0, second_plane = T::REGULAR ? s.N * HW : 0;
    auto x_at = [&](int q) { return T::REGULAR ? xoff[0] + (q & 1) * S + (q >> 1) * second : xoff[q]; };
    auto p_at = [&](int q) { return T::REGULAR ? poff[0] + (q & 1) * S + (q >> 1) * second_plane : poff[q]; };
    auto cell_at = [&](int q) { return T::REGULAR ? ucell[0] + 4u * (uint32_t)((q & 1) * (T::P - 2 * T::PL) + (q >> 1) * T::SLOT) : ucell[q]; };
    auto img_at = [&](int q) { return uimg[T::REGULAR ? 0 : q]; };

    float xv[UPT][QUAD];
    float dz[WPT];
    int bd[WPT];
#pragma unroll
    for (int q = 0; q < UPT; ++q)
#pragma unroll
        for (int i = 0; i < QUAD; ++i) xv[q][i] = 0.f;
    const float *gb = FM ? s.gy + (size_t)c * I * s.n_stride + n_lo : s.gy + ((size_t)n_lo * s.C + c) * I;
    const uint8_t *ab = s.amax + ((size_t)n_lo * s.C + c) * I;
    int left = n_hi - n_lo; // images from the next to be fetched on
    auto fetch = [&] {
#pragma unroll
        for (int q = 0; q < UPT; ++q)
            if (img_at(q) < left) {
                if constexpr (QUAD == 4) {
                    const float4 v = __ldg(reinterpret_cast<const float4 *>(xb + x_at(q)));
                    xv[q][0] = v.x, xv[q][1] = v.y, xv[q][2] = v.z, xv[q][3] = v.w;
                } else {
                    const float2 v = __ldg(reinterpret_cast<const float2 *>(xb + x_at(q)));
                    xv[q][0] = v.x, xv[q][1] = v.y;
                }
            }
#pragma unroll
        for (int j = 0; j < WPT; ++j) {
            const bool live = img_of[j] >= 0 && img_of[j] < left;
            dz[j] = live ? __ldg(gb + o_win[j]) : 0.f;
            bd[j] = live ? (int)__ldg(ab + a_win[j]) : 0;
        }
        xb += (size_t)NIMG * s.Ci * HW, ab += (size_t)NIMG * s.C * I;
        gb += FM ? NIMG : (size_t)NIMG * s.C * I;
        left -= NIMG;
    };
    fetch();
#pragma unroll 1
    for (int it = 0; it < iters; ++it) {
        // pixels 4q .. 4q + 3 are padded columns 4q + 1 .. 4q + 4: two of the odd plane, two of the even one (of a pair one each)
#pragma unroll
        for (int q = 0; q < UPT; ++q)
            if (T::UNITS % T::GSIZE == 0 || img_at(q) < NIMG) {
                if constexpr (QUAD == 4)
                    sts2<4 * T::PL>(cell_at(q), xv[q][0], xv[q][2]), sts2<0>(cell_at(q), xv[q][1], xv[q][3]);
                else
                    sts1<4 * T::PL>(cell_at(q), xv[q][0]), sts1<0>(cell_at(q), xv[q][1]);
            }
        float d[WPT];
        uint32_t pos[WPT];
#pragma unroll
        for (int j = 0; j < WPT; ++j) d[j] = dz[j], pos[j] = 0x9910u + 0x2222u * (uint32_t)bd[j];
        const int have = left + NIMG; // images from this iteration's first on
        group_sync();
        fetch();
        Gate<float> g[7]; // read again for every iteration: they need no registers while the gradients are added up
#pragma unroll
        for (int i = 0; i < 7; ++i) g[i] = lds_gate(gates + 16 * i);
        uint32_t cell[WPT][8];
        float tg[WPT][8];
#pragma unroll
        for (int j = 0; j < WPT; ++j) {
            float a[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                cell[j][k] = base[j] + pick16(off_lo[k], off_hi[k], pos[j]);
                a[k] = lds1<0>(cell[j][k]);
            }
            window_bwd(a, g, d[j], acc, tg[j]);
        }
        // One tap at a time: all windows of the group hit distinct pixels within one tap; a pixel outside the image is a halo cell
        // that is never written out.
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float cur[WPT];
#pragma unroll
            for (int j = 0; j < WPT; ++j) cur[j] = lds1<GT>(cell[j][k]);
#pragma unroll
            for (int j = 0; j < WPT; ++j)
                if ((T::FULL && T::PASSES == WPT * T::WARPS) || img_of[j] >= 0) sts1<GT>(cell[j][k], cur[j] + tg[j][k]);
            group_sync();
        }
        // write the gradient planes out and clear them for the next iteration (whose first barrier orders that before its additions)
#pragma unroll
        for (int q = 0; q < UPT; ++q) {
            if (T::UNITS % T::GSIZE != 0 && img_at(q) >= NIMG) continue;
            const uint32_t at = cell_at(q);
            if constexpr (QUAD == 4) {
                const float2 odd = lds2<GT + 4 * T::PL>(at), even = lds2<GT>(at);
                sts2<GT + 4 * T::PL>(at, 0.f, 0.f), sts2<GT>(at, 0.f, 0.f);
                if (img_at(q) < have) *reinterpret_cast<float4 *>(pb + p_at(q)) = make_float4(odd.x, even.x, odd.y, even.y);
            } else {
                const float odd = lds1<GT + 4 * T::PL>(at), even = lds1<GT>(at);
                sts1<GT + 4 * T::PL>(at, 0.f), sts1<GT>(at, 0.f);
                if (img_at(q) < have) *reinterpret_cast<float2 *>(pb + p_at(q)) = make_float2(odd, even);
            }
        }
        pb += NIMG * HW;
    }

    const float sum = warp_sums28(acc, lane);
    float *out = s.partial + ((size_t)part * s.C + c) * 28;
    if (T::WARPS == 1) {
        if (lane < 28) out[lane] = sum;
    } else {
        if (lane < 28) red[warp][lane] = sum;
        __syncthreads();
        if (tid < 28) out[tid] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
    }
}

template <int S> static int parts_for(int N, int C) { return clb_plane_parts(N, C, Tile<S>::NIMG, Tile<S>::GROUPS, Tile<S>::BLOCKS); }

template <int S> static int launch(const ClbTileBwd &a, cudaStream_t st)
{
    using T = Tile<S>;
    auto k = a.fm ? convtree_bwd_plane_kernel<S, true> : convtree_bwd_plane_kernel<S, false>;
    if (clb_host::ensure_dynamic_smem(k, T::SMEM) != cudaSuccess) return clb_host::check_launch(0);
    const long long tasks = (long long)a.C * a.parts;
    CLB_TRACED("convtree_bwd_plane_kernel", st, k<<<(unsigned)((tasks + T::GROUPS - 1) / T::GROUPS), kThreads, T::SMEM, st>>>(a));
    return CLB_OK;
}

} // namespace plane
} // namespace clb

using namespace clb::plane;

int clb_tile_bwd_parts(int side, int N, int C)
{
    return side == 32 ? parts_for<32>(N, C) : side == 28 ? parts_for<28>(N, C) : side == 16 ? parts_for<16>(N, C) : side == 12 ? parts_for<12>(N, C)
           : parts_for<6>(N, C);
}

int clb_tile_bwd(int side, const ClbTileBwd &a, cudaStream_t st)
{
    return side == 32 ? launch<32>(a, st) : side == 28 ? launch<28>(a, st) : side == 16 ? launch<16>(a, st) : side == 12 ? launch<12>(a, st)
           : launch<6>(a, st);
}

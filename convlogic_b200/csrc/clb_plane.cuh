// What the plane kernels (convtree_plane.cu, convtree_tile.cu) share: blocks of which an output channel reads at most two input
// channels, whose planes a block or a warp keeps in shared memory.
#pragma once

#include "clb_common.cuh"

namespace clb {
namespace plane {

constexpr int kThreads = 128;

struct SlotInfo {
    int slot[8];
    int ch[2];
    int nslot; // 3 = the selection does not fit two staged planes (more channels, or taps outside the 3x3 window)
};

// channel -> slot map of an output channel's taps: the first channel that they name has slot 0, another one slot 1.  word: tap lane & 7 of
// the selection; the whole warp calls this.  (One thread that walked the taps took longer than the soft-max of the gates.  The map goes
// through shared memory because in registers it cost the kernels a resident block.)
__device__ __forceinline__ void fill_slots(SlotInfo &si, int word, int Ci, int lane)
{
    const int ch = (word >> 16) & 0xFFFF;
    const bool inside = __all_sync(0xffffffffu, word >= 0 && ch < Ci && ((word >> 8) & 0xFF) < 3 && (word & 0xFF) < 3);
    const int first = __shfl_sync(0xffffffffu, ch, 0);
    const unsigned rest = __ballot_sync(0xffffffffu, ch != first) & 0xffu;
    const int other = __shfl_sync(0xffffffffu, ch, rest ? __ffs((int)rest) - 1 : 0);
    const unsigned more = __ballot_sync(0xffffffffu, ch != first && ch != other);
    if (lane < 8) si.slot[lane] = (int)(rest >> lane & 1u);
    if (lane == 0) si.ch[0] = min(first, Ci - 1), si.ch[1] = min(other, Ci - 1), si.nslot = !inside || more ? 3 : rest ? 2 : 1;
}

// 28 per-lane sums: lane i ends up with the warp's sum i (a transposed butterfly over the 32 lanes)
__device__ __forceinline__ float warp_sums28(const float (&acc)[28], int lane)
{
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = i < 28 ? acc[i] : 0.f;
#pragma unroll
    for (int half = 16; half >= 1; half >>= 1) {
        const bool upper = (lane & half) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float keep = upper ? v[i + half] : v[i];
            const float send = upper ? v[i] : v[i + half];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
        }
    }
    return v[0];
}

// One window at its arg-max position: the taps a, the upstream gradient d; adds the 28 basis sums of the gate gradients and
// returns the gradients w.r.t. the eight taps.
__device__ __forceinline__ void window_bwd(const float (&a)[8], const Gate<float> (&g)[7], float d, float (&acc)[28], float (&tg)[8])
{
    const float g0 = gate_eval<float>(g[0], a[0], a[1]), g1 = gate_eval<float>(g[1], a[2], a[3]);
    const float g2 = gate_eval<float>(g[2], a[4], a[5]), g3 = gate_eval<float>(g[3], a[6], a[7]);
    const float t0 = gate_eval<float>(g[4], g0, g1), t1 = gate_eval<float>(g[5], g2, g3);
    const float dt0 = d * gate_da<float>(g[6], t1), dt1 = d * gate_db<float>(g[6], t0);
    float dg[4];
    dg[0] = dt0 * gate_da<float>(g[4], g1), dg[1] = dt0 * gate_db<float>(g[4], g0);
    dg[2] = dt1 * gate_da<float>(g[5], g3), dg[3] = dt1 * gate_db<float>(g[5], g2);
    acc[24] = fmaf(d, t0 * t1, acc[24]), acc[25] = fmaf(d, t0, acc[25]), acc[26] = fmaf(d, t1, acc[26]), acc[27] += d;
    acc[16] = fmaf(dt0, g0 * g1, acc[16]), acc[17] = fmaf(dt0, g0, acc[17]), acc[18] = fmaf(dt0, g1, acc[18]), acc[19] += dt0;
    acc[20] = fmaf(dt1, g2 * g3, acc[20]), acc[21] = fmaf(dt1, g2, acc[21]), acc[22] = fmaf(dt1, g3, acc[22]), acc[23] += dt1;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        acc[4 * p] = fmaf(dg[p], a[2 * p] * a[2 * p + 1], acc[4 * p]);
        acc[4 * p + 1] = fmaf(dg[p], a[2 * p], acc[4 * p + 1]);
        acc[4 * p + 2] = fmaf(dg[p], a[2 * p + 1], acc[4 * p + 2]);
        acc[4 * p + 3] += dg[p];
        tg[2 * p] = dg[p] * gate_da<float>(g[p], a[2 * p + 1]);
        tg[2 * p + 1] = dg[p] * gate_db<float>(g[p], a[2 * p]);
    }
}

} // namespace plane
} // namespace clb

// How many contiguous parts the batch is split into: a (channel, part) pair is the task of a group, a block has `groups` of them and
// an SM `resident` blocks.  The SM's shared-memory pipe is what its blocks wait for, so the time goes with the blocks per SM
// times the iterations of one (256 images, 1024 channels of 16x16: 1 to 12 parts took 288, 279, 275, 246, 255, 256, 259, 247, ..
// 253, 253 us, in proportion); but where the last few blocks leave an SM half empty it also goes with the rounds (28x28, 128
// channels: 3 parts 80 us, 4 parts 99).  The sum of both decides; a task's set-up (soft-max of 7 gates, tap table, first
// copies) counts as a few iterations (4x4, eight images an iteration, 8192 channels: 189, 212, 230, 255 us with 1 to 4 parts).
int clb_plane_parts(int N, int C, int images_per_iteration, int groups, int resident);

// Pass 1 of the backward of a block of square images of 32, 28, 16, 12 or 6 pixels (convtree_tile.cu): partial [parts][C][28] basis
// sums, planes [C][2][N][side * side] gradients of the two input channels of every output channel.  gy, amax and x are those
// of the first of the N images; fm: gy is [C][windows][n_stride].
struct ClbTileBwd {
    const float *gy, *x, *w;
    const int32_t *sel;
    const uint8_t *amax;
    float *partial, *planes;
    int N, Ci, C, wmode, parts, fm, n_stride;
};
int clb_tile_bwd_parts(int side, int N, int C);
int clb_tile_bwd(int side, const ClbTileBwd &a, cudaStream_t st);

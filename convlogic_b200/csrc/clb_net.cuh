// The compiled network as the one-launch kernel sees it (net_cluster.cu), filled by net.cu.
#pragma once

#include <stdint.h>

namespace clb {

constexpr int kNetMaxLayers = 12;
constexpr int kNetMaxLevels = 256; // thermometer levels (byte pixels take no more)

// n / d by a multiplication
struct FastDiv {
    unsigned d, magic; // magic = ceil(2^32 / d), unused for d = 1
    __host__ __device__ static FastDiv of(unsigned d) { return FastDiv{d, d > 1 ? (unsigned)((0x100000000ull + d - 1) / d) : 0u}; }
    // div(n) == n / d for every 0 <= n < dividends: magic exceeds 2^32 / d by less than one, so n * magic / 2^32 exceeds n / d by less than
    // n / 2^32, which stays below 1 / d, the distance of n / d from the next whole number, while n * d < 2^32.  That holds or
    // fails for one dividend as for many: 67599 / 67600 came out as 1.
    __host__ __device__ static bool exact(long long dividends, long long d) { return dividends * d < (1LL << 32); }
    __host__ __device__ __forceinline__ int div(int n) const { return d > 1 ? (int)(((unsigned long long)(unsigned)n * magic) >> 32) : n; }
};

// Where the units (4, 8 or 16 bytes = 32, 64 or 128 samples of one feature) of a layer's input live inside a slab's storage: channels of
// rows x pitch units, the feature's image inside a halo of `ph` rows and `pw` columns.  Flat features: one "channel".
struct NetStorage {
    int base;                // first unit (a multiple of 8)
    int W, image;            // image width and size (rows * W), 1-D features: image = features
    int pitch, per_channel;  // units per stored row / channel
    int rows, ph, pw;        // image rows, halo
    int halo_units;          // channels * per_channel when there is a halo, else 0
    FastDiv by_image, by_W, by_pitch, by_channel;
    // `channels` images of rows x W inside their halo from `first` on; false if 32-bit unit indices or the divisions do not cover it
    bool lay_out(long long first, long long channels, int rows_, int W_, int ph_, int pw_)
    {
        const long long img = (long long)rows_ * W_, p = W_ + 2LL * pw_, per = (rows_ + 2LL * ph_) * p, most = 1LL << 24;
        if (channels > most || img > most || per > most || first + channels * per > most) return false;
        base = (int)first, W = W_, image = (int)img, pitch = (int)p, per_channel = (int)per, rows = rows_, ph = ph_, pw = pw_;
        halo_units = ph || pw ? (int)(channels * per) : 0;
        if ((halo_units || channels > 1) && !(FastDiv::exact(channels * img, img) && FastDiv::exact(img, W) && FastDiv::exact(channels * per, per) && FastDiv::exact(per, p)))
            return false;
        by_image = FastDiv::of((unsigned)image), by_W = FastDiv::of((unsigned)W);
        by_pitch = FastDiv::of((unsigned)pitch), by_channel = FastDiv::of((unsigned)per_channel);
        return true;
    }
#ifdef __CUDACC__
    __device__ __forceinline__ int unit(int f) const // unit of feature f
    {
        if (!halo_units) return f;
        const int c = by_image.div(f), p = f - c * image, y = by_W.div(p);
        return c * per_channel + (y + ph) * pitch + (p - y * W) + pw;
    }
    __device__ __forceinline__ bool halo(int i) const // i < halo_units
    {
        const int r = i - by_channel.div(i) * per_channel, row = by_pitch.div(r);
        return (unsigned)(row - ph) >= (unsigned)rows || (unsigned)(r - row * pitch - pw) >= (unsigned)W;
    }
#endif
};

struct NetLayer {
    int kind;                    // 1 conv block, 2 flat layer, 3 gate tree of `levels` levels
    int C, stride, Hp, Wp;       // conv: output channels and pooled extent
    FastDiv by_windows, by_Wp;
    int out_dim, levels;
    unsigned long long off_a, off_b, off_ops; // tables in the parameter blob
};

struct NetPlan {
    int n_layers, classes, input_kind, levels; // input_kind: 0 bytes, 1 float pixels, 2 byte pixels
    long long in_features;
    long long slab_units;
    NetLayer layer[kNetMaxLayers];
    NetStorage store[kNetMaxLayers + 1]; // store[i] = input of layer i; the last layer's output is counted, not stored
};

} // namespace clb

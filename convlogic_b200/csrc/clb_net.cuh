// The compiled network as the one-launch kernel sees it (net_cluster.cu), filled by net.cu.
#pragma once

#include <stdint.h>

namespace clb {

constexpr int kNetMaxLayers = 12;
constexpr int kNetMaxLevels = 256; // thermometer levels (byte pixels take no more)

// n / d by a multiplication for n * d < 2^32 (what plan_one_launch admits)
struct FastDiv {
    unsigned d, magic; // magic = ceil(2^32 / d), unused for d = 1
    __host__ __device__ static FastDiv of(unsigned d) { return FastDiv{d, d > 1 ? (unsigned)((0x100000000ull + d - 1) / d) : 0u}; }
#ifdef __CUDACC__
    __device__ __forceinline__ int div(int n) const { return d > 1 ? (int)__umulhi((unsigned)n, magic) : n; }
#endif
};

// Where the units (16 bytes = 128 samples of one feature) of a layer's input live inside a slab's storage: channels of
// rows x pitch units, the feature's image inside a halo of `ph` rows and `pw` columns.  Flat features: one "channel".
struct NetStorage {
    int base;                // first unit (a multiple of 8: 128 bytes)
    int W, image;            // image width and size (rows * W), 1-D features: image = features
    int pitch, per_channel;  // units per stored row / channel
    int rows, ph, pw;        // image rows, halo
    int halo_units;          // channels * per_channel when there is a halo, else 0
    FastDiv by_image, by_W, by_pitch, by_channel;
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

// Flat LogicLayer kernels on feature-major activations: x [in,B], y [out,B], batch contiguous.
//
// The work is HBM-bound (two gathered input rows and one output row per neuron, three FMAs per
// element), so the layout of the loop is chosen for memory: a half-warp owns a neuron (forward, gate
// gradient), a warp a stretch of input features (input gradient), and sweeps the batch with the widest
// accesses that the rows allow.  The 16 gate values of a neuron are read once: each lane of the half-warp
// loads one value and the soft-max / 4-coefficient reduction runs on shuffles.
//
// Input gradient: segmented reduction over the consumer lists (CSR), no atomics, fixed order.
// A neuron whose two inputs are the same feature is listed twice in a row; the first entry takes the
// derivative w.r.t. its first input and the second w.r.t. its second input, so the sum is the true
// derivative (the reference kernel, src/difflogic/cuda/difflogic_kernel.cu:196-226, applies the
// first-input derivative twice in that case; its CPU path gives the sum used here).
#include "clb_common.cuh"
#include "clb_logic.cuh"

#include <cmath>
#include <type_traits>

namespace clb {

// ---------------------------------------------------------------------------------------- forward
// A half-warp per neuron.  V: elements per access, by the alignment that a row of B elements has; R: accesses of a row in flight per
// lane.  What bounds a neuron is its chain of dependent loads: its first rows are under way while the soft-max of its 16 values is
// taken, and the values and indices of the half-warp's next neuron are loaded a neuron ahead.  (A warp for two neurons in turn, rows
// behind the soft-max: 109660 neurons x 6 layers, 112 samples 228 us, now 124; 519000 neurons, 20 samples 128, now 80.)
template <typename T, int V, int R>
__global__ void __launch_bounds__(256) logic_fwd_kernel(const T *__restrict__ x, const int64_t *__restrict__ ia,
                                                        const int64_t *__restrict__ ib, const T *__restrict__ w, T *__restrict__ y,
                                                        T *__restrict__ coef /* [out][4] for the backward pass, or null */, long long out_dim,
                                                        long long B, int wmode)
{
    const int lane = threadIdx.x & 31, l = lane & 15;
    const long long step = ((long long)gridDim.x * blockDim.x) >> 4;
    long long j = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4, ja = 0, jb = 0;
    T v = T(0);
    auto fetch = [&](long long n) {
        if (n < out_dim) v = w[n * 16 + l], ja = ia[n], jb = ib[n];
    };
    fetch(j);
    for (; j - (lane >> 4) < out_dim; j += step) { // uniform over the warp
        const bool mine = j < out_dim;
        const T *xa = x + ja * B, *xb = x + jb * B;
        T a[R][V], b[R][V], p;
        auto load = [&](long long b0) {
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (b0 + 16 * V * i < B) vload<T, V>(xa + b0 + 16 * V * i, a[i]), vload<T, V>(xb + b0 + 16 * V * i, b[i]);
        };
        if (mine) load(l * V);
        const T mine_v = v;
        fetch(j + step);
        const Gate<T> g = half_warp_gate_of<T>(mine_v, wmode, lane, p);
        if (!mine) continue;
        if (coef != nullptr && l == 0) {
            T *o = coef + 4 * j;
            o[0] = g.k1, o[1] = g.ka, o[2] = g.kb, o[3] = g.kab;
        }
        T *yo = y + j * B;
        for (long long b0 = l * V; b0 < B; b0 += 16 * V * R) {
            if (b0 != l * V) load(b0);
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (b0 + 16 * V * i < B) {
                    T r[V];
#pragma unroll
                    for (int k = 0; k < V; ++k) r[k] = gate_eval<T>(g, a[i][k], b[i][k]);
                    vstore<T, V>(yo + b0 + 16 * V * i, r);
                }
        }
    }
}

// ------------------------------------------------------------------------------------ gate grads
// A half-warp per neuron, as in the forward pass and for its reason: the values and indices come a neuron ahead and the first rows
// are under way while the soft-max is taken.  (A warp for two neurons in turn, first layer of 125090 neurons, 472 samples 114 us, now
// 67; 109660 x 112 44, now 28; 256000 x 1024 269, now 228.  64 registers, so that four blocks are resident: at 74 and three 76, 29, 255.)
template <typename T, int V, int R>
__global__ void __launch_bounds__(256, 4) logic_bwd_w_kernel(const T *__restrict__ x, const int64_t *__restrict__ ia,
                                                             const int64_t *__restrict__ ib, const T *__restrict__ w,
                                                             const T *__restrict__ gy, T *__restrict__ gw, long long out_dim, long long B,
                                                             int wmode)
{
    const int lane = threadIdx.x & 31, l = lane & 15;
    const long long step = ((long long)gridDim.x * blockDim.x) >> 4;
    long long j = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4, ja = 0, jb = 0;
    T v = T(0);
    auto fetch = [&](long long n) {
        if (n < out_dim) v = w[n * 16 + l], ja = ia[n], jb = ib[n];
    };
    fetch(j);
    for (; j - (lane >> 4) < out_dim; j += step) { // uniform over the warp
        const bool mine = j < out_dim;
        const T *xa = x + ja * B, *xb = x + jb * B, *g = gy + j * B;
        T a[R][V], b[R][V], d[R][V], p = T(0);
        auto load = [&](long long b0) {
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (b0 + 16 * V * i < B) {
                    vload<T, V>(g + b0 + 16 * V * i, d[i]);
                    vload<T, V>(xa + b0 + 16 * V * i, a[i]);
                    vload<T, V>(xb + b0 + 16 * V * i, b[i]);
                }
        };
        if (mine) load(l * V);
        const T mine_v = v;
        fetch(j + step);
        if (wmode == CLB_W_SOFTMAX) (void)half_warp_gate_of<T>(mine_v, CLB_W_SOFTMAX, lane, p);
        T s[4] = {T(0), T(0), T(0), T(0)};
        if (mine)
            for (long long b0 = l * V; b0 < B; b0 += 16 * V * R) {
                if (b0 != l * V) load(b0);
#pragma unroll
                for (int i = 0; i < R; ++i)
                    if (b0 + 16 * V * i < B)
#pragma unroll
                        for (int k = 0; k < V; ++k) {
                            s[0] = fma_t<T>(d[i][k], a[i][k] * b[i][k], s[0]);
                            s[1] = fma_t<T>(d[i][k], a[i][k], s[1]);
                            s[2] = fma_t<T>(d[i][k], b[i][k], s[2]);
                            s[3] += d[i][k];
                        }
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        T gi = T(kcoef(0, l)) * s[0] + T(kcoef(1, l)) * s[1] + T(kcoef(2, l)) * s[2] + T(kcoef(3, l)) * s[3];
        if (wmode == CLB_W_SOFTMAX) {
            T dot = p * gi;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            gi = p * (gi - dot);
        }
        if (mine) gw[j * 16 + l] = gi;
    }
}

// ----------------------------------------------------------------------------------- input grads
// gx[f] = sum over the consumers j of feature f (CSR lists built at construction) of  gy[j] * d op_j / d x_f.
// A warp owns a unit = (FPU consecutive features, batch split); the consumer entries of consecutive features are
// one contiguous range of the CSR list, so the warp walks that range 32 entries at a time whatever the fan-out:
// lane l reads entry e0+l, finds the feature it belongs to (a 5-step search over the 32 list starts held by the
// lanes), reads the consumer's two input indices and 16 logits, takes the soft-max and keeps the two coefficients
// (k0, kab) of  d op / d x_f = k0 + kab * other.  The entries are then handed round by shuffles while all lanes
// stream each entry's two rows (gy[j] and the other operand's x row), U entries' loads in flight at a time; the
// running sum is stored and reset whenever the feature changes (features without consumers get zeros).  FPU is 1
// for wide fan-outs (one feature per warp) and up to 32 when a feature has one or two consumers, where a per-feature
// chain of dependent loads would otherwise dominate.  Entries are added in list order: no dependence on scheduling.
template <typename T, int V, int SLOTS>
__global__ void __launch_bounds__(256) logic_bwd_x_kernel(const T *__restrict__ x, const int64_t *__restrict__ ia,
                                                          const int64_t *__restrict__ ib, const T *__restrict__ w,
                                                          const T *__restrict__ gy, T *__restrict__ gx,
                                                          const int64_t *__restrict__ start, const int64_t *__restrict__ cons,
                                                          long long in_dim, long long out_dim, long long B, int wmode,
                                                          int batch_splits, int fpu)
{
    constexpr int U = 8 / SLOTS; // entries whose rows are loaded before the first is added
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    // a split is a multiple of 32*V elements
    const long long span = ((B + (long long)batch_splits * 32 * V - 1) / ((long long)batch_splits * 32 * V)) * 32 * V;
    const long long funits = (in_dim + fpu - 1) / fpu;
    for (long long unit = warp; unit < funits * batch_splits; unit += nwarps) {
        const long long f0 = (unit / batch_splits) * fpu, f1 = min(in_dim, f0 + fpu);
        const long long blo = (unit % batch_splits) * span, bhi = min(B, blo + span);
        const long long my_start = start[min(f0 + lane, f1)]; // lanes past the unit hold its end
        const long long lo = __shfl_sync(0xffffffffu, my_start, 0), hi = start[f1];
        for (long long bb = blo; bb < bhi; bb += (long long)SLOTS * 32 * V) {
            T acc[SLOTS][V];
#pragma unroll
            for (int q = 0; q < SLOTS; ++q)
#pragma unroll
                for (int k = 0; k < V; ++k) acc[q][k] = T(0);
            long long cur_f = f0; // the feature `acc` belongs to
            auto flush_to = [&](long long f_next) {
                while (cur_f < f_next) {
#pragma unroll
                    for (int q = 0; q < SLOTS; ++q) {
                        const long long b0 = bb + ((long long)q * 32 + lane) * V;
                        if (b0 < bhi) vstore<T, V>(gx + cur_f * B + b0, acc[q]);
#pragma unroll
                        for (int k = 0; k < V; ++k) acc[q][k] = T(0);
                    }
                    ++cur_f;
                }
            };
            for (long long c0 = lo; c0 < hi; c0 += 32) {
                const long long e = c0 + lane;
                int my_j = 0, my_other = 0, my_f = 0;
                T my_k0 = T(0), my_kab = T(0);
                {
                    // the feature of entry e: the last lane whose list start is <= e (entries past the range: any)
                    int sel = 0;
#pragma unroll
                    for (int step = 16; step >= 1; step >>= 1) {
                        const long long sv = __shfl_sync(0xffffffffu, my_start, sel + step);
                        if (sv <= e) sel += step;
                    }
                    const long long fs = __shfl_sync(0xffffffffu, my_start, sel);
                    if (e < hi) {
                        const long long f = f0 + sel;
                        const long long j = cons[e];
                        const long long a_j = ia[j], b_j = ib[j];
                        // a neuron fed twice by f is listed twice in a row: the first entry is w.r.t. a, the second w.r.t. b
                        const bool second = (a_j == f) && (b_j == f) && (e > fs) && (cons[e - 1] == j);
                        const bool wrt_a = (a_j == f) && !second;
                        const Gate<T> g = gate_load<T>(w + j * 16, wmode);
                        my_j = (int)j, my_other = (int)(wrt_a ? b_j : a_j), my_f = sel;
                        my_k0 = wrt_a ? g.ka : g.kb, my_kab = g.kab;
                    }
                }
                const int n = (int)min((long long)32, hi - c0);
                for (int i0 = 0; i0 < n; i0 += U) {
                    T o[U][SLOTS][V], d[U][SLOTS][V], k0[U], kab[U];
                    int fi[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int i = min(i0 + u, n - 1); // past the end: a repeated load that is not added
                        const T *xo = x + (long long)__shfl_sync(0xffffffffu, my_other, i) * B;
                        const T *gr = gy + (long long)__shfl_sync(0xffffffffu, my_j, i) * B;
                        k0[u] = __shfl_sync(0xffffffffu, my_k0, i), kab[u] = __shfl_sync(0xffffffffu, my_kab, i);
                        fi[u] = __shfl_sync(0xffffffffu, my_f, i);
#pragma unroll
                        for (int q = 0; q < SLOTS; ++q) {
                            const long long b0 = bb + ((long long)q * 32 + lane) * V;
                            if (b0 < bhi) {
                                vload<T, V>(xo + b0, o[u][q]);
                                vload<T, V>(gr + b0, d[u][q]);
                            } else {
#pragma unroll
                                for (int k = 0; k < V; ++k) o[u][q][k] = T(0), d[u][q][k] = T(0);
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (i0 + u < n) {
                            flush_to(f0 + fi[u]);
#pragma unroll
                            for (int q = 0; q < SLOTS; ++q)
#pragma unroll
                                for (int k = 0; k < V; ++k) acc[q][k] = fma_t<T>(d[u][q][k], fma_t<T>(kab[u], o[u][q][k], k0[u]), acc[q][k]);
                        }
                    }
                }
            }
            flush_to(f1);
        }
    }
}

// ----------------------------------------------------------------------------------- group sum
// GroupSum on the feature-major activations the flat layers produce ([F][B]; class c owns rows [c*S, (c+1)*S)):
// out[b][c] = (sum of the class's rows at sample b) / tau.  The rows of a class are 16 parts (one when there are few) of eight
// chains, row by row in turn; chains are added in order, then parts.  No transposed copy of the activations, no atomics.
constexpr int kGroupSumParts = 16;

// Block (batch tile, class, part): a warp per chain.
template <typename T>
__global__ void __launch_bounds__(256) group_sum_partial_kernel(const T *__restrict__ y, T *__restrict__ partial, long long S, long long B, int k)
{
    __shared__ T red[8][32];
    const int lane = threadIdx.x & 31, wv = threadIdx.x >> 5;
    const long long b = (long long)blockIdx.x * 32 + lane;
    const int c = blockIdx.y, part = blockIdx.z;
    const long long r0 = S * part / gridDim.z, r1 = S * (part + 1) / gridDim.z;
    T acc = T(0);
    if (b < B)
        for (long long r = r0 + wv; r < r1; r += 8) acc += y[((long long)c * S + r) * B + b];
    red[wv][lane] = acc;
    __syncthreads();
    if (wv == 0 && b < B) {
        T t = red[0][lane];
#pragma unroll
        for (int i = 1; i < 8; ++i) t += red[i][lane];
        partial[((long long)part * k + c) * B + b] = t;
    }
}

// Few rows and blocks (clb_group_sum_fwd): block (batch tile, class), two warps to a part and four chains to a warp, and no second launch.
template <typename T>
__global__ void __launch_bounds__(1024) group_sum_one_kernel(const T *__restrict__ y, T *__restrict__ out, long long S, long long B, int k, int parts, T tau)
{
    __shared__ T red[kGroupSumParts][8][32];
    const int lane = threadIdx.x & 31, wv = threadIdx.x >> 5, part = wv >> 1, w0 = (wv & 1) * 4;
    const long long b = (long long)blockIdx.x * 32 + lane;
    const int c = blockIdx.y;
    if (part < parts && b < B) {
        const long long r0 = S * part / parts, r1 = S * (part + 1) / parts;
        const T *col = y + (long long)c * S * B + b;
        T acc[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 4
        for (long long r = r0 + w0; r < r1; r += 8)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (r + j < r1) acc[j] += col[(r + j) * B];
#pragma unroll
        for (int j = 0; j < 4; ++j) red[part][w0 + j][lane] = acc[j];
    }
    __syncthreads();
    if (wv < parts) {
        T t = red[wv][0][lane];
#pragma unroll
        for (int i = 1; i < 8; ++i) t += red[wv][i][lane];
        red[wv][0][lane] = t;
    }
    __syncthreads();
    if (wv == 0 && b < B) {
        T t = T(0);
        for (int p = 0; p < parts; ++p) t += red[p][0][lane];
        out[b * k + c] = t / tau;
    }
}

template <typename T>
__global__ void group_sum_finalize_kernel(const T *__restrict__ partial, T *__restrict__ out, long long B, int k, int parts, T tau)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; // (c, b), b fastest
    if (i >= B * k) return;
    const long long c = i / B, b = i - c * B;
    T t = T(0);
    for (int p = 0; p < parts; ++p) t += partial[((long long)p * k + c) * B + b];
    out[b * k + c] = t / tau;
}

// GroupSum + cross-entropy finish (src/convlogic/model.py:137-152: CrossEntropyLoss on the GroupSum scores):
// scores[b][c] = (sum of the parts) / tau, loss = mean_b (logsumexp(scores[b]) - scores[b][label_b]), and
// dscore[b][c] = (softmax(scores[b])[c] - [c == label_b]) / B, the gradient of the mean loss w.r.t. the scores.
// A warp per sample, lane c = class c (k <= 32): the parts are added in part order with all loads in flight, the
// soft-max is two warp reductions.  The sample's loss overwrites partial[b] (part 0, class 0 of that sample: read by this
// warp alone, before the write); group_sum_loss_mean_kernel adds the B losses in a fixed tree.
__global__ void __launch_bounds__(256) group_sum_ce_sample_kernel(float *__restrict__ partial, const int64_t *__restrict__ labels,
                                                                  float *__restrict__ scores, float *__restrict__ dscore, long long B, int k,
                                                                  int parts, float tau)
{
    const int lane = threadIdx.x & 31;
    const long long b = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (b >= B) return; // the whole warp
    float sc = -3.0e38f;
    if (lane < k) {
        float t = 0.f;
        for (int p = 0; p < parts; p += 32) { // (a chain of loads eight at a time took 7.1 us for 59 parts of 256 samples)
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (p + j < parts) v[j] = partial[((long long)(p + j) * k + lane) * B + b];
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (p + j < parts) t += v[j];
        }
        sc = t / tau;
    }
    float mx = sc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e = lane < k ? expf(sc - mx) : 0.f;
    const float sum = warp_sum<float>(e);
    const int lab = (int)labels[b];
    const bool lab_ok = lab >= 0 && lab < k;
    const float sc_lab = __shfl_sync(0xffffffffu, sc, lab_ok ? lab : 0);
    if (lane < k) {
        if (scores != nullptr) scores[b * k + lane] = sc;
        dscore[b * k + lane] = (e / sum - (lane == lab ? 1.f : 0.f)) / (float)B;
    }
    __syncwarp();
    if (lane == 0) partial[b] = mx + logf(sum) - (lab_ok ? sc_lab : 0.f);
}

__global__ void __launch_bounds__(256) group_sum_loss_mean_kernel(const float *__restrict__ sample_loss, float *__restrict__ loss, long long B)
{
    __shared__ float red[256];
    float mine = 0.f;
    for (long long b = threadIdx.x; b < B; b += 256) mine += sample_loss[b];
    red[threadIdx.x] = mine;
    __syncthreads();
    for (int half = 128; half >= 1; half >>= 1) {
        if ((int)threadIdx.x < half) red[threadIdx.x] += red[threadIdx.x + half];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] / (float)B;
}

// out[c][r] = in[r][c]: 32 x 32 tiles through shared memory (33-float rows: no bank conflicts), both sides coalesced.
// The flat layers work on feature-major activations [features][batch]; this is the copy between that and the
// [batch][features] tensors of the layers around them.
__global__ void __launch_bounds__(256) transpose_f32_kernel(const float *__restrict__ in, float *__restrict__ out, long long R, long long Cc)
{
    __shared__ float tile[32][33];
    const long long c0 = (long long)blockIdx.x * 32, r0 = (long long)blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long r = r0 + ty + 8 * i, c = c0 + tx;
        if (r < R && c < Cc) tile[ty + 8 * i][tx] = __ldg(in + r * Cc + c);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long c = c0 + ty + 8 * i, r = r0 + tx;
        if (r < R && c < Cc) out[c * R + r] = tile[tx][ty + 8 * i];
    }
}

// Adam / AdamW over one flat parameter buffer (src/convlogic/model.py:179-180 uses torch.optim.AdamW): one thread per
// four elements, 128-bit accesses.  step_size = lr / (1 - beta1^t), bc2_sqrt = sqrt(1 - beta2^t).
__global__ void __launch_bounds__(256) adam_step_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                                                        float *__restrict__ v, long long n, float lr, float beta1, float beta2, float eps,
                                                        float weight_decay, float step_size, float bc2_sqrt, int decoupled)
{
    auto one = [&](float &pp, float gg, float &mm, float &vv) {
        if (weight_decay != 0.f) {
            if (decoupled)
                pp *= 1.f - lr * weight_decay;
            else
                gg = fmaf(weight_decay, pp, gg);
        }
        mm = fmaf(1.f - beta1, gg - mm, mm);           // exp_avg.lerp_(grad, 1 - beta1)
        vv = fmaf(1.f - beta2, gg * gg, beta2 * vv);   // exp_avg_sq.mul_(beta2).addcmul_(grad, grad, 1 - beta2)
        const float denom = sqrtf(vv) / bc2_sqrt + eps;
        pp -= step_size * (mm / denom);
    };
    const long long n4 = n >> 2;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        float4 pp = reinterpret_cast<float4 *>(p)[i], mm = reinterpret_cast<float4 *>(m)[i], vv = reinterpret_cast<float4 *>(v)[i];
        const float4 gg = reinterpret_cast<const float4 *>(g)[i];
        one(pp.x, gg.x, mm.x, vv.x), one(pp.y, gg.y, mm.y, vv.y), one(pp.z, gg.z, mm.z, vv.z), one(pp.w, gg.w, mm.w, vv.w);
        reinterpret_cast<float4 *>(p)[i] = pp, reinterpret_cast<float4 *>(m)[i] = mm, reinterpret_cast<float4 *>(v)[i] = vv;
    }
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
        const long long i = (n4 << 2) + threadIdx.x;
        one(p[i], g[i], m[i], v[i]);
    }
}

// gy[f][b] = gout[b][f / S] / tau.  grid (row chunks, k): a thread keeps the quotients of its batch positions -- V neighbours at
// a time -- in registers and writes them to every row of its chunk; a batch that needs fewer than 256 threads leaves the rest
// to further rows.
template <typename T, int V>
__global__ void __launch_bounds__(256) group_sum_bwd_kernel(const T *__restrict__ gout, const T *__restrict__ scale, T *__restrict__ gy,
                                                            long long S, long long B, int k, T tau)
{
    const int c = blockIdx.y;
    if (scale != nullptr) tau = tau / scale[0]; // an upstream scalar gradient, read on the device
    const long long r0 = S * blockIdx.x / gridDim.x, r1 = S * (blockIdx.x + 1) / gridDim.x;
    const int per_row = (int)min(256LL, (B + V - 1) / V), rows = 256 / per_row; // threads per row, rows at a time
    const int row = threadIdx.x / per_row, col = threadIdx.x - row * per_row;
    if (row >= rows) return;
    for (long long b0 = (long long)col * V; b0 < B; b0 += (long long)per_row * V) {
        T v[V];
#pragma unroll
        for (int q = 0; q < V; ++q) v[q] = gout[(b0 + q) * k + c] / tau;
        for (long long r = r0 + row; r < r1; r += rows) vstore<T, V>(gy + ((long long)c * S + r) * B + b0, v);
    }
}

// The same where rows of B floats are not whole 16-byte words: a chunk is one contiguous stretch of gy, written in aligned words of
// four from the class's B quotients in shared memory, so that the L2 gets whole sectors.  Bound by the writes (a float per store:
// 125090 x 473 65 us, now 40; 256000 x 1022 380, now 186: 86 % of the copy rate).  At most kGroupSumFlatMax quotients.
constexpr int kGroupSumFlatMax = 4096;
__global__ void __launch_bounds__(256) group_sum_bwd_flat_kernel(const float *__restrict__ gout, const float *__restrict__ scale, float *__restrict__ gy,
                                                                 long long S, int B, int k, float tau)
{
    extern __shared__ float quot[];
    const int c = blockIdx.y, tid = threadIdx.x;
    if (scale != nullptr) tau = tau / scale[0];
    for (int b = tid; b < B; b += 256) quot[b] = gout[(long long)b * k + c] / tau;
    __syncthreads();
    const long long r0 = S * blockIdx.x / gridDim.x, r1 = S * (blockIdx.x + 1) / gridDim.x;
    const long long first = (c * S + r0) * B, n = (r1 - r0) * B;
    const int lead = (int)min(n, (4 - (first & 3)) & 3);
    const long long words = (n - lead) >> 2;
    gy += first;
    if (tid < lead) gy[tid] = quot[tid % B];
    const int step = 1024 % B;
    int b = (lead + 4 * tid) % B;
    for (long long i = tid; i < words; i += 256) {
        const int b1 = b + 1 < B ? b + 1 : 0, b2 = b1 + 1 < B ? b1 + 1 : 0, b3 = b2 + 1 < B ? b2 + 1 : 0;
        reinterpret_cast<float4 *>(gy + lead)[i] = make_float4(quot[b], quot[b1], quot[b2], quot[b3]);
        b += step;
        if (b >= B) b -= B;
    }
    const long long done = lead + 4 * words;
    if (tid < n - done) gy[done + tid] = quot[(done + tid) % B];
}

// ----------------------------------------------------------------------------------- fused flat layers (training)
// Three consecutive flat layers whose outputs are each read at most once by the next one, as ONE differentiable
// gate tree per neuron of the last layer: leaf [T][8] are rows of the first layer's input (gate p of the first
// level reads leaves 2p, 2p+1), node [T][7] the neuron that sits at each tree position (4 of the first layer, 2 of
// the second, 1 of the third: its logits are the gate's).  The two intermediate activations are never written.
// Forward: a warp per tree, lanes along the batch.  Backward pass 1: the chain recomputed from the leaves, the
// gradient w.r.t. each leaf written as a row of `tapgrad` [T*8][B], the 28 basis sums of the 7 gates reduced over
// the batch and turned into the logit (or mixture) gradients of the 7 neurons.  Pass 2: gx[f] = sum of the
// tapgrad rows of the leaves that are feature f (CSR by feature, fixed order).
struct TreeTables {
    const int32_t *leaf; // [T][8]
    const int32_t *node; // [T][7]
    const float *w[3];   // logits (or mixtures) of the three layers
};

// ---- the seven gates of a tree on the warp's lanes: the quad of lanes 4g..4g+3 owns gate g (lanes 28..31 idle), lane
// q = lane & 3 of a quad holds entries 4q..4q+3 of the gate's 16.  Gate id j = 4q + i has truth-table bits (q >> 1,
// q & 1, i >> 1, i & 1), so the coefficients of the multilinear form follow from three sums of the lane's four entries.
__device__ __forceinline__ float quad_sum(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// the lane's four entries of the mixture over the 16 gates from those of the values p (zeros on an idle lane); every lane of the warp
// calls this
__device__ __forceinline__ void quad_mixture(int wmode, int q, float (&p)[4])
{
    if (wmode == CLB_W_SOFTMAX) {
        float m = fmaxf(fmaxf(p[0], p[1]), fmaxf(p[2], p[3]));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = expf(p[i] - m);
        const float inv = 1.f / quad_sum((p[0] + p[1]) + (p[2] + p[3]));
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] *= inv;
    } else if (wmode == CLB_W_ARGMAX) {   // the first largest entry, as a scan from entry 0 finds it
        float m = p[0];
        int best = 4 * q;
#pragma unroll
        for (int i = 1; i < 4; ++i)
            if (p[i] > m) m = p[i], best = 4 * q + i;
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            const float mo = __shfl_xor_sync(0xffffffffu, m, o);
            const int bo = __shfl_xor_sync(0xffffffffu, best, o);
            if (mo > m || (mo == m && bo < best)) m = mo, best = bo;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = (4 * q + i == best) ? 1.f : 0.f;
    }
}

// coefficients of the quad's gate from the four lanes' mixture entries (every lane of the quad gets them)
__device__ __forceinline__ Gate<float> quad_gate(const float (&p)[4], int q)
{
    const float q3 = (float)(q >> 1), q2 = (float)(q & 1);
    const float all = (p[0] + p[1]) + (p[2] + p[3]), hi = p[2] + p[3], odd = p[1] + p[3];
    Gate<float> g;
    g.k1 = quad_sum(q3 * all);
    g.ka = quad_sum(hi - q3 * all);
    g.kb = quad_sum((q2 - q3) * all);
    g.kab = quad_sum(odd - hi + (q3 - q2) * all);
    return g;
}

// the row of 16 values of neuron n behind the lane's gate (lane < 28)
__device__ __forceinline__ const float *tree_row(const TreeTables &tt, int lane, long long n)
{
    const int g = lane >> 2;
    return tt.w[g < 4 ? 0 : (g < 6 ? 1 : 2)] + n * 16;
}

// the lane's four of the values of its neuron n
__device__ __forceinline__ void tree_values(const TreeTables &tt, long long n, int lane, float (&p)[4])
{
    const bool active = lane < 28;
    const float *w16 = tree_row(tt, active ? lane : 0, n);
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = active ? __ldg(w16 + 4 * (lane & 3) + i) : 0.f;
}

// The seven gates of the warp's tree into sg (as k1, ka, kb, kab); p: the lane's four values, then its four mixture entries.
__device__ __forceinline__ void tree_gates_to(float4 *sg, int lane, int wmode, float (&p)[4])
{
    quad_mixture(wmode, lane & 3, p);
    const Gate<float> mine = quad_gate(p, lane & 3);
    __syncwarp(); // the tree before is done with them
    if (lane < 28 && (lane & 3) == 0) sg[lane >> 2] = make_float4(mine.k1, mine.ka, mine.kb, mine.kab);
    __syncwarp();
}
__device__ __forceinline__ Gate<float> tree_gate(const float4 *sg, int i)
{
    const float4 v = sg[i];
    return Gate<float>{v.x, v.y, v.z, v.w};
}
// the trees' output for the lane's V samples
template <int V> __device__ __forceinline__ void tree_eval(const float4 *sg, const float (&a)[8][V], float (&r)[V])
{
    float t[2][V];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const Gate<float> g0 = tree_gate(sg, 2 * h), g1 = tree_gate(sg, 2 * h + 1), g2 = tree_gate(sg, 4 + h);
#pragma unroll
        for (int e = 0; e < V; ++e)
            t[h][e] = gate_eval<float>(g2, gate_eval<float>(g0, a[4 * h][e], a[4 * h + 1][e]), gate_eval<float>(g1, a[4 * h + 2][e], a[4 * h + 3][e]));
    }
    const Gate<float> g = tree_gate(sg, 6);
#pragma unroll
    for (int e = 0; e < V; ++e) r[e] = gate_eval<float>(g, t[0][e], t[1][e]);
}

template <int V>
__global__ void __launch_bounds__(256, 3) logic_tree_fwd_kernel(const float *__restrict__ x, TreeTables tt, float *__restrict__ y, long long T,
                                                             long long B, int wmode)
{
    __shared__ float4 gates[8][7];
    float4 *sg = gates[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    // The tables of a tree (leaf rows on lanes 0..7, the gates' neurons on lanes 0..27) are fetched one tree ahead, so that
    // a tree's own chain of dependent loads is one hop (the rows, the logits) instead of two (index, then data).
    int my_leaf = (warp < T && lane < 8) ? __ldg(tt.leaf + warp * 8 + lane) : 0;
    int my_node = (warp < T && lane < 28) ? __ldg(tt.node + warp * 7 + (lane >> 2)) : 0;
    for (long long t = warp; t < T; t += nwarps) {
        const long long tn = t + nwarps;
        const int nx_leaf = (tn < T && lane < 8) ? __ldg(tt.leaf + tn * 8 + lane) : 0;
        const int nx_node = (tn < T && lane < 28) ? __ldg(tt.node + tn * 7 + (lane >> 2)) : 0;
        float pq[4];
        tree_values(tt, my_node, lane, pq);
        tree_gates_to(sg, lane, wmode, pq);
        const float *row[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) row[k] = x + (long long)__shfl_sync(0xffffffffu, my_leaf, k) * B;
        my_leaf = nx_leaf, my_node = nx_node;
        for (long long b0 = (long long)lane * V; b0 < B; b0 += 32 * V) {
            float a[8][V], r[V];
#pragma unroll
            for (int k = 0; k < 8; ++k) vload<float, V>(row[k] + b0, a[k]);
            tree_eval<V>(sg, a, r);
            vstore<float, V>(y + t * B + b0, r);
        }
    }
}

// Forward of the trees when they feed GroupSum: the class sums directly, without the activation [T][B] (nothing but the
// class sums reads it in a training step).  Block (part, class): its 8 warps share the trees of one part of one class
// (tree i of the part goes to warp i % 8), a lane adds up the outputs of its samples over the warp's trees in tree order, the
// 8 warps' sums are added in warp order: partial[(part * k + class) * B + b], the layout group_sum_ce_sample_kernel reads.
// Gates and running sums in shared memory, four rows at a time and a gate's values a tree ahead: 64 registers, so that four blocks of an SM
// take nearly all parts in one wave (k = 256, 256 samples 108 -> 104 us, k = 32, 100 samples 13.5 -> 11.7; it is a hundredth of
// the blocks that are left for a second one, and fewer parts would add in another order).
template <int TR>
__global__ void __launch_bounds__(256, 4) logic_tree_fwd_sum_kernel(const float *__restrict__ x, TreeTables tt, float *__restrict__ partial,
                                                                 long long T, long long batch, int k, int wmode)
{
    __shared__ __align__(16) float red[8][TR * 128]; // a lane's running sums: in registers they would cost a resident block
    __shared__ float4 gates[8][7];
    const int lane = threadIdx.x & 31, wv = threadIdx.x >> 5;
    const int cls = blockIdx.y, part = blockIdx.x, parts = gridDim.x;
    const long long S = T / k;
    const int t_lo = (int)(cls * S + S * part / parts), t_hi = (int)(cls * S + S * (part + 1) / parts), B = (int)batch;
    float4 *sg = gates[wv];
    float4 *const acc = reinterpret_cast<float4 *>(red[wv]) + lane;
#pragma unroll
    for (int tr = 0; tr < TR; ++tr) acc[tr * 32] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int t0 = t_lo + wv;
    int my_leaf = (t0 < t_hi && lane < 8) ? __ldg(tt.leaf + t0 * 8 + lane) : 0;   // index tables one tree ahead
    int my_node = (t0 < t_hi && lane < 28) ? __ldg(tt.node + t0 * 7 + (lane >> 2)) : 0;
    int nx_node = (t0 + 8 < t_hi && lane < 28) ? __ldg(tt.node + (t0 + 8) * 7 + (lane >> 2)) : 0;
    float raw[4]; // its values one tree ahead
    tree_values(tt, my_node, lane, raw);
    for (int t = t0; t < t_hi; t += 8) {
        const int tn = t + 8, tnn = t + 16;
        const int nx_leaf = (tn < t_hi && lane < 8) ? __ldg(tt.leaf + tn * 8 + lane) : 0;
        const int nn_node = (tnn < t_hi && lane < 28) ? __ldg(tt.node + tnn * 7 + (lane >> 2)) : 0;
        float pq[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pq[i] = raw[i];
        if (tn < t_hi) tree_values(tt, nx_node, lane, raw);
        tree_gates_to(sg, lane, wmode, pq);
#pragma unroll 1
        for (int tr = 0; tr < TR; ++tr) {
            const int b0 = (tr * 32 + lane) * 4;
            float t[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h) { // four rows at a time
                float a[4][4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float *row = x + ((long long)__shfl_sync(0xffffffffu, my_leaf, 4 * h + q) * B + b0);
                    if (b0 < B) vload<float, 4>(row, a[q]);
                }
                const Gate<float> g0 = tree_gate(sg, 2 * h), g1 = tree_gate(sg, 2 * h + 1), g2 = tree_gate(sg, 4 + h);
#pragma unroll
                for (int e = 0; e < 4; ++e) t[h][e] = gate_eval<float>(g2, gate_eval<float>(g0, a[0][e], a[1][e]), gate_eval<float>(g1, a[2][e], a[3][e]));
            }
            if (b0 < B) {
                float r[4];
                const Gate<float> g = tree_gate(sg, 6);
#pragma unroll
                for (int e = 0; e < 4; ++e) r[e] = gate_eval<float>(g, t[0][e], t[1][e]);
                float4 sum = acc[tr * 32];
                sum.x += r[0], sum.y += r[1], sum.z += r[2], sum.w += r[3];
                acc[tr * 32] = sum;
            }
        }
        my_leaf = nx_leaf, my_node = nx_node, nx_node = nn_node;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < TR * 128; i += 256) {
        if (i < B) {
            float t = red[0][i];
#pragma unroll
            for (int w = 1; w < 8; ++w) t += red[w][i];
            partial[((long long)part * k + cls) * B + i] = t;
        }
    }
}

// HEAD: the upstream gradient is not a tensor [T][B] but the GroupSum + cross-entropy head's d loss / d score [B][k]:
// tree t belongs to class t / S and gy[t][b] = dscore[b][class] / (tau / scale), exactly what group_sum_bwd_kernel would
// have written -- the [T][B] gradient is then neither written nor read.
struct TreeHead {
    const float *dscore, *scale; // scale: the scalar gradient that reaches the loss, on the device
    int k;
    unsigned S;                  // trees per class
    float tau;
};

constexpr long long kTreeRows = 1LL << 19; // outputs of the trees from which on their upstream gradients are laid out as rows

// The head's upstream gradients as rows, a class each: up [k][B].  Read straight from dscore, a lane's four values lie four lines
// apart (32 look-ups in the L1 per load instead of four) and are divided again for every tree.
__global__ void __launch_bounds__(256) tree_head_rows_kernel(float *__restrict__ up, long long B, TreeHead head)
{
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= B * head.k) return;
    const long long c = i / B, b = i - c * B;
    up[i] = __ldg(head.dscore + b * head.k + c) / (head.tau / __ldg(head.scale));
}

constexpr int kTreeStages = 2, // (k = 256, 256 samples: 202 us with two, 208 with three, 215 with four)
              kTreeStageBytes = 8 * 512, kTreeSmem = 4 * kTreeStages * kTreeStageBytes;

// !HEAD: tree t's upstream gradient is row t / head.S of gy
template <int V, bool HEAD, bool ONCE>
__global__ void __launch_bounds__(128, 3) logic_tree_bwd_kernel(const float *__restrict__ x, TreeTables tt, const float *__restrict__ gy,
                                                             float *__restrict__ tapgrad, float *__restrict__ gw0, float *__restrict__ gw1,
                                                             float *__restrict__ gw2, int T, int B, int wmode, TreeHead head)
{
    extern __shared__ __align__(16) unsigned char tree_smem[];
    __shared__ float4 gates[4][7];
    const int lane = threadIdx.x & 31;
    const int warp = (int)((blockIdx.x * 128u + threadIdx.x) >> 5), nwarps = (int)(gridDim.x * 4u);
    // V = 4: the leaf rows arrive kTreeStages - 1 trips of 128 samples ahead in shared memory, each lane's 16 bytes by its own copy (so that
    // nothing has to be synchronised), in one wave of blocks that walk on from tree to tree; a gate's values come a tree ahead.  What was
    // waited for before: the classes' upstream gradients (tree_head_rows_kernel), rows and values of a tree one after the other at
    // 12 warps per SM (k = 256, 256 samples: 269 us, now 193; k = 32, 100 samples 23 and 18).  The tree and trip fetched next:
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(tree_smem) + (threadIdx.x >> 5) * (kTreeStages * kTreeStageBytes) + lane * 16;
    int ft = warp, fb = 0, fslot = 0, f_leaf = 0, f_next = 0;
    auto fetch = [&] {
        if (ft < T) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float *row = x + ((long long)__shfl_sync(0xffffffffu, f_leaf, k) * B + fb + lane * 4);
                if (fb + lane * 4 < B) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring + fslot * kTreeStageBytes + k * 512), "l"(row) : "memory");
            }
            fb += 128;
            if (fb >= B) {
                fb = 0, ft += nwarps, f_leaf = f_next;
                f_next = (ft + nwarps < T && lane < 8) ? __ldg(tt.leaf + (ft + nwarps) * 8 + lane) : 0;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        fslot = fslot + 1 == kTreeStages ? 0 : fslot + 1;
    };
    int slot = 0;
    if (V == 4) {
        f_leaf = (warp < T && lane < 8) ? __ldg(tt.leaf + warp * 8 + lane) : 0;
        f_next = (warp + nwarps < T && lane < 8) ? __ldg(tt.leaf + (warp + nwarps) * 8 + lane) : 0;
#pragma unroll
        for (int i = 0; i < kTreeStages - 1; ++i) fetch();
    }
    // 128-thread blocks, three per SM: 168 registers, nothing spilled (at 256 threads x 2 blocks the limit of 128 registers
    // spilled 144 bytes).  The index tables are fetched one tree ahead, as in the forward kernel.
    int my_leaf = (V != 4 && warp < T && lane < 8) ? __ldg(tt.leaf + warp * 8 + lane) : 0;
    int my_node = (warp < T && lane < 28) ? __ldg(tt.node + warp * 7 + (lane >> 2)) : 0;
    int nx_node = (warp + nwarps < T && lane < 28) ? __ldg(tt.node + (warp + nwarps) * 7 + (lane >> 2)) : 0;
    float raw[4];
    tree_values(tt, my_node, lane, raw);
    for (int t = warp; t < T; t += nwarps) {
        const int tn = t + nwarps, tnn = tn + nwarps;
        const int nx_leaf = (V != 4 && tn < T && lane < 8) ? __ldg(tt.leaf + tn * 8 + lane) : 0;
        const int nn_node = (tnn < T && lane < 28) ? __ldg(tt.node + tnn * 7 + (lane >> 2)) : 0;
        Gate<float> g[7];
        float pq[4]; // the lane's four mixture entries, kept for the soft-max Jacobian at the end
#pragma unroll
        for (int i = 0; i < 4; ++i) pq[i] = raw[i];
        if (tn < T) tree_values(tt, nx_node, lane, raw); // a tree ahead
        tree_gates_to(gates[threadIdx.x >> 5], lane, wmode, pq);
#pragma unroll
        for (int i = 0; i < 7; ++i) g[i] = tree_gate(gates[threadIdx.x >> 5], i);
        float bs[28];
#pragma unroll
        for (int i = 0; i < 28; ++i) bs[i] = 0.f;
        // V = 1: rows found once per tree and numbers of 64 bits (at every trip of 32 samples, in 32 bits, 40960 trees of 131 samples took 142 us,
        // 120 with the rows alone, now 117)
        using Index = std::conditional_t<V == 4, int, long long>;
        const Index samples = B;
        const float *row[8];
        if constexpr (V != 4) {
#pragma unroll
            for (int k = 0; k < 8; ++k) row[k] = x + (long long)__shfl_sync(0xffffffffu, my_leaf, k) * B;
        }
        for (Index bb = V == 4 ? 0 : lane; bb < B; bb += 32 * V) { // V = 4: uniform over the warp, the rows' numbers are handed round
            const Index b0 = V == 4 ? bb + lane * V : bb;
            float a[8][V], dz[V], dg[4][V];
            if constexpr (V == 4) {
                fetch();
                asm volatile("cp.async.wait_group %0;" ::"n"(kTreeStages - 1) : "memory");
                if (b0 < B) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a[k][0]), "=f"(a[k][1]), "=f"(a[k][2]), "=f"(a[k][3])
                                     : "r"(ring + slot * kTreeStageBytes + k * 512));
                }
                slot = slot + 1 == kTreeStages ? 0 : slot + 1;
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) vload<float, V>(row[k] + b0, a[k]);
            }
            if (b0 >= B) continue;
            if (HEAD) {
                const float taus = head.tau / __ldg(head.scale);
                const float *ds = head.dscore + (long long)b0 * head.k + (unsigned)t / head.S;
#pragma unroll
                for (int e = 0; e < V; ++e) dz[e] = __ldg(ds + e * head.k) / taus;
            } else {
                vload<float, V>(gy + (long long)((unsigned)t / head.S) * B + b0, dz);
            }
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const float g0 = gate_eval<float>(g[0], a[0][e], a[1][e]), g1 = gate_eval<float>(g[1], a[2][e], a[3][e]);
                const float g2 = gate_eval<float>(g[2], a[4][e], a[5][e]), g3 = gate_eval<float>(g[3], a[6][e], a[7][e]);
                const float t0 = gate_eval<float>(g[4], g0, g1), t1 = gate_eval<float>(g[5], g2, g3);
                const float d = dz[e];
                const float dt0 = d * gate_da<float>(g[6], t1), dt1 = d * gate_db<float>(g[6], t0);
                dg[0][e] = dt0 * gate_da<float>(g[4], g1), dg[1][e] = dt0 * gate_db<float>(g[4], g0);
                dg[2][e] = dt1 * gate_da<float>(g[5], g3), dg[3][e] = dt1 * gate_db<float>(g[5], g2);
                bs[16] = fmaf(dt0, g0 * g1, bs[16]), bs[17] = fmaf(dt0, g0, bs[17]), bs[18] = fmaf(dt0, g1, bs[18]), bs[19] += dt0;
                bs[20] = fmaf(dt1, g2 * g3, bs[20]), bs[21] = fmaf(dt1, g2, bs[21]), bs[22] = fmaf(dt1, g3, bs[22]), bs[23] += dt1;
                bs[24] = fmaf(d, t0 * t1, bs[24]), bs[25] = fmaf(d, t0, bs[25]), bs[26] = fmaf(d, t1, bs[26]), bs[27] += d;
            }
            // leaf gradients pair by pair, stored at once so that they do not occupy registers
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                float ta[V], tb[V];
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const float x0 = a[2 * p][e], x1 = a[2 * p + 1][e], d = dg[p][e];
                    ta[e] = d * gate_da<float>(g[p], x1), tb[e] = d * gate_db<float>(g[p], x0);
                    bs[4 * p] = fmaf(d, x0 * x1, bs[4 * p]), bs[4 * p + 1] = fmaf(d, x0, bs[4 * p + 1]);
                    bs[4 * p + 2] = fmaf(d, x1, bs[4 * p + 2]), bs[4 * p + 3] += d;
                }
                float *const to = tapgrad + ((long long)(t * 8 + 2 * p) * samples + b0);
                if (ONCE)
                    vstore_once<float, V>(to, ta), vstore_once<float, V>(to + B, tb);
                else
                    vstore<float, V>(to, ta), vstore<float, V>(to + samples, tb);
            }
        }
        // batch totals: a transposed butterfly leaves total i on lane i, i.e. basis sum k = lane & 3 of gate lane >> 2 on
        // the lane that owns entries 4k..4k+3 of that gate; the quad then finishes the gate's 16 gradients together
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = i < 28 ? bs[i] : 0.f;
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
        float s4[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) s4[k] = __shfl_sync(0xffffffffu, v[0], (lane & ~3) + k);
        const float(&p)[4] = pq;
        const long long n = my_node;
        my_leaf = nx_leaf, my_node = nx_node, nx_node = nn_node;
        const int q = lane & 3;
        const float q3 = (float)(q >> 1), q2 = (float)(q & 1);
        const float base = (q3 - q2) * s4[0] - q3 * s4[1] + (q2 - q3) * s4[2] + q3 * s4[3];
        float gr[4] = {base, base + s4[0], base + (s4[1] - s4[0]), base + s4[1]}; // entry i adds (i & 1) s0 + (i >> 1) (s1 - s0)
        if (wmode == CLB_W_SOFTMAX) {
            const float dot = quad_sum((p[0] * gr[0] + p[1] * gr[1]) + (p[2] * gr[2] + p[3] * gr[3]));
#pragma unroll
            for (int i = 0; i < 4; ++i) gr[i] = p[i] * (gr[i] - dot);
        }
        if (lane < 28) {
            const int gi = lane >> 2;
            float *out = (gi < 4 ? gw0 : gi < 6 ? gw1 : gw2) + n * 16 + 4 * q;
#pragma unroll
            for (int i = 0; i < 4; ++i) out[i] = gr[i];
        }
    }
}

// gx[f][b] = sum over the entries e of feature f of rows[list[e]][b]  (rows = tapgrad, list = leaf slots t*8+k)
// ASK: read past the L2 where `once` tells; a branch at run time, which makes the better code of V = 4 (21.4 us for 84 MB of 64 samples, an
// instance of its own 28.6), but spilled for V = 1 (10240 trees, 99 samples, 32 MB: 17.3 us, without it 15.7; 40960, 131 samples: 63.8 and 69).
template <int V, bool ASK>
__global__ void __launch_bounds__(256) row_segment_sum_kernel(const float *__restrict__ rows, const int64_t *__restrict__ start,
                                                              const int32_t *__restrict__ list, float *__restrict__ gx, long long F,
                                                              long long B, bool once)
{
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long f = warp; f < F; f += nwarps) {
        const long long lo = start[f], hi = start[f + 1];
        for (long long bb = 0; bb < B; bb += 32 * V) { // uniform over the warp: the shuffles below need every lane
            const long long b0 = bb + (long long)lane * V;
            const bool in = b0 < B;
            float acc[V];
#pragma unroll
            for (int k = 0; k < V; ++k) acc[k] = 0.f;
            for (long long c0 = lo; c0 < hi; c0 += 32) {
                const int mine = c0 + lane < hi ? __ldg(list + c0 + lane) : 0;
                const int n = (int)min((long long)32, hi - c0);
                for (int i0 = 0; i0 < n; i0 += 4) {
                    float v[4][V];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int r = __shfl_sync(0xffffffffu, mine, min(i0 + u, n - 1));
                        if (in) {
                            const float *from = rows + (long long)r * B + b0;
                            if (ASK && once)
                                vload_once<float, V>(from, v[u]);
                            else
                                vload<float, V>(from, v[u]);
                        } else {
#pragma unroll
                            for (int k = 0; k < V; ++k) v[u][k] = 0.f;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i0 + u < n)
#pragma unroll
                            for (int k = 0; k < V; ++k) acc[k] += v[u][k];
                }
            }
            if (in)
                vstore<float, V>(gx + f * B + b0, acc);
        }
    }
}

} // namespace clb

using namespace clb;
using namespace clb_host;

static bool aligned8(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }
static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// per: blocks of an SM at most.  The resident ones (4 at 64 registers) where a warp loads ahead for its next unit.
static int logic_grid(long long units_of_warps, int per = 32)
{
    long long blocks = (units_of_warps + 7) / 8; // 8 warps per block
    const long long cap = (long long)sm_count() * per;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

int clb_logic_fwd_cols(const float *x, const int64_t *a, const int64_t *b, const float *w, float *y, float *coef, int64_t out_dim, int64_t B, int wmode,
                       cudaStream_t st); // logic_bwd.cu

// When the forward of a layer walks its rows in stretches of 64 samples (logic_fwd_cols_kernel).  The input has to be beyond half the L2
// (us without / with; 48 MB 18.4 / 18.5, 80 MB 36 / 32, 262144 x 1024 480 / 451, 65536 x 4096 480 / 422), a stretch worth the walk
// (196608 x 64 29 / 30, 131072 x 256 59 / 58, 87381 x 384 58 / 51) and nearly all of them whole (264 samples 129 / 175, 520 127 / 138, 1032
// 126 / 107), and its rows made of whole sectors unless they are long (500 samples 123 / 150, 1020 123 / 115, 2052 128 / 107).  A layer with
// fewer outputs than inputs reads a row once at most and gains nothing (200000 -> 100000, 512 samples 96 / 106); just above half the
// L2 the two are level there (66000 -> 33001, 260 samples 17 / 15, 57671 -> 28835, 300 15 / 16, 16962 -> 8481, 1020 14 / 16).
static bool cols_pay(int64_t in_dim, int64_t out_dim, int64_t B)
{
    const int64_t bytes = in_dim * B * 4;
    if (B < 256 || B > 4000000 || B % 4 || in_dim > 0x3fffffff || out_dim > 0x3fffffff || bytes <= (64LL << 20)) return false;
    if (out_dim < in_dim) return bytes <= (72LL << 20);
    return (B % 8 == 0 || B >= 1000) && 12 * ((B + 63) / 64 * 64) <= 13 * B;
}

extern "C" size_t clb_logic_fwd_scratch_bytes(int64_t in_dim, int64_t out_dim, int64_t B, int dtype)
{
    return dtype == CLB_F32 && in_dim > 0 && out_dim > 0 && B > 0 && cols_pay(in_dim, out_dim, B) ? (size_t)out_dim * 16 : 0;
}

extern "C" int clb_logic_fwd(const void *x, const int64_t *a, const int64_t *b, const void *w, void *y, int64_t in_dim,
                             int64_t out_dim, int64_t B, int wmode, int dtype, void *stream)
{
    return clb_logic_fwd_coef(x, a, b, w, y, nullptr, in_dim, out_dim, B, wmode, dtype, stream);
}

extern "C" int clb_logic_fwd_coef(const void *x, const int64_t *a, const int64_t *b, const void *w, void *y, void *coef, int64_t in_dim,
                                  int64_t out_dim, int64_t B, int wmode, int dtype, void *stream)
{
    if (!x || !a || !b || !w || !y || in_dim <= 0 || out_dim < 0 || B < 0 || wmode < 0 || wmode > 2) return CLB_ERR_ARG;
    if (out_dim == 0 || B == 0) return CLB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    // The resident blocks alone while the input is in the L2, or where the last accesses of a row leave more than a quarter of the lanes idle; for
    // larger inputs more of them, which the SMs take up as they come (us with 4 / 32 blocks per SM: 65536 x 128 12.4 / 14.3, 109660 x 112
    // 20.7 / 25.5; 131072 x 512 128 / 117, 262144 x 1024 525 / 480; but 258111 x 260 131 / 137).
    const bool beyond_l2 = in_dim * B * (dtype == CLB_F64 ? 8 : 4) > (96LL << 20) && 4 * B >= 3 * ((B + 127) / 128 * 128);
    const int grid = logic_grid((out_dim + 1) / 2, beyond_l2 ? 32 : 4);
    if (dtype == CLB_F32) {
        const bool vec = B % 4 == 0 && aligned16(x) && aligned16(y);
        if (coef && vec && aligned16(coef) && aligned16(w) && cols_pay(in_dim, out_dim, B))
            return clb_logic_fwd_cols((const float *)x, a, b, (const float *)w, (float *)y, (float *)coef, out_dim, B, wmode, st);
        if (vec)
            CLB_TRACED("logic_fwd_kernel", st,
                       logic_fwd_kernel<float, 4, 2><<<grid, 256, 0, st>>>((const float *)x, a, b, (const float *)w, (float *)y, (float *)coef, out_dim, B, wmode));
        else if (B % 2 == 0 && aligned8(x) && aligned8(y))
            CLB_TRACED("logic_fwd_kernel", st,
                       logic_fwd_kernel<float, 2, 4><<<grid, 256, 0, st>>>((const float *)x, a, b, (const float *)w, (float *)y, (float *)coef, out_dim, B, wmode));
        else
            CLB_TRACED("logic_fwd_kernel", st,
                       logic_fwd_kernel<float, 1, 8><<<grid, 256, 0, st>>>((const float *)x, a, b, (const float *)w, (float *)y, (float *)coef, out_dim, B, wmode));
    } else if (dtype == CLB_F64) {
        CLB_TRACED("logic_fwd_kernel", st,
                   logic_fwd_kernel<double, 1, 4><<<grid, 256, 0, st>>>((const double *)x, a, b, (const double *)w, (double *)y, (double *)coef, out_dim, B, wmode));
    } else
        return CLB_ERR_ARG;
    return check_launch();
}

extern "C" int clb_logic_bwd_w(const void *x, const int64_t *a, const int64_t *b, const void *w, const void *gy, void *gw,
                               int64_t in_dim, int64_t out_dim, int64_t B, int wmode, int dtype, void *stream)
{
    if (!x || !a || !b || !w || !gy || !gw || in_dim <= 0 || out_dim < 0 || B < 0 || wmode < 0 || wmode > 2) return CLB_ERR_ARG;
    if (out_dim == 0) return CLB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int grid = logic_grid((out_dim + 1) / 2, 4);
    if (dtype == CLB_F32) {
        if (B % 4 == 0 && aligned16(x) && aligned16(gy))
            CLB_TRACED("logic_bwd_w_kernel", st, logic_bwd_w_kernel<float, 4, 2><<<grid, 256, 0, st>>>((const float *)x, a, b, (const float *)w, (const float *)gy, (float *)gw, out_dim, B, wmode));
        else if (B % 2 == 0 && aligned8(x) && aligned8(gy))
            CLB_TRACED("logic_bwd_w_kernel", st, logic_bwd_w_kernel<float, 2, 4><<<grid, 256, 0, st>>>((const float *)x, a, b, (const float *)w, (const float *)gy, (float *)gw, out_dim, B, wmode));
        else
            CLB_TRACED("logic_bwd_w_kernel", st, logic_bwd_w_kernel<float, 1, 8><<<grid, 256, 0, st>>>((const float *)x, a, b, (const float *)w, (const float *)gy, (float *)gw, out_dim, B, wmode));
    } else if (dtype == CLB_F64) {
        // four accesses in flight once a row fills them (us with two / four: 64000 x 512 144 / 117, 64000 x 128 41 / 32, 64000 x 32 18 / 21)
        if (B >= 64)
            CLB_TRACED("logic_bwd_w_kernel", st, logic_bwd_w_kernel<double, 1, 4><<<grid, 256, 0, st>>>((const double *)x, a, b, (const double *)w, (const double *)gy, (double *)gw, out_dim, B, wmode));
        else
            CLB_TRACED("logic_bwd_w_kernel", st, logic_bwd_w_kernel<double, 1, 2><<<grid, 256, 0, st>>>((const double *)x, a, b, (const double *)w, (const double *)gy, (double *)gw, out_dim, B, wmode));
    } else
        return CLB_ERR_ARG;
    return check_launch();
}

extern "C" int clb_logic_bwd_x(const void *x, const int64_t *a, const int64_t *b, const void *w, const void *gy, void *gx,
                               const int64_t *start, const int64_t *consumers, int64_t in_dim, int64_t out_dim, int64_t B,
                               int wmode, int dtype, void *stream)
{
    if (!x || !a || !b || !w || !gy || !gx || !start || !consumers || in_dim <= 0 || out_dim < 0 || B < 0 || wmode < 0 || wmode > 2)
        return CLB_ERR_ARG;
    if (B == 0) return CLB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const bool vec = dtype == CLB_F32 && B % 4 == 0 && aligned16(x) && aligned16(gy) && aligned16(gx);
    const int V = vec ? 4 : 1;
    // features per warp: about 32 consumer entries per unit (one feature when the fan-out 2*out/in is wide)
    long long fpu = out_dim > 0 ? (16 * in_dim + out_dim - 1) / out_dim : 1;
    if (fpu > 32) fpu = 32;
    if (fpu < 1) fpu = 1;
    while (fpu > 1 && (in_dim + fpu - 1) / fpu < (long long)sm_count() * 8 * 8) fpu /= 2; // keep enough units to occupy the GPU
    const long long funits = (in_dim + fpu - 1) / fpu;
    // split the batch when there are too few units to occupy the GPU
    long long splits = 1;
    const long long max_splits = (B + 32LL * V * 4 - 1) / (32LL * V * 4);
    while (funits * splits < (long long)sm_count() * 8 * 8 && splits < max_splits) splits *= 2;
    if (splits > max_splits) splits = max_splits;
    const int grid = logic_grid(funits * splits);
    if (out_dim > 0x7fffffffLL || in_dim > 0x7fffffffLL) return CLB_ERR_SHAPE; // consumer and row indices travel as 32-bit shuffles
    // vector slots a lane needs for its share of a split: 1, 2 or 4 at a time
    const long long span = ((B + splits * 32 * V - 1) / (splits * 32 * V));
    const int slots = span <= 1 ? 1 : span <= 2 ? 2 : 4;
#define CLB_BWD_X(T, VV, SS)                                                                                                     \
    logic_bwd_x_kernel<T, VV, SS><<<grid, 256, 0, st>>>((const T *)x, a, b, (const T *)w, (const T *)gy, (T *)gx, start, consumers, \
                                                        in_dim, out_dim, B, wmode, (int)splits, (int)fpu)
    clb_host::TraceScope trace_scope("logic_bwd_x_kernel", st);
    if (dtype == CLB_F32) {
        if (vec) {
            if (slots == 1) CLB_BWD_X(float, 4, 1);
            else if (slots == 2) CLB_BWD_X(float, 4, 2);
            else CLB_BWD_X(float, 4, 4);
        } else {
            if (slots == 1) CLB_BWD_X(float, 1, 1);
            else if (slots == 2) CLB_BWD_X(float, 1, 2);
            else CLB_BWD_X(float, 1, 4);
        }
    } else if (dtype == CLB_F64) {
        if (slots == 1) CLB_BWD_X(double, 1, 1);
        else if (slots == 2) CLB_BWD_X(double, 1, 2);
        else CLB_BWD_X(double, 1, 4);
    } else
        return CLB_ERR_ARG;
#undef CLB_BWD_X
    return check_launch();
}

static int group_sum_parts(long long S) { return S >= 8 * kGroupSumParts ? kGroupSumParts : 1; }

extern "C" size_t clb_group_sum_scratch_bytes(int64_t F, int64_t B, int k, int dtype)
{
    if (F <= 0 || B <= 0 || k <= 0 || F % k) return 0;
    return (size_t)group_sum_parts(F / k) * (size_t)k * (size_t)B * (dtype == CLB_F64 ? 8 : 4);
}

extern "C" int clb_group_sum_fwd(const void *y, void *out, void *scratch, size_t scratch_bytes, int64_t F, int64_t B, int k, double tau,
                                 int dtype, void *stream)
{
    if (!y || !out || F < 0 || B < 0 || k <= 0 || tau == 0.0 || (dtype != CLB_F32 && dtype != CLB_F64)) return CLB_ERR_ARG;
    if (F % k) return CLB_ERR_SHAPE;
    if (B == 0) return CLB_OK;
    if (F == 0) return CLB_ERR_SHAPE;
    if (!scratch || scratch_bytes < clb_group_sum_scratch_bytes(F, B, k, dtype)) return CLB_ERR_SCRATCH;
    const long long S = F / k;
    const int parts = group_sum_parts(S);
    if (k > 65535) return CLB_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    dim3 grid((unsigned)((B + 31) / 32), (unsigned)k, (unsigned)parts);
    const int fb = (int)((B * k + 255) / 256);
    // One launch while a block is short and there are few of them.  Sixteen parts: up to 1024 rows in at most two blocks per SM, else up to
    // 448 (us with one launch / two; 500 rows, 2000 samples, 2 classes 4.3 / 8.6; 2000 rows, 512 x 10 11.8 / 11.1; 400 rows, 4096 x 10 28
    // / 37; 512 rows, 2000 x 80 154 / 134).  One part, which two of the 32 warps add up: below 64 rows in at most a block per SM
    // (40 rows, 100 x 10 3.1 / 3.8, 944 x 10 6.8 / 4.4; 100 rows, 20001 x 10 201 / 20; 2 rows, 512 x 1000 133 / 24).
    const long long blocks = (B + 31) / 32 * k;
    const bool one = parts > 1 ? S <= (blocks <= 2LL * sm_count() ? 1024 : 448) : S < 64 && blocks <= sm_count();
    auto go = [&](auto t) {
        using T = decltype(t);
        if (one) {
            grid.z = 1;
            CLB_TRACED("group_sum_one_kernel", st, group_sum_one_kernel<T><<<grid, 1024, 0, st>>>((const T *)y, (T *)out, S, B, k, parts, (T)tau));
            return 1;
        }
        CLB_TRACED("group_sum_partial_kernel", st, group_sum_partial_kernel<T><<<grid, 256, 0, st>>>((const T *)y, (T *)scratch, S, B, k));
        CLB_TRACED("group_sum_finalize_kernel", st, group_sum_finalize_kernel<T><<<fb, 256, 0, st>>>((const T *)scratch, (T *)out, B, k, parts, (T)tau));
        return 2;
    };
    return check_launch(dtype == CLB_F32 ? go(0.f) : go(0.0));
}

extern "C" int clb_group_sum_ce(const float *y, const int64_t *labels, float *scores, float *dscore, float *loss, void *scratch,
                                size_t scratch_bytes, int64_t F, int64_t B, int k, double tau, void *stream)
{
    if (!y || !labels || !dscore || !loss || F <= 0 || B <= 0 || k <= 0 || tau == 0.0) return CLB_ERR_ARG;
    if (F % k || k > 32) return CLB_ERR_SHAPE;
    if (!scratch || scratch_bytes < clb_group_sum_scratch_bytes(F, B, k, CLB_F32)) return CLB_ERR_SCRATCH;
    const long long S = F / k;
    const int parts = group_sum_parts(S);
    cudaStream_t st = (cudaStream_t)stream;
    dim3 grid((unsigned)((B + 31) / 32), (unsigned)k, (unsigned)parts);
    CLB_TRACED("group_sum_partial_kernel", st, group_sum_partial_kernel<float><<<grid, 256, 0, st>>>(y, (float *)scratch, S, B, k));
    CLB_TRACED("group_sum_ce_sample_kernel", st,
               group_sum_ce_sample_kernel<<<(unsigned)((B + 7) / 8), 256, 0, st>>>((float *)scratch, labels, scores, dscore, B, k, parts, (float)tau));
    CLB_TRACED("group_sum_loss_mean_kernel", st, group_sum_loss_mean_kernel<<<1, 256, 0, st>>>((const float *)scratch, loss, B));
    return check_launch(3);
}

extern "C" int clb_transpose_f32(const float *in, float *out, int64_t rows, int64_t cols, void *stream)
{
    if (!in || !out || rows < 0 || cols < 0 || in == out) return CLB_ERR_ARG;
    if (rows == 0 || cols == 0) return CLB_OK;
    const long long gx = (cols + 31) / 32, gy = (rows + 31) / 32;
    if (gy > 65535 || gx > 0x7fffffffLL) return CLB_ERR_TOO_LARGE;
    cudaStream_t st = (cudaStream_t)stream;
    CLB_TRACED("transpose_f32_kernel", st, transpose_f32_kernel<<<dim3((unsigned)gx, (unsigned)gy), 256, 0, st>>>(in, out, rows, cols));
    return check_launch();
}

extern "C" int clb_adam_step(float *p, const float *g, float *m, float *v, int64_t n, double lr, double beta1, double beta2, double eps,
                             double weight_decay, int64_t step, int decoupled, void *stream)
{
    if (!p || !g || !m || !v || n < 0 || step < 1 || beta1 < 0 || beta1 >= 1 || beta2 < 0 || beta2 >= 1) return CLB_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15)
        return CLB_ERR_ARG;
    if (n == 0) return CLB_OK;
    const double bc1 = 1.0 - std::pow(beta1, (double)step), bc2 = 1.0 - std::pow(beta2, (double)step);
    cudaStream_t st = (cudaStream_t)stream;
    long long blocks = ((n >> 2) + 255) / 256;
    const long long cap = (long long)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    CLB_TRACED("adam_step_kernel", st,
               adam_step_kernel<<<(unsigned)blocks, 256, 0, st>>>(p, g, m, v, n, (float)lr, (float)beta1, (float)beta2, (float)eps, (float)weight_decay,
                                                                  (float)(lr / bc1), (float)std::sqrt(bc2), decoupled));
    return check_launch();
}

extern "C" int clb_group_sum_bwd_scaled(const void *gout, const void *scale, void *gy, int64_t F, int64_t B, int k, double tau, int dtype,
                                        void *stream);
extern "C" int clb_group_sum_bwd(const void *gout, void *gy, int64_t F, int64_t B, int k, double tau, int dtype, void *stream)
{
    return clb_group_sum_bwd_scaled(gout, nullptr, gy, F, B, k, tau, dtype, stream);
}

extern "C" int clb_group_sum_bwd_scaled(const void *gout, const void *scale, void *gy, int64_t F, int64_t B, int k, double tau, int dtype,
                                        void *stream)
{
    if (!gout || !gy || F < 0 || B < 0 || k <= 0 || tau == 0.0 || (dtype != CLB_F32 && dtype != CLB_F64)) return CLB_ERR_ARG;
    if (F % k) return CLB_ERR_SHAPE;
    if (B == 0 || F == 0) return CLB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const long long S = F / k;
    if (k > 65535) return CLB_ERR_SHAPE;
    long long chunks = ((long long)sm_count() * 16 + k - 1) / k; // about sixteen blocks per SM in all, at least 16 rows each
    if (chunks > (S + 15) / 16) chunks = (S + 15) / 16;
    dim3 grid((unsigned)chunks, (unsigned)k);
    if (dtype == CLB_F32 && B % 4 == 0 && aligned16(gy))
        CLB_TRACED("group_sum_bwd_kernel", st, group_sum_bwd_kernel<float, 4><<<grid, 256, 0, st>>>((const float *)gout, (const float *)scale, (float *)gy, S, B, k, (float)tau));
    else if (dtype == CLB_F32 && B <= kGroupSumFlatMax && aligned16(gy))
        CLB_TRACED("group_sum_bwd_kernel", st, group_sum_bwd_flat_kernel<<<grid, 256, (size_t)B * 4, st>>>((const float *)gout, (const float *)scale, (float *)gy, S, (int)B, k, (float)tau));
    else if (dtype == CLB_F32)
        CLB_TRACED("group_sum_bwd_kernel", st, group_sum_bwd_kernel<float, 1><<<grid, 256, 0, st>>>((const float *)gout, (const float *)scale, (float *)gy, S, B, k, (float)tau));
    else
        CLB_TRACED("group_sum_bwd_kernel", st, group_sum_bwd_kernel<double, 1><<<grid, 256, 0, st>>>((const double *)gout, (const double *)scale, (double *)gy, S, B, k, tau));
    return check_launch();
}

// ---- fused flat layers (training) ------------------------------------------------------------------
static bool tree_args_ok(const void *x, const int32_t *leaf, const int32_t *node, const void *w0, const void *w1, const void *w2, int64_t T,
                         int64_t B, int wmode)
{
    return x && leaf && node && w0 && w1 && w2 && T >= 0 && B >= 0 && wmode >= 0 && wmode <= 2;
}

extern "C" int clb_logic_tree_fwd(const float *x, const int32_t *leaf, const int32_t *node, const float *w0, const float *w1, const float *w2,
                                  float *y, int64_t T, int64_t B, int wmode, void *stream)
{
    if (!tree_args_ok(x, leaf, node, w0, w1, w2, T, B, wmode) || !y) return CLB_ERR_ARG;
    if (T == 0 || B == 0) return CLB_OK;
    TreeTables tt{leaf, node, {w0, w1, w2}};
    const int grid = logic_grid(T);
    cudaStream_t st = (cudaStream_t)stream;
    if (B % 4 == 0 && aligned16(x) && aligned16(y))
        CLB_TRACED("logic_tree_fwd_kernel", st, logic_tree_fwd_kernel<4><<<grid, 256, 0, st>>>(x, tt, y, T, B, wmode));
    else
        CLB_TRACED("logic_tree_fwd_kernel", st, logic_tree_fwd_kernel<1><<<grid, 256, 0, st>>>(x, tt, y, T, B, wmode));
    return check_launch();
}

// tapgrad: scratch of T*8*B floats.  gw0/gw1/gw2 must be zeroed by the caller: neurons no tree uses keep zero.
// start int64 [in_dim + 1], list int32 [T*8]: the leaf slots (t*8 + k) grouped by the input feature they read.
// parts of a class for the fused forward + class sums: enough blocks to fill the GPU a few times over
static int tree_sum_parts(int64_t T, int k)
{
    long long parts = ((long long)sm_count() * 4 + k - 1) / k;
    const long long most = T / k / 8; // at least eight trees (one per warp) per part
    if (parts > most) parts = most;
    return (int)(parts < 1 ? 1 : parts);
}

extern "C" size_t clb_logic_tree_fwd_ce_scratch_bytes(int64_t T, int64_t B, int k)
{
    if (T <= 0 || B <= 0 || k <= 0 || T % k) return 0;
    return (size_t)tree_sum_parts(T, k) * (size_t)k * (size_t)B * sizeof(float);
}

extern "C" int clb_logic_tree_fwd_ce(const float *x, const int32_t *leaf, const int32_t *node, const float *w0, const float *w1,
                                     const float *w2, const int64_t *labels, float *dscore, float *loss, void *scratch,
                                     size_t scratch_bytes, int64_t T, int64_t B, int k, double tau, int wmode, void *stream)
{
    if (!tree_args_ok(x, leaf, node, w0, w1, w2, T, B, wmode) || !labels || !dscore || !loss || k <= 0 || tau == 0.0) return CLB_ERR_ARG;
    if (T <= 0 || B <= 0 || T % k || k > 32 || B % 4 || B > 512 || !aligned16(x) || T * 8 > 0x7fffffffLL) return CLB_ERR_SHAPE;
    if (!scratch || scratch_bytes < clb_logic_tree_fwd_ce_scratch_bytes(T, B, k)) return CLB_ERR_SCRATCH;
    TreeTables tt{leaf, node, {w0, w1, w2}};
    cudaStream_t st = (cudaStream_t)stream;
    const int parts = tree_sum_parts(T, k);
    const dim3 grid((unsigned)parts, (unsigned)k);
    float *partial = (float *)scratch;
    if (B <= 128)
        CLB_TRACED("logic_tree_fwd_sum_kernel", st, logic_tree_fwd_sum_kernel<1><<<grid, 256, 0, st>>>(x, tt, partial, T, B, k, wmode));
    else if (B <= 256)
        CLB_TRACED("logic_tree_fwd_sum_kernel", st, logic_tree_fwd_sum_kernel<2><<<grid, 256, 0, st>>>(x, tt, partial, T, B, k, wmode));
    else
        CLB_TRACED("logic_tree_fwd_sum_kernel", st, logic_tree_fwd_sum_kernel<4><<<grid, 256, 0, st>>>(x, tt, partial, T, B, k, wmode));
    CLB_TRACED("group_sum_ce_sample_kernel", st,
               group_sum_ce_sample_kernel<<<(unsigned)((B + 7) / 8), 256, 0, st>>>(partial, labels, nullptr, dscore, B, k, parts, (float)tau));
    CLB_TRACED("group_sum_loss_mean_kernel", st, group_sum_loss_mean_kernel<<<1, 256, 0, st>>>(partial, loss, B));
    return check_launch(3);
}

static int logic_tree_bwd_impl(const float *x, const int32_t *leaf, const int32_t *node, const float *w0, const float *w1, const float *w2,
                               const float *gy, const TreeHead *head, float *tapgrad, float *gw0, float *gw1, float *gw2, float *gx,
                               const int64_t *start, const int32_t *list, int64_t in_dim, int64_t T, int64_t B, int wmode, void *stream)
{
    if (!tree_args_ok(x, leaf, node, w0, w1, w2, T, B, wmode) || (!gy && !head) || !tapgrad || !gw0 || !gw1 || !gw2 || in_dim <= 0) return CLB_ERR_ARG;
    if (gx && (!start || !list)) return CLB_ERR_ARG;
    if (T * 8 > 0x7fffffffLL || B > 0x7fffff00LL) return CLB_ERR_SHAPE;
    if (B == 0) return CLB_OK;
    TreeTables tt{leaf, node, {w0, w1, w2}};
    cudaStream_t st = (cudaStream_t)stream;
    const bool vec = B % 4 == 0 && aligned16(x) && (head || aligned16(gy)) && aligned16(tapgrad) && (!gx || aligned16(gx));
    const TreeHead none{nullptr, nullptr, 1, 1u, 1.f};
    // leaf gradients beyond half the L2 go past it, both ways: x stays there (k = 256, 256 samples, 671 MB: 202 -> 193 us, their sums 129 -> 121;
    // at k = 32, 33 MB, the sums 7.3 -> 8.5)
    const bool once = T * 8 * B * 4 > (64LL << 20);
    int launched = 0;
    if (T > 0) {
        const long long resident = (long long)sm_count() * 3; // vec: one wave, whose warps fetch ahead from tree to tree
        const int grid = vec && (T + 3) / 4 > resident ? (int)resident : 2 * logic_grid(T);
        TreeHead rows = none;
        // Classes' upstream gradients as rows: a launch of 1.8 us, and one more to wait for, which the trees make good from there on (us of their kernel,
        // from dscore / from rows: 5120 trees, 128 samples 12.8 / 10.6, 10240, 16 19.2 / 17.1; 10240, 100 22.2 / 18.1, 2560, 256 13.3 / 9.8)
        if (head && vec && gx && in_dim >= head->k && T * B >= kTreeRows) { // (in the input gradient's memory, until the sums are written to it)
            CLB_TRACED("tree_head_rows_kernel", st, tree_head_rows_kernel<<<(unsigned)((B * head->k + 255) / 256), 256, 0, st>>>(gx, B, *head));
            gy = gx, rows.S = head->S, head = nullptr;
            ++launched;
        }
        bool ok = true;
        auto go = [&](auto kern, int smem, const TreeHead &h) {
            if (smem) ok = ensure_dynamic_smem(kern, smem) == cudaSuccess;
            if (ok) CLB_TRACED("logic_tree_bwd_kernel", st, kern<<<grid, 128, smem, st>>>(x, tt, gy, tapgrad, gw0, gw1, gw2, (int)T, (int)B, wmode, h));
        };
        if (head && vec)
            go(logic_tree_bwd_kernel<4, true, false>, kTreeSmem, *head);
        else if (head)
            go(logic_tree_bwd_kernel<1, true, false>, 0, *head);
        else if (vec && once)
            go(logic_tree_bwd_kernel<4, false, true>, kTreeSmem, rows);
        else if (vec)
            go(logic_tree_bwd_kernel<4, false, false>, kTreeSmem, rows);
        else
            go(logic_tree_bwd_kernel<1, false, false>, 0, rows);
        if (!ok) return check_launch(0);
        ++launched;
    }
    if (gx) {
        if (vec)
            CLB_TRACED("row_segment_sum_kernel", st, row_segment_sum_kernel<4, true><<<logic_grid(in_dim), 256, 0, st>>>(tapgrad, start, list, gx, in_dim, B, once));
        else if (once)
            CLB_TRACED("row_segment_sum_kernel", st, row_segment_sum_kernel<1, true><<<logic_grid(in_dim), 256, 0, st>>>(tapgrad, start, list, gx, in_dim, B, true));
        else
            CLB_TRACED("row_segment_sum_kernel", st, row_segment_sum_kernel<1, false><<<logic_grid(in_dim), 256, 0, st>>>(tapgrad, start, list, gx, in_dim, B, false));
        ++launched;
    }
    return check_launch(launched);
}

extern "C" int clb_logic_tree_bwd(const float *x, const int32_t *leaf, const int32_t *node, const float *w0, const float *w1, const float *w2,
                                  const float *gy, float *tapgrad, float *gw0, float *gw1, float *gw2, float *gx, const int64_t *start,
                                  const int32_t *list, int64_t in_dim, int64_t T, int64_t B, int wmode, void *stream)
{
    if (!gy) return CLB_ERR_ARG;
    return logic_tree_bwd_impl(x, leaf, node, w0, w1, w2, gy, nullptr, tapgrad, gw0, gw1, gw2, gx, start, list, in_dim, T, B, wmode, stream);
}

extern "C" int clb_logic_tree_bwd_scores(const float *x, const int32_t *leaf, const int32_t *node, const float *w0, const float *w1,
                                         const float *w2, const float *dscore, const float *scale, int k, double tau, float *tapgrad,
                                         float *gw0, float *gw1, float *gw2, float *gx, const int64_t *start, const int32_t *list,
                                         int64_t in_dim, int64_t T, int64_t B, int wmode, void *stream)
{
    if (!dscore || !scale || k <= 0 || tau == 0.0) return CLB_ERR_ARG;
    if (T % k) return CLB_ERR_SHAPE;
    const TreeHead head{dscore, scale, k, (unsigned)(T / k > 0 ? T / k : 1), (float)tau};
    return logic_tree_bwd_impl(x, leaf, node, w0, w1, w2, nullptr, &head, tapgrad, gw0, gw1, gw2, gx, start, list, in_dim, T, B, wmode, stream);
}

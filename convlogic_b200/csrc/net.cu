// Compiled network: a discretised stack (fused ConvLogic blocks, flat LogicLayers, GroupSum) serialised into one
// blob and run by a single host call that enqueues the packed kernels of this library back to back.
// It plays the part of the reference's CompiledLogicNet (src/difflogic/compiled_model.py:41-361), which writes
// the gates out as C source and compiles it with gcc for the CPU and which cannot hold conv blocks; here the
// artefact is data (the blob), the code is this library, and the network runs on the GPU from any host
// language that can call C.
//
// Blob, little-endian, every array 16-byte aligned relative to the blob start:
//   header  (64 bytes): "CLBNET01", u32 n_layers, u32 num_classes, u32 in_channels, u32 in_h, u32 in_w,
//                       u32 in_features (flat input: in_channels = 0), u64 total_bytes, zero padding
//   layer i (64 bytes): u32 kind (1 fused conv block, 2 flat layer), u32 p[7], u64 off_a, u64 off_b, u64 off_ops, pad
//       conv: p = {Ci, C, kh, kw, stride, pad_h, pad_w}; off_a -> int32 sel[C][8]; off_ops -> u8 ops[C][7]
//       flat: p = {in_dim (lo), out_dim (lo), in_dim (hi), out_dim (hi)}; off_a / off_b -> int64 idx[out]; off_ops -> u8 ops[out]
//       kind 3, two or three flat layers fused into a gate tree (clb_packed_tree): p = {in_dim (lo), out_dim (lo), in_dim (hi),
//             out_dim (hi), levels}; off_a -> int32 leaf[out][2^levels]; off_ops -> u8 ops[out][2^levels - 1]
//   arrays
// The last flat layer's outputs are summed per class (GroupSum): counts[b][k].
#include "clb_common.cuh"
#include "clb_net.cuh"
#include "clb_slab.cuh"

#include <cstring>
#include <new>
#include <vector>

using namespace clb_host;

namespace {

constexpr char kMagic[8] = {'C', 'L', 'B', 'N', 'E', 'T', '0', '1'};
constexpr size_t kHeaderBytes = 64, kLayerBytes = 64;
// The one-launch kernel (net_cluster.cu) against layer-by-layer launches, us per call on B200: mnist k=64 (cost 0.1 M) batch 1 16.5 / 51,
// batch 8192 104 / 146; cifar k=32 (0.13 M) batch 1 21 / 40, batch 1000 41 / 41, batch 2000 52 / 58, batch 8192 133 / 124; cifar k=48 (0.19 M) batch 1 23 / 39,
// batch 1000 50 / 51; cifar k=64 (0.25 M) batch 1 27 / 39, batch 500 43 / 43, batch 1000 64 / 56, batch 8192 236 / 178.  The line was drawn when slabs had 128
// samples and k=64 took 43 / 39 at batch 1; calls of a slab or two beyond it would be faster in one launch now (cifar k=128 batch 1 39 / 47, mnist k=128
// 25 / 55, k=256 37 / 63; batch 500 of cifar k=128 68 / 61).  Beyond one slab per SM the clusters come in waves and the layered kernels win from k=32 on.
constexpr long long kOneLaunchCost = 200000;

struct Header {
    char magic[8];
    uint32_t n_layers, num_classes, in_channels, in_h, in_w, in_features;
    uint64_t total_bytes;
};

struct LayerRec {
    uint32_t kind, p[7];
    uint64_t off_a, off_b, off_ops;
};

struct Layer {
    int kind;
    // conv
    int Ci, C, kh, kw, stride, ph, pw, H, W, Hp, Wp; // input extent and pooled output extent
    // flat (kind 2) and fused flat tree (kind 3)
    long long in_dim, out_dim;
    int levels;
    size_t off_a, off_b, off_ops;
    bool slab3 = false;   // a 3x3 block of the stacks' geometry, which works from tap records ...
    size_t off_recs = 0;  // ... in the records memory, where the caller gave some, with the table of their order behind them
    std::vector<int32_t> order; // (clb_slab3_order)
};

} // namespace

struct clb_net {
    std::vector<Layer> layers;
    int num_classes = 0;
    int in_channels = 0, in_h = 0, in_w = 0;
    long long in_features = 0; // features of one sample at the input
    size_t param_bytes = 0;    // the blob is copied to the device as it is
    size_t record_bytes = 0;   // tap records of all 3x3 blocks
    const unsigned char *records = nullptr; // device memory that holds them, or null: laid out in the workspace on every call
    const unsigned char *dev = nullptr;
    size_t max_conv_channels = 0;
    clb::NetPlan plan = {};     // for the one-launch kernel
    bool one_launch = false;    // the stack has the form that kernel takes
    long long slab_cost = 0;    // gate trees per 128-sample slab, a conv window counting as four
};
 // packed.cu
int clb_net_cluster_launch(const clb::NetPlan &net, const void *input, const float *thresholds, const unsigned char *params, void *work,
                           int32_t *counts, int64_t batch, cudaStream_t st); // net_cluster.cu

static size_t align256(size_t v) { return (v + 255) / 256 * 256; }

static bool parse(const void *blob, size_t bytes, clb_net &net)
{
    if (!blob || bytes < kHeaderBytes) return false;
    Header h;
    std::memcpy(&h, blob, sizeof(Header));
    if (std::memcmp(h.magic, kMagic, 8) != 0 || h.total_bytes != bytes || h.n_layers == 0 || h.n_layers > 4096 || h.num_classes == 0)
        return false;
    if (bytes < kHeaderBytes + (size_t)h.n_layers * kLayerBytes) return false;
    net.num_classes = (int)h.num_classes;
    net.in_channels = (int)h.in_channels, net.in_h = (int)h.in_h, net.in_w = (int)h.in_w;
    net.in_features = h.in_channels ? (long long)h.in_channels * h.in_h * h.in_w : (long long)h.in_features;
    if (net.in_features <= 0) return false;
    net.param_bytes = bytes;
    int C = net.in_channels, H = net.in_h, W = net.in_w; // running conv extent
    long long feat = net.in_features;
    bool flat_seen = false;
    auto in_blob = [&](uint64_t off, unsigned long long n) { return off % 16 == 0 && off <= bytes && n <= bytes - off; };
    const unsigned char *base = (const unsigned char *)blob; // arrays sit at 16-byte aligned offsets of a caller buffer
    for (uint32_t i = 0; i < h.n_layers; ++i) {
        LayerRec r;
        std::memcpy(&r, (const unsigned char *)blob + kHeaderBytes + (size_t)i * kLayerBytes, sizeof(LayerRec));
        Layer L{};
        L.kind = (int)r.kind;
        L.off_a = r.off_a, L.off_b = r.off_b, L.off_ops = r.off_ops;
        if (r.kind == 1) {
            if (flat_seen || C <= 0) return false; // conv blocks come first and need an image input
            L.Ci = (int)r.p[0], L.C = (int)r.p[1], L.kh = (int)r.p[2], L.kw = (int)r.p[3], L.stride = (int)r.p[4], L.ph = (int)r.p[5],
            L.pw = (int)r.p[6];
            if (L.Ci != C || L.C <= 0 || L.C > 65535 || L.stride <= 0 || !conv_args_ok(1, L.Ci, H, W, L.C, L.stride, L.stride, L.ph, L.pw, L.kh, L.kw))
                return false;
            const int Ho = conv_out(H, L.ph, L.kh, L.stride), Wo = conv_out(W, L.pw, L.kw, L.stride);
            if (Ho <= 0 || Wo <= 0 || (Ho & 1) || (Wo & 1)) return false;
            L.H = H, L.W = W, L.Hp = Ho / 2, L.Wp = Wo / 2;
            if (!in_blob(r.off_a, (unsigned long long)L.C * 32) || !in_blob(r.off_ops, (unsigned long long)L.C * 7)) return false;
            { // every tap must name a channel of the input and a cell of the window, every gate id one of the 16 gates
                const int32_t *selw = reinterpret_cast<const int32_t *>(base + r.off_a);
                for (long long t = 0; t < (long long)L.C * 8; ++t) {
                    const int32_t word = selw[t];
                    if (word < 0 || ((word >> 16) & 0xFFFF) >= L.Ci || ((word >> 8) & 0xFF) >= L.kh || (word & 0xFF) >= L.kw) return false;
                }
                const uint8_t *opsb = base + r.off_ops;
                for (long long t = 0; t < (long long)L.C * 7; ++t)
                    if (opsb[t] > 15) return false;
            }
            C = L.C, H = L.Hp, W = L.Wp;
            feat = (long long)C * H * W;
            if ((size_t)L.C > net.max_conv_channels) net.max_conv_channels = (size_t)L.C;
        } else if (r.kind == 2) {
            flat_seen = true;
            L.in_dim = (long long)r.p[0] | ((long long)r.p[2] << 32), L.out_dim = (long long)r.p[1] | ((long long)r.p[3] << 32);
            if (L.in_dim != feat || L.out_dim <= 0) return false;
            if (!in_blob(r.off_a, (unsigned long long)L.out_dim * 8) || !in_blob(r.off_b, (unsigned long long)L.out_dim * 8) ||
                !in_blob(r.off_ops, (unsigned long long)L.out_dim))
                return false;
            { // connection indices must name input features, gate ids one of the 16 gates
                const int64_t *ia = reinterpret_cast<const int64_t *>(base + r.off_a), *ib = reinterpret_cast<const int64_t *>(base + r.off_b);
                const uint8_t *opsb = base + r.off_ops;
                for (long long t = 0; t < L.out_dim; ++t)
                    if (ia[t] < 0 || ia[t] >= L.in_dim || ib[t] < 0 || ib[t] >= L.in_dim || opsb[t] > 15) return false;
            }
            feat = L.out_dim;
        } else if (r.kind == 3) {
            flat_seen = true;
            L.in_dim = (long long)r.p[0] | ((long long)r.p[2] << 32), L.out_dim = (long long)r.p[1] | ((long long)r.p[3] << 32);
            L.levels = (int)r.p[4];
            if (L.in_dim != feat || L.out_dim <= 0 || (L.levels != 2 && L.levels != 3) || L.in_dim > 0x7fffffffLL) return false;
            const unsigned long long leaves = 1ull << L.levels;
            if (!in_blob(r.off_a, (unsigned long long)L.out_dim * leaves * 4) || !in_blob(r.off_ops, (unsigned long long)L.out_dim * (leaves - 1)))
                return false;
            {
                const int32_t *leaf = reinterpret_cast<const int32_t *>(base + r.off_a);
                for (unsigned long long t = 0; t < (unsigned long long)L.out_dim * leaves; ++t)
                    if (leaf[t] < 0 || leaf[t] >= L.in_dim) return false;
                const uint8_t *opsb = base + r.off_ops;
                for (unsigned long long t = 0; t < (unsigned long long)L.out_dim * (leaves - 1); ++t)
                    if (opsb[t] > 15) return false;
            }
            feat = L.out_dim;
        } else {
            return false;
        }
        if (L.kind == 1 && clb_slab3_covers(L.H, L.W, L.stride, L.stride, L.ph, L.pw, L.kh, L.kw)) {
            L.slab3 = true, L.off_recs = net.record_bytes;
            net.record_bytes += align256(clb_slab3_record_bytes(L.C)) + align256((size_t)L.C * 12);
        }
        net.layers.push_back(L);
    }
    return feat % net.num_classes == 0;
}

// The layout of a slab for the one-launch kernel: conv blocks first, at least one flat layer last, sizes that 32-bit unit
// indices cover.
static void plan_one_launch(clb_net &net)
{
    const size_t n = net.layers.size();
    if (n > (size_t)clb::kNetMaxLayers || net.layers.back().kind == 1) return;
    clb::NetPlan &P = net.plan;
    P.n_layers = (int)n, P.classes = net.num_classes, P.in_features = net.in_features;
    long long units = 0;
    auto store = [&](size_t i, long long channels, int rows, int W, int ph, int pw) {
        if (!P.store[i].lay_out(units, channels, rows, W, ph, pw)) return false;
        units += (channels * P.store[i].per_channel + 7) / 8 * 8;
        return true;
    };
    auto flat_store = [&](size_t i, long long features) { return features <= (1 << 24) && store(i, 1, 1, (int)features, 0, 0); };
    const Layer &first = net.layers.front();
    if (!(net.in_channels > 0 ? store(0, net.in_channels, net.in_h, net.in_w, first.kind == 1 ? first.ph : 0, first.kind == 1 ? first.pw : 0)
                              : flat_store(0, net.in_features)))
        return;
    for (size_t i = 0; i < n; ++i) {
        const Layer &L = net.layers[i];
        clb::NetLayer &o = P.layer[i];
        o.kind = L.kind, o.C = L.C, o.stride = L.stride, o.Hp = L.Hp, o.Wp = L.Wp, o.levels = L.levels;
        o.off_a = L.off_a, o.off_b = L.off_b, o.off_ops = L.off_ops;
        if (L.kind == 1) {
            const Layer &next = net.layers[i + 1];
            const bool conv = next.kind == 1;
            if (!store(i + 1, L.C, L.Hp, L.Wp, conv ? next.ph : 0, conv ? next.pw : 0)) return;
            const long long windows = (long long)L.Hp * L.Wp;
            if (!clb::FastDiv::exact(L.C * windows, windows) || !clb::FastDiv::exact(windows, L.Wp)) return;
            o.by_windows = clb::FastDiv::of((unsigned)(L.Hp * L.Wp)), o.by_Wp = clb::FastDiv::of((unsigned)L.Wp);
            net.slab_cost += 4LL * L.C * L.Hp * L.Wp;
        } else {
            if (L.out_dim > (1 << 24)) return;
            o.out_dim = (int)L.out_dim;
            if (i + 1 < n && !flat_store(i + 1, L.out_dim)) return;
            net.slab_cost += L.out_dim;
        }
    }
    P.slab_units = units;
    net.one_launch = true;
}

// When the one-launch kernel is used: small stacks (a slab is one cluster's work) and at most a slab per SM, see kOneLaunchCost.
static bool use_one_launch(const clb_net *net, int input_kind, int64_t batch)
{
    if (!net->one_launch || input_kind == 3 || tune_get(CLB_TUNE_NET_ONE_LAUNCH) == 0) return false;
    const long long slabs = (batch + 127) / 128;
    if (slabs * net->plan.slab_units > (1LL << 27)) return false; // 2 GB of activations
    return tune_get(CLB_TUNE_NET_ONE_LAUNCH) == 2 || (net->slab_cost <= kOneLaunchCost && slabs <= sm_count());
}

extern "C" int clb_net_device_bytes(const void *blob, size_t bytes, size_t *device_bytes)
{
    clb_net tmp;
    if (!device_bytes) return CLB_ERR_ARG;
    if (!parse(blob, bytes, tmp)) return CLB_ERR_SHAPE;
    *device_bytes = tmp.param_bytes;
    return CLB_OK;
}

extern "C" int clb_net_create(const void *blob, size_t bytes, void *device_mem, void *stream, clb_net **out)
{
    if (!out || !device_mem || (reinterpret_cast<uintptr_t>(device_mem) & 15)) return CLB_ERR_ARG;
    clb_net *net = new (std::nothrow) clb_net;
    if (!net) return CLB_ERR_ARG;
    if (!parse(blob, bytes, *net)) {
        delete net;
        return CLB_ERR_SHAPE;
    }
    // the parameters travel as one copy; `blob` must stay valid until the stream has run it
    if (cudaMemcpyAsync(device_mem, blob, bytes, cudaMemcpyHostToDevice, (cudaStream_t)stream) != cudaSuccess) {
        delete net;
        return check_launch(0);
    }
    net->dev = (const unsigned char *)device_mem;
    for (Layer &L : net->layers) {
        if (!L.slab3) continue;
        L.order.resize((size_t)L.C * 3);
        if (!clb_slab3_order((const int32_t *)((const unsigned char *)blob + L.off_a), L.Ci, L.C, L.order.data())) L.order.clear();
    }
    plan_one_launch(*net);
    *out = net;
    return CLB_OK;
}

extern "C" size_t clb_net_record_bytes(const clb_net *net) { return net ? net->record_bytes : 0; }

extern "C" int clb_net_records(clb_net *net, void *records, void *stream)
{
    if (!net || (net->record_bytes && (!records || (reinterpret_cast<uintptr_t>(records) & 15)))) return CLB_ERR_ARG;
    for (const Layer &L : net->layers) {
        if (!L.slab3) continue;
        unsigned char *recs = (unsigned char *)records + L.off_recs;
        int32_t *order = L.order.empty() ? nullptr : (int32_t *)(recs + align256(clb_slab3_record_bytes(L.C)));
        if (order && cudaMemcpyAsync(order, L.order.data(), L.order.size() * sizeof(int32_t), cudaMemcpyHostToDevice, (cudaStream_t)stream) != cudaSuccess)
            return check_launch(0);
        const int rc = clb_slab3_records(net->dev + L.off_ops, (const int32_t *)(net->dev + L.off_a), order, recs, L.Ci, L.H, L.C, (cudaStream_t)stream);
        if (rc != CLB_OK) return rc;
    }
    net->records = (const unsigned char *)records;
    return CLB_OK;
}

extern "C" void clb_net_destroy(clb_net *net) { delete net; }

extern "C" int clb_net_info(const clb_net *net, int64_t *in_features, int *num_classes, int *n_layers)
{
    if (!net) return CLB_ERR_ARG;
    if (in_features) *in_features = net->in_features;
    if (num_classes) *num_classes = net->num_classes;
    if (n_layers) *n_layers = (int)net->layers.size();
    return CLB_OK;
}

// Activations ping-pong between two buffers sized for the widest layer; the batch is padded to 128 samples so
// that every pixel row is a whole number of 16-byte units (slab layout, 128-bit kernels).
static size_t row_bytes(int64_t batch) { return (size_t)((batch + 127) / 128) * 16; }

static size_t widest(const clb_net *net)
{
    long long m = net->in_features;
    for (const Layer &L : net->layers) {
        const long long f = L.kind == 1 ? (long long)L.C * L.Hp * L.Wp : L.out_dim;
        if (f > m) m = f;
    }
    return (size_t)m;
}

extern "C" size_t clb_net_workspace_bytes(const clb_net *net, int64_t batch)
{
    if (!net || batch <= 0) return 0;
    const size_t act = align256(widest(net) * row_bytes(batch));
    const size_t layers = 2 * act + align256((size_t)clb_packed_convtree_slab_scratch_bytes((int)net->max_conv_channels)) + 256;
    const size_t slabs = use_one_launch(net, 0, batch) ? (size_t)((batch + 127) / 128) * (size_t)net->plan.slab_units * 16 : 0;
    return slabs > layers ? slabs : layers;
}

// input_kind: 0 = bool / uint8 bits [batch][in_features]; 1 = float32 pixels, 2 = uint8 pixels [batch][pc][H*W] with
// `levels` thresholds (in_channels == levels * pc); 3 = packed rows [in_features][ceil(batch/128)*2] of 64-bit words.
extern "C" int clb_net_forward(const clb_net *net, int input_kind, const void *input, const float *thresholds, int levels, int64_t batch,
                               int32_t *counts, void *workspace, size_t workspace_bytes, void *stream)
{
    if (!net || !input || !counts || !workspace || batch <= 0 || input_kind < 0 || input_kind > 3) return CLB_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255)) return CLB_ERR_ARG;
    if (workspace_bytes < clb_net_workspace_bytes(net, batch)) return CLB_ERR_SCRATCH;
    if (use_one_launch(net, input_kind, batch) && levels <= clb::kNetMaxLevels) {
        if (input_kind != 0 && (net->in_channels <= 0 || !thresholds || levels <= 0 || net->in_channels % levels)) return CLB_ERR_SHAPE;
        clb::NetPlan plan = net->plan;
        plan.input_kind = input_kind, plan.levels = levels;
        return clb_net_cluster_launch(plan, input, thresholds, net->dev, workspace, counts, batch, (cudaStream_t)stream);
    }
    const size_t rb = row_bytes(batch);
    const int64_t words = (int64_t)(rb / 8), U = (int64_t)(rb / 16);
    const size_t act = align256(widest(net) * rb);
    unsigned char *buf[2] = {(unsigned char *)workspace, (unsigned char *)workspace + act};
    void *scratch = (unsigned char *)workspace + 2 * act;
    const bool image = net->in_channels > 0;
    const Layer &first = net->layers.front();
    // conv blocks run on slabs where a kernel covers them (stride 1, <= 256 pooled outputs per image), and the stacks' own geometry
    // takes and gives them in split order; the order of the activations that a layer wants:
    auto wanted = [&](size_t i) {
        if (i >= net->layers.size() || net->layers[i].kind != 1) return clb::kRows;
        const Layer &L = net->layers[i];
        return L.slab3 ? clb::kSplitSlabs : L.stride == 1 && L.Hp * L.Wp <= 256 ? clb::kSlabs : clb::kRows;
    };
    clb::Order order = image ? wanted(0) : clb::kRows; // of the current activations
    const int64_t in_hw = (int64_t)net->in_h * net->in_w;
    cudaStream_t cs = (cudaStream_t)stream;
    int cur = 0, st;

    // ---- input stage
    if (input_kind == 0) {
        st = clb_pack_bits_units((const uint8_t *)input, buf[0], batch, net->in_features, U, in_hw, net->in_w, order, cs);
        if (st != CLB_OK) return st;
    } else if (input_kind == 1 || input_kind == 2) {
        if (!image || !thresholds || levels <= 0 || net->in_channels % levels) return CLB_ERR_SHAPE;
        st = clb_thermometer_pack_units(input, input_kind == 2, thresholds, levels, buf[0], batch, net->in_channels / levels, in_hw, words, net->in_w, order, cs);
        if (st != CLB_OK) return st;
    } else if (order != clb::kRows) {
        st = clb_packed_rows_to_slabs(input, buf[0], net->in_channels, in_hw, U, net->in_w, order, cs);
        if (st != CLB_OK) return st;
    } else {
        if (cudaMemcpyAsync(buf[0], input, (size_t)net->in_features * rb, cudaMemcpyDeviceToDevice, cs) != cudaSuccess) return check_launch(0);
    }

    // ---- layers
    const unsigned char *P = net->dev;
    long long feat = net->in_features;
    for (size_t i = 0; i < net->layers.size(); ++i) {
        const Layer &L = net->layers[i];
        if (L.kind == 1) {
            const clb::Order want = wanted(i), next = wanted(i + 1);
            if ((order == clb::kRows) != (want == clb::kRows)) { // change of layout between blocks
                st = want == clb::kRows ? clb_packed_layout(buf[cur], buf[cur ^ 1], L.Ci, (int64_t)L.H * L.W, U, 0, stream)
                                        : clb_packed_rows_to_slabs(buf[cur], buf[cur ^ 1], L.Ci, (int64_t)L.H * L.W, U, L.W, want, cs);
                if (st != CLB_OK) return st;
                cur ^= 1, order = want;
            }
            if (L.slab3) { // takes either slab order and writes what the next layer reads
                const void *recs = net->records ? (const void *)(net->records + L.off_recs) : scratch;
                if (!net->records) {
                    st = clb_slab3_records(P + L.off_ops, (const int32_t *)(P + L.off_a), nullptr, scratch, L.Ci, L.H, L.C, cs);
                    if (st != CLB_OK) return st;
                }
                st = clb_slab3_block(buf[cur], recs, buf[cur ^ 1], L.Ci, L.H, L.C, U, order, next, cs);
                order = next;
            } else if (order != clb::kRows) {
                st = clb_packed_convtree_slab(buf[cur], P + L.off_ops, (const int32_t *)(P + L.off_a), buf[cur ^ 1], scratch, L.Ci, L.H, L.W,
                                              L.C, 1, 1, L.ph, L.pw, L.kh, L.kw, U, stream);
                if (st == CLB_ERR_SHAPE) { // a tile the slab kernel cannot hold: this block runs on the rows layout
                    st = clb_packed_layout(buf[cur], buf[cur ^ 1], L.Ci, (int64_t)L.H * L.W, U, 0, stream);
                    if (st != CLB_OK) return st;
                    cur ^= 1, order = clb::kRows;
                }
            }
            if (!L.slab3 && order == clb::kRows)
                st = clb_packed_convtree(buf[cur], P + L.off_ops, (const int32_t *)(P + L.off_a), buf[cur ^ 1], L.Ci, L.H, L.W, L.C,
                                         L.stride, L.stride, L.ph, L.pw, L.kh, L.kw, words, 64, stream);
            if (st != CLB_OK) return st;
            cur ^= 1;
            feat = (long long)L.C * L.Hp * L.Wp;
            const bool last_conv = i + 1 == net->layers.size() || net->layers[i + 1].kind != 1;
            if (last_conv && order != clb::kRows) { // Flatten: back to feature rows
                st = clb_packed_layout(buf[cur], buf[cur ^ 1], L.C, (int64_t)L.Hp * L.Wp, U, 0, stream);
                if (st != CLB_OK) return st;
                cur ^= 1, order = clb::kRows;
            }
        } else if (L.kind == 2) {
            st = clb_packed_logic(buf[cur], (const int64_t *)(P + L.off_a), (const int64_t *)(P + L.off_b), P + L.off_ops, buf[cur ^ 1],
                                  L.in_dim, L.out_dim, words, 64, stream);
            if (st != CLB_OK) return st;
            cur ^= 1;
            feat = L.out_dim;
        } else {
            if (i + 1 == net->layers.size()) { // with their class sums
                st = clb_packed_tree_count(buf[cur], (const int32_t *)(P + L.off_a), P + L.off_ops, counts, L.in_dim, L.out_dim, L.levels, U, batch,
                                           net->num_classes, cs);
                if (st != CLB_ERR_SHAPE) return st;
            }
            st = clb_packed_tree(buf[cur], (const int32_t *)(P + L.off_a), P + L.off_ops, buf[cur ^ 1], L.in_dim, L.out_dim, L.levels, words,
                                 64, stream);
            if (st != CLB_OK) return st;
            cur ^= 1;
            feat = L.out_dim;
        }
    }
    // ---- GroupSum over the samples of the batch: gates such as NOT turn the zero samples behind them on
    return clb_group_popcount_units(buf[cur], counts, feat, U, batch, net->num_classes, cs);
}

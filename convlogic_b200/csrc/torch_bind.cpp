// Torch binding of the C-ABI library: tensors in, tensors out, autograd nodes in C++.
//
// What bounds a small call is the host: through ctypes and Python autograd Functions a layer cost 50 to 100 us of host
// time (measured on a three-layer flat stack, batch 100: 506 us forward + backward, of which the kernels take 91), the
// launches themselves about 2.5 us each.  Here a layer is one call: checks, output allocation, launch and the autograd
// node, and its backward runs on autograd's own thread without entering Python (except for the gradient-bucket callback
// of a parameter that carries one).  No arithmetic happens here; every number comes from the kernels behind
// include/convlogic_b200.h.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/accumulate_grad.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/convlogic_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::edge_list;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// ------------------------------------------------------------------------------------------------ helpers
// the exception the reference raises for the same condition (the Python side's `check`)
void check(int status)
{
    if (status == CLB_OK) return;
    const std::string text = std::string("convlogic_b200: ") + clb_status_string(status);
    if (status == CLB_ERR_LAUNCH) TORCH_CHECK(false, text, " (cudaError ", clb_last_cuda_error(), ")");
    TORCH_CHECK_VALUE(status != CLB_ERR_SHAPE && status != CLB_ERR_TOO_LARGE, text);
    TORCH_CHECK(false, text);
}

void need_input(const Tensor &t)
{
    TORCH_CHECK(t.is_cuda(), "convlogic_b200: tensor must be a CUDA tensor");
    TORCH_CHECK(t.is_contiguous(), "convlogic_b200: tensor must be contiguous");
}
template <typename... Ts> void need_inputs(const Ts &...ts) { (need_input(ts), ...); }

int dtype_code(const Tensor &t)
{
    if (t.scalar_type() == at::kFloat) return CLB_F32;
    TORCH_CHECK(t.scalar_type() == at::kDouble, "convlogic_b200: expected a float32 or float64 tensor, got ", t.scalar_type());
    return CLB_F64;
}

void *cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
template <typename T = void> T *ptr(const Tensor &t) { return t.defined() ? static_cast<T *>(t.data_ptr()) : nullptr; }
// device memory from torch's caching allocator, without the dispatcher's detour (about half a microsecond each) unless a trace
// has to see where an operation's result comes from
Tensor alloc(at::IntArrayRef sizes, const Tensor &like, at::ScalarType type)
{
    if (torch::jit::tracer::isTracing()) return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device()));
    return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}
Tensor alloc(at::IntArrayRef sizes, const Tensor &like) { return alloc(sizes, like, like.scalar_type()); }
Tensor alloc_strided(at::IntArrayRef sizes, at::IntArrayRef strides, const Tensor &like)
{
    if (torch::jit::tracer::isTracing()) return at::empty_strided(sizes, strides, like.options());
    return at::detail::empty_strided_cuda(sizes, strides, like.scalar_type(), like.device());
}
Tensor scratch_bytes(size_t n, const Tensor &like) { return alloc({(int64_t)(n < 16 ? 16 : n)}, like, at::kByte); }

// Raw calls run below autograd and view tracking: their results get a history from our own nodes only.
struct Below {
    at::AutoDispatchBelowADInplaceOrView guard;
    c10::cuda::CUDAGuard device;
    explicit Below(const Tensor &t) : device(t.device()) {}
};

bool wants_grad(std::initializer_list<std::reference_wrapper<const Tensor>> ts)
{
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor &t : ts)
        if (t.defined() && t.requires_grad()) return true;
    return false;
}

// Does torch follow this call by something that knows Python Functions only: torch.jit.trace, which would take a result made here for
// a constant, or forward-mode AD, whose tangents would be dropped?  Then it is handed to convlogic_b200.functional.
bool followed(std::initializer_list<std::reference_wrapper<const Tensor>> ts)
{
    if (torch::jit::tracer::isTracing()) return true;
    for (const Tensor &t : ts)
        if (t.defined() && t._fw_grad(0).defined()) return true;
    return false;
}
template <typename... Args> py::object in_python(const char *name, Args &&...args)
{
    return py::module_::import("convlogic_b200.functional").attr(name)(std::forward<Args>(args)...);
}

// SavedVariable of an input (never an output) of a node
SavedVariable saved(const Tensor &t) { return SavedVariable(t, false); }

// One node kind per operation: `Derived` has fields, run(grads) and clear().
template <typename Derived> std::shared_ptr<Derived> new_node() { return std::shared_ptr<Derived>(new Derived(), torch::autograd::deleteNode); }

// A node's upstream gradient.  Where nothing comes in (a consumer whose backward gives no gradient) it is zeros, as for a Python Function: the
// parameters' gradients are then zeros too, and a gradient slice is overwritten and not left with the last step's values.
Tensor upstream(const Node &n, const variable_list &grads) { return grads[0].defined() ? grads[0] : n.input_metadata(0).zeros_like(); }

// [rows, cols] fp32 -> contiguous [cols, rows]
Tensor transpose2d(const Tensor &x)
{
    need_input(x);
    TORCH_CHECK(x.dim() == 2 && x.scalar_type() == at::kFloat, "convlogic_b200: transpose2d expects a contiguous 2-D float32 tensor");
    Below below(x);
    Tensor out = alloc({x.size(1), x.size(0)}, x);
    check(clb_transpose_f32(ptr<float>(x), ptr<float>(out), x.size(0), x.size(1), cur_stream()));
    return out;
}

// contiguous copy of t's transpose (t 2-D), with the library's tiled kernel where it applies
Tensor transposed_copy(const Tensor &t)
{
    if (t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel()) return transpose2d(t);
    return t.t().contiguous();
}

// Is a [B, F] activation stored feature-major ([F, B], what a flat layer returns)?  Then its storage is read as it is.
bool stored_feature_major(const Tensor &x)
{
    return x.dim() == 2 && (x.size(0) <= 1 || x.stride(0) == 1) && (x.size(1) <= 1 || x.stride(1) == x.size(0));
}
// a tensor whose storage is [F, B], from a [B, F] activation (x itself where possible; the shape of the result is not to be used)
Tensor feature_major_storage(const Tensor &x) { return stored_feature_major(x) ? x : transposed_copy(x); }

// A [B, F] gradient of feature-major storage: made in that form, and turned round at the end for a leaf that stores [B, F] itself (`.grad`
// takes the leaf's strides).
Tensor feature_major_grad(int64_t batch, int64_t features, const Tensor &like)
{
    return alloc_strided({batch, features}, {1, std::max<int64_t>(batch, 1)}, like);
}
Tensor finished_grad(const Tensor &g, const Node &n) // of the node's first input
{
    if (g.is_contiguous()) return g;
    const auto *leaf = dynamic_cast<const torch::autograd::AccumulateGrad *>(n.next_edge(0).function.get());
    return leaf && !stored_feature_major(leaf->variable) ? transposed_copy(g.t()) : g;
}

// ------------------------------------------------------------------------------------------------ gradient sinks
// A parameter may carry `_clb_grad_sink` = (slice of a flat gradient buffer, ready callback, ranges callback, range): its
// gradient is then written into the slice by the kernel and the callback told, and autograd gets no gradient for it.
struct Sink {
    Tensor slice;
    py::object ready, ranges, range;
};
std::optional<Sink> sink_of(const Tensor &w) // GIL held
{
    py::object obj = py::reinterpret_steal<py::object>(THPVariable_Wrap(w));
    PyObject *s = nullptr;
    if (PyObject_HasAttrString(obj.ptr(), "_clb_grad_sink")) s = PyObject_GetAttrString(obj.ptr(), "_clb_grad_sink");
    if (!s) return std::nullopt;
    py::object held = py::reinterpret_steal<py::object>(s);
    if (held.is_none()) return std::nullopt;
    py::tuple t = held.cast<py::tuple>();
    Sink out;
    out.slice = t[0].cast<Tensor>();
    out.ready = t[1];
    if (t.size() > 3) out.ranges = t[2], out.range = t[3];
    return out;
}

std::atomic<int64_t> g_sinks{0}; // parameters that carry one: while there are none, no backward pass needs to ask Python

// The slices of one backward call's parameters: all of them or none (a kernel writes them together).
class Sinks {
public:
    explicit Sinks(std::initializer_list<std::reference_wrapper<const Tensor>> ws)
    {
        if (g_sinks.load(std::memory_order_relaxed) <= 0) return;
        py::gil_scoped_acquire gil;
        for (const Tensor &w : ws) {
            auto s = sink_of(w);
            if (!s) {
                list_.clear();
                return;
            }
            list_.push_back(std::move(*s));
        }
    }
    ~Sinks()
    {
        if (list_.empty()) return;
        py::gil_scoped_acquire gil;
        list_.clear();
    }
    bool any() const { return !list_.empty(); }
    Tensor slice(size_t i) const { return any() ? list_[i].slice : Tensor(); }
    // the kernels that write the slices are enqueued: neighbouring slices of one bucket are reported as one exchange
    void ready()
    {
        if (list_.empty()) return;
        py::gil_scoped_acquire gil;
        bool one_bucket = list_.size() > 1;
        for (const Sink &s : list_) one_bucket = one_bucket && s.ranges && s.ranges.equal(list_[0].ranges);
        if (one_bucket) {
            py::list ranges;
            for (const Sink &s : list_) ranges.append(s.range);
            list_[0].ranges(ranges);
        } else {
            for (const Sink &s : list_) s.ready();
        }
    }

private:
    std::vector<Sink> list_;
};

// ------------------------------------------------------------------------------------------------ fused block
struct Geom {
    int sh, sw, ph, pw, kh, kw;
    bool operator==(const Geom &o) const { return sh == o.sh && sw == o.sw && ph == o.ph && pw == o.pw && kh == o.kh && kw == o.kw; }
};

// What the kernels need to know about a selection: checked and laid out once per (selection tensor and version, geometry,
// input channels), kept on the selection tensor object as `_clb_plan` (nothing outlives the tensor).
struct BlockPlan {
    Geom g;
    int C, ci;
    int64_t version;
    const void *data;
    int flag;                        // CLB_SEL_UNBOUNDED when a tap lies outside the window
    int many;                        // CLB_SEL_MANY when an output channel reads more than two input channels
    bool channels_ok;
    std::vector<int32_t> sel;        // host copy
    std::mutex mu;
    int lists = -1;                  // channel lists: -1 not built, 0 the selection does not fit two planes, 1 built
    Tensor start, entry;
    struct Groups {
        Tensor start, list;
        int cg, nb;
    };
    std::map<std::tuple<int64_t, int64_t, int64_t, int>, Groups> groups; // (N, H, W, dtype), at most 16 kept
    c10::Device device{c10::kCUDA};

    Tensor to_device(const std::vector<int32_t> &v)
    {
        return at::tensor(at::ArrayRef<int32_t>(v.data(), v.size()), at::TensorOptions().dtype(at::kInt)).to(device);
    }
    bool channel_lists()
    {
        std::lock_guard<std::mutex> lock(mu);
        if (lists < 0) {
            std::vector<int32_t> st((size_t)ci + 1, 0), en((size_t)(2 * C > 0 ? 2 * C : 1), 0);
            const int n = clb_conv_channel_lists(sel.data(), C, ci, g.kh, g.kw, st.data(), en.data(), (int)en.size());
            if (n < 0 && n != CLB_ERR_SHAPE) check(n);
            if (n >= 0) {
                en.resize((size_t)(n > 0 ? n : 1));
                start = to_device(st), entry = to_device(en);
            }
            lists = n >= 0;
        }
        return lists == 1;
    }
    Groups group_tables(int64_t n, int64_t h, int64_t w, int dtype)
    {
        std::lock_guard<std::mutex> lock(mu);
        const auto key = std::make_tuple(n, h, w, dtype);
        auto it = groups.find(key);
        if (it != groups.end()) return it->second;
        Groups out;
        check(clb_conv_group_plan((int)n, ci, (int)h, (int)w, C, g.sh, g.sw, g.ph, g.pw, g.kh, g.kw, dtype, &out.cg, &out.nb));
        const int count = (ci + out.cg - 1) / out.cg;
        std::vector<int32_t> st((size_t)count + 1, 0), ls((size_t)std::max<long long>(1, (long long)C * std::min(count, 8)), 0);
        const int got = clb_conv_build_groups(sel.data(), C, ci, out.cg, st.data(), ls.data(), (int)ls.size());
        TORCH_CHECK(got != CLB_ERR_ARG, "convlogic_b200: selection refers to a channel the input does not have");
        if (got < 0) check(got);
        ls.resize((size_t)(got > 0 ? got : 1));
        out.start = to_device(st), out.list = to_device(ls);
        if (groups.size() >= 16) groups.clear();
        groups.emplace(key, out);
        return out;
    }
};
using PlanPtr = std::shared_ptr<BlockPlan>;

// What a plan is on a copied or unpickled tensor (Tensor.__deepcopy__ and __reduce_ex__ take a tensor's attributes along): nothing
// that `kept` accepts, so that the copy's first use lays its own out.  An empty OrderedDict is what torch.load reads without
// this extension and under weights_only.
template <typename Plan> void copies_as_nothing(py::class_<Plan, std::shared_ptr<Plan>> c)
{
    c.def("__deepcopy__", [](const Plan &, const py::object &) { return py::none(); });
    c.def("__reduce__", [](const Plan &) { return py::make_tuple(py::module_::import("collections").attr("OrderedDict"), py::tuple()); });
}
template <typename Plan> std::shared_ptr<Plan> kept(const py::handle &tensor) // GIL held
{
    static PyObject *const name = PyUnicode_InternFromString("_clb_plan");
    const py::object o = py::reinterpret_steal<py::object>(PyObject_GetAttr(tensor.ptr(), name));
    if (!o) {
        PyErr_Clear();
        return nullptr;
    }
    return py::isinstance<Plan>(o) ? o.cast<std::shared_ptr<Plan>>() : nullptr;
}

PlanPtr plan_for(const py::handle &sel_obj, const Tensor &sel, const Geom &g, int64_t ci) // GIL held
{
    const int64_t version = (int64_t)sel._version(); // raises for a tensor made in inference mode: nothing would tell that it has changed
    if (PlanPtr p = kept<BlockPlan>(sel_obj); p && p->version == version && p->data == sel.data_ptr() && p->g == g && p->ci == ci) return p;
    auto p = std::make_shared<BlockPlan>();
    p->g = g, p->C = (int)sel.size(0), p->ci = (int)ci, p->version = version, p->data = sel.data_ptr(), p->device = sel.device();
    const Tensor host = sel.detach().to(at::kCPU).contiguous();
    p->sel.assign(host.data_ptr<int32_t>(), host.data_ptr<int32_t>() + host.numel());
    bool inside = true, channels = true, two = true;
    for (size_t c = 0; c < p->sel.size(); c += 8) {
        int first = -1, second = -1;
        for (size_t k = c; k < c + 8; ++k) {
            const int32_t word = p->sel[k];
            const int ch = (word >> 16) & 0xFFFF;
            inside = inside && ((word >> 8) & 0xFF) < g.kh && (word & 0xFF) < g.kw;
            channels = channels && word >= 0 && ch < ci;
            if (first < 0) first = ch;
            else if (ch != first && second < 0) second = ch;
            two = two && (ch == first || ch == second);
        }
    }
    p->flag = inside ? 0 : CLB_SEL_UNBOUNDED, p->many = two ? 0 : CLB_SEL_MANY, p->channels_ok = channels;
    sel_obj.attr("_clb_plan") = p;
    return p;
}

bool is_feature_major(const Tensor &t) // [N, C, h, w] on the contiguous storage [C, h, w, N]
{
    if (t.dim() != 4 || t.is_contiguous()) return false;
    const int64_t n = t.size(0), c = t.size(1), h = t.size(2), w = t.size(3);
    auto ok = [](int64_t size, int64_t stride, int64_t want) { return size == 1 || stride == want; };
    return ok(n, t.stride(0), 1) && ok(w, t.stride(3), n) && ok(h, t.stride(2), n * w) && ok(c, t.stride(1), n * w * h);
}

struct BlockDims {
    int n, ci, h, w, c, ho, wo;
};
BlockDims block_dims(const Tensor &x, const Tensor &w, const Tensor &sel, const Geom &g)
{
    TORCH_CHECK(x.dim() == 4, "convlogic_b200: x must be [N, C, H, W]");
    const int64_t c = w.size(0);
    TORCH_CHECK(w.dim() == 3 && w.size(1) == 7 && w.size(2) == 16 && w.scalar_type() == x.scalar_type(), "convlogic_b200: gate tensor must be [", c,
                ", 7, 16] ", x.scalar_type());
    TORCH_CHECK(sel.scalar_type() == at::kInt && sel.dim() == 2 && sel.size(0) == c && sel.size(1) == 8,
                "convlogic_b200: selection must be int32 [", c, ", 8], got ", sel.scalar_type(), " ", sel.sizes());
    BlockDims d{(int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), (int)c, 0, 0};
    d.ho = (d.h + 2 * g.ph - g.kh) / g.sh + 1, d.wo = (d.w + 2 * g.pw - g.kw) / g.sw + 1;
    return d;
}

struct BlockOut {
    Tensor y, amax, x2, x3, idx;
};

BlockOut block_fwd(const Tensor &x, const Tensor &w, const Tensor &sel, const Geom &g, const std::function<PlanPtr()> &get_plan, int wmode,
                   bool want_amax, bool want_inter, bool want_idx, bool y_fm)
{
    need_inputs(x, w, sel);
    const BlockDims d = block_dims(x, w, sel, g);
    TORCH_CHECK(d.ho > 0 && d.wo > 0, "Invalid output shape: H_out=", d.ho, ", W_out=", d.wo);
    TORCH_CHECK(d.ho % 2 == 0 && d.wo % 2 == 0, "Output height and width after convolution must be divisible by 2 for 2x2 max pooling, but got H_out=",
                d.ho, ", W_out=", d.wo);
    const int hp = d.ho / 2, wp = d.wo / 2, dt = dtype_code(x);
    Below below(x);
    BlockOut o;
    if (want_amax) o.amax = alloc({d.n, d.c, hp, wp}, x, at::kByte);
    if (want_inter) o.x2 = alloc({d.n, d.c, d.ho, d.wo, 4}, x), o.x3 = alloc({d.n, d.c, d.ho, d.wo, 2}, x);
    if (want_idx) o.idx = alloc({d.n, d.c, (int64_t)hp * wp}, x, at::kInt);
    if (d.n == 0 || d.c == 0) { // empty batch: nothing to launch
        o.y = alloc({d.n, d.c, hp, wp}, x);
        return o;
    }
    const PlanPtr plan = get_plan();
    TORCH_CHECK(plan->channels_ok, "convlogic_b200: selection refers to a channel the input does not have");
    if (y_fm && dt == CLB_F32 && !want_inter && !want_idx && !plan->flag) {
        // the flat layers' layout, storage [C, h, w, N]; only the plane kernels write it
        o.y = alloc_strided({d.n, d.c, hp, wp}, {1, (int64_t)hp * wp * d.n, (int64_t)wp * d.n, d.n}, x);
        const int rc = clb_convtree_fwd(ptr(x), ptr(w), ptr<int32_t>(sel), ptr(o.y), ptr<uint8_t>(o.amax), nullptr, nullptr, nullptr, d.n, d.ci, d.h, d.w,
                                        d.c, g.sh, g.sw, g.ph, g.pw, g.kh, g.kw, wmode | CLB_Y_FEATURE_MAJOR | plan->many, dt, cur_stream());
        if (rc != CLB_ERR_SHAPE) {
            check(rc);
            return o;
        }
    }
    o.y = alloc({d.n, d.c, hp, wp}, x);
    check(clb_convtree_fwd(ptr(x), ptr(w), ptr<int32_t>(sel), ptr(o.y), ptr<uint8_t>(o.amax), ptr(o.x2), ptr(o.x3), ptr<int32_t>(o.idx), d.n, d.ci, d.h,
                           d.w, d.c, g.sh, g.sw, g.ph, g.pw, g.kh, g.kw, wmode | plan->flag | plan->many, dt, cur_stream()));
    return o;
}

// (gx or undefined, gw or undefined); gw_out: where the gate gradient goes (a slice of a flat bucket)
std::pair<Tensor, Tensor> block_bwd(Tensor gy, const Tensor &x, const Tensor &w, const Tensor &sel, const Tensor &amax, const Geom &g,
                                    const std::function<PlanPtr()> &get_plan, int wmode, bool need_gx, bool need_gw, const Tensor &gw_out)
{
    const bool fm = gy.is_cuda() && is_feature_major(gy);
    need_inputs(x, w, sel);
    if (!fm) need_input(gy);
    const BlockDims d = block_dims(x, w, sel, g);
    const int64_t hp = d.ho / 2, wp = d.wo / 2;
    const std::vector<int64_t> want{d.n, d.c, hp, wp};
    TORCH_CHECK(gy.sizes() == at::IntArrayRef(want) && gy.scalar_type() == x.scalar_type(), "convlogic_b200: upstream gradient must be ",
                at::IntArrayRef(want), " ", x.scalar_type(), ", got ", gy.sizes(), " ", gy.scalar_type());
    TORCH_CHECK(!amax.defined() || (amax.sizes() == at::IntArrayRef(want) && amax.scalar_type() == at::kByte),
                "convlogic_b200: arg-max tensor must be uint8 ", at::IntArrayRef(want));
    const int dt = dtype_code(x);
    Below below(x);
    Tensor gx, gw;
    if (need_gx) gx = alloc(x.sizes(), x);
    if (need_gw) {
        gw = gw_out.defined() ? gw_out : alloc(w.sizes(), w);
        TORCH_CHECK(gw.sizes() == w.sizes() && gw.scalar_type() == w.scalar_type() && gw.is_contiguous(),
                    "convlogic_b200: `gw_out` must be contiguous with the gate tensor's shape and dtype");
    }
    if (d.n == 0 || d.c == 0) { // empty batch: the gate gradient is an empty sum
        if (gw.defined()) gw.zero_();
        return {gx, gw};
    }
    const PlanPtr plan = get_plan();
    TORCH_CHECK(plan->channels_ok, "convlogic_b200: selection refers to a channel the input does not have");
    if (!plan->flag && dt == CLB_F32 && amax.defined()) {
        // The plane kernels (two channel planes per output channel in shared memory): both gradients of 3x3 blocks on images of 32 to 4
        // pixels, the gate gradient alone of a 32x32 first block.
        const size_t bytes = clb_convtree_bwd_plane_scratch_bytes(d.n, d.ci, d.h, d.w, d.c, g.sh, g.sw, g.ph, g.pw, g.kh, g.kw, dt);
        if (bytes && plan->channel_lists()) {
            Tensor scratch = scratch_bytes(bytes, x);
            const int rc = clb_convtree_bwd_plane(ptr(gy), ptr(x), ptr(w), ptr<int32_t>(sel), ptr<uint8_t>(amax), ptr(gx), ptr(gw), ptr<int32_t>(plan->start),
                                                  ptr<int32_t>(plan->entry), ptr(scratch), bytes, d.n, d.ci, d.h, d.w, d.c, g.sh, g.sw, g.ph, g.pw, g.kh,
                                                  g.kw, wmode | (fm ? CLB_Y_FEATURE_MAJOR : 0), dt, cur_stream());
            if (rc != CLB_ERR_SHAPE) {
                check(rc);
                return {gx, gw};
            }
        }
    }
    if (fm) gy = transposed_copy(gy.permute({1, 2, 3, 0}).reshape({(int64_t)d.c * hp * wp, d.n})).view({d.n, d.c, hp, wp});
    const size_t bytes = clb_convtree_bwd_scratch_bytes(d.n, d.ci, d.h, d.w, d.c, g.sh, g.sw, g.ph, g.pw, g.kh, g.kw, need_gx, need_gw, dt);
    Tensor scratch = scratch_bytes(bytes, x);
    BlockPlan::Groups gr{Tensor(), Tensor(), 1, 1};
    if (need_gx) gr = plan->group_tables(d.n, d.h, d.w, dt);
    check(clb_convtree_bwd(ptr(gy), ptr(x), ptr(w), ptr<int32_t>(sel), ptr<uint8_t>(amax), ptr(gx), ptr(gw), ptr<int32_t>(gr.start),
                           ptr<int32_t>(gr.list), gr.cg, gr.nb, ptr(scratch), bytes, d.n, d.ci, d.h, d.w, d.c, g.sh, g.sw, g.ph, g.pw, g.kh, g.kw,
                           wmode | plan->flag, dt, cur_stream()));
    return {gx, gw};
}

struct BlockNode : public Node {
    SavedVariable x, w, amax; // what the call made or was given goes through saved-tensor hooks; `sel` belongs to the module
    Tensor sel;
    PlanPtr plan;
    Geom g;
    int wmode;
    std::string name() const override { return "FullConvLogicFunctionBackward"; }
    void release_variables() override { x.reset_data(), w.reset_data(), amax.reset_data(); }
    variable_list apply(variable_list &&grads) override
    {
        const Tensor xx = x.unpack(), ww = w.unpack(), best = amax.unpack(), &ss = sel;
        TORCH_CHECK(plan->version == (int64_t)ss._version(), "convlogic_b200: the selection was modified between forward and backward");
        const bool need_gx = task_should_compute_output(0), need_gw = task_should_compute_output(1) && wmode != CLB_W_ARGMAX;
        if (!need_gx && !need_gw) return {Tensor(), Tensor()};
        Tensor gy = upstream(*this, grads);
        if (!is_feature_major(gy)) gy = gy.contiguous(); // a feature-major gradient (from flat layers behind this block) is read as it is
        if (!need_gw) return {block_bwd(gy, xx, ww, ss, best, g, [&] { return plan; }, wmode, need_gx, false, Tensor()).first, Tensor()};
        Sinks sinks({ww});
        auto out = block_bwd(gy, xx, ww, ss, best, g, [&] { return plan; }, wmode, need_gx, true, sinks.slice(0));
        if (!sinks.any()) return {out.first, out.second};
        sinks.ready();
        return {out.first, Tensor()};
    }
};

// y, or (y[, x2, x3][, idx]) when extras are asked for
py::object block(Tensor x, Tensor w, py::object sel_obj, int sh, int sw, int ph, int pw, int kh, int kw, bool want_inter, bool want_idx, int wmode,
                 bool y_fm)
{
    if (followed({x, w})) return in_python("followed_block", x, w, sel_obj, sh, sw, ph, pw, kh, kw, want_inter, want_idx, wmode, y_fm);
    const Tensor sel = sel_obj.cast<Tensor>();
    x = x.contiguous(), w = w.contiguous();
    const Geom g{sh, sw, ph, pw, kh, kw};
    const bool graph = wants_grad({x, w});
    PlanPtr plan;
    auto get_plan = [&] { return plan = plan_for(sel_obj, sel, g, x.size(1)); };
    BlockOut o = block_fwd(x, w, sel, g, get_plan, wmode, graph, want_inter, want_idx, y_fm);
    if (graph) {
        auto node = new_node<BlockNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(x, w));
        if (!plan) get_plan();
        node->x = saved(x), node->w = saved(w), node->sel = sel, node->amax = saved(o.amax), node->plan = plan, node->g = g, node->wmode = wmode;
        torch::autograd::set_history(o.y, node);
    }
    if (!want_inter && !want_idx) return py::cast(o.y);
    py::list out;
    out.append(o.y);
    if (want_inter) out.append(o.x2), out.append(o.x3);
    if (want_idx) out.append(o.idx);
    return py::tuple(out);
}

// ------------------------------------------------------------------------------------------------ flat layer
struct LogicDims {
    int64_t in, out, batch;
};
LogicDims logic_dims(const Tensor &x_fm, const Tensor &a, const Tensor &b, const Tensor &w)
{
    TORCH_CHECK(x_fm.dim() == 2, "convlogic_b200: x must be [in_dim, batch], got ", x_fm.sizes());
    const int64_t out = w.size(0);
    TORCH_CHECK(w.dim() == 2 && w.size(1) == 16 && w.scalar_type() == x_fm.scalar_type(), "convlogic_b200: gate tensor must be [", out, ", 16] ",
                x_fm.scalar_type());
    TORCH_CHECK(a.scalar_type() == at::kLong && b.scalar_type() == at::kLong && a.dim() == 1 && b.dim() == 1 && a.size(0) == out && b.size(0) == out,
                "convlogic_b200: connection indices must be int64 [out_dim]");
    return {x_fm.size(0), out, x_fm.size(1)};
}

// The consumer lists as the combined backward reads them, laid out once per layer and kept on the list tensor object as
// `_clb_plan` (checked by the tensors' addresses and versions).
using LogicKey = std::array<std::pair<const void *, int64_t>, 4>; // a, b, start, consumers: address and version
LogicKey logic_key(const Tensor &a, const Tensor &b, const Tensor &start, const Tensor &cons)
{
    auto id = [](const Tensor &t) { return std::make_pair((const void *)t.data_ptr(), (int64_t)t._version()); };
    return {id(a), id(b), id(start), id(cons)};
}
struct LogicPlan {
    LogicKey key;
    int64_t in = 0, out = 0;
    Tensor start32, entry;
    bool paths = false;
    Tensor rec, open;    // (paths) neurons in the order of paths, features whose gradient a path does not complete; undefined: lists and connections disagree
    int64_t n_open = 0;
    bool captured = false; // a stream capture reads it: its tables stay with the plan that replaces it, for the graph holds their addresses
    std::shared_ptr<LogicPlan> held;
    c10::Stream stream{c10::Stream::UNSAFE, c10::Device(c10::kCPU), 0}; // of the tables' memory
    void used() const // on the current stream: the memory of a plan that goes waits for what that stream still reads
    {
        const c10::Stream now = c10::cuda::getCurrentCUDAStream().unwrap();
        if (now == stream) return;
        for (const Tensor &t : {start32, entry, rec, open})
            if (t.defined()) t.record_stream(now);
    }
    bool path_fwd(int64_t batch) const { return rec.defined() && clb_logic_path_pays(in, out, batch, n_open, 0); }
    bool path_bwd(int64_t batch) const { return rec.defined() && clb_logic_path_pays(in, out, batch, n_open, 1); }
};
using LogicPlanPtr = std::shared_ptr<LogicPlan>;

// paths: with the neurons in the order of paths (a plan is never changed: one without is replaced by one that shares its lists)
LogicPlanPtr logic_plan_for(const py::handle &start_obj, const Tensor &a, const Tensor &b, const Tensor &start, const Tensor &cons, int64_t in, int64_t out,
                            bool paths)
{
    const LogicKey key = logic_key(a, b, start, cons);
    const LogicPlanPtr last = kept<LogicPlan>(start_obj);
    // (the default stream, which cannot be captured, is not asked: it would cost half a microsecond per layer and step)
    const bool capture = c10::cuda::getCurrentCUDAStream().stream() && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
    LogicPlanPtr old = last;
    if (old && !(old->key == key && old->in == in && old->out == out)) old = nullptr;
    if (old && capture) old->captured = true;
    if (old && (old->paths || !paths)) {
        old->used();
        return old;
    }
    need_inputs(a, b, start, cons);
    TORCH_CHECK(start.scalar_type() == at::kLong && cons.scalar_type() == at::kLong && start.numel() == in + 1 && cons.numel() == 2 * out,
                "convlogic_b200: consumer lists must be int64 [in_dim + 1] and [2 * out_dim]");
    if (in > 0x3fffffff || out > 0x3fffffff) return nullptr;
    // inside a stream capture nothing would be laid out before the replay: this call runs the two separate gradient kernels
    if (capture) return old;
    auto p = std::make_shared<LogicPlan>();
    p->key = key, p->in = in, p->out = out, p->paths = paths;
    p->stream = c10::cuda::getCurrentCUDAStream().unwrap();
    if (last) p->held = last->captured ? last : last->held;
    Below below(start);
    if (old) {
        old->used();
        p->start32 = old->start32, p->entry = old->entry;
    } else {
        p->start32 = alloc({in + 1}, start, at::kInt), p->entry = alloc({2 * out, 2}, start, at::kInt);
        check(clb_logic_entries(ptr<int64_t>(a), ptr<int64_t>(b), ptr<int64_t>(start), ptr<int64_t>(cons), ptr<int32_t>(p->start32), ptr(p->entry), in, out,
                                cur_stream()));
    }
    if (paths && out) {
        const size_t bytes = clb_logic_path_scratch_bytes(in, out);
        const Tensor scratch = scratch_bytes(bytes, start), count = alloc({2}, start, at::kInt);
        p->rec = alloc({out, 4}, start, at::kInt), p->open = alloc({in}, start, at::kInt);
        check(clb_logic_path(ptr<int64_t>(a), ptr<int64_t>(b), ptr<int32_t>(p->start32), ptr(p->entry), ptr(p->rec), ptr<int32_t>(p->open), ptr<int32_t>(count),
                             ptr(scratch), bytes, in, out, cur_stream()));
        const Tensor host = count.to(at::kCPU);
        p->n_open = host.data_ptr<int32_t>()[1];
        if (host.data_ptr<int32_t>()[0] != out) p->rec = p->open = Tensor();
    }
    // the plan outlives this call: work of other streams may read it next
    c10::cuda::getCurrentCUDAStream().synchronize();
    start_obj.attr("_clb_plan") = p;
    return p;
}

void logic_fwd(const Tensor &x_fm, const Tensor &a, const Tensor &b, const Tensor &w, int wmode, const Tensor &y_storage)
{
    need_inputs(x_fm, a, b, w);
    const LogicDims d = logic_dims(x_fm, a, b, w);
    if (d.batch == 0 || d.out == 0) return;
    const Tensor coef = clb_logic_fwd_scratch_bytes(d.in, d.out, d.batch, dtype_code(x_fm)) ? alloc({d.out, 4}, x_fm) : Tensor();
    check(clb_logic_fwd_coef(ptr(x_fm), ptr<int64_t>(a), ptr<int64_t>(b), ptr(w), ptr(y_storage), ptr(coef), d.in, d.out, d.batch, wmode, dtype_code(x_fm),
                             cur_stream()));
}

Tensor logic_bwd_w(const Tensor &x_fm, const Tensor &a, const Tensor &b, const Tensor &w, const Tensor &gy_fm, int wmode, const Tensor &gw_out)
{
    need_inputs(x_fm, a, b, w, gy_fm);
    const LogicDims d = logic_dims(x_fm, a, b, w);
    Below below(x_fm);
    Tensor gw = gw_out.defined() ? gw_out : alloc(w.sizes(), w);
    if (d.batch == 0 || d.out == 0) return gw.zero_();
    check(clb_logic_bwd_w(ptr(x_fm), ptr<int64_t>(a), ptr<int64_t>(b), ptr(w), ptr(gy_fm), ptr(gw), d.in, d.out, d.batch, wmode, dtype_code(x_fm),
                          cur_stream()));
    return gw;
}

Tensor logic_bwd_x(const Tensor &x_fm, const Tensor &a, const Tensor &b, const Tensor &w, const Tensor &gy_fm, const Tensor &start, const Tensor &cons,
                   int wmode)
{
    need_inputs(x_fm, a, b, w, gy_fm, start, cons);
    const LogicDims d = logic_dims(x_fm, a, b, w);
    TORCH_CHECK(start.scalar_type() == at::kLong && cons.scalar_type() == at::kLong && start.numel() == d.in + 1 && cons.numel() == 2 * d.out,
                "convlogic_b200: consumer lists must be int64 [in_dim + 1] and [2 * out_dim]");
    Below below(x_fm);
    Tensor gx = alloc(x_fm.sizes(), x_fm);
    if (d.batch == 0) return gx;
    check(clb_logic_bwd_x(ptr(x_fm), ptr<int64_t>(a), ptr<int64_t>(b), ptr(w), ptr(gy_fm), ptr(gx), ptr<int64_t>(start), ptr<int64_t>(cons), d.in, d.out,
                          d.batch, wmode, dtype_code(x_fm), cur_stream()));
    return gx;
}

struct LogicNode : public Node {
    SavedVariable x, w;      // x: a tensor on the feature-major storage the forward read
    Tensor a, b, start, cons; // connections, checked against `key`
    LogicKey key;
    SavedVariable coef;      // gate coefficients and the laid-out lists (fp32 with an input gradient)
    LogicPlanPtr plan;
    int64_t in, out, batch;
    int wmode;
    bool fm; // the call's own tensors are feature-major ([in, B] -> [out, B])
    std::string name() const override { return "LogicLayerCudaFunctionBackward"; }
    void release_variables() override { x.reset_data(), w.reset_data(), coef.reset_data(); }
    variable_list apply(variable_list &&grads) override
    {
        const Tensor xx = x.unpack(), ww = w.unpack();
        TORCH_CHECK(key == logic_key(a, b, start, cons), "convlogic_b200: the connections of a layer were modified between forward and backward");
        const bool need_gx = task_should_compute_output(0), need_gw = task_should_compute_output(1) && wmode != CLB_W_ARGMAX;
        Below below(xx);
        const Tensor up = upstream(*this, grads), gy = fm ? up.contiguous() : feature_major_storage(up);
        TORCH_CHECK(gy.numel() == out * batch && gy.scalar_type() == xx.scalar_type(), "convlogic_b200: upstream gradient must be [", out, ", ", batch, "] ",
                    xx.scalar_type());
        const int dt = dtype_code(xx);
        Tensor gx, gw;
        Sinks sinks(need_gw ? std::initializer_list<std::reference_wrapper<const Tensor>>{ww} : std::initializer_list<std::reference_wrapper<const Tensor>>{});
        if (need_gx) gx = fm ? alloc({in, batch}, xx) : feature_major_grad(batch, in, xx);
        if (need_gw) {
            gw = sinks.any() ? sinks.slice(0) : alloc(ww.sizes(), ww);
            TORCH_CHECK(gw.sizes() == ww.sizes() && gw.is_contiguous() && gw.scalar_type() == ww.scalar_type(),
                        "convlogic_b200: a gradient slice must be contiguous with the gate tensor's shape and dtype");
        }
        if (batch == 0 || out == 0) {
            if (gw.defined()) gw.zero_();
            if (gx.defined()) gx.zero_();
        } else {
            int rc = CLB_ERR_SHAPE;
            if (need_gx && need_gw && plan && plan->path_bwd(batch)) {
                const Tensor cc = coef.unpack();
                const size_t bytes = clb_logic_path_bwd_scratch_bytes(out, batch);
                Tensor scratch = scratch_bytes(bytes, xx);
                rc = clb_logic_path_bwd(ptr<float>(xx), ptr<float>(ww), ptr<float>(cc), ptr<float>(gy), ptr<float>(gx), ptr<float>(gw),
                                        ptr<int32_t>(plan->start32), ptr(plan->entry), ptr(plan->rec), ptr<int32_t>(plan->open), plan->n_open, ptr(scratch),
                                        bytes, in, out, batch, wmode, cur_stream());
                if (rc != CLB_ERR_SHAPE) check(rc);
            }
            const size_t bytes = rc == CLB_ERR_SHAPE && need_gx && need_gw && plan ? clb_logic_bwd_scratch_bytes(in, out, batch) : 0;
            if (rc == CLB_ERR_SHAPE && need_gx && plan && (bytes || !need_gw)) { // both gradients in one pass, where that is the faster way
                const Tensor cc = coef.unpack();
                Tensor scratch;
                if (need_gw) scratch = scratch_bytes(bytes, xx);
                rc = clb_logic_bwd(ptr<float>(xx), ptr<float>(ww), ptr<float>(cc), ptr<float>(gy), ptr<float>(gx), ptr<float>(gw),
                                   ptr<int32_t>(plan->start32), ptr(plan->entry), ptr(scratch), bytes, in, out, batch, wmode, cur_stream());
                if (rc != CLB_ERR_SHAPE) check(rc);
            }
            if (rc == CLB_ERR_SHAPE && need_gx)
                check(clb_logic_bwd_x(ptr(xx), ptr<int64_t>(a), ptr<int64_t>(b), ptr(ww), ptr(gy), ptr(gx), ptr<int64_t>(start), ptr<int64_t>(cons), in, out, batch,
                                      wmode, dt, cur_stream()));
            if (rc == CLB_ERR_SHAPE && need_gw)
                check(clb_logic_bwd_w(ptr(xx), ptr<int64_t>(a), ptr<int64_t>(b), ptr(ww), ptr(gy), ptr(gw), in, out, batch, wmode, dt, cur_stream()));
        }
        if (gx.defined() && !fm) gx = finished_grad(gx, *this);
        if (sinks.any()) {
            sinks.ready();
            gw = Tensor();
        }
        return {gx, gw};
    }
};

// fm: x [in, B] -> y [out, B] (the reference's Function); else x [B, in] -> y [B, out] on the storage [out, B]
Tensor logic(const Tensor &x, const Tensor &a, const Tensor &b, const Tensor &w_in, py::object start_obj, const Tensor &cons, int wmode, bool fm)
{
    if (followed({x, w_in})) return in_python("followed_logic", x, a, b, w_in, start_obj, cons, wmode, fm).cast<Tensor>();
    const Tensor start = start_obj.cast<Tensor>();
    const bool graph = wants_grad({x, w_in});
    TORCH_CHECK(x.is_cuda(), "convlogic_b200: tensor must be a CUDA tensor");
    TORCH_CHECK(x.dim() == 2, "convlogic_b200: x must be 2-D, got ", x.sizes());
    const int64_t in = x.size(fm ? 0 : 1), batch = x.size(fm ? 1 : 0), out = w_in.size(0);
    const int dt = dtype_code(x);
    TORCH_CHECK(w_in.dim() == 2 && w_in.size(1) == 16 && w_in.scalar_type() == x.scalar_type(), "convlogic_b200: gate tensor must be [", out, ", 16] ",
                x.scalar_type());
    TORCH_CHECK(a.scalar_type() == at::kLong && b.scalar_type() == at::kLong && a.dim() == 1 && b.dim() == 1 && a.size(0) == out && b.size(0) == out,
                "convlogic_b200: connection indices must be int64 [out_dim]");
    need_inputs(a, b);
    Tensor y, x_fm, w, coef;
    LogicPlanPtr plan;
    {
        Below below(x);
        w = w_in.contiguous();
        need_input(w);
        x_fm = fm ? x.contiguous() : feature_major_storage(x);
        y = fm ? alloc({out, batch}, x) : alloc_strided({batch, out}, {1, std::max<int64_t>(batch, 1)}, x);
        if (graph && x.requires_grad() && dt == CLB_F32 && out) { // the backward takes both gradients in one pass
            plan = logic_plan_for(start_obj, a, b, start, cons, in, out, clb_logic_path_pays(in, out, batch, 0, 0) || clb_logic_path_pays(in, out, batch, 0, 1));
            if (plan) coef = alloc({out, 4}, x);
        }
        if (!coef.defined() && clb_logic_fwd_scratch_bytes(in, out, batch, dt)) coef = alloc({out, 4}, x); // (then not kept)
        int rc = CLB_ERR_SHAPE;
        if (batch && out && plan && plan->path_fwd(batch)) {
            const Tensor live = alloc({out, 4}, x, at::kInt); // the order is the plan's, the connections are those of this call
            rc = clb_logic_path_fwd_live(ptr<float>(x_fm), ptr<int64_t>(a), ptr<int64_t>(b), ptr(plan->rec), ptr(live), ptr<float>(w), ptr<float>(y),
                                         ptr<float>(coef), in, out, batch, wmode, cur_stream());
            if (rc != CLB_ERR_SHAPE) check(rc);
        }
        if (batch && out && rc == CLB_ERR_SHAPE)
            check(clb_logic_fwd_coef(ptr(x_fm), ptr<int64_t>(a), ptr<int64_t>(b), ptr(w), ptr(y), ptr(coef), in, out, batch, wmode, dt, cur_stream()));
    }
    if (graph) {
        auto node = new_node<LogicNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(x, w_in));
        need_inputs(start, cons);
        TORCH_CHECK(start.scalar_type() == at::kLong && cons.scalar_type() == at::kLong && start.numel() == in + 1 && cons.numel() == 2 * out,
                    "convlogic_b200: consumer lists must be int64 [in_dim + 1] and [2 * out_dim]");
        // the parameter itself is saved (it may carry a gradient sink); its contiguous copy only where it is not contiguous
        node->x = saved(x_fm), node->w = saved(w_in.is_contiguous() ? w_in : w);
        node->a = a, node->b = b, node->start = start, node->cons = cons, node->key = plan ? plan->key : logic_key(a, b, start, cons);
        if (plan) node->coef = saved(coef);
        node->plan = plan, node->in = in, node->out = out, node->batch = batch, node->wmode = wmode, node->fm = fm;
        torch::autograd::set_history(y, node);
    }
    return y;
}

// ------------------------------------------------------------------------------------------------ class sums
// [B, k] -> the [B, F] gradient on feature-major storage
Tensor group_sum_bwd(const Tensor &gout, int64_t f, int k, double tau, const Tensor &scale)
{
    need_input(gout);
    if (scale.defined()) {
        need_input(scale);
        TORCH_CHECK(scale.numel() == 1 && scale.scalar_type() == gout.scalar_type(),
                    "convlogic_b200: `scale` must be a one-element tensor of the gradient's dtype");
    }
    Below below(gout);
    Tensor gy = feature_major_grad(gout.size(0), f, gout);
    check(clb_group_sum_bwd_scaled(ptr(gout), ptr(scale), ptr(gy), f, gout.size(0), k, tau, dtype_code(gout), cur_stream()));
    return gy;
}

// y: [B, F] on feature-major storage
Tensor group_sum_fwd(const Tensor &y, int k, double tau)
{
    TORCH_CHECK_VALUE(k > 0, "the number of classes has to be positive, got ", k);
    TORCH_CHECK(y.is_cuda() && stored_feature_major(y), "convlogic_b200: class sums are taken from a flat layer's output");
    const int64_t f = y.size(1), b = y.size(0);
    const int dt = dtype_code(y);
    Below below(y);
    Tensor out = alloc({b, k}, y);
    const size_t bytes = clb_group_sum_scratch_bytes(f, b, k, dt);
    Tensor scratch = scratch_bytes(bytes, y);
    check(clb_group_sum_fwd(ptr(y), ptr(out), ptr(scratch), bytes, f, b, k, tau, dt, cur_stream()));
    return out;
}

struct GroupSumNode : public Node {
    int64_t f;
    int k;
    double tau;
    std::string name() const override { return "GroupSumFunctionBackward"; }
    variable_list apply(variable_list &&grads) override
    {
        const Tensor gout = upstream(*this, grads);
        Below below(gout);
        return {finished_grad(group_sum_bwd(gout.contiguous(), f, k, tau, Tensor()), *this)};
    }
};

// x [B, F] on feature-major storage -> [B, k]
Tensor group_sum(const Tensor &x, int k, double tau)
{
    if (followed({x})) return in_python("followed_group_sum", x, k, tau).cast<Tensor>();
    Tensor out;
    {
        Below below(x);
        out = group_sum_fwd(x, k, tau);
    }
    if (wants_grad({x})) {
        auto node = new_node<GroupSumNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(x));
        node->f = x.size(1), node->k = k, node->tau = tau;
        torch::autograd::set_history(out, node);
    }
    return out;
}

// (loss [1], dscore [B, k], scores [B, k] or undefined)
// y_fm: a tensor whose storage is [F, B]
std::tuple<Tensor, Tensor, Tensor> group_sum_ce_raw(const Tensor &y_fm, int64_t f, int64_t b, const Tensor &labels, int k, double tau, bool want_scores)
{
    need_input(labels);
    TORCH_CHECK(y_fm.is_cuda() && y_fm.scalar_type() == at::kFloat && labels.scalar_type() == at::kLong && labels.dim() == 1 && labels.size(0) == b,
                "convlogic_b200: group_sum_ce expects float32 [F, B] activations and int64 [B] labels");
    TORCH_CHECK_VALUE(f % k == 0, "in_dim (", f, ") has to be divisible by k (", k, ") but it is not");
    Below below(y_fm);
    Tensor loss = alloc({1}, y_fm), dscore = alloc({b, k}, y_fm), scores;
    if (want_scores) scores = alloc({b, k}, y_fm);
    const size_t bytes = clb_group_sum_scratch_bytes(f, b, k, CLB_F32);
    Tensor scratch = scratch_bytes(bytes, y_fm);
    check(clb_group_sum_ce(ptr<float>(y_fm), ptr<int64_t>(labels), ptr<float>(scores), ptr<float>(dscore), ptr<float>(loss), ptr(scratch), bytes, f, b, k,
                           tau, cur_stream()));
    return {loss, dscore, scores};
}

struct GroupSumCeNode : public Node {
    SavedVariable dscore;
    int64_t f;
    int k;
    double tau;
    std::string name() const override { return "GroupSumCrossEntropyFunctionBackward"; }
    void release_variables() override { dscore.reset_data(); }
    variable_list apply(variable_list &&grads) override
    {
        const Tensor ds = dscore.unpack();
        Below below(ds);
        const Tensor scale = upstream(*this, grads).reshape({1}).to(ds.scalar_type()).contiguous();
        return {finished_grad(group_sum_bwd(ds, f, k, tau, scale), *this)};
    }
};

Tensor group_sum_ce(const Tensor &x, const Tensor &labels, int k, double tau)
{
    TORCH_CHECK_VALUE(k > 0, "the number of classes has to be positive, got ", k);
    if (followed({x})) return in_python("followed_group_sum_ce", x, labels, k, tau).cast<Tensor>();
    Tensor loss, dscore;
    {
        Below below(x);
        std::tie(loss, dscore, std::ignore) = group_sum_ce_raw(x, x.size(1), x.size(0), labels.contiguous(), k, tau, false);
        loss = loss.reshape({});
    }
    if (wants_grad({x})) {
        auto node = new_node<GroupSumCeNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(x));
        node->dscore = saved(dscore), node->f = x.size(1), node->k = k, node->tau = tau;
        torch::autograd::set_history(loss, node);
    }
    return loss;
}

// ------------------------------------------------------------------------------------------------ fused flat layers
struct TreeTables {
    Tensor leaf, node, start, slots;
    bool covers_all; // every neuron of the first two layers sits in some tree: gate-gradient buffers need no clearing
};

// x_fm: a tensor whose storage is [in, B]
void tree_fwd(const Tensor &x_fm, int64_t batch, const TreeTables &t, const Tensor &w0, const Tensor &w1, const Tensor &w2, int wmode, const Tensor &y)
{
    check(clb_logic_tree_fwd(ptr<float>(x_fm), ptr<int32_t>(t.leaf), ptr<int32_t>(t.node), ptr<float>(w0), ptr<float>(w1), ptr<float>(w2), ptr<float>(y),
                             t.leaf.size(0), batch, wmode, cur_stream()));
}

// upstream gradient: gy on the storage [T, B], or the head (dscore [B, k], scale [1]) of GroupSum + cross-entropy
std::array<Tensor, 4> tree_bwd(const Tensor &x_fm, int64_t in, int64_t b, const TreeTables &t, const Tensor &w0, const Tensor &w1, const Tensor &w2, const Tensor &gy,
                               const Tensor &dscore, const Tensor &scale, int k, double tau, int wmode, bool need_gx, std::array<Tensor, 3> gw)
{
    const int64_t trees = t.leaf.size(0);
    Below below(x_fm);
    Tensor tapgrad = alloc({std::max<int64_t>(trees * 8, 1), b}, x_fm);
    const Tensor *ws[3] = {&w0, &w1, &w2};
    for (int i = 0; i < 3; ++i) {
        if (!gw[i].defined()) gw[i] = alloc(ws[i]->sizes(), *ws[i]);
        if (!t.covers_all) gw[i].zero_();
    }
    Tensor gx;
    if (need_gx) gx = feature_major_grad(b, in, x_fm);
    if (gy.defined()) {
        check(clb_logic_tree_bwd(ptr<float>(x_fm), ptr<int32_t>(t.leaf), ptr<int32_t>(t.node), ptr<float>(w0), ptr<float>(w1), ptr<float>(w2),
                                 ptr<float>(gy), ptr<float>(tapgrad), ptr<float>(gw[0]), ptr<float>(gw[1]), ptr<float>(gw[2]), ptr<float>(gx),
                                 ptr<int64_t>(t.start), ptr<int32_t>(t.slots), in, trees, b, wmode, cur_stream()));
    } else {
        check(clb_logic_tree_bwd_scores(ptr<float>(x_fm), ptr<int32_t>(t.leaf), ptr<int32_t>(t.node), ptr<float>(w0), ptr<float>(w1), ptr<float>(w2),
                                        ptr<float>(dscore), ptr<float>(scale), k, tau, ptr<float>(tapgrad), ptr<float>(gw[0]), ptr<float>(gw[1]),
                                        ptr<float>(gw[2]), ptr<float>(gx), ptr<int64_t>(t.start), ptr<int32_t>(t.slots), in, trees, b, wmode, cur_stream()));
    }
    return {gx, gw[0], gw[1], gw[2]};
}

struct TreeNode : public Node {
    SavedVariable x, w0, w1, w2; // x: a tensor on feature-major storage [in, batch]
    TreeTables t;
    int64_t in, batch;
    int wmode;
    SavedVariable dscore; // head: GroupSum + cross-entropy
    int k = 0;
    double tau = 1.0;
    std::string name() const override { return k ? "LogicTreeCrossEntropyFunctionBackward" : "LogicTreeFunctionBackward"; }
    void release_variables() override { x.reset_data(), w0.reset_data(), w1.reset_data(), w2.reset_data(), dscore.reset_data(); }
    variable_list apply(variable_list &&grads) override
    {
        const Tensor xx = x.unpack(), a = w0.unpack(), b = w1.unpack(), c = w2.unpack();
        Below below(xx);
        const Tensor up = upstream(*this, grads);
        Tensor gy, scale;
        if (k)
            scale = up.reshape({1}).to(at::kFloat).contiguous();
        else
            gy = feature_major_storage(up);
        Sinks sinks({a, b, c});
        const bool direct = sinks.any() && wmode != CLB_W_ARGMAX;
        auto out = tree_bwd(xx, in, batch, t, a, b, c, gy, k ? dscore.unpack() : Tensor(), scale, k, tau, wmode, task_should_compute_output(0),
                            direct ? std::array<Tensor, 3>{sinks.slice(0), sinks.slice(1), sinks.slice(2)} : std::array<Tensor, 3>{});
        Tensor gx = out[0].defined() ? finished_grad(out[0], *this) : Tensor();
        if (direct) sinks.ready();
        if (direct || wmode == CLB_W_ARGMAX) return {gx, Tensor(), Tensor(), Tensor()};
        return {gx, out[1], out[2], out[3]};
    }
};

// x [B, in] -> [B, T] (k == 0), or with labels the mean cross-entropy of GroupSum(k, tau) over the trees
Tensor trees(const Tensor &x, const Tensor &w0, const Tensor &w1, const Tensor &w2, const Tensor &leaf, const Tensor &node_t, const Tensor &start,
             const Tensor &slots, int wmode, bool covers_all, const std::optional<Tensor> &labels_in, int k, double tau)
{
    if (followed({x, w0, w1, w2}))
        return in_python("followed_trees", x, w0, w1, w2, leaf, node_t, start, slots, wmode, covers_all, labels_in, k, tau).cast<Tensor>();
    const bool graph = wants_grad({x, w0, w1, w2});
    const TreeTables t{leaf, node_t, start, slots, covers_all};
    TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kFloat, "convlogic_b200: the fused flat layers take float32 [B, in] CUDA tensors");
    need_inputs(leaf, node_t, w0, w1, w2, start, slots);
    const int64_t T = leaf.size(0), B = x.size(0);
    Tensor x_fm, out, dscore;
    {
        Below below(x);
        x_fm = feature_major_storage(x);
        if (!k) {
            out = alloc_strided({B, T}, {1, std::max<int64_t>(B, 1)}, x);
            tree_fwd(x_fm, B, t, w0, w1, w2, wmode, out);
        } else {
            const Tensor labels = labels_in->contiguous();
            need_input(labels);
            TORCH_CHECK(labels.scalar_type() == at::kLong && labels.dim() == 1 && labels.size(0) == B, "convlogic_b200: labels must be int64 [B]");
            const size_t bytes = clb_logic_tree_fwd_ce_scratch_bytes(T, B, k);
            int rc = CLB_ERR_SHAPE;
            if (bytes && B % 4 == 0 && B <= 512 && k <= 32) { // class sums without the activation
                out = alloc({1}, x), dscore = alloc({B, k}, x);
                Tensor scratch = scratch_bytes(bytes, x);
                rc = clb_logic_tree_fwd_ce(ptr<float>(x_fm), ptr<int32_t>(leaf), ptr<int32_t>(node_t), ptr<float>(w0), ptr<float>(w1), ptr<float>(w2),
                                           ptr<int64_t>(labels), ptr<float>(dscore), ptr<float>(out), ptr(scratch), bytes, T, B, k, tau, wmode, cur_stream());
                if (rc != CLB_ERR_SHAPE) check(rc);
            }
            if (rc == CLB_ERR_SHAPE) {
                Tensor y = alloc({T, B}, x);
                tree_fwd(x_fm, B, t, w0, w1, w2, wmode, y);
                std::tie(out, dscore, std::ignore) = group_sum_ce_raw(y, T, B, labels, k, tau, false);
            }
            out = out.reshape({});
        }
    }
    if (graph) {
        auto node = new_node<TreeNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(x, w0, w1, w2));
        node->x = saved(x_fm), node->w0 = saved(w0), node->w1 = saved(w1), node->w2 = saved(w2), node->t = t, node->in = x.size(1), node->batch = B,
        node->wmode = wmode;
        if (k) node->dscore = saved(dscore);
        node->k = k, node->tau = tau;
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ------------------------------------------------------------------------------------------------ optimiser
void adam_step(const Tensor &p, const Tensor &g, const Tensor &m, const Tensor &v, double lr, double beta1, double beta2, double eps, double weight_decay,
               int64_t step, bool decoupled)
{
    need_inputs(p, g, m, v);
    const int64_t n = p.numel();
    for (const Tensor *t : {&p, &g, &m, &v})
        TORCH_CHECK(t->numel() == n && t->scalar_type() == at::kFloat, "convlogic_b200: adam_step expects four float32 buffers of equal size");
    c10::cuda::CUDAGuard device(p.device());
    check(clb_adam_step(ptr<float>(p), ptr<float>(g), ptr<float>(m), ptr<float>(v), n, lr, beta1, beta2, eps, weight_decay, step, decoupled, cur_stream()));
}

// ------------------------------------------------------------------------------------------------ packed inference
at::ScalarType word_type(int bits)
{
    TORCH_CHECK_VALUE(bits == 8 || bits == 16 || bits == 32 || bits == 64, "`bit_count` has to be in { 8, 16, 32, 64 }");
    return bits == 8 ? at::kChar : bits == 16 ? at::kShort : bits == 32 ? at::kInt : at::kLong;
}

std::pair<Tensor, int64_t> pack_bits(const Tensor &t, int bits, bool sample_major)
{
    const at::ScalarType type = word_type(bits);
    need_input(t);
    TORCH_CHECK(t.dim() == 2 && (t.scalar_type() == at::kBool || t.scalar_type() == at::kByte), "convlogic_b200: pack_bits expects a bool or uint8 tensor");
    const int64_t b = t.size(sample_major ? 0 : 1), f = t.size(sample_major ? 1 : 0);
    Below below(t);
    Tensor packed = alloc({f, (b + bits - 1) / bits}, t, type);
    check(sample_major ? clb_pack_bits_nmajor(ptr<uint8_t>(t), ptr(packed), b, f, bits, cur_stream()) : clb_pack_bits(ptr<uint8_t>(t), ptr(packed), f, b, bits, cur_stream()));
    return {packed, (bits - b % bits) % bits};
}

// The order in which large packed layers are walked, laid out once and kept on the tensor object of the connections' first halves as
// `_clb_plan`.  The walk reads the connections themselves, so that an order of others is never wrong, and little slower (64000 neurons, 10000
// samples: 45.1 us in the neurons' own order, 33.9 in this, 37.9 in that of other connections): connections that are written to keep it, and
// captured graphs, which hold its address, with them.
struct PackedOrder {
    int64_t out = 0;
    Tensor order;
    c10::Stream stream{c10::Stream::UNSAFE, c10::Device(c10::kCPU), 0}; // of its memory
};
using PackedOrderPtr = std::shared_ptr<PackedOrder>;

PackedOrderPtr packed_order_for(const py::handle &keep, const Tensor &a, const Tensor &b, int64_t in, int64_t out) // GIL held
{
    const c10::Stream now = c10::cuda::getCurrentCUDAStream().unwrap();
    if (PackedOrderPtr p = kept<PackedOrder>(keep); p && p->out == out && p->order.defined() && p->order.device() == a.device()) {
        if (now != p->stream) p->order.record_stream(now);
        return p;
    }
    // inside a stream capture nothing would be laid out before the replay
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return nullptr;
    auto p = std::make_shared<PackedOrder>();
    p->out = out, p->stream = now;
    p->order = alloc({out}, a, at::kInt);
    const size_t bytes = clb_packed_order_scratch_bytes(in, out);
    const Tensor scratch = scratch_bytes(bytes, a);
    check(clb_packed_order(ptr<int64_t>(a), ptr<int64_t>(b), ptr<int32_t>(p->order), ptr(scratch), bytes, in, out, cur_stream()));
    c10::cuda::getCurrentCUDAStream().synchronize(); // work of other streams may read it next
    keep.attr("_clb_plan") = p;
    return p;
}

// keep: the object of the layer's connections `a`, or None: the neurons in their own order
Tensor packed_logic(const Tensor &x, const Tensor &a, const Tensor &b, const Tensor &ops, const py::object &keep)
{
    need_inputs(x, a, b, ops);
    TORCH_CHECK(ops.scalar_type() == at::kByte, "convlogic_b200: gate ids must be uint8");
    Below below(x);
    Tensor y = alloc({ops.size(0), x.size(1)}, x);
    const int bits = (int)x.element_size() * 8;
    if (!keep.is_none() && a.numel() == ops.size(0) && b.numel() == ops.size(0) && clb_packed_path_pays(x.size(0), ops.size(0), x.size(1), bits)) {
        if (const PackedOrderPtr p = packed_order_for(keep, a, b, x.size(0), ops.size(0))) {
            const int rc = clb_packed_walk(ptr(x), ptr<int64_t>(a), ptr<int64_t>(b), ptr<int32_t>(p->order), ptr<uint8_t>(ops), ptr(y), x.size(0), ops.size(0),
                                           x.size(1), bits, cur_stream());
            if (rc == CLB_OK) return y;
            if (rc != CLB_ERR_SHAPE) check(rc);
        }
    }
    check(clb_packed_logic(ptr(x), ptr<int64_t>(a), ptr<int64_t>(b), ptr<uint8_t>(ops), ptr(y), x.size(0), ops.size(0), x.size(1), (int)x.element_size() * 8,
                           cur_stream()));
    return y;
}

Tensor group_popcount(const Tensor &x, int64_t pad, int k)
{
    TORCH_CHECK_VALUE(k > 0, "the number of classes has to be positive, got ", k);
    need_input(x);
    const int64_t f = x.size(0), words = x.size(1), bits = x.element_size() * 8;
    TORCH_CHECK_VALUE(f % k == 0, "in_dim (", f, ") has to be divisible by k (", k, ") but it is not");
    Below below(x);
    Tensor counts = alloc({words * bits - pad, k}, x, at::kInt);
    check(clb_group_popcount(ptr(x), ptr<int32_t>(counts), f, words, (int)bits, (int)pad, k, cur_stream()));
    return counts;
}

// A compiled network on one device: the handle and the device copy of its parameters.  The workspace of a call comes from
// torch's caching allocator, so calls on several streams or threads do not share one.
class Net {
public:
    Net(const py::bytes &blob, const c10::Device &device)
        : device_(device.has_index() ? device : c10::Device(c10::kCUDA, c10::cuda::current_device()))
    {
        TORCH_CHECK(device.is_cuda(), "convlogic_b200: a compiled network runs on a CUDA device, got ", device.str());
        const std::string_view data(blob);
        size_t need = 0;
        check(clb_net_device_bytes(data.data(), data.size(), &need));
        c10::cuda::CUDAGuard guard(device_);
        params_ = at::empty({(int64_t)(need < 16 ? 16 : need)}, at::TensorOptions().dtype(at::kByte).device(device_));
        clb_net *made = nullptr;
        check(clb_net_create(data.data(), data.size(), ptr(params_), cur_stream(), &made));
        net_.reset(made); // released also when something below throws
        if (const size_t bytes = clb_net_record_bytes(made)) {
            records_ = at::empty({(int64_t)bytes}, params_.options());
            check(clb_net_records(made, ptr(records_), cur_stream()));
        }
        c10::cuda::getCurrentCUDAStream().synchronize(); // the blob is pageable host memory: wait for the copy
        check(clb_net_info(made, &features, &classes, &layers));
    }
    Net(const Net &) = delete;
    // bool / uint8 bits [B, ...] -> counts
    Tensor forward(const Tensor &x_in) const
    {
        TORCH_CHECK(x_in.scalar_type() == at::kBool || x_in.scalar_type() == at::kByte, "convlogic_b200: CompiledLogicNet.forward expects bool inputs");
        const int64_t batch = x_in.size(0), bits = batch ? x_in.numel() / batch : features;
        TORCH_CHECK_VALUE(bits == features, "expected ", features, " input bits per sample, got ", bits);
        return run(0, x_in.device() == device_ ? x_in.contiguous() : x_in.to(device_).contiguous(), std::nullopt, batch);
    }
    // float32 / uint8 pixels [B, C, H, W] and thermometer thresholds -> counts
    Tensor pixels(const Tensor &x_in, const Tensor &thresholds) const
    {
        const Tensor x = x_in.device() == device_ ? x_in.contiguous() : x_in.to(device_).contiguous();
        TORCH_CHECK(x.scalar_type() == at::kFloat || x.scalar_type() == at::kByte, "convlogic_b200: pixels must be float32 or uint8");
        return run(x.scalar_type() == at::kByte ? 2 : 1, x, thresholds.to(device_, at::kFloat).contiguous(), x.size(0));
    }
    Tensor run(int kind, const Tensor &x, const std::optional<Tensor> &thresholds, int64_t batch) const
    {
        need_input(x);
        Below below(params_);
        const size_t bytes = clb_net_workspace_bytes(net_.get(), batch);
        Tensor workspace = scratch_bytes(bytes, params_);
        Tensor counts = alloc({batch, classes}, params_, at::kInt);
        check(clb_net_forward(net_.get(), kind, ptr(x), thresholds ? ptr<float>(*thresholds) : nullptr, thresholds ? (int)thresholds->numel() : 0, batch,
                              ptr<int32_t>(counts), ptr(workspace), bytes, cur_stream()));
        return counts;
    }
    int64_t features = 0;
    int classes = 0, layers = 0;

private:
    c10::Device device_;
    Tensor params_, records_;
    struct Destroy {
        void operator()(clb_net *n) const { clb_net_destroy(n); }
    };
    std::unique_ptr<clb_net, Destroy> net_;
};

// raw forward / backward of the fused block for callers that handle autograd themselves
py::tuple block_fwd_py(const Tensor &x, const Tensor &w, py::object sel_obj, const std::array<int, 6> &geom, int wmode, bool want_amax, bool want_inter,
                       bool want_idx, bool y_fm)
{
    const Tensor sel = sel_obj.cast<Tensor>();
    const Geom g{geom[0], geom[1], geom[2], geom[3], geom[4], geom[5]};
    BlockOut o = block_fwd(x, w, sel, g, [&] { return plan_for(sel_obj, sel, g, x.size(1)); }, wmode, want_amax, want_inter, want_idx, y_fm);
    auto opt = [](const Tensor &t) { return t.defined() ? py::cast(t) : py::object(py::none()); };
    return py::make_tuple(o.y, opt(o.amax), opt(o.x2), opt(o.x3), opt(o.idx));
}
py::tuple block_bwd_py(const Tensor &gy, const Tensor &x, const Tensor &w, py::object sel_obj, const std::optional<Tensor> &amax,
                       const std::array<int, 6> &geom, int wmode, bool need_gx, bool need_gw, const std::optional<Tensor> &gw_out)
{
    const Tensor sel = sel_obj.cast<Tensor>();
    const Geom g{geom[0], geom[1], geom[2], geom[3], geom[4], geom[5]};
    auto out = block_bwd(gy, x, w, sel, amax.value_or(Tensor()), g, [&] { return plan_for(sel_obj, sel, g, x.size(1)); }, wmode, need_gx, need_gw,
                         gw_out.value_or(Tensor()));
    auto opt = [](const Tensor &t) { return t.defined() ? py::cast(t) : py::object(py::none()); };
    return py::make_tuple(opt(out.first), opt(out.second));
}

Tensor logic_fwd_py(const Tensor &x, const Tensor &a, const Tensor &b, const Tensor &w, int wmode)
{
    Below below(x);
    Tensor y = alloc({w.size(0), x.size(1)}, x);
    logic_fwd(x, a, b, w, wmode, y);
    return y;
}

} // namespace

PYBIND11_MODULE(_clb_torch, m)
{
    copies_as_nothing(py::class_<BlockPlan, PlanPtr>(m, "BlockPlan").def(py::init<>()));
    copies_as_nothing(py::class_<LogicPlan, LogicPlanPtr>(m, "LogicPlan").def(py::init<>()));
    copies_as_nothing(py::class_<PackedOrder, PackedOrderPtr>(m, "PackedOrder").def(py::init<>()));
    m.def("block", &block);
    m.def("block_fwd", &block_fwd_py);
    m.def("block_bwd", &block_bwd_py);
    m.def("is_feature_major", &is_feature_major);
    m.def("logic", &logic);
    m.def("logic_fwd", &logic_fwd_py);
    m.def("logic_bwd_w", [](const Tensor &x, const Tensor &a, const Tensor &b, const Tensor &w, const Tensor &gy, int wmode, const std::optional<Tensor> &out) {
        return logic_bwd_w(x, a, b, w, gy, wmode, out.value_or(Tensor()));
    });
    m.def("logic_bwd_x", &logic_bwd_x);
    m.def("group_sum", &group_sum);
    m.def("group_sum_ce", &group_sum_ce);
    m.def("trees", &trees);
    m.def("transpose2d", &transpose2d);
    m.def("adam_step", &adam_step);
    m.def("count_sinks", [](int64_t change) { g_sinks += change; });
    m.def("pack_bits", &pack_bits);
    m.def("packed_logic", &packed_logic, py::arg("x"), py::arg("a"), py::arg("b"), py::arg("ops"), py::arg("keep") = py::none());
    m.def("group_popcount", &group_popcount);
    py::class_<Net>(m, "Net")
        .def(py::init([](const py::bytes &blob, const std::string &device) { return std::make_unique<Net>(blob, c10::Device(device)); }))
        .def("run", &Net::run)
        .def("forward", &Net::forward)
        .def("pixels", &Net::pixels)
        .def_readonly("features", &Net::features)
        .def_readonly("classes", &Net::classes)
        .def_readonly("layers", &Net::layers);
}

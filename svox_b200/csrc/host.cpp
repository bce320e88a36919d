// Host side of the hot calls: reads the spec objects, allocates the results and calls the C-ABI
// library, and the autograd nodes of the training step and of the point query.
//
// A small call is bound by the host: packing the specs into ctypes structures, entering a device
// guard, looking up the stream and going through a Python autograd function took 47 us for a
// query of 1000 points and 370 us for a training step of 4096 rays whose kernels need 5 and 65.
// The nodes' backward runs on autograd's thread without taking the interpreter lock.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <array>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/svox_b200.h"

namespace {

using at::Tensor;
using std::optional;

// The library's functions, from the file that the Python side has loaded.
struct Library {
#define SVOXB_FUNCTIONS(X)                                                                      \
    X(query_vertical) X(query_vertical_backward) X(query_scatter) X(volume_render) X(volume_render_image)        \
    X(volume_render_prepared) X(volume_render_image_prepared) X(volume_render_backward)         \
    X(volume_render_image_backward) X(volume_render_logged) X(volume_render_image_logged)       \
    X(volume_render_backward_replay) X(volume_render_image_backward_replay)                     \
    X(se_grad_replay) X(se_grad_image_replay) X(item_log_words) X(item_log_watch)               \
    X(item_log_used)                                                                            \
    X(volume_render_logged_clear) X(volume_render_image_logged_clear) X(log_is_sorted)          \
    X(strerror) X(last_cuda_error)
#define SVOXB_MEMBER(name) decltype(&svoxb_##name) name = nullptr;
    SVOXB_FUNCTIONS(SVOXB_MEMBER)
} lib;

void load(const std::string& path) {
    void* handle = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (!handle) throw std::runtime_error(std::string("svox_b200: ") + dlerror());
#define SVOXB_LOOKUP(name)                                                                      \
    lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(handle, "svoxb_" #name));             \
    if (!lib.name) throw std::runtime_error("svox_b200: the library lacks svoxb_" #name);
    SVOXB_FUNCTIONS(SVOXB_LOOKUP)
}

[[noreturn]] void fail(const std::string& text) { throw std::runtime_error(text); }

void check(int status, const char* what) {
    if (status == SVOXB_OK) return;
    std::string text = std::string("svox_b200.") + what + ": " + lib.strerror(status);
    const char* cuda = lib.last_cuda_error();
    if (cuda && *cuda) text += std::string(" (") + cuda + ")";
    fail(text);
}

// ---------------------------------------------------------------------------
// Spec objects -> C structures.  The checks and their words are those of the reference's
// CHECK_INPUT (svox/csrc/include/data_spec.hpp:37-42) plus the dtype.

void check_input(const Tensor& t, const char* name, at::ScalarType dtype = at::kFloat) {
    if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor");
    if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
    if (t.scalar_type() != dtype)
        fail(std::string(name) + " must be " + (dtype == at::kInt ? "torch.int32" : "torch.float32") +
             " (this build computes in float32 only)");
}

Tensor tensor_of(py::handle obj, const char* name) {
    if (!THPVariable_Check(obj.ptr())) fail(std::string(name) + " must be a tensor");
    return THPVariable_Unpack(obj.ptr());
}

// One attribute; the names are interned once.
struct Name {
    PyObject* key;
    explicit Name(const char* s) : key(PyUnicode_InternFromString(s)) {}
    py::object of(py::handle obj) const {
        PyObject* v = PyObject_GetAttr(obj.ptr(), key);
        if (!v) throw py::error_already_set();
        return py::reinterpret_steal<py::object>(v);
    }
    double number(py::handle obj) const {
        const double v = PyFloat_AsDouble(of(obj).ptr());
        if (v == -1.0 && PyErr_Occurred()) throw py::error_already_set();
        return v;
    }
    long whole(py::handle obj) const { return (long)number(obj); }
};
#define SVOXB_NAME(id) static const Name id(#id);

// A tree as a call sees it: the spec's tensors, and the pointers and sizes read from them.  A tensor
// can be given another storage while a node waits for its backward (`data.data = x`, `tree.to()`),
// which pins neither the old one nor counts as a version: `bind` is repeated there.
struct Tree {
    Tensor data, child, offset, scaling, weight, extra;
    bool weight_max = false;
    svoxb_tree c{};

    void bind();
    // Whether the records still lie where `other` was bound to them.
    bool same_records(const svoxb_tree& other) const {
        return c.data == other.data && c.M == other.M && c.N == other.N && c.K == other.K;
    }
};

void Tree::bind() {
    check_input(data, "data");
    check_input(offset, "offset");
    check_input(scaling, "scaling");
    check_input(child, "child", at::kInt);
    if (data.dim() != 5 || child.dim() != 4 || child.sizes() != data.sizes().slice(0, 4))
        fail("data must be (M,N,N,N,K) and child (M,N,N,N)");
    const auto dev = data.device();
    if (child.device() != dev) fail("child must be on the same device as data");
    if (offset.device() != dev) fail("offset must be on the same device as data");
    if (scaling.device() != dev) fail("scaling must be on the same device as data");
    c = svoxb_tree{};
    if (weight.defined() && weight.numel()) {
        check_input(weight, "_weight_accum");
        if (weight.sizes() != child.sizes() || weight.device() != dev)
            fail("_weight_accum must have the shape and device of child");
        c.weight_accum = weight.data_ptr<float>();
    }
    c.weight_accum_max = weight_max;
    if (extra.defined() && extra.numel()) {
        check_input(extra, "extra_data");
        if (extra.dim() != 2 || extra.device() != dev)
            fail("extra_data must be (basis_dim, C) on the device of data");
        c.extra_data = extra.data_ptr<float>();
        c.extra_rows = (int32_t)extra.size(0);
        c.extra_cols = (int32_t)extra.size(1);
    }
    c.data = data.data_ptr<float>();
    c.child = child.data_ptr<int32_t>();
    c.offset = offset.data_ptr<float>();
    c.scaling = scaling.data_ptr<float>();
    c.M = data.size(0);
    c.N = (int32_t)data.size(1);
    c.K = (int32_t)data.size(4);
}

Tree read_tree(py::handle spec) {
    SVOXB_NAME(data) SVOXB_NAME(child) SVOXB_NAME(offset) SVOXB_NAME(scaling)
    SVOXB_NAME(extra_data) SVOXB_NAME(_weight_accum) SVOXB_NAME(_weight_accum_max)
    Tree t;
    t.data = tensor_of(data.of(spec), "data");
    t.child = tensor_of(child.of(spec), "child");
    t.offset = tensor_of(offset.of(spec), "offset");
    t.scaling = tensor_of(scaling.of(spec), "scaling");
    py::object w = _weight_accum.of(spec), e = extra_data.of(spec);
    if (!w.is_none()) {
        t.weight = tensor_of(w, "_weight_accum");
        t.weight_max = PyObject_IsTrue(_weight_accum_max.of(spec).ptr()) == 1;
    }
    if (!e.is_none()) t.extra = tensor_of(e, "extra_data");
    t.bind();
    return t;
}

svoxb_render_options read_options(py::handle opt) {
    SVOXB_NAME(step_size) SVOXB_NAME(background_brightness) SVOXB_NAME(format)
    SVOXB_NAME(basis_dim) SVOXB_NAME(ndc_width) SVOXB_NAME(ndc_height) SVOXB_NAME(ndc_focal)
    SVOXB_NAME(min_comp) SVOXB_NAME(max_comp) SVOXB_NAME(sigma_thresh) SVOXB_NAME(stop_thresh)
    SVOXB_NAME(density_softplus) SVOXB_NAME(rgb_padding)
    svoxb_render_options o;
    o.step_size = (float)step_size.number(opt);
    o.background_brightness = (float)background_brightness.number(opt);
    o.format = (int32_t)format.whole(opt);
    o.basis_dim = (int32_t)basis_dim.whole(opt);
    o.ndc_width = (int32_t)ndc_width.whole(opt);
    o.ndc_height = (int32_t)ndc_height.whole(opt);
    o.ndc_focal = (float)ndc_focal.number(opt);
    o.min_comp = (int32_t)min_comp.whole(opt);
    o.max_comp = (int32_t)max_comp.whole(opt);
    o.sigma_thresh = (float)sigma_thresh.number(opt);
    o.stop_thresh = (float)stop_thresh.number(opt);
    o.density_softplus = PyObject_IsTrue(density_softplus.of(opt).ptr()) == 1;
    o.rgb_padding = (float)rgb_padding.number(opt);
    return o;
}

// Rays or the pixels of a camera.
struct Source {
    bool image = false;
    Tensor origins, dirs, vdirs, c2w;
    svoxb_rays rays{};
    svoxb_camera cam{};

    void bind(const Tree& tree);      // repeated for a backward, as Tree::bind
    int64_t count() const { return image ? (int64_t)cam.width * cam.height : rays.Q; }
    std::vector<int64_t> shape(int64_t channels) const {
        if (image) return {cam.height, cam.width, channels};
        return {rays.Q, channels};
    }
};

void Source::bind(const Tree& tree) {
    const auto dev = tree.data.device();
    if (image) {
        check_input(c2w, "c2w");
        if (c2w.dim() != 2 || c2w.size(1) != 4 || (c2w.size(0) != 3 && c2w.size(0) != 4))
            fail("c2w must be (3, 4) or (4, 4)");
        if (c2w.device() != dev) fail("c2w must be on the same device as the tree");
        cam.c2w = c2w.data_ptr<float>();
        return;
    }
    const std::array<std::pair<const Tensor*, const char*>, 3> all{
        {{&origins, "origins"}, {&dirs, "dirs"}, {&vdirs, "vdirs"}}};
    for (const auto& [t, name] : all) {
        check_input(*t, name);
        if (t->dim() != 2 || t->size(1) != 3) fail(std::string(name) + " must be (Q, 3)");
        if (t->device() != dev) fail(std::string(name) + " must be on the same device as the tree");
    }
    rays.Q = origins.size(0);
    if (dirs.size(0) != rays.Q || vdirs.size(0) != rays.Q)
        fail("origins, dirs and vdirs must have the same length");
    rays.origins = origins.data_ptr<float>();
    rays.dirs = dirs.data_ptr<float>();
    rays.vdirs = vdirs.data_ptr<float>();
}

Source read_source(py::handle spec, bool image, const Tree& tree) {
    SVOXB_NAME(origins) SVOXB_NAME(dirs) SVOXB_NAME(vdirs) SVOXB_NAME(c2w) SVOXB_NAME(fx)
    SVOXB_NAME(fy) SVOXB_NAME(width) SVOXB_NAME(height)
    Source s;
    s.image = image;
    if (image) {
        s.c2w = tensor_of(c2w.of(spec), "c2w");
        s.cam.fx = (float)fx.number(spec);
        s.cam.fy = (float)fy.number(spec);
        s.cam.width = (int32_t)width.whole(spec);
        s.cam.height = (int32_t)height.whole(spec);
    } else {
        s.origins = tensor_of(origins.of(spec), "origins");
        s.dirs = tensor_of(dirs.of(spec), "dirs");
        s.vdirs = tensor_of(vdirs.of(spec), "vdirs");
    }
    s.bind(tree);
    return s;
}

void check_points(const Tensor& indices) {
    check_input(indices, "indices");
    if (indices.dim() != 2 || indices.size(1) != 3) fail("indices must be (Q, 3)");
}

int64_t out_dim(const svoxb_tree& t, const svoxb_render_options& o) {
    // get_out_data_dim, svox/csrc/rt_kernel.cu:1009-1015
    if (o.format == SVOXB_FORMAT_RGBA) return t.K - 1;
    return o.basis_dim > 0 ? (t.K - 1) / o.basis_dim : 0;
}

void* stream_of(const Tensor& t) {
    return at::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

bool capturing() {      // on the current stream of the current device
    return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
}

// ---------------------------------------------------------------------------
// How large the item log has to be, learnt without making the host wait: after a logged forward
// the counts at the head of its log are copied to a slot of pinned memory that holds -1 until
// they arrive.
class LogWatch {
  public:
    struct Seen { int64_t used, batches, rays, capacity; };

    void watch(const Tensor& log, int64_t capacity, int64_t rays) {
        // a forward that is captured would write to its slot at every replay, also when the slot
        // has long been another forward's
        if (capturing()) return;
        std::lock_guard<std::mutex> lock(mutex_);
        if (!slots_.defined())
            slots_ = torch::full({kSlots, 2}, -1, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
        for (int i = 0; i < kSlots; ++i) {
            if (pending_[i].capacity >= 0) continue;
            volatile int32_t* to = slots_.data_ptr<int32_t>() + 2 * i;
            to[0] = to[1] = -1;
            check(lib.item_log_watch(log.data_ptr<int32_t>(), const_cast<int32_t*>(to),
                                     stream_of(log)), "item_log_watch");
            pending_[i] = Seen{0, 0, rays, capacity};
            return;
        }
        // every slot is under way: this forward is not watched
    }
    std::vector<Seen> poll() {
        std::lock_guard<std::mutex> lock(mutex_);
        std::vector<Seen> seen;
        if (!slots_.defined()) return seen;
        volatile int32_t* all = slots_.data_ptr<int32_t>();
        for (int i = 0; i < kSlots; ++i) {
            if (pending_[i].capacity < 0 || all[2 * i] < 0 || all[2 * i + 1] < 0) continue;
            pending_[i].used = all[2 * i];
            pending_[i].batches = all[2 * i + 1];
            seen.push_back(pending_[i]);
            pending_[i].capacity = -1;
        }
        return seen;
    }
    bool waiting() {
        std::lock_guard<std::mutex> lock(mutex_);
        for (const Seen& s : pending_)
            if (s.capacity >= 0) return true;
        return false;
    }

  private:
    static constexpr int kSlots = 16;
    std::mutex mutex_;
    Tensor slots_;
    std::vector<Seen> pending_ = std::vector<Seen>(kSlots, Seen{0, 0, 0, -1});
};
LogWatch& log_watch() {
    static LogWatch* w = new LogWatch;      // outlives the interpreter's tear-down
    return *w;
}

// ---------------------------------------------------------------------------
// Calls

std::pair<Tensor, Tensor> run_query(const Tree& t, const Tensor& indices) {
    const c10::cuda::CUDAGuard guard(indices.device());
    const int64_t Q = indices.size(0);
    Tensor values = at::empty({Q, t.c.K}, indices.options());
    Tensor ids = at::empty({Q}, indices.options().dtype(at::kLong));
    check(lib.query_vertical(&t.c, indices.data_ptr<float>(), Q, values.data_ptr<float>(),
                             ids.data_ptr<int64_t>(), stream_of(indices)), "query_vertical");
    return {values, ids};
}

Tensor run_query_backward(const Tree& t, const Tensor& indices, const Tensor& grad_out,
                          const optional<Tensor>& zeroed) {
    check_input(grad_out, "grad_output");
    const int64_t Q = indices.size(0);
    if (grad_out.dim() != 2 || grad_out.size(0) != Q) fail("grad_output must be (Q, K)");
    const int64_t Kg = grad_out.size(1);
    const c10::cuda::CUDAGuard guard(indices.device());
    const std::vector<int64_t> shape{t.c.M, t.c.N, t.c.N, t.c.N, Kg};
    if (zeroed) {
        check_input(*zeroed, "zeroed");
        if (zeroed->sizes() != at::IntArrayRef(shape)) fail("zeroed must be (M, N, N, N, Kg)");
    }
    Tensor grad = zeroed ? *zeroed : at::empty(shape, grad_out.options());
    check(lib.query_vertical_backward(&t.c, indices.data_ptr<float>(), Q,
                                      grad_out.data_ptr<float>(), (int32_t)Kg,
                                      grad.data_ptr<float>(), zeroed ? 0 : 1, stream_of(indices)),
          "query_vertical_backward");
    return grad;
}

Tensor run_render(const Tree& t, const Source& s, const svoxb_render_options& o,
                  const optional<Tensor>& prepared) {
    const c10::cuda::CUDAGuard guard(t.data.device());
    Tensor out = at::empty(s.shape(out_dim(t.c, o)), t.data.options());
    float* to = out.data_ptr<float>();
    void* stream = stream_of(t.data);
    int st;
    if (prepared) {
        const int32_t* index = prepared->data_ptr<int32_t>();
        st = s.image ? lib.volume_render_image_prepared(&t.c, &s.cam, &o, index, to, stream)
                     : lib.volume_render_prepared(&t.c, &s.rays, &o, index, to, stream);
    } else {
        st = s.image ? lib.volume_render_image(&t.c, &s.cam, &o, to, stream)
                     : lib.volume_render(&t.c, &s.rays, &o, to, stream);
    }
    check(st, s.image ? "volume_render_image" : "volume_render");
    return out;
}

// Gradients that the backward does not clear on its way are cleared on a side stream beside the
// forward's march, which leaves memory bandwidth unused -- unless they are so small that the two
// events cost more than the fill.
constexpr int64_t kFillBeside = 16 << 20;   // bytes; 16 MB are cleared in about 4 us

struct Zeroed {
    std::vector<Tensor> buffers;
    at::cuda::CUDAEvent done;
    c10::cuda::CUDAStream side;

    Zeroed(const Tensor& like, int count) : side(side_stream(like.device().index())) {
        for (int i = 0; i < count; ++i) buffers.push_back(at::empty(like.sizes(), like.options()));
    }
    float* pointer(size_t i) { return i < buffers.size() ? buffers[i].data_ptr<float>() : nullptr; }
    Zeroed(const Zeroed&) = delete;
    // A buffer dropped before anyone waited for its fill: its memory must not be handed out again
    // while the side stream still writes to it.
    ~Zeroed() {
        for (const Tensor& b : buffers)
            if (b.defined())
                c10::cuda::CUDACachingAllocator::recordStream(b.storage().data_ptr(), side);
    }
    void enqueued() { done.record(side); }      // after the call that enqueued the fills
    Tensor claim(size_t i) {
        done.block(at::cuda::getCurrentCUDAStream(buffers[i].device().index()));
        return std::move(buffers[i]);
    }
    static c10::cuda::CUDAStream side_stream(c10::DeviceIndex dev) {
        static std::mutex mutex;
        static std::vector<optional<c10::cuda::CUDAStream>> streams(64);
        std::lock_guard<std::mutex> lock(mutex);
        auto& s = streams.at((size_t)dev);
        if (!s) s = c10::cuda::getStreamFromPool(false, dev);
        return *s;
    }
};

std::pair<Tensor, Tensor> run_logged(const Tree& t, const Source& s, const svoxb_render_options& o,
                                     int64_t capacity, Zeroed* zeroed = nullptr,
                                     bool watch = true) {
    const c10::cuda::CUDAGuard guard(t.data.device());
    Tensor out = at::empty(s.shape(3), t.data.options());
    Tensor log = at::empty({lib.item_log_words(capacity)}, t.child.options());
    float* to = out.data_ptr<float>();
    int32_t* words = log.data_ptr<int32_t>();
    void* stream = stream_of(t.data);
    int st;
    if (zeroed) {
        float *c0 = zeroed->pointer(0), *c1 = zeroed->pointer(1);
        void* side = zeroed->side.stream();
        st = s.image ? lib.volume_render_image_logged_clear(&t.c, &s.cam, &o, to, words, capacity,
                                                            stream, c0, c1, side)
                     : lib.volume_render_logged_clear(&t.c, &s.rays, &o, to, words, capacity,
                                                      stream, c0, c1, side);
        zeroed->enqueued();
    } else {
        st = s.image ? lib.volume_render_image_logged(&t.c, &s.cam, &o, to, words, capacity, stream)
                     : lib.volume_render_logged(&t.c, &s.rays, &o, to, words, capacity, stream);
    }
    check(st, "volume_render_logged");
    if (watch) log_watch().watch(log, capacity, s.count());
    return {out, log};
}

// Gradient by replay of the log, into `zeroed` or a tensor that the call clears.
Tensor run_replay(const Tree& t, const Source& s, const svoxb_render_options& o,
                  const Tensor& grad_out, const Tensor& fwd, const Tensor& log, int64_t capacity,
                  int64_t used, const optional<Tensor>& zeroed) {
    check_input(grad_out, "grad_output");
    check_input(fwd, "fwd_out");
    check_input(log, "log", at::kInt);
    if (grad_out.numel() != 3 * s.count() || fwd.numel() != 3 * s.count())
        fail("grad_output and fwd_out must have the shape of the render");
    if (log.numel() < lib.item_log_words(capacity)) fail("the item log is smaller than its capacity");
    if (used > capacity) fail("the item log overflowed: it cannot be replayed");
    if (zeroed) {
        check_input(*zeroed, "zeroed");
        if (zeroed->numel() != t.data.numel()) fail("zeroed must be like data");
    }
    const c10::cuda::CUDAGuard guard(t.data.device());
    Tensor grad = zeroed ? *zeroed : at::empty(t.data.sizes(), t.data.options());
    const float *g = grad_out.data_ptr<float>(), *f = fwd.data_ptr<float>();
    int32_t* words = log.data_ptr<int32_t>();
    float* to = grad.data_ptr<float>();
    void* stream = stream_of(t.data);
    check(s.image ? lib.volume_render_image_backward_replay(&t.c, &s.cam, &o, g, f, words, capacity,
                                                            used, to, zeroed ? 0 : 1, stream)
                  : lib.volume_render_backward_replay(&t.c, &s.rays, &o, g, f, words, capacity,
                                                      used, to, zeroed ? 0 : 1, stream),
          "volume_render_backward_replay");
    return grad;
}

Tensor run_backward(const Tree& t, const Source& s, const svoxb_render_options& o,
                    const Tensor& grad_out, const optional<Tensor>& fwd) {
    check_input(grad_out, "grad_output");
    const std::vector<int64_t> shape = s.shape(out_dim(t.c, o));
    if (grad_out.sizes() != at::IntArrayRef(shape)) fail("grad_output must have the render's shape");
    const float* f = nullptr;
    if (fwd) {
        check_input(*fwd, "fwd_out");
        if (fwd->sizes() != at::IntArrayRef(shape))
            fail("fwd_out must have the shape of the forward output");
        f = fwd->data_ptr<float>();
    }
    const c10::cuda::CUDAGuard guard(t.data.device());
    Tensor grad = at::empty(t.data.sizes(), t.data.options());
    const float* g = grad_out.data_ptr<float>();
    float* to = grad.data_ptr<float>();
    void* stream = stream_of(t.data);
    check(s.image ? lib.volume_render_image_backward(&t.c, &s.cam, &o, g, f, to, 1, stream)
                  : lib.volume_render_backward(&t.c, &s.rays, &o, g, f, to, 1, stream),
          s.image ? "volume_render_image_backward" : "volume_render_backward");
    return grad;
}

bool fills_beside(const Tree& t, const Source& s, int64_t capacity) {
    return s.count() > 0 && t.data.numel() * 4 >= kFillBeside &&
           !lib.log_is_sorted(&t.c, s.count(), s.image, capacity);
}

// ---------------------------------------------------------------------------
// Autograd nodes

template <class T>
struct Holder : torch::CustomClassHolder {
    T value;
    explicit Holder(T v) : value(std::move(v)) {}
};
template <class T>
void keep(torch::autograd::AutogradContext* ctx, T value) {
    ctx->saved_data["call"] = c10::IValue::make_capsule(c10::make_intrusive<Holder<T>>(std::move(value)));
}
template <class T>
T& kept(torch::autograd::AutogradContext* ctx) {
    return static_cast<Holder<T>*>(ctx->saved_data["call"].toCapsule().get())->value;
}

// What the backward of a render needs (svox/renderer.py:57-89).
struct RenderCall {
    Tree tree;
    Source source;
    svoxb_render_options options;
    int64_t capacity = 0;      // of the item log; 0: none is written
    Tensor epoch;              // the owning tree's count of edits that go through data.data
    int64_t epoch_then = 0;
    uint32_t version_then = 0;
    bool keeps_out = false;
    std::shared_ptr<Zeroed> zeroed;

    int64_t epoch_now() const { return epoch.defined() ? epoch.data_ptr<int64_t>()[0] : -1; }
};

class RenderNode : public torch::autograd::Function<RenderNode> {
  public:
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& data,
                          std::shared_ptr<RenderCall> call) {
        RenderCall& c = *call;
        c.version_then = data._version();
        c.epoch_then = c.epoch_now();
        // The backward differentiates the render without thresholds (svox/csrc/rt_kernel.cu:377,
        // 441); the forward's output equals that render only when both are off.  Its dot product
        // with the upstream gradient then replaces the reference's first march.
        c.keeps_out = c.options.sigma_thresh == 0.f && c.options.stop_thresh == 0.f;
        Tensor out, log;
        if (c.capacity > 0) {
            if (fills_beside(c.tree, c.source, c.capacity))
                c.zeroed = std::make_shared<Zeroed>(c.tree.data, 1);
            std::tie(out, log) =
                run_logged(c.tree, c.source, c.options, c.capacity, c.zeroed.get());
        } else {
            out = run_render(c.tree, c.source, c.options, {});
        }
        // saved, so that an in-place edit of the returned render raises in the backward
        if (c.keeps_out) ctx->save_for_backward({out, log});
        keep(ctx, std::move(call));
        return out;
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                   torch::autograd::variable_list grads) {
        if (!ctx->needs_input_grad(0)) return {Tensor(), Tensor()};
        RenderCall& c = *kept<std::shared_ptr<RenderCall>>(ctx);
        const Tensor grad_out = grads[0].contiguous();
        const svoxb_tree then = c.tree.c;
        c.tree.bind();
        c.source.bind(c.tree);
        optional<Tensor> fwd;
        if (c.keeps_out) {
            const auto saved = ctx->get_saved_variables();
            if (c.tree.data._version() == c.version_then && c.epoch_now() == c.epoch_then &&
                c.tree.same_records(then)) {
                // (a log of another size: a saved-tensor hook ran the forward again, and it was
                // given another log by then)
                if (saved[1].defined() && saved[1].numel() == lib.item_log_words(c.capacity)) {
                    optional<Tensor> zeroed;
                    if (auto z = std::move(c.zeroed)) zeroed = z->claim(0);
                    return {run_replay(c.tree, c.source, c.options, grad_out, saved[0], saved[1],
                                       c.capacity, 0, zeroed),
                            Tensor()};
                }
                fwd = saved[0];
            }
        }
        // `data` was edited since the forward, or thresholds are on: everything is recomputed
        // from the current `data`, as the reference does
        c.zeroed.reset();
        return {run_backward(c.tree, c.source, c.options, grad_out, fwd), Tensor()};
    }
};

struct QueryCall {
    Tree tree;
    Tensor ids;                // the leaves found, for as long as nobody writes to them or to
    uint32_t ids_version = 0, child_version = 0;   // the tree's structure, or replaces that
};

class QueryNode : public torch::autograd::Function<QueryNode> {
  public:
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx,
                                                  const Tensor& data, const Tensor& indices,
                                                  std::shared_ptr<QueryCall> call) {
        auto [values, ids] = run_query(call->tree, indices);
        ctx->mark_non_differentiable({ids});
        ctx->save_for_backward({indices});
        call->ids = ids;
        call->ids_version = ids._version();
        call->child_version = call->tree.child._version();
        keep(ctx, std::move(call));
        return {values, ids};
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                   torch::autograd::variable_list grads) {
        if (!ctx->needs_input_grad(0)) return {Tensor(), Tensor(), Tensor()};
        QueryCall& c = *kept<std::shared_ptr<QueryCall>>(ctx);
        const Tensor indices = ctx->get_saved_variables()[0], grad_out = grads[0].contiguous();
        const svoxb_tree then = c.tree.c;
        c.tree.bind();
        if (c.ids._version() != c.ids_version || c.tree.child._version() != c.child_version ||
            c.tree.c.child != then.child || c.tree.c.M != then.M)
            return {run_query_backward(c.tree, indices, grad_out, {}), Tensor(), Tensor()};
        const c10::cuda::CUDAGuard guard(indices.device());
        const int64_t Kg = grad_out.size(1);
        Tensor grad = at::empty({then.M, then.N, then.N, then.N, Kg}, grad_out.options());
        check(lib.query_scatter(&c.tree.c, c.ids.data_ptr<int64_t>(), c.ids.numel(),
                                grad_out.data_ptr<float>(), (int32_t)Kg, grad.data_ptr<float>(), 1,
                                stream_of(indices)),
              "query_scatter");
        return {grad, Tensor(), Tensor()};
    }
};

// ---------------------------------------------------------------------------
// The functions Python sees: arguments are read with the interpreter lock held, the calls run
// without it.

template <class F>
auto unlocked(F f) {
    py::gil_scoped_release release;
    return f();
}

PYBIND11_MODULE(_host, m) {
    m.def("load", &load);

    m.def("query_vertical", [](py::handle tree, const Tensor& indices) {
        const Tree t = read_tree(tree);
        check_points(indices);
        return unlocked([&] { return run_query(t, indices); });
    });
    m.def("query_vertical_backward", [](py::handle tree, const Tensor& indices,
                                        const Tensor& grad_out, const optional<Tensor>& zeroed) {
        const Tree t = read_tree(tree);
        check_points(indices);
        return unlocked([&] { return run_query_backward(t, indices, grad_out, zeroed); });
    });
    m.def("query_node", [](const Tensor& data, py::handle tree, const Tensor& indices) {
        auto call = std::make_shared<QueryCall>(QueryCall{read_tree(tree)});
        check_points(indices);
        return unlocked([&] {
            auto out = QueryNode::apply(data, indices, call);
            return std::make_pair(out[0], out[1]);
        });
    });

    m.def("volume_render", [](py::handle tree, py::handle source, py::handle opt, bool image,
                              const optional<Tensor>& prepared) {
        const Tree t = read_tree(tree);
        const Source s = read_source(source, image, t);
        const svoxb_render_options o = read_options(opt);
        return unlocked([&] { return run_render(t, s, o, prepared); });
    });
    m.def("volume_render_logged", [](py::handle tree, py::handle source, py::handle opt, bool image,
                                     int64_t capacity) {
        const Tree t = read_tree(tree);
        const Source s = read_source(source, image, t);
        const svoxb_render_options o = read_options(opt);
        return unlocked([&] { return run_logged(t, s, o, capacity); });
    });
    m.def("volume_render_backward_replay",
          [](py::handle tree, py::handle source, py::handle opt, bool image, const Tensor& grad_out,
             const Tensor& fwd, const Tensor& log, int64_t capacity, int64_t used,
             const optional<Tensor>& zeroed) {
              const Tree t = read_tree(tree);
              const Source s = read_source(source, image, t);
              const svoxb_render_options o = read_options(opt);
              return unlocked(
                  [&] { return run_replay(t, s, o, grad_out, fwd, log, capacity, used, zeroed); });
          });
    m.def("volume_render_backward",
          [](py::handle tree, py::handle source, py::handle opt, bool image, const Tensor& grad_out,
             const optional<Tensor>& fwd) {
              const Tree t = read_tree(tree);
              const Source s = read_source(source, image, t);
              const svoxb_render_options o = read_options(opt);
              return unlocked([&] { return run_backward(t, s, o, grad_out, fwd); });
          });
    m.def("render_node", [](const Tensor& data, py::handle tree, py::handle source, py::handle opt,
                            bool image, int64_t capacity, const optional<Tensor>& epoch) {
        auto call = std::make_shared<RenderCall>();
        if (epoch && !(epoch->device().is_cpu() && epoch->scalar_type() == at::kLong &&
                       epoch->numel() == 1))
            fail("the tree's edit counter must be one int64 in host memory");
        call->tree = read_tree(tree);
        call->source = read_source(source, image, call->tree);
        call->options = read_options(opt);
        call->capacity = capacity;
        if (epoch) call->epoch = *epoch;
        return unlocked([&] { return RenderNode::apply(data, std::move(call)); });
    });

    // -> (render, gradient, diagonal, chunks the forward asked for).  `checked`: the host waits for
    // the forward, while the replay runs, to learn whether the log was large enough; if it was not,
    // gradient and diagonal are not filled and the call is for the caller to repeat.  Otherwise 0
    // chunks are returned, and a march behind the replay covers a log that was too small.
    m.def("se_grad", [](py::handle tree, py::handle source, py::handle opt, bool image,
                        const Tensor& colors, int64_t capacity, bool checked, bool watch) {
        const Tree t = read_tree(tree);
        const Source s = read_source(source, image, t);
        const svoxb_render_options o = read_options(opt);
        return unlocked([&] {
            const c10::cuda::CUDAGuard guard(t.data.device());
            if (capturing()) checked = false;       // nobody can wait for a captured stream
            Tensor grad, hess;
            const bool beside = fills_beside(t, s, capacity);
            optional<Zeroed> zeroed;
            if (beside) {
                zeroed.emplace(t.data, 2);
            } else {
                grad = at::empty(t.data.sizes(), t.data.options());
                hess = at::empty(t.data.sizes(), t.data.options());
            }
            auto [out, log] = run_logged(t, s, o, capacity, beside ? &*zeroed : nullptr, watch);
            at::cuda::CUDAEvent rendered;
            if (checked) rendered.record(at::cuda::getCurrentCUDAStream(t.data.device().index()));
            const Tensor resid = at::sub(out, colors.reshape(out.sizes())).contiguous();
            check_input(resid, "colors");
            if (beside) {
                grad = zeroed->claim(0);
                hess = zeroed->claim(1);
            }
            const float *r = resid.data_ptr<float>(), *f = out.template data_ptr<float>();
            int32_t* words = log.template data_ptr<int32_t>();
            float *g = grad.data_ptr<float>(), *h = hess.data_ptr<float>();
            const int64_t known = checked ? capacity : 0;
            void* stream = stream_of(t.data);
            check(s.image ? lib.se_grad_image_replay(&t.c, &s.cam, &o, r, f, words, capacity, known,
                                                     g, h, !beside, stream)
                          : lib.se_grad_replay(&t.c, &s.rays, &o, r, f, words, capacity, known, g,
                                               h, !beside, stream),
                  "se_grad_replay");
            int64_t used = 0;
            if (checked) {
                const auto side = Zeroed::side_stream(t.data.device().index());
                rendered.block(side);
                check(lib.item_log_used(words, &used, side.stream()), "item_log_used");
            }
            return std::make_tuple(out, grad, hess, used);
        });
    });

    m.def("log_is_sorted", [](py::handle tree, int64_t rays, bool image, int64_t capacity) {
        const Tree t = read_tree(tree);
        return lib.log_is_sorted(&t.c, rays, image, capacity) != 0;
    });
    m.def("poll_logs", [] {
        py::list out;
        for (const auto& s : log_watch().poll())
            out.append(py::make_tuple(s.used, s.batches, s.rays, s.capacity));
        return out;
    });
    m.def("logs_pending", [] { return log_watch().waiting(); });
}

}  // namespace

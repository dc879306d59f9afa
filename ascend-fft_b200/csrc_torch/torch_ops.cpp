// The transforms of bfly/ops.py on torch tensors without Python between the call and the launch,
// and their autograd nodes in C++ (a backward pass then runs without the interpreter).  Same
// entry points, checks and values as the Python functions there, which keep every call this file
// does not take: each function returns None for those (another device or type, a tensor subclass,
// forward-mode or functorch transforms, tracing, dispatch modes, lengths without a one-kernel
// gradient).
//
// Plans belong to Python (ops.plan_for).  A lookup table keeps a reference to each plan it has
// asked for, so that a plan cannot go away under a call; ops.autotune empties it, and it is emptied
// at kMaxPlans entries.  Nodes hold no plan: a backward pass looks its own up.
#include <torch/extension.h>

#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/custom_class.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <unordered_map>

#include "bfly_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using Maybe = std::optional<Tensor>;

// ------------------------------------------------------------------ plans
struct Held {   // a bfly.Plan and its handle
    PyObject* owner;
    bfly_plan* plan;
    Held(PyObject* o, bfly_plan* p) : owner(o), plan(p) {}
    Held(const Held&) = delete;
    ~Held() {
        py::gil_scoped_acquire gil;
        Py_DECREF(owner);
    }
};
using Plan = std::shared_ptr<Held>;
constexpr size_t kMaxPlans = 4096;
struct Table {
    std::mutex mu;
    std::unordered_map<uint64_t, Plan> plans;
    uint64_t forgotten = 0;      // times forgetPlans has emptied it
    PyObject* find = nullptr;    // find(device, real, n) -> (plan object, handle)
    PyObject* error = nullptr;   // bfly.BflyError
};
Table& table() {
    static Table* t = new Table;   // never destroyed: it may outlive the interpreter
    return *t;
}

[[noreturn]] void raisePython() {   // the Python error that is set
    python_error e;
    e.persist();
    throw e;
}

Plan planFor(int device, bool real, int64_t n) {
    Table& t = table();
    uint64_t forgotten;
    const uint64_t key = ((uint64_t)device << 33) | ((uint64_t)real << 32) | (uint32_t)n;
    {
        std::lock_guard<std::mutex> lock(t.mu);
        const auto it = t.plans.find(key);
        if (it != t.plans.end()) return it->second;
        forgotten = t.forgotten;
    }
    Plan p;
    {
        py::gil_scoped_acquire gil;
        PyObject* r = PyObject_CallFunction(t.find, "iiL", device, (int)real, (long long)n);
        if (!r) raisePython();
        PyObject* owner = PyTuple_GetItem(r, 0);
        void* handle = owner ? PyLong_AsVoidPtr(PyTuple_GetItem(r, 1)) : nullptr;
        if (!handle) {
            Py_DECREF(r);
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "bfly: no plan");
            raisePython();
        }
        Py_INCREF(owner);
        Py_DECREF(r);
        p = std::make_shared<Held>(owner, static_cast<bfly_plan*>(handle));
    }
    std::unordered_map<uint64_t, Plan> old;   // released after the lock: a Held takes the interpreter's
    {
        std::lock_guard<std::mutex> lock(t.mu);
        if (t.forgotten != forgotten) return p;   // asked for before the table was emptied: not kept
        if (t.plans.size() >= kMaxPlans) old.swap(t.plans);
        t.plans[key] = p;
    }
    return p;
}

void forgetPlans() {
    std::unordered_map<uint64_t, Plan> old;
    std::lock_guard<std::mutex> lock(table().mu);
    old.swap(table().plans);
    ++table().forgotten;
}

void bind(py::object find, py::object error) {
    table().find = find.release().ptr();
    table().error = error.release().ptr();
}

[[noreturn]] void raiseStatus(int rc, const std::string& what) {
    py::gil_scoped_acquire gil;
    PyObject* e = PyObject_CallFunction(table().error, "si", what.c_str(), rc);
    if (e) {
        PyErr_SetObject(table().error, e);
        Py_DECREF(e);
    }
    raisePython();
}
template <class What>   // what(): the call's text, made for a failure alone
void check(int rc, What&& what) {
    if (rc) raiseStatus(rc, what());
}

// ------------------------------------------------------------------ what is taken here
// A plain CUDA tensor of `type` outside every transform that has to see the call itself.  Empty ones
// stay with Python, whose scales divide by the length.
bool takes(const Tensor& x, at::ScalarType type) {
    if (!x.defined() || !x.is_cuda() || x.scalar_type() != type || x.layout() != at::kStrided ||
        x.unsafeGetTensorImpl()->key_set().has_any(c10::python_ks) || !x.numel() || x._fw_grad(0).defined())
        return false;
    for (const int64_t d : x.sizes())
        if (d > INT32_MAX) return false;
    return true;
}
// Contiguous memory that holds the values themselves (a conjugate view's does not).
Tensor dense(const Tensor& x) { return x.resolve_conj().resolve_neg().contiguous(); }
// No functorch transform around the call (its front key is included while one is active; the
// thread's functorch state itself outlives the first of them), no tracing, no dispatch mode.
bool plainMode() {
    return !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
           !torch::jit::tracer::isTracing() && !c10::impl::dispatch_mode_enabled();
}
bool wantsGrad(const Tensor& x) { return at::GradMode::is_enabled() && x.requires_grad(); }
void* streamOf(const Tensor& x) { return c10::cuda::getCurrentCUDAStream(x.get_device()).stream(); }
std::string text(const char* f, int64_t a, int64_t b) {
    return std::string(f) + "(n=" + std::to_string(a) + ", batch=" + std::to_string(b) + ")";
}

// ------------------------------------------------------------------ launches (contiguous results)
Tensor execC2C(const Tensor& in, int64_t direction, double scale) {
    const Tensor x = dense(in);
    Tensor y = at::empty_like(x);
    if (!x.numel()) return y;
    const int64_t n = x.size(-1), batch = x.numel() / n;
    const Plan p = planFor(x.get_device(), false, n);
    check(bfly_plan_exec_c2c_async(p->plan, x.data_ptr(), y.data_ptr(), (uint32_t)n, (uint64_t)batch, (int)direction,
                                   (float)scale, streamOf(x)),
          [&] { return text("exec_c2c", n, batch); });
    return y;
}

Tensor execAxis(const Tensor& in, int64_t dim, int64_t direction, double scale) {
    dim = dim < 0 ? dim + in.dim() : dim;
    if (dim == in.dim() - 1) return execC2C(in, direction, scale);
    const Tensor x = dense(in);
    Tensor y = at::empty_like(x);
    if (!x.numel()) return y;
    const int64_t n = x.size(dim);
    int64_t outer = 1, inner = 1;
    for (int64_t d = 0; d < dim; ++d) outer *= x.size(d);
    for (int64_t d = dim + 1; d < x.dim(); ++d) inner *= x.size(d);
    const Plan p = planFor(x.get_device(), false, n);
    check(bfly_plan_exec_c2c_axis_async(p->plan, x.data_ptr(), y.data_ptr(), (uint32_t)n, (uint64_t)outer,
                                        (uint64_t)inner, (int)direction, (float)scale, streamOf(x)),
          [&] { return "exec_c2c_axis(n=" + std::to_string(n) + ", outer=" + std::to_string(outer) + ", inner=" +
              std::to_string(inner) + ")"; });
    return y;
}

Tensor exec2D(const Tensor& in, int64_t direction, double scale) {
    const Tensor x = dense(in);
    Tensor y = at::empty_like(x);
    if (!x.numel()) return y;
    const int64_t ny = x.size(-2), nx = x.size(-1), batch = x.numel() / (ny * nx);
    const Plan p = planFor(x.get_device(), false, nx);
    check(bfly_plan_exec_c2c_2d_async(p->plan, x.data_ptr(), y.data_ptr(), (uint32_t)ny, (uint32_t)nx,
                                      (uint64_t)batch, (int)direction, (float)scale, streamOf(x)),
          [&] { return "exec_c2c_2d(ny=" + std::to_string(ny) + ", nx=" + std::to_string(nx) + ", batch=" +
              std::to_string(batch) + ")"; });
    return y;
}

Tensor emptyLast(const Tensor& x, int64_t last, at::ScalarType type) {
    auto shape = x.sizes().vec();
    shape.back() = last;
    return at::empty(shape, x.options().dtype(type));
}

Tensor execR2C(const Tensor& in, double edge, double inside) {
    const Tensor x = dense(in);
    const int64_t n = x.size(-1);
    Tensor y = emptyLast(x, n / 2 + 1, at::kComplexFloat);
    if (!x.numel()) return y;
    const int64_t batch = x.numel() / n;
    const Plan p = planFor(x.get_device(), true, n);
    check(bfly_plan_exec_r2c_async(p->plan, x.data_ptr(), y.data_ptr(), (uint32_t)n, (uint64_t)batch, (float)edge,
                                   (float)inside, streamOf(x)),
          [&] { return text("exec_r2c", n, batch); });
    return y;
}

Tensor execC2R(const Tensor& in, int64_t n, double edge, double inside, double scale) {
    const Tensor x = dense(in);
    Tensor y = emptyLast(x, n, at::kFloat);
    if (!x.numel()) return y;
    const int64_t batch = x.numel() / x.size(-1);
    const Plan p = planFor(x.get_device(), true, n);
    check(bfly_plan_exec_c2r_async(p->plan, x.data_ptr(), y.data_ptr(), (uint32_t)n, (uint64_t)batch, (float)edge,
                                   (float)inside, (float)scale, streamOf(x)),
          [&] { return text("exec_c2r", n, batch); });
    return y;
}

Tensor execR2C2D(const Tensor& in, double scale) {
    const Tensor x = dense(in);
    const int64_t ny = x.size(-2), nx = x.size(-1);
    Tensor y = emptyLast(x, nx / 2 + 1, at::kComplexFloat);
    if (!x.numel()) return y;
    const Plan p = planFor(x.get_device(), true, nx);
    check(bfly_plan_exec_r2c_2d_async(p->plan, x.data_ptr(), y.data_ptr(), (uint32_t)ny, (uint32_t)nx,
                                      (uint64_t)(x.numel() / (ny * nx)), (float)scale, streamOf(x)),
          [&] { return "exec_r2c_2d(ny=" + std::to_string(ny) + ", nx=" + std::to_string(nx) + ", batch=" +
              std::to_string(x.numel() / (ny * nx)) + ")"; });
    return y;
}

// The column pass goes to a tensor of the call's own, not to the plan's buffer (exec_c2r_2d's), which
// calls on other streams and captured graphs would share.
Tensor execC2R2D(const Tensor& in, int64_t nx, double scale) {
    return execC2R(execAxis(in, -2, 1, 1.0), nx, 1.0, 1.0, scale);
}

const void* windowPtr(const Tensor& w) { return w.defined() ? w.data_ptr() : nullptr; }
std::string frameText(const char* f, int64_t n, const char* b, int64_t vb, const char* c, int64_t vc, int64_t hop) {
    return std::string(f) + "(n=" + std::to_string(n) + ", " + b + "=" + std::to_string(vb) + ", " + c + "=" +
           std::to_string(vc) + ", hop=" + std::to_string(hop) + ")";
}

Tensor execStft(const Tensor& x, int64_t n, int64_t hop, bool center, const Tensor& window) {
    const int64_t signals = x.size(0), length = x.size(1);
    const int64_t frames = center ? 1 + length / hop : 1 + (length - n) / hop;
    Tensor y = at::empty({signals, frames, n / 2 + 1}, x.options().dtype(at::kComplexFloat));
    const Plan p = planFor(x.get_device(), true, n);
    uint64_t got = 0;
    check(bfly_plan_exec_stft_async(p->plan, x.data_ptr(), y.data_ptr(), (uint32_t)n, (uint64_t)signals,
                                    (uint64_t)length, (uint32_t)hop, center, windowPtr(window), &got, streamOf(x)),
          [&] { return frameText("exec_stft", n, "signals", signals, "length", length, hop); });
    return y;
}

Tensor execIstft(const Tensor& spec, int64_t n, int64_t hop, bool center, const Tensor& window, int64_t outLen,
                 double scale) {
    const int64_t signals = spec.size(0), frames = spec.size(1);
    Tensor y = at::empty({signals, outLen}, spec.options().dtype(at::kFloat));
    const Plan p = planFor(spec.get_device(), true, n);
    check(bfly_plan_exec_istft_async(p->plan, spec.data_ptr(), y.data_ptr(), (uint32_t)n, (uint64_t)signals,
                                     (uint32_t)frames, (uint32_t)hop, center, windowPtr(window), (uint64_t)outLen,
                                     (float)scale, streamOf(spec)),
          [&] { return frameText("exec_istft", n, "signals", signals, "frames", frames, hop); });
    return y;
}

// The gradients of a short-time transform's input: one kernel each.
Tensor execStftAdjoint(const Tensor& grad, int64_t n, int64_t hop, bool center, const Tensor& window, int64_t length) {
    const Tensor g = dense(grad);
    const int64_t signals = g.size(0);
    Tensor gx = at::empty({signals, length}, g.options().dtype(at::kFloat));
    const Plan p = planFor(g.get_device(), true, n);
    check(bfly_plan_exec_stft_backward_async(p->plan, g.data_ptr(), gx.data_ptr(), (uint32_t)n, (uint64_t)signals,
                                             (uint64_t)length, (uint32_t)hop, center, windowPtr(window), streamOf(g)),
          [&] { return frameText("exec_stft_backward", n, "signals", signals, "length", length, hop); });
    return gx;
}

Tensor execIstftAdjoint(const Tensor& grad, int64_t n, int64_t hop, bool center, const Tensor& window, int64_t frames,
                        double scale) {
    const Tensor g = dense(grad);
    Tensor gs = at::empty({g.size(0), frames, n / 2 + 1}, g.options().dtype(at::kComplexFloat));
    const Plan p = planFor(g.get_device(), true, n);
    check(bfly_plan_exec_istft_backward_async(p->plan, g.data_ptr(), gs.data_ptr(), (uint32_t)n, (uint64_t)g.size(0),
                                              (uint32_t)frames, (uint32_t)hop, center, windowPtr(window),
                                              (uint64_t)g.size(1), (float)scale, streamOf(g)),
          [&] { return "exec_istft_backward(n=" + std::to_string(n) + ", frames=" + std::to_string(frames) + ", hop=" +
              std::to_string(hop) + ")"; });
    return gs;
}

// ------------------------------------------------------------------ autograd nodes (adjoints as in ops.py)
// Every transform here is linear, so the adjoint of an adjoint is the transform: a backward pass runs
// its launches through the same functions as a forward one, and those record a node of their own
// where the gradient itself needs a gradient.  Windows are constants.
bool wantsFrames(const Tensor& x, const Maybe& w) { return wantsGrad(x) || (w && wantsGrad(*w)); }
Tensor c2cAxis(const Tensor& x, int64_t dim, int64_t direction, double scale);
Tensor c2c2D(const Tensor& x, int64_t direction, double scale);
// Bins 0 and n/2 times scale * edge, the others times scale * inside.
Tensor r2c(const Tensor& x, double scale, double edge = 1.0, double inside = 1.0);
Tensor c2r(const Tensor& x, int64_t n, double scale, double edge = 1.0, double inside = 1.0);
Tensor stftOf(const Tensor& x, int64_t n, int64_t hop, bool center, const Maybe& w);
Tensor istftOf(const Tensor& spec, int64_t n, int64_t hop, bool center, const Maybe& w, int64_t outLen, double scale);
Tensor stftAdjoint(const Tensor& g, int64_t n, int64_t hop, bool center, const Maybe& w, int64_t length);
Tensor istftAdjoint(const Tensor& g, int64_t n, int64_t hop, bool center, const Maybe& w, int64_t frames, double scale);

// What a node keeps for its backward pass, in one entry of saved_data: each entry is a string, a hash and
// an allocation (rfft of 1024 rows of 4096 with its gradient: 52.0 us with an entry per value, 50.0 so).
struct Saved : torch::CustomClassHolder {
    int64_t n = 0, hop = 0, size = 0, direction = 0;   // n: length or dimension; size: signal length or frames
    double scale = 1.0, edge = 1.0, inside = 1.0;
    bool center = false;
};
void save(AutogradContext* ctx, Saved s) {
    ctx->saved_data["p"] = c10::IValue::make_capsule(c10::make_intrusive<Saved>(std::move(s)));
}
Saved saved(AutogradContext* ctx) { return static_cast<const Saved&>(*ctx->saved_data["p"].toCapsule()); }
// The nodes of the short-time transforms keep their window too.
void saveFrames(AutogradContext* ctx, const Maybe& w, int64_t n, int64_t hop, bool center, int64_t size, double scale) {
    Saved s;
    s.n = n, s.hop = hop, s.size = size, s.scale = scale, s.center = center;
    save(ctx, s);
    ctx->save_for_backward({w.value_or(Tensor())});
}
Maybe savedWindow(AutogradContext* ctx) {
    const Tensor w = ctx->get_saved_variables()[0];
    return w.defined() ? Maybe(w) : std::nullopt;
}

struct C2CNode : Function<C2CNode> {   // dim: the transformed dimension
    static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t dim, int64_t direction, double scale) {
        Saved s;
        s.n = dim, s.direction = direction, s.scale = scale;
        save(ctx, s);
        return execAxis(x, dim, direction, scale);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        const Saved s = saved(ctx);
        return {c2cAxis(g[0], s.n, -s.direction, s.scale), Tensor(), Tensor(), Tensor()};
    }
};

struct C2C2DNode : Function<C2C2DNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t direction, double scale) {
        Saved s;
        s.direction = direction, s.scale = scale;
        save(ctx, s);
        return exec2D(x, direction, scale);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        const Saved s = saved(ctx);
        return {c2c2D(g[0], -s.direction, s.scale), Tensor(), Tensor()};
    }
};

struct R2CNode : Function<R2CNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, double scale, double edge, double inside) {
        Saved s;
        s.n = x.size(-1), s.scale = scale, s.edge = edge, s.inside = inside;
        save(ctx, s);
        return execR2C(x, scale * edge, scale * inside);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        const Saved s = saved(ctx);
        return {c2r(g[0], s.n, s.scale, s.edge, 0.5 * s.inside), Tensor(), Tensor(), Tensor()};
    }
};

struct C2RNode : Function<C2RNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t n, double scale, double edge, double inside) {
        Saved s;
        s.scale = scale, s.edge = edge, s.inside = inside;
        save(ctx, s);
        return execC2R(x, n, edge, inside, scale);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        const Saved s = saved(ctx);
        return {r2c(g[0], s.scale, s.edge, 2.0 * s.inside), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

struct R2C2DNode : Function<R2C2DNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, double scale) {
        Saved s;
        s.n = x.size(-1), s.scale = scale;
        save(ctx, s);
        return execR2C2D(x, scale);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        const Saved s = saved(ctx);
        return {c2r(c2cAxis(g[0], -2, 1, 1.0), s.n, s.scale, 1.0, 0.5), Tensor()};
    }
};

struct C2R2DNode : Function<C2R2DNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t nx, double scale) {
        Saved s;
        s.scale = scale;
        save(ctx, s);
        return execC2R2D(x, nx, scale);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        return {c2cAxis(r2c(g[0], saved(ctx).scale, 1.0, 2.0), -2, -1, 1.0), Tensor(), Tensor()};
    }
};

// `w` is optional: apply() asks every plain Tensor argument for its device, an undefined one included.
struct StftNode : Function<StftNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Maybe& w, int64_t n, int64_t hop, bool center) {
        saveFrames(ctx, w, n, hop, center, x.size(1), 1.0);
        return execStft(x, n, hop, center, w.value_or(Tensor()));
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        const Saved s = saved(ctx);
        return {stftAdjoint(g[0], s.n, s.hop, s.center, savedWindow(ctx), s.size), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

struct StftAdjointNode : Function<StftAdjointNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& g, const Maybe& w, int64_t n, int64_t hop, bool center,
                          int64_t length) {
        saveFrames(ctx, w, n, hop, center, length, 1.0);
        return execStftAdjoint(g, n, hop, center, w.value_or(Tensor()), length);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& h) {
        const Saved s = saved(ctx);
        return {stftOf(dense(h[0]), s.n, s.hop, s.center, savedWindow(ctx)), Tensor(), Tensor(), Tensor(), Tensor(),
                Tensor()};
    }
};

struct IstftNode : Function<IstftNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& spec, const Maybe& w, int64_t n, int64_t hop, bool center,
                          int64_t outLen, double scale) {
        saveFrames(ctx, w, n, hop, center, spec.size(1), scale);
        return execIstft(spec, n, hop, center, w.value_or(Tensor()), outLen, scale);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& g) {
        const Saved s = saved(ctx);
        return {istftAdjoint(g[0], s.n, s.hop, s.center, savedWindow(ctx), s.size, s.scale), Tensor(), Tensor(), Tensor(),
                Tensor(), Tensor(), Tensor()};
    }
};

struct IstftAdjointNode : Function<IstftAdjointNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& g, const Maybe& w, int64_t n, int64_t hop, bool center,
                          int64_t frames, double scale) {
        saveFrames(ctx, w, n, hop, center, g.size(1), scale);
        return execIstftAdjoint(g, n, hop, center, w.value_or(Tensor()), frames, scale);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& h) {
        const Saved s = saved(ctx);
        return {istftOf(dense(h[0]), s.n, s.hop, s.center, savedWindow(ctx), s.size, s.scale), Tensor(), Tensor(), Tensor(),
                Tensor(), Tensor(), Tensor()};
    }
};

Tensor c2cAxis(const Tensor& x, int64_t dim, int64_t direction, double scale) {
    return wantsGrad(x) ? C2CNode::apply(x, dim, direction, scale) : execAxis(x, dim, direction, scale);
}
Tensor c2c2D(const Tensor& x, int64_t direction, double scale) {
    return wantsGrad(x) ? C2C2DNode::apply(x, direction, scale) : exec2D(x, direction, scale);
}
Tensor r2c(const Tensor& x, double scale, double edge, double inside) {
    return wantsGrad(x) ? R2CNode::apply(x, scale, edge, inside) : execR2C(x, scale * edge, scale * inside);
}
Tensor c2r(const Tensor& x, int64_t n, double scale, double edge, double inside) {
    return wantsGrad(x) ? C2RNode::apply(x, n, scale, edge, inside) : execC2R(x, n, edge, inside, scale);
}
Tensor stftOf(const Tensor& x, int64_t n, int64_t hop, bool center, const Maybe& w) {
    return wantsFrames(x, w) ? StftNode::apply(x, w, n, hop, center) : execStft(x, n, hop, center, w.value_or(Tensor()));
}
Tensor istftOf(const Tensor& spec, int64_t n, int64_t hop, bool center, const Maybe& w, int64_t outLen, double scale) {
    return wantsFrames(spec, w) ? IstftNode::apply(spec, w, n, hop, center, outLen, scale)
                                : execIstft(spec, n, hop, center, w.value_or(Tensor()), outLen, scale);
}
Tensor stftAdjoint(const Tensor& g, int64_t n, int64_t hop, bool center, const Maybe& w, int64_t length) {
    return wantsGrad(g) ? StftAdjointNode::apply(g, w, n, hop, center, length)
                        : execStftAdjoint(g, n, hop, center, w.value_or(Tensor()), length);
}
Tensor istftAdjoint(const Tensor& g, int64_t n, int64_t hop, bool center, const Maybe& w, int64_t frames, double scale) {
    return wantsGrad(g) ? IstftAdjointNode::apply(g, w, n, hop, center, frames, scale)
                        : execIstftAdjoint(g, n, hop, center, w.value_or(Tensor()), frames, scale);
}

// ------------------------------------------------------------------ entry points
double scaleOf(int norm, double n, bool forward) {   // norm: 0 backward, 1 ortho, 2 forward
    return norm == 1 ? 1.0 / std::sqrt(n) : (norm == 0) == forward ? 1.0 : 1.0 / n;
}

Maybe fft(const Tensor& x, int64_t dim, int64_t direction, int64_t norm) {
    if (!takes(x, at::kComplexFloat) || !plainMode() || x.dim() < 1) return std::nullopt;
    dim = dim < 0 ? dim + x.dim() : dim;
    if (dim < 0 || dim >= x.dim()) return std::nullopt;
    const double s = scaleOf((int)norm, (double)x.size(dim), direction < 0);
    return c2cAxis(x, dim, direction, s);
}

Maybe fft2(const Tensor& x, int64_t direction, int64_t norm) {
    if (!takes(x, at::kComplexFloat) || !plainMode() || x.dim() < 2) return std::nullopt;
    const double s = scaleOf((int)norm, (double)x.size(-2) * (double)x.size(-1), direction < 0);
    return c2c2D(x, direction, s);
}

Maybe rfft(const Tensor& x, int64_t norm) {
    if (!takes(x, at::kFloat) || !plainMode() || x.dim() < 1) return std::nullopt;
    return r2c(x, scaleOf((int)norm, (double)x.size(-1), true));
}

Maybe irfft(const Tensor& x, int64_t n, int64_t norm) {
    if (!takes(x, at::kComplexFloat) || !plainMode() || x.dim() < 1 || n < 1 || x.size(-1) != n / 2 + 1)
        return std::nullopt;
    return c2r(x, n, scaleOf((int)norm, (double)n, false));
}

Maybe rfft2(const Tensor& x, int64_t norm) {
    if (!takes(x, at::kFloat) || !plainMode() || x.dim() < 2) return std::nullopt;
    const double s = scaleOf((int)norm, (double)x.size(-2) * (double)x.size(-1), true);
    return wantsGrad(x) ? R2C2DNode::apply(x, s) : execR2C2D(x, s);
}

Maybe irfft2(const Tensor& x, int64_t nx, int64_t norm) {
    if (!takes(x, at::kComplexFloat) || !plainMode() || x.dim() < 2 || nx < 1 || x.size(-1) != nx / 2 + 1)
        return std::nullopt;
    const double s = scaleOf((int)norm, (double)x.size(-2) * (double)nx, false);
    return wantsGrad(x) ? C2R2DNode::apply(x, nx, s) : execC2R2D(x, nx, s);
}

bool oneKernelFrames(int64_t n) { return n >= 64 && n <= 8192 && (n & (n - 1)) == 0; }

Maybe stft(const Tensor& x, int64_t n, int64_t hop, bool center, const Maybe& w) {
    if (!takes(x, at::kFloat) || !plainMode() || x.dim() != 2 || !x.is_contiguous() || x.is_neg() || hop < 1 ||
        !oneKernelFrames(n) || x.size(1) < (center ? n + 2 : n) || x.size(0) < 1 ||
        (w && !takes(*w, at::kFloat)))
        return std::nullopt;
    return stftOf(x, n, hop, center, w);
}

Maybe istft(const Tensor& spec, int64_t n, int64_t hop, bool center, const Maybe& w, int64_t outLen, double scale) {
    if (!takes(spec, at::kComplexFloat) || !plainMode() || spec.dim() != 3 || !spec.is_contiguous() ||
        spec.is_conj() || spec.is_neg() ||
        !oneKernelFrames(n) || (w && !takes(*w, at::kFloat)))
        return std::nullopt;
    return istftOf(spec, n, hop, center, w, outLen, scale);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", &bind);
    m.def("forget_plans", &forgetPlans, py::call_guard<py::gil_scoped_release>());
    m.def("fft", torch::wrap_pybind_function_no_gil(fft));
    m.def("fft2", torch::wrap_pybind_function_no_gil(fft2));
    m.def("rfft", torch::wrap_pybind_function_no_gil(rfft));
    m.def("irfft", torch::wrap_pybind_function_no_gil(irfft));
    m.def("rfft2", torch::wrap_pybind_function_no_gil(rfft2));
    m.def("irfft2", torch::wrap_pybind_function_no_gil(irfft2));
    m.def("stft", torch::wrap_pybind_function_no_gil(stft));
    m.def("istft", torch::wrap_pybind_function_no_gil(istft));
}

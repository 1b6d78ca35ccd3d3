// Host side of one call, in native code: what `jit.__call__` runs for ordinary eager CUDA tensors.
//
// A call of a compiled step function has to find its specialisation, check its arguments, allocate the results,
// encode the TMA tensor maps of this call's addresses, launch one or a few kernels and hang a node into the autograd
// graph.  Through a Python custom op that took 0.12 ms for a forward and 0.5 ms for a forward and backward (B200 host,
// problems small enough that the GPU time does not count); here it is a few tens of microseconds.  The custom ops stay
// for everything that traces or transforms a call (torch.compile, fake tensors, functorch, dispatch modes, subclasses).
//
// Kernels are launched through the C ABI of libfrnn_b200.so (include/frnn.h), whose entry points are handed over by
// address; this file links against PyTorch only.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>

#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

namespace py = pybind11;
using at::Tensor;
using torch::autograd::variable_list;

namespace {

typedef int (*launch_fn)(void*, int, const unsigned*, const unsigned*, unsigned, void*, void* const*, int);
typedef int (*encode_fn)(void*, const void*, unsigned, unsigned, const uint64_t*, const uint64_t*, const uint32_t*);
typedef const char* (*error_fn)();
launch_fn g_launch = nullptr;
encode_fn g_encode = nullptr;
error_fn g_error = nullptr;

struct Meta {
    std::vector<int64_t> sizes, strides;
    at::ScalarType dtype;
};

Meta meta_of(const Tensor& t) { return {t.sizes().vec(), t.strides().vec(), t.scalar_type()}; }

// A saved tensor in the layout it was saved with, on a 16-byte boundary if `aligned`.  Kernels are built for that layout,
// but a saved-tensor hook may hand back another one (torch.autograd.graph.save_on_cpu returns contiguous copies): the
// values are then copied into it.  Another shape, data type or device is refused.
Tensor as_saved(const Tensor& t, const Meta& m, const c10::Device& dev, bool aligned) {
    TORCH_CHECK(t.defined() && t.layout() == at::kStrided && t.sizes().equals(m.sizes) && t.scalar_type() == m.dtype && t.device() == dev,
                "flex_rnn_b200: a saved-tensor hook returned another shape, data type or device than was saved (shape ", at::IntArrayRef(m.sizes),
                ", ", m.dtype, " on ", dev, ")");
    bool same = !aligned || !((uintptr_t)t.data_ptr() & 15);
    for (size_t d = 0; d < m.sizes.size(); d++) same = same && (m.sizes[d] <= 1 || t.stride(d) == m.strides[d]);
    if (same) return t;
    Tensor r = at::empty_strided(m.sizes, m.strides, t.options()), to = r, from = t;
    for (size_t d = 0; d < m.sizes.size(); d++)
        if (m.sizes[d] > 1 && m.strides[d] == 0) {       // an expanded dimension: one element, whose copies are all alike
            to = to.narrow(d, 0, 1);
            from = from.narrow(d, 0, 1);
        }
    to.copy_(from);
    return r;
}

struct TensorMap {                 // a TMA tensor map to encode per call (it embeds the tensor's address)
    int src;                       // parameter whose tensor it describes
    int64_t off;                   // bytes from that tensor's first element
    unsigned elt;
    uint64_t dims[4], strides[3];
    uint32_t box[4];
};

struct Kernel {
    void* module = nullptr;
    unsigned grid[3], block[3], smem = 0;
    std::vector<int> params;       // buffer index of every pointer parameter
    std::vector<TensorMap> maps;   // by-value parameters after the pointers
};

// One launch sequence.  Buffers are numbered: the caller's tensors, then `alloc` in order, then the error word.
struct Program {
    std::vector<Kernel> kernels;
    std::vector<Meta> alloc;
    std::vector<int> zeroed;       // members of `alloc` that must start at zero: fp32, carved out of one zeroed buffer
    std::vector<int> cast_from;    // member of `alloc` to convert into member i of the results, or -1
    int returned = 0;              // the first `returned` members of `alloc` are results
};

struct alignas(64) RawMap { unsigned char b[128]; };

enum { MAX_PARAMS = 64, MAX_MAPS = 24 };

void run_program(const Program& p, const std::vector<void*>& given, std::vector<Tensor>& made, const c10::Device& dev, int* err) {
    made.resize(p.alloc.size());
    if (!p.zeroed.empty()) {
        int64_t total = 0;
        for (int i : p.zeroed) {
            int64_t n = 1;
            for (int64_t s : p.alloc[i].sizes) n *= s;
            total += (n + 63) / 64 * 64;
        }
        Tensor flat = at::detail::empty_strided_cuda({total}, {1}, at::kFloat, dev);
        flat.zero_();
        int64_t at_ = 0;
        for (int i : p.zeroed) {
            int64_t n = 1;
            for (int64_t s : p.alloc[i].sizes) n *= s;
            made[i] = flat.as_strided(p.alloc[i].sizes, p.alloc[i].strides, at_);
            at_ += (n + 63) / 64 * 64;
        }
    }
    for (size_t i = 0; i < p.alloc.size(); i++)
        if (!made[i].defined()) made[i] = at::detail::empty_strided_cuda(p.alloc[i].sizes, p.alloc[i].strides, p.alloc[i].dtype, dev);
    void* stream = (void*)c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const size_t ng = given.size(), na = made.size();
    for (const Kernel& k : p.kernels) {
        void* vals[MAX_PARAMS];
        void* args[MAX_PARAMS + MAX_MAPS];
        RawMap maps[MAX_MAPS];
        int n = 0;
        for (int b : k.params) {
            vals[n] = (size_t)b < ng ? given[b] : (size_t)b < ng + na ? made[b - ng].data_ptr() : (void*)err;
            args[n] = &vals[n];
            n++;
        }
        int m = 0;
        for (const TensorMap& t : k.maps) {
            if (g_encode(&maps[m], (const char*)vals[t.src] + t.off, t.elt, 4, t.dims, t.strides, t.box))
                TORCH_CHECK(false, "flex_rnn_b200: ", g_error());
            args[n++] = &maps[m++];
        }
        if (g_launch(k.module, 0, k.grid, k.block, k.smem, stream, args, n)) TORCH_CHECK(false, "flex_rnn_b200: ", g_error());
    }
    for (size_t i = 0; i < p.cast_from.size(); i++)
        if (p.cast_from[i] >= 0) made[i].copy_(made[p.cast_from[i]]);
}

// A specialisation: shapes, strides and data types of one call, its launch programs, and the Python closures that
// serve until those are there (the first call of each kind compiles) and wherever a check fails (they name it).
struct Spec : std::enable_shared_from_this<Spec> {
    int nin = 0, nst = 0, nout = 0;
    c10::DeviceIndex device = 0;
    int* err = nullptr;                  // the device's error word, in pinned host memory
    std::vector<char> aligned;           // argument i was 16-byte aligned at compilation
    std::vector<int64_t> reach;          // bytes from argument i's first element to the end of its last one
    // of the results and of what a forward saves (the arguments first), the same for every call; filled by the first one
    std::vector<Meta> result_meta, saved_meta;
    std::atomic<const Program*> forward{nullptr}, infer{nullptr}, backward{nullptr};   // set once, by a Python closure's first run
    py::object py_forward, py_infer, py_backward;    // (spec, args) -> results and saved; (spec, args) -> results; (spec, grads, args, saved, whether the custom op is not needed) -> gradients
    ~Spec() {
        delete forward.load();
        delete infer.load();
        delete backward.load();
        if (!Py_IsInitialized()) {
            py_forward.release(); py_infer.release(); py_backward.release();
            return;
        }
        py::gil_scoped_acquire g;
        py_forward = py_infer = py_backward = py::object();
    }
    bool args_ok(const variable_list& a, size_t n) const {
        if (*(volatile int*)err) return false;           // a kernel of an earlier call gave up: the closure reports it
        for (size_t i = 0; i < n; i++) {
            if (aligned[i] && ((uintptr_t)a[i].data_ptr() & 15)) return false;
            if (a[i].numel() && (size_t)reach[i] + a[i].storage_offset() * a[i].element_size() > a[i].storage().nbytes()) return false;
        }
        return true;
    }
};

variable_list to_list(const py::object& o) {
    variable_list v;
    for (auto x : py::cast<py::tuple>(o)) v.push_back(py::cast<Tensor>(x));
    return v;
}

py::tuple to_tuple(const variable_list& v, size_t lo, size_t hi) {
    py::tuple t(hi - lo);
    for (size_t i = lo; i < hi; i++) t[i - lo] = py::cast(v[i]);
    return t;
}

// run a Python closure from any thread; its exception keeps its type
template <class F> variable_list with_python(F f) {
    py::gil_scoped_acquire g;
    try {
        return f();
    } catch (py::error_already_set& e) {
        e.restore();
        python_error err;
        err.persist();
        throw std::move(err);
    }
}

// Run a program of a call's arguments, from a thread that holds the interpreter lock: allocations and launches may wait (a
// full launch queue), and other Python threads go on meanwhile.
variable_list launch(const Program& p, const variable_list& args, const Spec& s) {
    std::vector<void*> given;
    for (const Tensor& t : args) given.push_back(t.data_ptr());
    variable_list made;
    py::gil_scoped_release others;
    run_program(p, given, made, c10::Device(c10::kCUDA, s.device), s.err);
    return made;
}

variable_list run_forward(Spec& s, const variable_list& args) {      // results, final states, saved tensors
    const Program* p = s.forward.load(std::memory_order_acquire);
    if (!p || !s.args_ok(args, args.size()))
        return with_python([&] { return to_list(s.py_forward(s.shared_from_this(), to_tuple(args, 0, args.size()))); });
    variable_list made = launch(*p, args, s);
    made.resize(p->returned);
    return made;
}

// Whether something that traces or transforms calls is active, which only the custom ops serve.
bool transformed() {
    return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Functionalize) ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Tracer);
}

// Whether a tensor is a wrapper of some kind (subclass, batched, lazily conjugated ...), which only the custom ops serve.
bool wrapped(const Tensor& t) {
    static const c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot,
        c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
        c10::DispatchKey::Batched, c10::DispatchKey::ZeroTensor, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative, c10::DispatchKey::BatchedNestedTensor});
    return t.key_set().has_any(special);
}

// The node of one call in the autograd graph.
struct RecurrenceBackward : torch::autograd::Node {
    std::shared_ptr<Spec> spec;
    std::vector<torch::autograd::SavedVariable> saved;   // the arguments, then what the forward saved

    explicit RecurrenceBackward(torch::autograd::edge_list&& e) : Node(std::move(e)) {}
    std::string name() const override { return "RecurrenceBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto& v : saved) v.reset_data();
        released = true;
    }
    bool released = false;

    variable_list apply(variable_list&& up) override {
        Spec& s = *spec;
        variable_list kept;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
            for (auto& v : saved) kept.push_back(v.unpack(shared_from_this()));
        }
        c10::cuda::CUDAGuard guard(s.device);
        const c10::Device dev(c10::kCUDA, s.device);
        for (size_t i = 0; i < up.size(); i++) {
            const Meta& m = s.result_meta[i];      // absent upstream gradients are zeros
            if (!up[i].defined()) {
                up[i] = at::detail::empty_cuda(m.sizes, at::TensorOptions().dtype(m.dtype).device(dev)).zero_();
            } else {
                up[i] = up[i].contiguous();
            }
        }
        const int narg = s.nin + s.nst;
        // a gradient that is itself traced or transformed (a dispatch mode, batched upstream gradients) is the custom op's;
        // with create_graph=True too, which refuses to be differentiated in its turn
        bool direct = !transformed() && !at::GradMode::is_enabled();
        for (const Tensor& t : up) direct = direct && !wrapped(t);
        for (const Tensor& t : kept) direct = direct && t.defined() && !wrapped(t);
        if (direct)
            for (size_t i = 0; i < kept.size(); i++) kept[i] = as_saved(kept[i], s.saved_meta[i], dev, i >= (size_t)narg || s.aligned[i]);
        const Program* p = s.backward.load(std::memory_order_acquire);
        bool ok = p && direct && s.args_ok(kept, s.nin);
        for (const Tensor& t : up) ok = ok && t.device() == dev && !((uintptr_t)t.data_ptr() & 15);
        for (size_t i = 0; i < up.size() && ok; i++) ok = up[i].scalar_type() == s.result_meta[i].dtype;
        variable_list g;
        if (!ok) {
            g = with_python([&] {
                return to_list(s.py_backward(s.shared_from_this(), to_tuple(up, 0, up.size()), to_tuple(kept, 0, narg), to_tuple(kept, narg, kept.size()), direct));
            });
        } else {
            std::vector<void*> given;
            for (int i = 0; i < s.nin; i++) given.push_back(kept[i].data_ptr());
            for (const Tensor& t : up) given.push_back(t.data_ptr());
            for (size_t i = narg; i < kept.size(); i++) given.push_back(kept[i].data_ptr());
            run_program(*p, given, g, dev, s.err);
            g.resize(p->returned);
        }
        for (size_t i = 0; i < g.size(); i++)
            if (!task_should_compute_output(i)) g[i] = Tensor();
        return g;
    }
};

struct KeyHash {
    size_t operator()(const std::vector<int64_t>& k) const {
        uint64_t h = 1469598103934665603ull;
        for (int64_t v : k) h = (h ^ (uint64_t)v) * 1099511628211ull;
        return (size_t)(h ^ (h >> 29));
    }
};

struct HostOp {
    int nargs;
    py::object on_miss;        // (args) -> Spec, or None where the custom op has to be used
    std::unordered_map<std::vector<int64_t>, std::shared_ptr<Spec>, KeyHash> table;

    HostOp(int n, py::object miss) : nargs(n), on_miss(std::move(miss)) {}

    // The results of a direct call, or None: the caller then goes through the custom op.
    py::object call(py::tuple args) {
        if ((int)args.size() != nargs) return py::none();
        if (transformed()) return py::none();
        variable_list a;
        a.reserve(nargs);
        std::vector<int64_t> key;
        key.reserve(nargs * 11 + 1);
        bool grad = false;
        for (int i = 0; i < nargs; i++) {
            PyObject* o = PyTuple_GET_ITEM(args.ptr(), i);
            if (!THPVariable_CheckExact(o)) return py::none();
            const Tensor& t = THPVariable_Unpack(o);
            if (!t.is_cuda() || t.layout() != at::kStrided || wrapped(t) || t._fw_grad(0).defined()) return py::none();
            if (t.device() != THPVariable_Unpack(PyTuple_GET_ITEM(args.ptr(), 0)).device()) return py::none();
            grad = grad || t.requires_grad();
            auto sz = t.sizes();
            auto st = t.strides();
            key.push_back((int64_t)sz.size() | ((int64_t)t.scalar_type() << 8));
            for (size_t d = 0; d < sz.size(); d++) {
                key.push_back(sz[d]);
                key.push_back(sz[d] > 1 ? st[d] : 0);
            }
            a.push_back(t);
        }
        key.push_back(a[0].device().index());
        auto it = table.find(key);
        if (it == table.end()) {
            py::object found = on_miss(args);
            if (found.is_none()) return py::none();
            it = table.emplace(std::move(key), py::cast<std::shared_ptr<Spec>>(found)).first;
        }
        std::shared_ptr<Spec> s = it->second;
        c10::cuda::CUDAGuard guard(s->device);
        grad = grad && at::GradMode::is_enabled();
        const size_t nres = s->nout + s->nst;
        variable_list res;
        if (!grad) {
            at::AutoDispatchBelowADInplaceOrView below;
            const Program* p = s->infer.load(std::memory_order_acquire);
            if (p && s->args_ok(a, a.size()))
                res = launch(*p, a, *s);
            else
                res = to_list(s->py_infer(s, args));
            res.resize(nres);
        } else {
            auto node = std::shared_ptr<RecurrenceBackward>(
                new RecurrenceBackward(torch::autograd::collect_next_edges(a)), torch::autograd::deleteNode);
            {
                at::AutoDispatchBelowADInplaceOrView below;
                at::NoGradGuard no_grad;
                res = run_forward(*s, a);
            }
            node->spec = s;
            if (s->result_meta.empty()) {           // (no saving hook has run yet: the interpreter lock is held throughout)
                for (const Tensor& t : a) s->saved_meta.push_back(meta_of(t));
                for (size_t i = 0; i < res.size(); i++) (i < nres ? s->result_meta : s->saved_meta).push_back(meta_of(res[i]));
            }
            for (const Tensor& t : a) node->saved.emplace_back(t, false);
            for (size_t i = nres; i < res.size(); i++) node->saved.emplace_back(res[i], false);
            res.resize(nres);
            for (Tensor& t : res) torch::autograd::create_gradient_edge(t, node);
        }
        py::tuple out(res.size());
        for (size_t i = 0; i < res.size(); i++) out[i] = py::reinterpret_steal<py::object>(THPVariable_Wrap(res[i]));
        return std::move(out);
    }
};

Meta meta_from(const py::handle& h) {
    auto t = py::cast<py::tuple>(h);
    Meta m;
    m.sizes = py::cast<std::vector<int64_t>>(t[0]);
    m.strides = py::cast<std::vector<int64_t>>(t[1]);
    m.dtype = reinterpret_cast<THPDtype*>(t[2].ptr())->scalar_type;
    return m;
}

std::unique_ptr<Program> program_of(const py::dict& d) {
    std::unique_ptr<Program> p(new Program());
    for (auto h : d["alloc"]) p->alloc.push_back(meta_from(h));
    p->zeroed = py::cast<std::vector<int>>(d["zeroed"]);
    p->cast_from = py::cast<std::vector<int>>(d["cast_from"]);
    p->returned = py::cast<int>(d["returned"]);
    for (auto h : d["kernels"]) {
        auto k = py::cast<py::dict>(h);
        Kernel q;
        q.module = (void*)py::cast<uintptr_t>(k["module"]);
        auto grid = py::cast<std::vector<unsigned>>(k["grid"]);
        for (int i = 0; i < 3; i++) { q.grid[i] = grid[i]; q.block[i] = 1; }
        q.block[0] = py::cast<unsigned>(k["block"]);
        q.smem = py::cast<unsigned>(k["smem"]);
        q.params = py::cast<std::vector<int>>(k["params"]);
        for (auto mh : k["maps"]) {
            auto m = py::cast<py::dict>(mh);
            TensorMap t;
            t.src = py::cast<int>(m["src_index"]);
            t.off = py::cast<int64_t>(m["off_bytes"]);
            t.elt = py::cast<unsigned>(m["elt"]);
            auto dims = py::cast<std::vector<uint64_t>>(m["dims"]);
            auto str = py::cast<std::vector<uint64_t>>(m["strides_bytes"]);
            auto box = py::cast<std::vector<uint32_t>>(m["box"]);
            for (int i = 0; i < 4; i++) { t.dims[i] = dims[i]; t.box[i] = box[i]; }
            for (int i = 0; i < 3; i++) t.strides[i] = str[i];
            q.maps.push_back(t);
        }
        TORCH_CHECK(q.params.size() <= MAX_PARAMS && q.maps.size() <= MAX_MAPS, "flex_rnn_b200: too many kernel parameters");
        p->kernels.push_back(std::move(q));
    }
    return p;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", [](uintptr_t launch, uintptr_t encode, uintptr_t error) {
        g_launch = (launch_fn)launch;
        g_encode = (encode_fn)encode;
        g_error = (error_fn)error;
    });
    m.def("as_saved", [](const Tensor& t, const py::object& meta, const Tensor& device_of, bool aligned) {
        return as_saved(t, meta_from(meta), device_of.device(), aligned);
    });
    py::class_<Spec, std::shared_ptr<Spec>>(m, "Spec")
        .def(py::init([](int nin, int nst, int nout, int device, uintptr_t err, std::vector<bool> aligned, std::vector<int64_t> reach,
                         py::object fwd, py::object infer, py::object bwd) {
            auto s = std::make_shared<Spec>();
            s->nin = nin; s->nst = nst; s->nout = nout;
            s->device = (c10::DeviceIndex)device;
            s->err = (int*)err;
            s->aligned.assign(aligned.begin(), aligned.end());
            s->reach = std::move(reach);
            s->py_forward = std::move(fwd); s->py_infer = std::move(infer); s->py_backward = std::move(bwd);
            return s;
        }))
        .def("set", [](Spec& s, const std::string& which, py::dict d) {
            auto& slot = which == "forward" ? s.forward : which == "infer" ? s.infer : s.backward;
            if (!slot.load()) slot.store(program_of(d).release(), std::memory_order_release);     // the GIL serialises this
        })
        .def("has", [](Spec& s, const std::string& which) {
            return (which == "forward" ? s.forward : which == "infer" ? s.infer : s.backward).load() != nullptr;
        });
    py::class_<HostOp>(m, "HostOp").def(py::init<int, py::object>()).def("call", &HostOp::call);
}

// The operator on torch tensors: argument checks, output allocation, the C-ABI call and the autograd node,
// in one native call per direction.
//
// A small problem's kernels take about ten microseconds, so what the host does around them decides its speed.
// Done in Python (ctypes structures, a torch allocation for every buffer, a Python autograd function, a status
// word that is cleared on the device before and copied back after every call) that was 76 microseconds per
// forward call at B1 H2 N256 D64 w 64/16.
//
// Only plain calls are made here: tensors that are torch.Tensor or Parameter themselves, and for the autograd node no
// tracing, functorch transform or forward-mode tangent, which the Python autograd function records or refuses.  For
// other calls the entry points return None and the Python layer takes over.
//
// Device-side timeouts: the kernels record them straight into a pinned host word per device and direction
// (sa_forward_status / sa_backward_status), which every later call looks at before it launches.  Nothing is
// cleared, copied or waited for per call.
#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAContext.h>
#include <Python.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <atomic>
#include <mutex>

#include "../../include/simplicial_attn_b200.h"

namespace {

using at::Tensor;

struct Config {
    int64_t w1, w2, halo1, halo2;
    double scale, k2_bias, v2_bias;
    int algo;
};

// ---- status words: pinned host memory, 256 bytes per device and direction ({code, wait site, block, 0})
constexpr int kMaxDevices = 64;
constexpr int kSlotInts = 64;
enum Direction { kForward = 0, kBackward = 1 };
const char* const kLabel[2] = {"sa_forward", "sa_backward"};

std::atomic<volatile int*> g_slots{nullptr};
std::atomic<uint64_t> g_devices{0};               // bit per device that has been called on

volatile int* slot(int device, Direction d) {
    volatile int* base = g_slots.load(std::memory_order_acquire);
    if (base == nullptr) {
        static std::mutex mu;
        std::lock_guard<std::mutex> lock(mu);
        base = g_slots.load(std::memory_order_acquire);
        if (base == nullptr) {
            void* p = nullptr;
            const size_t bytes = sizeof(int) * kSlotInts * 2 * kMaxDevices;
            C10_CUDA_CHECK(cudaHostAlloc(&p, bytes, cudaHostAllocPortable | cudaHostAllocMapped));
            memset(p, 0, bytes);
            base = static_cast<volatile int*>(p);
            g_slots.store(base, std::memory_order_release);
        }
    }
    return base + (device * 2 + d) * kSlotInts;
}

void* status_word(int device, Direction d) { return const_cast<int*>(slot(device, d)); }

PyObject* g_on_error = nullptr;       // Python callable (function name, status, detail or None) that raises

[[noreturn]] void raise_status(const char* fn, int status, const char* detail = nullptr) {
    pybind11::gil_scoped_acquire gil;
    PyObject* r = PyObject_CallFunction(g_on_error, "siz", fn, status, detail);
    Py_XDECREF(r);
    if (r != nullptr) PyErr_SetString(PyExc_RuntimeError, fn);      // (the callable always raises)
    python_error e;
    e.persist();
    throw python_error(std::move(e));
}

// Raises if a kernel of an earlier call on the device gave up on a bounded wait, and clears the word.  (While that kernel
// still runs, another of its blocks may give up and leave a second report.)
void poll_device(int device) {
    g_devices.fetch_or(1ull << device, std::memory_order_relaxed);
    for (Direction d : {kForward, kBackward}) {
        volatile int* s = slot(device, d);
        if (s[0] != 0) {
            const int code = s[0], where = s[1], block = s[2];      // (the device writes the code last)
            s[0] = s[1] = s[2] = 0;
            char text[96];
            snprintf(text, sizeof(text), "device side: wait site %d, block %d", where, block);
            raise_status(kLabel[d], code, text);
        }
    }
}

// ---- arguments
Tensor unit_inner(const Tensor& t) { return t.dim() > 0 && t.stride(-1) != 1 ? t.contiguous() : t; }

sa_strides strides_of(const Tensor& t) {
    return t.defined() ? sa_strides{t.stride(0), t.stride(1), t.stride(2)} : sa_strides{0, 0, 0};
}

void check_inputs(const Tensor& q, const Tensor& k1, const Tensor& k2, const Tensor& v1, const Tensor& v2, const Config& c) {
    TORCH_CHECK(q.is_cuda(), "simplical_attn_b200 runs on CUDA tensors only; there is no CPU path");
    TORCH_CHECK_VALUE(q.dim() == 4, "q must be [batch, seq_len, num_heads, head_dim]");
    const auto st = q.scalar_type();
    TORCH_CHECK_TYPE(st == at::kBFloat16 || st == at::kHalf || st == at::kFloat, "unsupported dtype ", st);
    const Tensor* const kv[4] = {&k1, &v1, &k2, &v2};
    static const char* const names[4] = {"k1", "v1", "k2", "v2"};
    const int64_t B = q.size(0), N = q.size(1), H = q.size(2), D = q.size(3);
    for (int i = 0; i < 4; ++i) {
        const Tensor& t = *kv[i];
        TORCH_CHECK_TYPE(t.scalar_type() == st && t.device() == q.device(), names[i], " must match q's dtype and device");
        const int64_t halo = i < 2 ? c.halo1 : c.halo2;
        TORCH_CHECK_VALUE(t.dim() == 4 && t.size(0) == B && t.size(1) == N + halo && t.size(3) == D, names[i],
                          " must be [batch, seq_len + halo, kv_heads, head_dim], got ", t.sizes());
        TORCH_CHECK_VALUE(t.size(2) > 0 && t.size(2) == k1.size(2) && H % t.size(2) == 0,
                          "K/V tensors must share a head count that divides the query head count");
    }
}

sa_params make_params(const Tensor& q, const Tensor& k1, const Tensor& k2, const Tensor& v1, const Tensor& v2, const Tensor& o,
                      const Config& c) {
    sa_params p{};
    p.B = (int32_t)q.size(0); p.N = (int32_t)q.size(1); p.H = (int32_t)q.size(2); p.D = (int32_t)q.size(3);
    p.Hkv = (int32_t)k1.size(2);
    p.w1 = (int32_t)c.w1; p.w2 = (int32_t)c.w2; p.halo1 = (int32_t)c.halo1; p.halo2 = (int32_t)c.halo2;
    p.dtype = q.scalar_type() == at::kBFloat16 ? SA_BF16 : q.scalar_type() == at::kHalf ? SA_F16 : SA_F32;
    p.algo = c.algo;
    p.scale = (float)c.scale; p.k2_bias = (float)c.k2_bias; p.v2_bias = (float)c.v2_bias;
    p.q = strides_of(q); p.k1 = strides_of(k1); p.k2 = strides_of(k2); p.v1 = strides_of(v1); p.v2 = strides_of(v2);
    p.o = strides_of(o);
    return p;
}

constexpr size_t kStatusBytes = 256;      // the part of a workspace that a separate status word makes unnecessary

// A workspace from torch's allocator, if the call needs more than the status word.
struct Workspace {
    Tensor t;
    void* ptr = nullptr;
    size_t bytes = 0;
    Workspace(size_t need, const Tensor& like) {
        if (need > kStatusBytes) {
            t = at::empty({(int64_t)need}, like.options().dtype(at::kByte));
            ptr = t.data_ptr();
            bytes = need;
        }
    }
};

std::pair<Tensor, Tensor> forward_call(const Tensor& q_, const Tensor& k1_, const Tensor& k2_, const Tensor& v1_, const Tensor& v2_,
                                       const Config& c) {
    const Tensor q = unit_inner(q_), k1 = unit_inner(k1_), k2 = unit_inner(k2_), v1 = unit_inner(v1_), v2 = unit_inner(v2_);
    check_inputs(q, k1, k2, v1, v2, c);
    const c10::cuda::CUDAGuard guard(q.device());
    const int device = q.device().index();
    poll_device(device);
    Tensor o = at::empty_like(q);
    Tensor lse = at::empty({q.size(0), q.size(2), q.size(1)}, q.options().dtype(at::kFloat));
    const sa_params p = make_params(q, k1, k2, v1, v2, o, c);
    const Workspace ws(sa_forward_workspace_size(&p), q);
    const int rc = sa_forward_status(&p, q.data_ptr(), k1.data_ptr(), k2.data_ptr(), v1.data_ptr(), v2.data_ptr(), o.data_ptr(),
                                     (float*)lse.data_ptr(), ws.ptr, ws.bytes, status_word(device, kForward),
                                     at::cuda::getCurrentCUDAStream(device).stream());
    if (rc != SA_OK) raise_status("sa_forward", rc);
    return {std::move(o), std::move(lse)};
}

std::array<Tensor, 5> backward_call(const Tensor& q_, const Tensor& k1_, const Tensor& k2_, const Tensor& v1_, const Tensor& v2_,
                                    const Tensor& o_, const Tensor& lse, const Tensor& d_o_, const Config& c,
                                    const std::array<bool, 5>& need) {
    const Tensor q = unit_inner(q_), k1 = unit_inner(k1_), k2 = unit_inner(k2_), v1 = unit_inner(v1_), v2 = unit_inner(v2_),
                 o = unit_inner(o_), d_o = unit_inner(d_o_);
    check_inputs(q, k1, k2, v1, v2, c);
    const c10::cuda::CUDAGuard guard(q.device());
    const int device = q.device().index();
    poll_device(device);
    const Tensor* const in[5] = {&q, &k1, &k2, &v1, &v2};
    std::array<Tensor, 5> g;
    void* gp[5];
    for (int i = 0; i < 5; ++i) {
        if (need[i]) g[i] = at::empty_like(*in[i]);
        gp[i] = need[i] ? g[i].data_ptr() : nullptr;
    }
    sa_params p = make_params(q, k1, k2, v1, v2, o, c);
    p.d_o = strides_of(d_o);
    p.dq = strides_of(g[0]); p.dk1 = strides_of(g[1]); p.dk2 = strides_of(g[2]); p.dv1 = strides_of(g[3]); p.dv2 = strides_of(g[4]);
    const Workspace ws(sa_backward_workspace_size(&p), q);
    const int rc = sa_backward_status(&p, q.data_ptr(), k1.data_ptr(), k2.data_ptr(), v1.data_ptr(), v2.data_ptr(), o.data_ptr(),
                                      (const float*)lse.data_ptr(), d_o.data_ptr(), gp[0], gp[1], gp[2], gp[3], gp[4], ws.ptr, ws.bytes,
                                      status_word(device, kBackward), at::cuda::getCurrentCUDAStream(device).stream());
    if (rc != SA_OK) raise_status("sa_backward", rc);
    return g;
}

// ---- autograd
struct AttentionBackward : public torch::autograd::Node {
    torch::autograd::SavedVariable q, k1, k2, v1, v2, o, lse;
    Config cfg;

    torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        torch::autograd::variable_list out(5);
        if (!grads[0].defined()) return out;
        std::array<bool, 5> need;
        bool any = false;
        for (int i = 0; i < 5; ++i) any |= need[i] = task_should_compute_output(i);
        if (!any) return out;
        const auto self = getptr();
        const Tensor q_ = q.unpack(), k1_ = k1.unpack(), k2_ = k2.unpack(), v1_ = v1.unpack(), v2_ = v2.unpack(), o_ = o.unpack(self),
                     lse_ = lse.unpack();
        at::AutoDispatchBelowADInplaceOrView below;
        std::array<Tensor, 5> g = backward_call(q_, k1_, k2_, v1_, v2_, o_, lse_, grads[0], cfg, need);
        for (int i = 0; i < 5; ++i) out[i] = std::move(g[i]);
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto* v : {&q, &k1, &k2, &v1, &v2, &o, &lse}) v->reset_data();
    }
    std::string name() const override { return "TwoSimplicialAttentionBackward"; }
};

Tensor attention(const Tensor& q, const Tensor& k1, const Tensor& k2, const Tensor& v1, const Tensor& v2, const Config& c) {
    std::shared_ptr<AttentionBackward> node;
    if (torch::autograd::compute_requires_grad(q, k1, k2, v1, v2)) {
        node = std::shared_ptr<AttentionBackward>(new AttentionBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(q, k1, k2, v1, v2));
        node->cfg = c;
        node->q = torch::autograd::SavedVariable(q, false);
        node->k1 = torch::autograd::SavedVariable(k1, false);
        node->k2 = torch::autograd::SavedVariable(k2, false);
        node->v1 = torch::autograd::SavedVariable(v1, false);
        node->v2 = torch::autograd::SavedVariable(v2, false);
    }
    std::pair<Tensor, Tensor> r;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        r = forward_call(q, k1, k2, v1, v2, c);
    }
    if (node) {
        torch::autograd::set_history(r.first, node);
        node->o = torch::autograd::SavedVariable(r.first, true);
        node->lse = torch::autograd::SavedVariable(r.second, false);
    }
    return r.first;
}

// ---- Python entry points (plain C calls: a generic argument converter would cost as much as the launch)
const Tensor& tensor_arg(PyObject* o, const char* name) {
    TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a tensor");
    return THPVariable_Unpack(o);
}
int64_t int_arg(PyObject* o) {
    PyObject* l = PyNumber_Long(o);
    const int64_t v = l ? PyLong_AsLongLong(l) : -1;
    Py_XDECREF(l);
    if (PyErr_Occurred()) throw python_error();
    return v;
}
double float_arg(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
}
// w1, w2, scale, k2_bias, v2_bias, halo1, halo2, algo
Config config_args(PyObject* const* a) {
    Config c;
    c.w1 = int_arg(a[0]);
    c.w2 = int_arg(a[1]);
    c.scale = float_arg(a[2]);
    c.k2_bias = float_arg(a[3]);
    c.v2_bias = float_arg(a[4]);
    c.halo1 = int_arg(a[5]);
    c.halo2 = int_arg(a[6]);
    c.algo = (int)int_arg(a[7]);
    return c;
}
// Whether every one of the five inputs is a torch.Tensor or Parameter itself: what a subclass does with the tensors that
// are allocated for it is up to its __torch_function__.
bool exact(PyObject* const* a) {
    for (int i = 0; i < 5; ++i)
        if (!THPVariable_CheckTypeExact(Py_TYPE(a[i]))) return false;
    return true;
}
// ... and the call is neither traced nor under a functorch transform, and no input carries a forward-mode tangent.
bool plain(PyObject* const* a) {
    if (!exact(a) || at::tracer::impl::is_dispatch_enabled() ||
        c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode))
        return false;
    for (int i = 0; i < 5; ++i) {
        const Tensor& t = THPVariable_Unpack(a[i]);
        if (t.unsafeGetTensorImpl()->autograd_meta() != nullptr && t._fw_grad(0).defined()) return false;
    }
    return true;
}

void expect(Py_ssize_t have, Py_ssize_t want) { TORCH_CHECK_TYPE(have == want, "expected ", want, " arguments, got ", have); }

PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect(n, 13);
    if (!plain(a)) Py_RETURN_NONE;
    const Config c = config_args(a + 5);
    const Tensor &q = tensor_arg(a[0], "q"), &k1 = tensor_arg(a[1], "k1"), &k2 = tensor_arg(a[2], "k2"), &v1 = tensor_arg(a[3], "v1"),
                 &v2 = tensor_arg(a[4], "v2");
    Tensor o;
    {
        pybind11::gil_scoped_release no_gil;
        o = attention(q, k1, k2, v1, v2, c);
    }
    return THPVariable_Wrap(std::move(o));
    END_HANDLE_TH_ERRORS
}

PyObject* py_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect(n, 13);
    if (!exact(a)) Py_RETURN_NONE;
    const Config c = config_args(a + 5);
    const Tensor &q = tensor_arg(a[0], "q"), &k1 = tensor_arg(a[1], "k1"), &k2 = tensor_arg(a[2], "k2"), &v1 = tensor_arg(a[3], "v1"),
                 &v2 = tensor_arg(a[4], "v2");
    std::pair<Tensor, Tensor> r;
    {
        pybind11::gil_scoped_release no_gil;
        at::AutoDispatchBelowADInplaceOrView below;
        r = forward_call(q, k1, k2, v1, v2, c);
    }
    PyObject* t = PyTuple_New(2);
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(r.first)));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(r.second)));
    return t;
    END_HANDLE_TH_ERRORS
}

// q, k1, k2, v1, v2, o, lse, d_o, <8 configuration values>, need (bit i: gradient i)
PyObject* py_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect(n, 17);
    if (!exact(a)) Py_RETURN_NONE;
    static const char* const names[8] = {"q", "k1", "k2", "v1", "v2", "o", "lse", "d_o"};
    const Tensor* t[8];
    for (int i = 0; i < 8; ++i) t[i] = &tensor_arg(a[i], names[i]);
    const Config c = config_args(a + 8);
    const int64_t bits = int_arg(a[16]);
    std::array<bool, 5> need;
    for (int i = 0; i < 5; ++i) need[i] = (bits >> i) & 1;
    std::array<Tensor, 5> g;
    {
        pybind11::gil_scoped_release no_gil;
        at::AutoDispatchBelowADInplaceOrView below;
        g = backward_call(*t[0], *t[1], *t[2], *t[3], *t[4], *t[5], *t[6], *t[7], c, need);
    }
    PyObject* r = PyTuple_New(5);
    for (int i = 0; i < 5; ++i) {
        if (g[i].defined()) PyTuple_SET_ITEM(r, i, THPVariable_Wrap(std::move(g[i])));
        else PyTuple_SET_ITEM(r, i, Py_NewRef(Py_None));
    }
    return r;
    END_HANDLE_TH_ERRORS
}

PyObject* py_plain(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect(n, 5);
    return PyBool_FromLong(plain(a));
    END_HANDLE_TH_ERRORS
}

PyObject* py_poll(PyObject*, PyObject* device) {
    HANDLE_TH_ERRORS
    poll_device((int)int_arg(device));
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// device, direction (0: forward, 1: backward)
PyObject* py_status_word(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    expect(n, 2);
    const int64_t device = int_arg(a[0]), direction = int_arg(a[1]);
    TORCH_CHECK_INDEX(device >= 0 && device < kMaxDevices && (direction == kForward || direction == kBackward), "no such status word");
    return PyLong_FromVoidPtr(status_word((int)device, (Direction)direction));
    END_HANDLE_TH_ERRORS
}

PyObject* py_devices(PyObject*, PyObject*) {
    const uint64_t bits = g_devices.load();
    PyObject* l = PyList_New(0);
    for (int i = 0; i < kMaxDevices; ++i) {
        if (!((bits >> i) & 1)) continue;
        PyObject* v = PyLong_FromLong(i);
        PyList_Append(l, v);
        Py_DECREF(v);
    }
    return l;
}

PyObject* py_on_error(PyObject*, PyObject* fn) {
    Py_XDECREF(g_on_error);
    g_on_error = Py_NewRef(fn);
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"attention", (PyCFunction)(void*)py_attention, METH_FASTCALL, "O with its autograd history; None if the call is not plain"},
    {"plain", (PyCFunction)(void*)py_plain, METH_FASTCALL, "whether `attention` makes the call for these five inputs"},
    {"forward", (PyCFunction)(void*)py_forward, METH_FASTCALL, "(O, LSE); None for tensor subclasses"},
    {"backward", (PyCFunction)(void*)py_backward, METH_FASTCALL, "(dq, dk1, dk2, dv1, dv2); None for tensor subclasses"},
    {"poll", py_poll, METH_O, "raises if an earlier call on the device left a status"},
    {"status_word", (PyCFunction)(void*)py_status_word, METH_FASTCALL, "address of the word that calls of a device and direction report to"},
    {"devices", py_devices, METH_NOARGS, "indices of the devices that have been called on"},
    {"on_error", py_on_error, METH_O, "sets the callable that raises for a status"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "sa_torch", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_sa_torch(void) { return PyModule_Create(&kModule); }

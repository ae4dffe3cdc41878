// Host path of the package in native code: the CPython module `_native`.
//
// A forward of the model is 8 launches per block.  Driven from Python each of them costs 10 - 20 us of host time (argument
// checks, torch.empty, ctypes conversions), which is more than the GPU needs for a decode step or a short prompt; here a
// launch costs about 2 us and a whole forward allocates three tensors.  The module holds no kernels: it calls the C ABI of
// libmmfree_b200.so through a table of function pointers, so that the configuration-sweep tests can point it at the
// experiments build of the same library (use_library).
//
//   use_library(path)                    resolve the C ABI from this shared object
//   set_hooks(error_class, workspace, require_device)     exception class for negative status codes, workspace(device_index) ->
//                                        tensor, require_device(device_index) raises if the GPU is not one the library runs on
//   take_launches()                      kernels launched since the last call of it
//   bitlinear(x, norm_w, packed, scale, N, eps)       RMSNorm + int8 quantisation + contraction, [..., K] -> [..., N]
//   hgrn_scan(x, g, h0 | None, want_state, gate_is_log, state_dtype)      -> (o, final state | None)
//   check_gave_up(device_index), take_gave_up()       raise if a decode step gave up waiting; forget that any did
//   watch(slots), unchanged(watch)       cheap "has any parameter been replaced, cast or modified" over (dict, name) slots
//   chain(...), chain_forward(...), prepare_step(...)     the fused forward of a model (engine.FusedRunner)
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Dtype.h>

#include <atomic>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/mmfree_b200.h"

namespace {

struct Api {
#define MMF_FN(name) decltype(&::name) name = nullptr;
#define MMF_FNS(F)                                                                                                      \
    F(mmf_last_error) F(mmf_act_quant) F(mmf_bitlinear) F(mmf_hgrn_workspace_bytes) F(mmf_hgrn_scan) F(mmf_hgrn_gated_masked) \
    F(mmf_prenorm_quant) F(mmf_gatenorm_quant) F(mmf_decode_mix_masked) F(mmf_swiglu_quant) F(mmf_embedding) \
    F(mmf_decode_linear) F(mmf_decode_step_layer_bytes) F(mmf_decode_step_pack) F(mmf_decode_step_workspace_bytes) F(mmf_decode_step)
    MMF_FNS(MMF_FN)
#undef MMF_FN
};
std::map<std::string, Api> g_apis;   // by path; the pointers stay valid because the libraries are never closed
const Api* g_api = nullptr;

int64_t g_launches = 0;    // guarded by the GIL

// Rows of a decode step that take the fused kernels, and from how many on the row work is a kernel of its own.  Step times, row
// work repeated in every CTA / in row kernels: one row, width 256 (12 blocks) 156 / 198 us, 1024 (24) 338 / 397, 2048 (24) 434 / 513,
// 2560 (32) 687 / 797, 3072 (16) 472 / 493, 4096 (16) 574 / 590; two rows, 256 181 / 194, 1024 376 / 404, 2048 498 / 526, but 2304 (24)
// 588 / 564, 2560 934 / 805, 3072 558 / 500, 4096 689 / 618.  Above 16 rows the contraction on tcgen05 with row kernels around it is
// faster (2048 wide, 24 blocks, 32 rows: 828 us against 1000).
constexpr int64_t DECODE_ROWS = MMF_DECODE_LINEAR_MAX_M;
bool rows_in_contraction(int64_t M, int64_t h) { return M == 1 || (M <= MMF_DECODE_LINEAR_FUSED_MAX_M && h <= 2048); }
// lm_head (32000 outputs) alone: tcgen05 above.  Whole steps, this kernel / tcgen05: two rows of 2560 788 / 801 us, four to eight rows
// within 0.5 % either way (256, 2048 and 2560 wide), 12 rows 1166 / 1149 (2560) and 639 / 637 (2048), 16 rows 1181 / 1154 and 651 / 647.
constexpr int64_t HEAD_ROWS = 8;
bool on16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }
constexpr int64_t FUSED_MAX_N = 262144;       // partial sums of more output rows would not fit in shared memory

PyObject* g_error_class = nullptr;
PyObject* g_workspace_fn = nullptr;
PyObject* g_require_device_fn = nullptr;
uint64_t g_device_ok = 0;         // devices that require_device has accepted (guarded by the GIL)

// a C-ABI call returned a negative status: carried as a C++ exception so that it can cross code that runs without the GIL
struct MmfStatus {
    const char* fn;
    int code;
    std::string text;
};
#define MMF_CALL(fn, ...)                                                        \
    do {                                                                         \
        const int rc__ = g_api->fn(__VA_ARGS__);                                 \
        if (rc__ != MMF_OK) throw MmfStatus{#fn, rc__, g_api->mmf_last_error()}; \
    } while (0)

struct PythonError {};            // a Python call failed and its exception is set

// run `body` and turn C++ exceptions into Python ones
template <typename F> PyObject* guarded(F&& body) {
    try {
        return body();
    } catch (const PythonError&) {
    } catch (const MmfStatus& s) {
        PyObject* e = PyObject_CallFunction(g_error_class, "sis", s.fn, s.code, s.text.c_str());
        if (e) {
            PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(e)), e);
            Py_DECREF(e);
        }
    } catch (const std::invalid_argument& e) {
        PyErr_SetString(PyExc_ValueError, e.what());
    } catch (const std::domain_error& e) {
        PyErr_SetString(PyExc_TypeError, e.what());
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

struct NoGil {
    PyThreadState* s = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(s); }
};

const at::Tensor& tensor(PyObject* o, const char* what) {
    if (!THPVariable_Check(o)) throw std::domain_error(std::string(what) + " must be a tensor");
    return THPVariable_Unpack(o);
}
at::Tensor maybe_tensor(PyObject* o, const char* what) { return o == Py_None ? at::Tensor() : tensor(o, what); }

int dtype_code(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return MMF_F32;
        case at::kBFloat16: return MMF_BF16;
        case at::kHalf: return MMF_F16;
        default: throw std::domain_error("unsupported dtype; expected float32, bfloat16 or float16");
    }
}
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// The C entry points launch on the current device: every tensor has to live there, and the device is checked before its first launch.
int need_cuda(std::initializer_list<const at::Tensor*> ts) {
    int dev = -1;
    for (const at::Tensor* t : ts) {
        if (!t->defined()) continue;
        if (!t->is_cuda()) throw std::runtime_error("matmulfreellm_b200 kernels take CUDA tensors only (no CPU fallback exists)");
        if (dev < 0) dev = t->get_device();
        else if (t->get_device() != dev) throw std::runtime_error("tensors on different devices");
    }
    const int cur = c10::cuda::current_device();
    if (dev >= 0 && dev != cur)
        throw std::runtime_error("tensors live on cuda:" + std::to_string(dev) + " but the current device is cuda:" + std::to_string(cur) +
                                 "; wrap the call in `with torch.cuda.device(" + std::to_string(dev) + "):`");
    if (cur >= 64 || !(g_device_ok >> cur & 1)) {
        PyObject* o = PyObject_CallFunction(g_require_device_fn, "i", cur);
        if (!o) throw PythonError{};
        Py_DECREF(o);
        if (cur < 64) g_device_ok |= 1ull << cur;
    }
    return cur;
}

// status word (and split-K scratch) of a stream: handed out by the Python side once per (device, stream) and never released
struct Ws { int dev; void* stream; void* p; int64_t bytes; };
std::vector<Ws> g_ws;     // guarded by the GIL
Ws workspace(int dev, void* stream) {
    for (const Ws& w : g_ws)
        if (w.dev == dev && w.stream == stream) return w;
    PyObject* o = PyObject_CallFunction(g_workspace_fn, "i", dev);
    if (!o) throw PythonError{};
    const at::Tensor t = THPVariable_Unpack(o);
    Py_DECREF(o);
    g_ws.push_back(Ws{dev, stream, t.data_ptr(), t.numel()});
    return g_ws.back();
}

// One word of pinned host memory per device, which a decode step sets when it gives up waiting (mmf_decode_step_args.gave_up_host).  Never
// released: a captured graph may point at it.
std::atomic<int*> g_gave_up[64];
void make_gave_up_word(int dev) {
    static std::mutex lock;
    const std::lock_guard<std::mutex> hold(lock);
    if (dev >= 64 || g_gave_up[dev].load()) return;
    const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);      // (allocating is no part of a capture under way)
    g_gave_up[dev] = (new at::Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true))))->data_ptr<int>();
}
bool take_gave_up_word(int dev) {
    volatile int* w = dev >= 0 && dev < 64 ? g_gave_up[dev].load() : nullptr;
    const bool set = w && *w;
    if (set) *w = 0;
    return set;
}
void require_not_given_up(int dev) {
    if (take_gave_up_word(dev))
        throw MmfStatus{"mmf_decode_step", MMF_ERR_TIMEOUT, "an earlier decode step on cuda:" + std::to_string(dev) +
                        " gave up waiting: its outputs and the recurrent states are undefined"};
}

// carve 256-byte aligned pieces out of one allocation
struct Slab {
    uint8_t* base = nullptr;
    int64_t used = 0;
    int64_t take(int64_t bytes) {
        const int64_t at = used;
        used += (bytes + 255) / 256 * 256;
        return at;
    }
};

at::Tensor rows_of(const at::Tensor& x) {   // [..., K] -> [M, K] with unit inner stride
    at::Tensor r = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
    return r.stride(1) == 1 || r.size(1) == 1 ? r : r.contiguous();
}

// ---------------------------------------------------------------------------------------------------------------
PyObject* use_library(PyObject*, PyObject* path) {
    return guarded([&]() -> PyObject* {
        const char* p = PyUnicode_AsUTF8(path);
        if (!p) return nullptr;
        auto it = g_apis.find(p);
        if (it == g_apis.end()) {
            void* h = dlopen(p, RTLD_NOW | RTLD_LOCAL);
            if (!h) throw std::runtime_error(dlerror());
            Api api;
#define MMF_RESOLVE(name)                                                                            \
    api.name = reinterpret_cast<decltype(api.name)>(dlsym(h, #name));                                 \
    if (!api.name) throw std::runtime_error(std::string(p) + " does not export " #name);
            MMF_FNS(MMF_RESOLVE)
            it = g_apis.emplace(p, api).first;
        }
        g_api = &it->second;
        Py_RETURN_NONE;
    });
}

PyObject* set_hooks(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 3) { PyErr_SetString(PyExc_TypeError, "set_hooks(error_class, workspace, require_device)"); return nullptr; }
    Py_INCREF(args[0]); Py_XSETREF(g_error_class, args[0]);
    Py_INCREF(args[1]); Py_XSETREF(g_workspace_fn, args[1]);
    Py_INCREF(args[2]); Py_XSETREF(g_require_device_fn, args[2]);
    g_device_ok = 0;
    Py_RETURN_NONE;
}

// bitlinear(x, norm_w, packed, scale, N, eps)
PyObject* bitlinear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 6) throw std::domain_error("bitlinear takes 6 arguments");
        const at::Tensor& x = tensor(args[0], "x");
        const at::Tensor nw = maybe_tensor(args[1], "norm weight");
        const at::Tensor &packed = tensor(args[2], "packed"), &scale = tensor(args[3], "scale");
        const int64_t N = PyLong_AsLongLong(args[4]);
        const double eps = PyFloat_AsDouble(args[5]);
        if (PyErr_Occurred()) return nullptr;
        const int dev = need_cuda({&x, &nw, &packed, &scale});
        const int dt = dtype_code(x);
        const int64_t K = x.size(-1);
        if (nw.defined() && (nw.scalar_type() != at::kFloat || nw.numel() != K || !nw.is_contiguous()))
            throw std::domain_error("norm weight must be contiguous float32 [K]");
        if (packed.numel() != (N + MMF_TILE_ROWS - 1) / MMF_TILE_ROWS * MMF_TILE_ROWS * K / 4)
            throw std::invalid_argument("x does not have the layer's in_features columns");
        const at::Tensor x2 = rows_of(x);
        const int64_t M = x2.size(0), ld = M == 1 ? K : x2.stride(0);      // the pitch of a single row means nothing
        std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
        shape.back() = N;
        at::Tensor out = at::empty(shape, x.options());
        // one or two rows: one kernel, no scratch
        if (M > 0 && M <= MMF_DECODE_LINEAR_FUSED_MAX_M && dt != MMF_F32 && K <= 8192 && N <= FUSED_MAX_N && on16(x2.data_ptr()) &&
            ld % 8 == 0 && on16(ptr(nw)) && on16(packed.data_ptr())) {
            mmf_decode_linear_args a = {};
            a.prologue = MMF_PRO_QUANT;
            a.epilogue = MMF_EPI_STORE;
            a.dtype = dt;
            a.M = M; a.N = N; a.K = K;
            a.packed = packed.data_ptr();
            a.w_scale = scale.data_ptr<float>();
            a.x = x2.data_ptr();
            a.ld_x = ld;
            a.bl_norm_w[0] = (const float*)ptr(nw);
            a.eps_bl = (float)eps;
            a.out = out.data_ptr();
            a.ld_out = N;
            MMF_CALL(mmf_decode_linear, &a, c10::cuda::getCurrentCUDAStream(dev).stream());
            ++g_launches;
        } else if (M > 0) {
            void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
            const Ws ws = workspace(dev, st);
            Slab s;
            const int64_t q = s.take(M * K), dq = s.take(M * 4), rs = s.take(M * 4);
            const at::Tensor mem = at::empty({s.used}, x.options().dtype(at::kByte));
            uint8_t* b = mem.data_ptr<uint8_t>();
            MMF_CALL(mmf_act_quant, x2.data_ptr(), dt, ld, (const float*)ptr(nw), 1, (float)eps, (int8_t*)(b + q), (float*)(b + dq),
                     (int32_t*)(b + rs), M, K, st);
            MMF_CALL(mmf_bitlinear, (const int8_t*)(b + q), (const float*)(b + dq), (const int32_t*)(b + rs), packed.data_ptr(),
                     scale.data_ptr<float>(), 1, out.data_ptr(), dt, N, nullptr, M, N, K, ws.p, ws.bytes, MMF_KERNEL_AUTO, st);
            g_launches += 2;
        }
        return THPVariable_Wrap(std::move(out));
    });
}

// hgrn_scan(x, g, h0, want_state, gate_is_log, state_dtype): x, g [..., T, D]
PyObject* hgrn_scan(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 6) throw std::domain_error("hgrn_scan takes 6 arguments");
        const at::Tensor x = tensor(args[0], "x").contiguous(), g = tensor(args[1], "g").contiguous();
        at::Tensor h0 = maybe_tensor(args[2], "initial_state");
        const bool want = PyObject_IsTrue(args[3]), is_log = PyObject_IsTrue(args[4]);
        if (!THPDtype_Check(args[5])) throw std::domain_error("state dtype");
        const at::ScalarType sdt = reinterpret_cast<THPDtype*>(args[5])->scalar_type;
        const int dev = need_cuda({&x, &g, &h0});
        if (x.dim() < 2 || x.sizes() != g.sizes()) throw std::invalid_argument("x and g must have the same shape [..., T, D]");
        const int64_t D = x.size(-1), T = x.size(-2), B = D * T ? x.numel() / (D * T) : 0;
        if (h0.defined()) {
            if (h0.numel() != B * D) throw std::invalid_argument("initial_state must hold one value per (sequence, channel)");
            h0 = h0.detach().to(sdt).contiguous();
        }
        at::Tensor ht;
        if (want) {
            std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 2);
            shape.push_back(D);
            ht = at::empty(shape, x.options().dtype(sdt));
        }
        at::Tensor o = at::empty_like(x);
        const int state_code = sdt == at::kFloat ? MMF_F32 : sdt == at::kBFloat16 ? MMF_BF16 : sdt == at::kHalf ? MMF_F16 : -1;
        const int64_t bytes = g_api->mmf_hgrn_workspace_bytes(B, T, D);
        at::Tensor ws;
        if (bytes) ws = at::empty({bytes}, x.options().dtype(at::kByte));
        MMF_CALL(mmf_hgrn_scan, x.data_ptr(), dtype_code(x), g.data_ptr(), dtype_code(g), ptr(h0), ptr(ht), state_code, o.data_ptr(), B, T, D,
                 (int)is_log, ptr(ws), bytes, c10::cuda::getCurrentCUDAStream(dev).stream());
        if (x.numel()) g_launches += bytes ? 2 : 1;          // a scan whose time is split makes two passes
        PyObject* po = THPVariable_Wrap(std::move(o));
        PyObject* ph = want ? THPVariable_Wrap(std::move(ht)) : Py_NewRef(Py_None);
        PyObject* t = PyTuple_Pack(2, po, ph);
        Py_DECREF(po);
        Py_DECREF(ph);
        return t;
    });
}

// ---------------------------------------------------------------------------------------------------------------
// parameter watch
// ---------------------------------------------------------------------------------------------------------------
// What a slot holds is told by addresses and a version number.  The weak references keep the addresses of the tensor and of its
// storage from being used again for others (they do not keep the memory of the values): without them a parameter that was dropped
// and replaced could leave every address as it was.
struct Held {
    const void *impl = nullptr, *storage = nullptr, *data = nullptr;
    int64_t version = 0;
    at::ScalarType dtype = at::kByte;
    bool operator==(const Held& o) const {
        return impl == o.impl && storage == o.storage && data == o.data && version == o.version && dtype == o.dtype;
    }
};
struct Slot {
    PyObject *dict, *name;        // owned references
    Held held;                    // what the slot held when the watch was made
};
struct Watch {
    std::vector<Slot> slots;
    std::vector<c10::weak_intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl>> impls;
    std::vector<c10::weak_intrusive_ptr<c10::StorageImpl>> storages;
    ~Watch() {
        for (Slot& s : slots) { Py_DECREF(s.dict); Py_DECREF(s.name); }
    }
};
const at::Tensor* in_slot(PyObject* dict, PyObject* name) {
    PyObject* v = PyDict_GetItemWithError(dict, name);     // borrowed; a str key raises nothing
    return v && THPVariable_Check(v) ? &THPVariable_Unpack(v) : nullptr;
}
Held look(const at::Tensor* t) {
    Held h;
    if (t) {
        c10::TensorImpl* impl = t->unsafeGetTensorImpl();
        h.impl = impl;
        if (impl->has_storage()) {
            const c10::StorageImpl* storage = impl->unsafe_storage().unsafeGetStorageImpl();
            h.storage = storage;
            h.data = static_cast<const uint8_t*>(storage->data()) + impl->storage_offset() * impl->itemsize();
        }
        h.version = t->is_inference() ? 0 : (int64_t)t->_version();
        h.dtype = t->scalar_type();
    }
    return h;
}
PyObject* watch(PyObject*, PyObject* slots) {
    return guarded([&]() -> PyObject* {
        auto w = std::make_unique<Watch>();
        PyObject* seq = PySequence_Fast(slots, "slots must be a sequence of (dict, name)");
        if (!seq) return nullptr;
        for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) {
            PyObject* item = PySequence_Fast_GET_ITEM(seq, i);
            if (!PyTuple_Check(item) || PyTuple_GET_SIZE(item) != 2 || !PyDict_Check(PyTuple_GET_ITEM(item, 0)) ||
                !PyUnicode_Check(PyTuple_GET_ITEM(item, 1))) {
                Py_DECREF(seq);
                throw std::domain_error("slots must be a sequence of (dict, name)");
            }
            w->slots.emplace_back();
            Slot& s = w->slots.back();
            s.dict = Py_NewRef(PyTuple_GET_ITEM(item, 0));
            s.name = Py_NewRef(PyTuple_GET_ITEM(item, 1));
            if (const at::Tensor* t = in_slot(s.dict, s.name)) {
                s.held = look(t);
                w->impls.emplace_back(t->getIntrusivePtr());
                if (t->has_storage()) w->storages.push_back(t->storage().getWeakStorageImpl());
            }
        }
        Py_DECREF(seq);
        return PyCapsule_New(w.release(), "mmf.watch", [](PyObject* c) { delete static_cast<Watch*>(PyCapsule_GetPointer(c, "mmf.watch")); });
    });
}
PyObject* unchanged(PyObject*, PyObject* cap) {
    return guarded([&]() -> PyObject* {
        auto* w = static_cast<Watch*>(PyCapsule_GetPointer(cap, "mmf.watch"));
        if (!w) return nullptr;
        for (const Slot& s : w->slots) {
            if (!(look(in_slot(s.dict, s.name)) == s.held)) Py_RETURN_FALSE;
        }
        Py_RETURN_TRUE;
    });
}

// ---------------------------------------------------------------------------------------------------------------
// the fused forward of a model
// ---------------------------------------------------------------------------------------------------------------
struct Linear {
    const void* packed;
    const float* scale;
    int64_t N, K;
    int groups;
};
struct Layer {
    const float *attn_norm_w, *ifg_nw[3], *gnorm_w, *o_nw, *mlp_norm_w, *gate_nw, *down_nw;
    Linear ifg, o, gate, down;
    const void* lb;
    const void* step = nullptr;        // weights, norm weights and scales as the resident decode step reads them (see step_ready)
    float gnorm_eps, eps_bl;
};
enum { STEP_OPEN, STEP_READY, STEP_NEVER };
struct Chain {
    std::vector<Layer> layers;
    std::vector<at::Tensor> keep;      // everything the raw pointers above point into
    at::Tensor table;                  // token embeddings [V, h]
    const float *final_norm_w, *head_nw;
    Linear head;
    int64_t h = 0, inner = 0;
    std::atomic<int> step{STEP_OPEN};  // are the blocks' weights laid out for the resident decode step as well?
    std::mutex step_lock;              // held by the thread that does it
    float eps = 0, head_eps = 0;
    int dtype = 0;
};
struct Fields {      // positional reader of a Python tuple
    PyObject* t;
    Chain& c;
    Py_ssize_t i = 0;
    PyObject* next() {
        if (i >= PyTuple_GET_SIZE(t)) throw std::domain_error("chain: too few fields");
        return PyTuple_GET_ITEM(t, i++);
    }
    const void* data() {
        PyObject* o = next();
        if (o == Py_None) return nullptr;
        c.keep.push_back(tensor(o, "chain field"));
        return c.keep.back().data_ptr();
    }
    const float* f32() {
        PyObject* o = next();
        if (o == Py_None) return nullptr;
        c.keep.push_back(tensor(o, "chain field"));
        return c.keep.back().data_ptr<float>();
    }
    float num() { return (float)PyFloat_AsDouble(next()); }
    Linear linear() {      // packed, scale, N, K, groups
        Linear l;
        l.packed = data();
        l.scale = f32();
        l.N = PyLong_AsLongLong(next());
        l.K = PyLong_AsLongLong(next());
        l.groups = (int)PyLong_AsLong(next());
        return l;
    }
};
// The blocks' weights once more, in the layout of the resident decode step: as many bytes again as the blocks' packed weights, so only once
// a step wants them (a model that never decodes up to 16 sequences holds none), in one allocation.  True: they are there.  Called without the
// GIL, by several threads at once.  Made on the caller's stream and complete before any other stream can use them; not while that stream is
// captured (the memory would be the graph's and the packing a part of it), and not again once memory was refused: the chain of kernels needs
// none of it.
bool step_ready(Chain& c, int dev) {
    int s = c.step.load(std::memory_order_acquire);
    if (s != STEP_OPEN) return s == STEP_READY;
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return false;
    const std::lock_guard<std::mutex> lock(c.step_lock);
    if ((s = c.step.load(std::memory_order_acquire)) != STEP_OPEN) return s == STEP_READY;
    const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(dev);
    const int64_t bytes = (g_api->mmf_decode_step_layer_bytes(c.h, c.inner) + 255) / 256 * 256;
    at::Tensor mem;
    try {
        mem = at::empty({bytes * (int64_t)c.layers.size()}, c.table.options().dtype(at::kByte));
    } catch (const c10::OutOfMemoryError&) {
        c.step.store(STEP_NEVER, std::memory_order_release);
        return false;
    }
    make_gave_up_word(dev);
    uint8_t* at = mem.data_ptr<uint8_t>();
    for (Layer& L : c.layers) {
        const mmf_decode_step_weights w = {L.attn_norm_w, {L.ifg_nw[0], L.ifg_nw[1], L.ifg_nw[2]}, L.gnorm_w, L.o_nw, L.mlp_norm_w, L.gate_nw, L.down_nw,
                                           L.ifg.packed, L.o.packed, L.gate.packed, L.down.packed, L.ifg.scale, L.o.scale, L.gate.scale, L.down.scale};
        MMF_CALL(mmf_decode_step_pack, &w, c.h, c.inner, at, stream.stream());
        L.step = at;
        at += bytes;
    }
    stream.synchronize();
    c.keep.push_back(mem);
    c.step.store(STEP_READY, std::memory_order_release);
    return true;
}
// scratch of the resident decode step for M rows, 0: this chain or these sizes do not take it
int64_t step_workspace(const Chain& c, int64_t M) {
    return c.step.load(std::memory_order_relaxed) == STEP_NEVER ? 0 : g_api->mmf_decode_step_workspace_bytes(M, c.h, c.inner, (int64_t)c.layers.size());
}
// chain(table, layers, (final_norm_w, head (5 fields), head_nw, eps, head_eps), resident): layers is a list of tuples in the order read
// below; resident: decode steps may use the resident kernel, which takes a second copy of the blocks' weights
PyObject* chain(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 4 || !PyList_Check(args[1]) || !PyTuple_Check(args[2])) throw std::domain_error("chain(table, layers, tail, resident)");
        auto c = std::make_unique<Chain>();
        c->table = tensor(args[0], "table").detach().contiguous();
        c->h = c->table.size(1);
        c->dtype = dtype_code(c->table);
        for (Py_ssize_t i = 0; i < PyList_GET_SIZE(args[1]); ++i) {
            Fields f{PyList_GET_ITEM(args[1], i), *c};
            Layer L;
            L.attn_norm_w = f.f32();
            L.ifg = f.linear();
            for (int k = 0; k < 3; ++k) L.ifg_nw[k] = f.f32();
            L.lb = f.data();
            L.gnorm_w = f.f32();
            L.gnorm_eps = f.num();
            L.o = f.linear();
            L.o_nw = f.f32();
            L.mlp_norm_w = f.f32();
            L.gate = f.linear();
            L.gate_nw = f.f32();
            L.down = f.linear();
            L.down_nw = f.f32();
            L.eps_bl = f.num();
            if (L.ifg.K != c->h || L.ifg.N != 3 * c->h || L.o.K != c->h || L.o.N != c->h || L.gate.K != c->h || L.gate.N % 2 ||
                L.down.K != L.gate.N / 2 || L.down.N != c->h)
                throw std::invalid_argument("chain: a block's projections do not fit together");
            c->inner = std::max(c->inner, L.down.K);
            c->layers.push_back(L);
        }
        bool resident = PyObject_IsTrue(args[3]) && c->dtype != MMF_F32 && !c->layers.empty();
        for (const Layer& L : c->layers) resident = resident && L.down.K == c->inner;       // (its MLPs are all as wide)
        if (!resident) c->step = STEP_NEVER;
        Fields f{args[2], *c};
        c->final_norm_w = f.f32();
        c->head = f.linear();
        c->head_nw = f.f32();
        c->eps = f.num();
        c->head_eps = f.num();
        if (PyErr_Occurred()) return nullptr;
        return PyCapsule_New(c.release(), "mmf.chain", [](PyObject* o) { delete static_cast<Chain*>(PyCapsule_GetPointer(o, "mmf.chain")); });
    });
}

// The blocks of a decode step for a few token rows: four calls per block (decode_linear.cuh).  z: last block's MLP output and
// the attention output; x / next: residual stream.
template <typename ArgsOf, typename Run, typename Advance>
void decode_blocks(const Chain& c, ArgsOf&& args_of, Run&& run, const int64_t* gather, uint8_t* z, uint8_t* g, uint8_t* o, uint8_t* act,
                   const uint8_t* mask, const std::vector<float*>& states, const uint8_t*& x, uint8_t*& next, Advance&& advance) {
    const int64_t h = c.h;
    for (size_t i = 0; i < c.layers.size(); ++i) {
        const Layer& L = c.layers[i];
        const bool first = i == 0;
        auto norm = [&](mmf_decode_linear_args& a, const void* row, const void* res, bool round, const float* w, void* res_out) {
            a.x = row; a.ld_x = h;
            a.residual = res; a.ld_residual = h;
            a.round_sum_first = round;
            a.norm_w = w; a.eps_norm = c.eps;
            a.eps_bl = L.eps_bl;
            a.residual_out = res_out;
        };
        // i / f / g projections, gates, state; the reference adds residual + mlp output as a tensor op, then normalises the rounded sum
        mmf_decode_linear_args a = args_of(L.ifg, MMF_PRO_PRENORM, MMF_EPI_GATES, o, h);
        norm(a, first ? x : z, first ? nullptr : x, !first, L.attn_norm_w, first && !gather ? nullptr : next);
        if (first && gather) {
            a.row_ids = gather;
            a.x_rows = c.table.size(0);
        }
        for (int k = 0; k < 3; ++k) a.bl_norm_w[k] = L.ifg_nw[k];
        a.g_out = g;
        a.lower_bound = L.lb;
        a.mask = mask;
        a.state = states[i];
        run(a);
        if (!first || gather) advance();
        // gate norm, o_proj
        a = args_of(L.o, MMF_PRO_GATENORM, MMF_EPI_STORE, z, h);
        a.x = g; a.ld_x = h;
        a.residual = o; a.ld_residual = h;
        a.norm_w = L.gnorm_w; a.eps_norm = L.gnorm_eps;
        a.bl_norm_w[0] = L.o_nw; a.eps_bl = L.eps_bl;
        run(a);
        // mlp norm, gate / up projections, silu(gate) * up
        a = args_of(L.gate, MMF_PRO_PRENORM, MMF_EPI_SWIGLU, act, L.down.K);
        norm(a, z, x, false, L.mlp_norm_w, next);
        a.bl_norm_w[0] = L.gate_nw;
        run(a);
        advance();
        // down_proj
        a = args_of(L.down, MMF_PRO_QUANT, MMF_EPI_STORE, z, h);
        a.x = act; a.ld_x = L.down.K;
        a.bl_norm_w[0] = L.down_nw; a.eps_bl = L.eps_bl;
        run(a);
    }
}

// chain_forward(chain, ids | None, embeds | None, states, mask | None, last_only, want_logits, want_hidden)
//   ids int64 [B, T] or embeds [B, T, h]; states: list of fp32 tensors of B * h elements, advanced in place; mask uint8 [B, T]
//   -> (logits | None, hidden | None)
PyObject* chain_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 8) throw std::domain_error("chain_forward takes 8 arguments");
        auto* cp = static_cast<Chain*>(PyCapsule_GetPointer(args[0], "mmf.chain"));
        if (!cp) return nullptr;
        Chain& c = *cp;
        at::Tensor ids = maybe_tensor(args[1], "input_ids"), emb = maybe_tensor(args[2], "inputs_embeds");
        at::Tensor mask = maybe_tensor(args[4], "attention_mask");
        const bool last_only = PyObject_IsTrue(args[5]), want_logits = PyObject_IsTrue(args[6]), want_hidden = PyObject_IsTrue(args[7]);
        const at::Tensor& src = ids.defined() ? ids : emb;
        if (!src.defined() || src.dim() != (ids.defined() ? 2 : 3)) throw std::invalid_argument("input_ids [B, T] or inputs_embeds [B, T, h] expected");
        const int dev = need_cuda({&c.table, &src, &mask});
        require_not_given_up(dev);
        const int64_t B = src.size(0), T = src.size(1), M = B * T, h = c.h;
        const int64_t es = c.dtype == MMF_F32 ? 4 : 2;
        if (ids.defined()) ids = ids.to(at::kLong).contiguous();
        else {
            if (emb.size(2) != h) throw std::invalid_argument("inputs_embeds must have hidden_size columns");
            emb = emb.to(c.table.scalar_type()).contiguous();
        }
        if (mask.defined() && (mask.scalar_type() != at::kByte || mask.numel() != M || !mask.is_contiguous()))
            throw std::invalid_argument("attention_mask must be contiguous uint8 [B, T]");
        if (!PyList_Check(args[3]) || PyList_GET_SIZE(args[3]) != (Py_ssize_t)c.layers.size()) throw std::invalid_argument("one state per block expected");
        std::vector<float*> states;
        for (Py_ssize_t i = 0; i < PyList_GET_SIZE(args[3]); ++i) {
            const at::Tensor& s = tensor(PyList_GET_ITEM(args[3], i), "state");
            if (!s.is_cuda() || s.get_device() != dev || s.scalar_type() != at::kFloat || s.numel() != B * h || !s.is_contiguous())
                throw std::invalid_argument("states must be contiguous float32 CUDA tensors with batch * hidden elements");
            states.push_back(s.data_ptr<float>());
        }
        if (last_only && T == 0) throw std::invalid_argument("last_token_only needs at least one token");
        void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
        const Ws ws = workspace(dev, st);
        const int64_t Tn = last_only ? 1 : T, Mn = B * Tn;
        at::Tensor logits, hidden;
        int64_t launches = 0;
        {
            NoGil nogil;
            const auto opt = c.table.options();
            if (want_logits) logits = at::empty({B, Tn, c.head.N}, opt);
            if (want_hidden) hidden = at::empty({B, Tn, h}, opt);
            // One allocation for everything between the kernels.  The projections of the mixer (i | f | g and o) and the MLP's
            // gate | up are never alive together; the attention output and the MLP output share a buffer (each is consumed by
            // the norm that follows it); the residual stream alternates between two.
            Slab s;
            const int64_t x0 = s.take(M * h * es), x1 = s.take(M * h * es), z = s.take(M * h * es);
            const int64_t mix = s.used, ifg = s.take(3 * M * h * es), o = s.take(M * h * es), mix_end = s.used;
            s.used = mix;
            const int64_t gu = s.take(2 * M * c.inner * es);
            s.used = std::max(s.used, mix_end);
            // codes: decode-step contractions want rows of whole 256-column groups, up to 16 of them
            const int64_t Mc = M <= 8 ? 8 : M <= 16 ? 16 : M;
            const int64_t q = s.take(Mc * std::max(3 * ((h + 255) & ~255ll), (c.inner + 255) & ~255ll)), dq = s.take(3 * M * 4), rs = s.take(3 * M * 4);
            // one token per sequence and few sequences: contractions with the element-wise work around them in one kernel
            bool decode = T == 1 && M > 0 && M <= DECODE_ROWS && c.dtype != MMF_F32 && h % MMF_TILE_ROWS == 0 && h <= 4096 && c.inner <= 8192 &&
                          (ids.defined() || on16(emb.data_ptr()));
            for (const float* s : states) decode = decode && on16(s);
            // ... and all blocks in one where they fit on the chip's shared memory
            int64_t step_bytes = decode ? step_workspace(c, M) : 0;
            if (step_bytes && !step_ready(c, dev)) step_bytes = 0;
            const int64_t step = s.take(step_bytes);
            const int64_t hg_bytes = T > 1 ? g_api->mmf_hgrn_workspace_bytes(B, T, h) : 0, hg = s.take(hg_bytes);
            const at::Tensor mem = at::empty({s.used}, opt.dtype(at::kByte));
            uint8_t* b = mem.data_ptr<uint8_t>();
            int8_t* Q = reinterpret_cast<int8_t*>(b + q);
            float* DQ = reinterpret_cast<float*>(b + dq);
            int32_t* RS = reinterpret_cast<int32_t*>(b + rs);
            const uint8_t* mk = mask.defined() ? mask.data_ptr<uint8_t>() : nullptr;
            auto linear = [&](const Linear& l, void* out, int64_t rows) {
                MMF_CALL(mmf_bitlinear, Q, DQ, RS, l.packed, l.scale, l.groups, out, c.dtype, l.N, nullptr, rows, l.N, l.K, ws.p, ws.bytes,
                         MMF_KERNEL_AUTO, st);
                ++launches;
            };
            const int64_t* gather = decode && ids.defined() && !c.layers.empty() ? ids.data_ptr<int64_t>() : nullptr;
            const uint8_t* x = b + x0;            // residual stream
            if (gather) {                         // the first block reads the embedding rows itself
                x = static_cast<const uint8_t*>(c.table.data_ptr());
            } else if (ids.defined()) {
                MMF_CALL(mmf_embedding, c.table.data_ptr(), c.dtype, c.table.size(0), h, ids.data_ptr<int64_t>(), b + x0, M, st);
                ++launches;
            } else {
                x = static_cast<const uint8_t*>(emb.data_ptr());
            }
            uint8_t* next = b + x1;               // where the next residual stream goes
            auto advance = [&]() {
                x = next;
                next = next == b + x1 ? b + x0 : b + x1;
            };
            bool first = true;
            auto args_of = [&](const Linear& l, int pro, int epi, void* out, int64_t ld_out) {
                mmf_decode_linear_args a = {};
                a.prologue = pro;
                a.epilogue = epi;
                a.dtype = c.dtype;
                a.M = M; a.N = l.N; a.K = l.K;
                a.packed = l.packed;
                a.w_scale = l.scale;
                a.out = out;
                a.ld_out = ld_out;
                if (!rows_in_contraction(M, h)) {
                    a.codes = Q;
                    a.dq = DQ;
                    a.rowsum = RS;
                }
                return a;
            };
            auto run = [&](const mmf_decode_linear_args& a) {
                MMF_CALL(mmf_decode_linear, &a, st);
                launches += a.codes ? 2 : 1;
            };
            if (step_bytes) {
                std::vector<mmf_decode_step_layer> layers;
                for (size_t i = 0; i < c.layers.size(); ++i) layers.push_back({c.layers[i].step, c.layers[i].lb, states[i], c.layers[i].gnorm_eps, c.layers[i].eps_bl});
                mmf_decode_step_args a = {};
                a.dtype = c.dtype;
                a.M = M; a.hidden = h; a.inner = c.inner; a.layers = (int64_t)layers.size();
                a.layer = layers.data();
                a.x = x; a.ld_x = h;
                a.row_ids = gather; a.x_rows = c.table.size(0);
                a.mask = mk;
                a.eps_norm = c.eps;
                a.out = b + z; a.residual_out = next;
                a.workspace = b + step; a.workspace_bytes = step_bytes;
                a.status = static_cast<int*>(ws.p);
                a.gave_up_host = dev < 64 ? g_gave_up[dev].load() : nullptr;
                const int rc = g_api->mmf_decode_step(&a, st);
                ++launches;                       // fill
                if (rc == MMF_ERR_NOT_RESIDENT) {       // this context cannot hold it: the chain of kernels, now and from now on
                    c.step.store(STEP_NEVER, std::memory_order_release);
                    step_bytes = 0;
                } else if (rc != MMF_OK) {
                    throw MmfStatus{"mmf_decode_step", rc, g_api->mmf_last_error()};
                } else {
                    ++launches;                   // blocks
                    advance();
                }
            }
            if (decode && !step_bytes) decode_blocks(c, args_of, run, gather, b + z, b + ifg, b + o, b + gu, mk, states, x, next, advance);
            for (size_t i = 0; i < c.layers.size() && !decode; ++i) {
                const Layer& L = c.layers[i];
                if (first) {
                    MMF_CALL(mmf_prenorm_quant, x, h, nullptr, 0, c.dtype, 0, L.attn_norm_w, c.eps, nullptr, nullptr, 3, L.ifg_nw[0], L.ifg_nw[1],
                             L.ifg_nw[2], L.eps_bl, Q, DQ, RS, M, h, st);
                } else {       // the reference adds residual + mlp output as a tensor op, then normalises the rounded sum
                    MMF_CALL(mmf_prenorm_quant, b + z, h, x, h, c.dtype, 1, L.attn_norm_w, c.eps, next, nullptr, 3, L.ifg_nw[0], L.ifg_nw[1],
                             L.ifg_nw[2], L.eps_bl, Q, DQ, RS, M, h, st);
                    advance();
                }
                first = false;
                linear(L.ifg, b + ifg, M);
                if (T == 1) {  // decode: gates, state update, gate norm and o_proj's prologue in one kernel
                    MMF_CALL(mmf_decode_mix_masked, b + ifg, 3 * h, c.dtype, L.lb, mk, states[i], L.gnorm_w, L.gnorm_eps, L.o_nw, L.eps_bl, Q, DQ,
                             RS, M, h, st);
                } else {
                    MMF_CALL(mmf_hgrn_gated_masked, b + ifg, b + ifg + h * es, 3 * h, c.dtype, L.lb, mk, states[i], b + o, B, T, h,
                             hg_bytes ? b + hg : nullptr, hg_bytes, st);
                    MMF_CALL(mmf_gatenorm_quant, b + ifg + 2 * h * es, 3 * h, b + o, h, c.dtype, L.gnorm_w, L.gnorm_eps, L.o_nw, L.eps_bl, Q, DQ, RS,
                             M, h, st);
                    launches += hg_bytes ? 2 : 1;
                }
                linear(L.o, b + z, M);
                MMF_CALL(mmf_prenorm_quant, b + z, h, x, h, c.dtype, 0, L.mlp_norm_w, c.eps, next, nullptr, 1, L.gate_nw, nullptr, nullptr, L.eps_bl,
                         Q, DQ, RS, M, h, st);
                advance();
                linear(L.gate, b + gu, M);
                const int64_t inner = L.down.K;
                MMF_CALL(mmf_swiglu_quant, b + gu, b + gu + inner * es, 2 * inner, c.dtype, L.down_nw, L.eps_bl, Q, DQ, RS, M, inner, st);
                linear(L.down, b + z, M);
                launches += 4;
            }
            // final norm: only the last position of every sequence when only that feeds lm_head
            const int64_t skip = last_only ? (T - 1) * h * es : 0, ld = last_only ? T * h : h;
            first = c.layers.empty();
            const uint8_t* rows = first ? x : b + z;
            if (decode && M <= HEAD_ROWS && c.head.N <= FUSED_MAX_N && want_logits && !want_hidden) {
                mmf_decode_linear_args a = args_of(c.head, MMF_PRO_PRENORM, MMF_EPI_STORE, logits.data_ptr(), c.head.N);
                a.x = rows; a.ld_x = h;
                a.residual = first ? nullptr : x; a.ld_residual = h;
                a.round_sum_first = !first;
                a.norm_w = c.final_norm_w; a.eps_norm = c.eps;
                a.bl_norm_w[0] = c.head_nw; a.eps_bl = c.head_eps;
                run(a);
            } else {
                MMF_CALL(mmf_prenorm_quant, rows + skip, ld, first ? nullptr : x + skip, ld, c.dtype, first ? 0 : 1, c.final_norm_w, c.eps, nullptr,
                         ptr(hidden), want_logits ? 1 : 0, c.head_nw, nullptr, nullptr, c.head_eps, Q, DQ, RS, Mn, h, st);
                ++launches;
                if (want_logits) linear(c.head, logits.data_ptr(), Mn);
            }
        }
        g_launches += launches;
        PyObject* pl = logits.defined() ? THPVariable_Wrap(std::move(logits)) : Py_NewRef(Py_None);
        PyObject* ph = hidden.defined() ? THPVariable_Wrap(std::move(hidden)) : Py_NewRef(Py_None);
        return Py_BuildValue("(NN)", pl, ph);
    });
}

// prepare_step(chain, M): what the first decode step of M sequences would do once for all (step_ready), on the current stream; for a caller that
// takes its steps on another one.  True if those steps take the resident kernel.
PyObject* prepare_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 2) throw std::domain_error("prepare_step takes 2 arguments");
        auto* c = static_cast<Chain*>(PyCapsule_GetPointer(args[0], "mmf.chain"));
        if (!c) return nullptr;
        const int64_t M = PyLong_AsLongLong(args[1]);
        if (PyErr_Occurred()) return nullptr;
        const int dev = need_cuda({&c->table});
        bool ready;
        {
            NoGil nogil;
            ready = step_workspace(*c, M) && step_ready(*c, dev);
        }
        return PyBool_FromLong(ready);
    });
}

PyObject* take_launches(PyObject*, PyObject*) {
    const int64_t n = g_launches;
    g_launches = 0;
    return PyLong_FromLongLong(n);
}

// check_gave_up(device index): raises if a decode step there gave up waiting since the last look; take_gave_up(): forget all of them
PyObject* check_gave_up(PyObject*, PyObject* index) {
    return guarded([&]() -> PyObject* {
        const long dev = PyLong_AsLong(index);
        if (dev == -1 && PyErr_Occurred()) return nullptr;
        require_not_given_up((int)dev);
        Py_RETURN_NONE;
    });
}
PyObject* take_gave_up(PyObject*, PyObject*) {
    for (int dev = 0; dev < 64; ++dev) take_gave_up_word(dev);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"check_gave_up", check_gave_up, METH_O, nullptr},
    {"take_gave_up", take_gave_up, METH_NOARGS, nullptr},
    {"take_launches", take_launches, METH_NOARGS, nullptr},
    {"use_library", use_library, METH_O, nullptr},
    {"set_hooks", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(set_hooks)), METH_FASTCALL, nullptr},
    {"bitlinear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bitlinear)), METH_FASTCALL, nullptr},
    {"hgrn_scan", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(hgrn_scan)), METH_FASTCALL, nullptr},
    {"watch", watch, METH_O, nullptr},
    {"unchanged", unchanged, METH_O, nullptr},
    {"chain", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(chain)), METH_FASTCALL, nullptr},
    {"prepare_step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(prepare_step)), METH_FASTCALL, nullptr},
    {"chain_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(chain_forward)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "native host path of matmulfreellm_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }

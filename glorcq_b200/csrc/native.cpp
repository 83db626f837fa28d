// Host path of the Python classes: argument checks, output and scratch allocation and the C-ABI call of one
// operation in one native call (module glorcq_b200._native).
//
// Why: a decode-sized call runs for 5 to 10 us on the GPU, and the same steps in Python (a ctypes call with
// twenty arguments, two workspace queries, device and stream look-ups, torch.empty) took 20 to 60 us of host time, so
// eager calls were bound by the interpreter.  The functions take tensors as they come (METH_FASTCALL, no argument
// parsing) and raise RuntimeError exactly where the ctypes path did.
//
// The launches run without the interpreter lock (struct Launching): a launch into a full queue waits for the GPU, and
// the process's other threads have other GPUs to feed meanwhile.
//
// The library itself is not linked: bind() receives the entry points' addresses from the loaded library, so that a
// checking build selected with GLQ_LIB serves this module too.
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "../../include/glorcq_b200.h"

namespace {

struct Api {
#define GLQ_FN(name) decltype(&::name) name = nullptr;
#define GLQ_FNS                                                                                                     \
    GLQ_FN(glq_status_string)                                                                                       \
    GLQ_FN(glq_last_cuda_error)                                                                                     \
    GLQ_FN(glq_linear_workspace_bytes)                                                                              \
    GLQ_FN(glq_linear_counters)                                                                                     \
    GLQ_FN(glq_linear_forward)                                                                                      \
    GLQ_FN(glq_linear_rht_workspace_bytes)                                                                          \
    GLQ_FN(glq_linear_rht_forward)                                                                                  \
    GLQ_FN(glq_mm_workspace_bytes)                                                                                  \
    GLQ_FN(glq_mm_counters)                                                                                         \
    GLQ_FN(glq_grouped_matmul)                                                                                      \
    GLQ_FN(glq_grouped_matmul_pair)                                                                                 \
    GLQ_FN(glq_turbo_dequant_matmul)                                                                                \
    GLQ_FN(glq_turbo_dequant_grouped_gemv)                                                                          \
    GLQ_FN(glq_gptq_dequant_matmul)                                                                                 \
    GLQ_FN(glq_moe_workspace_bytes)                                                                                 \
    GLQ_FN(glq_moe_counters)                                                                                        \
    GLQ_FN(glq_moe_forward_ep)                                                                                      \
    GLQ_FN(glq_add_rmsnorm)
    GLQ_FNS
#undef GLQ_FN
} api;

struct Error {
    std::string msg;
};
[[noreturn]] void fail(std::string msg) { throw Error{std::move(msg)}; }

void check(int status, const char* what) {
    if (status == GLQ_OK) return;
    std::string m = std::string(what) + ": " + api.glq_status_string(status);
    if (status == GLQ_ERR_CUDA) m += " (cudaError " + std::to_string(api.glq_last_cuda_error()) + ")";
    fail(m);
}

template <class F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const Error& e) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.msg.c_str());
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* cls = nullptr;
        if (PyObject* m = PyImport_ImportModule("torch")) {
            cls = PyObject_GetAttrString(m, "OutOfMemoryError");
            Py_DECREF(m);
        }
        PyErr_SetString(cls ? cls : PyExc_RuntimeError, e.what_without_backtrace());
        Py_XDECREF(cls);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

void nargs_are(Py_ssize_t got, Py_ssize_t want) {
    if (got != want) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
        throw Error{};
    }
}
const at::Tensor& tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) fail(std::string(name) + " must be a tensor");
    return THPVariable_Unpack(o);
}
const at::Tensor* tensor_or_none(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor(o, name); }
long integer(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw Error{};
    return v;
}
float number(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1 && PyErr_Occurred()) throw Error{};
    return (float)v;
}
void need_cuda(const at::Tensor& t, const char* name) {
    if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor (glorcq_b200 has no CPU path)");
    if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
}
// the last dimension is the row: an element count that fits by chance would be read as other rows than it has (no rows: any width)
void need_rows(const at::Tensor& t, const char* name, int64_t K) {
    if (t.dim() == 0) fail(std::string(name) + " must have at least one dimension");
    const auto lead = t.sizes().slice(0, t.dim() - 1);
    if (t.size(-1) != K && std::find(lead.begin(), lead.end(), 0) == lead.end())
        fail(std::string(name) + " must have rows of " + std::to_string(K) + " values, got " + std::to_string(t.size(-1)));
}
void need(const at::Tensor& t, const char* name, at::ScalarType dtype, const char* dtype_name) {
    if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor");
    if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
    if (t.scalar_type() != dtype) fail(std::string(name) + " must be " + dtype_name);
}
at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const at::Tensor& like) {
    return at::detail::empty_cuda(shape, dtype, like.device(), std::nullopt);
}
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }
const void* ptr(const at::Tensor* t) { return t ? t->const_data_ptr() : nullptr; }
inline size_t up256(size_t v) { return (v + 255) / 256 * 256; }

bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &s) == cudaSuccess && s != cudaStreamCaptureStatusNone;
}

// ---- scratch of a stream -------------------------------------------------------------------------------------
// One scratch buffer and one array of arrival counters per (device, stream); torch hands out a bounded set of
// streams, the buffers grow to the largest call and clear_workspaces() gives them back.  The counters must be zero
// before a call and every kernel leaves them zero, so they are cleared only when the array is made.  Buffers that a call
// under capture was given are kept when a larger call outgrows them: the graph goes on using them (asking the stream costs
// 40 ns a call; at most one buffer per growth is kept).
struct Scratch {
    at::Tensor ws, ctr;
    bool captured = false;
};
using ScratchMap = std::map<std::pair<int, cudaStream_t>, Scratch>;
ScratchMap& g_scratch = *new ScratchMap;      // never destroyed: the process may end after the driver has gone
std::vector<Scratch>& g_outgrown = *new std::vector<Scratch>;

// Scratch of calls larger than this is shared by all blocks on a stream: they run one after another, and a private
// copy for every block and prompt length would not fit.  16 MB lie between the calls that graphs capture (64 tokens of the
// benchmark's models: 3 to 7 MB) and their prompts (512 tokens: 54 to 128 MB).
constexpr size_t kSharedScratchFrom = 16u << 20;
ScratchMap& g_big = *new ScratchMap;

Scratch& scratch(int dev, cudaStream_t st, size_t nbytes, size_t nctr) {
    Scratch& s = g_scratch[{dev, st}];
    const bool small_ws = !s.ws.defined() || (size_t)s.ws.numel() < nbytes, small_ctr = !s.ctr.defined() || (size_t)s.ctr.numel() < nctr;
    const bool capture = capturing(st);
    if (!small_ws && !small_ctr) {
        s.captured |= capture;
        return s;
    }
    if ((!s.ws.defined() || !s.ctr.defined()) && capture) {
        // no allocation (and no zero fill) inside a capture: the scratch of the warm-up calls on this device serves
        // the captured calls too (they run in stream order after them)
        for (auto& kv : g_scratch)
            if (kv.first.first == dev && kv.second.ws.defined() && kv.second.ctr.defined() &&
                (size_t)kv.second.ws.numel() >= nbytes && (size_t)kv.second.ctr.numel() >= nctr) {
                kv.second.captured = true;
                s = kv.second;
                return s;
            }
    }
    if (s.captured) g_outgrown.push_back(s);
    s.captured = capture;
    const auto opt = at::TensorOptions().device(at::kCUDA, dev);
    if (small_ws) {
        s.ws = at::Tensor();
        s.ws = at::empty({(int64_t)std::max<size_t>(nbytes, 1 << 20)}, opt.dtype(at::kByte));
    }
    if (small_ctr) s.ctr = at::zeros({(int64_t)std::max<size_t>(nctr, 1 << 16)}, opt.dtype(at::kInt));
    return s;
}

// The launches of one call: the interpreter lock is given back, and one lock per stream keeps the launches of a call
// together when several threads share the stream, since they also share its scratch.  The locks are taken in this order
// and given back in the other, so a thread that waits for the stream never holds the interpreter.  Whatever the call
// launches on is held by references of its own: other threads may grow the scratch or clear the maps meanwhile.
// Costs 0.15 us a call.
struct Launching {
    PyThreadState* state;
    std::mutex& m;
    static std::mutex& of(cudaStream_t st) {         // (a few streams may share a lock)
        static std::mutex* locks = new std::mutex[64];
        return locks[(reinterpret_cast<uintptr_t>(st) >> 4) % 61];
    }
    explicit Launching(cudaStream_t st) : state(PyEval_SaveThread()), m(of(st)) { m.lock(); }
    ~Launching() {
        m.unlock();
        PyEval_RestoreThread(state);
    }
    Launching(const Launching&) = delete;
};

template <class F> void launch(cudaStream_t st, const char* what, F&& f) {
    int status;
    {
        Launching unlocked(st);
        status = f();
    }
    check(status, what);
}

PyObject* py_workspace(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 3);
        const int dev = (int)integer(a[0]);
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
        Scratch& s = scratch(dev, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(), (size_t)integer(a[1]), (size_t)integer(a[2]));
        return Py_BuildValue("NN", wrap(s.ws), wrap(s.ctr));
    });
}
PyObject* py_clear_workspaces(PyObject*, PyObject*) {
    g_scratch.clear();
    g_outgrown.clear();
    g_big.clear();
    Py_RETURN_NONE;
}

// ---- one quantized layer -------------------------------------------------------------------------------------
struct Layer {
    int fmt, gs;
    glq_weight_t w;
    std::unordered_map<int64_t, std::pair<size_t, size_t>> needs;   // 4 * rows + route -> scratch bytes, counters
};
template <class T> void free_capsule(PyObject* c) { delete static_cast<T*>(PyCapsule_GetPointer(c, PyCapsule_GetName(c))); }
template <class T> T* capsule(PyObject* o, const char* name) {
    T* p = static_cast<T*>(PyCapsule_GetPointer(o, name));
    if (!p) throw Error{};
    return p;
}

PyObject* py_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {   // fmt, group size, bytes of a glq_weight_t
    return guarded([&]() -> PyObject* {
        nargs_are(n, 3);
        char* raw;
        Py_ssize_t len;
        if (PyBytes_AsStringAndSize(a[2], &raw, &len) < 0) throw Error{};
        if (len != (Py_ssize_t)sizeof(glq_weight_t)) fail("descriptor size mismatch");
        auto* L = new Layer{(int)integer(a[0]), (int)integer(a[1]), {}, {}};
        std::memcpy(&L->w, raw, sizeof(L->w));
        return PyCapsule_New(L, "glq.layer", free_capsule<Layer>);
    });
}

// layer, x (..., K) fp16, tiled U^T or None, Hadamard signs or None, precomputed x.U or None -> (..., N)
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 5);
        Layer* L = capsule<Layer>(a[0], "glq.layer");
        const at::Tensor& x = tensor(a[1], "x");
        const at::Tensor* ut = tensor_or_none(a[2], "ut");
        const at::Tensor* signs = tensor_or_none(a[3], "signs");
        const at::Tensor* xu = tensor_or_none(a[4], "precomputed x@U");
        if (x.scalar_type() != at::kHalf) fail("x must be fp16");
        need_rows(x, "x", L->w.K);
        need_cuda(x, "x");
        const int64_t K = L->w.K, rows = x.dim() == 2 ? x.size(0) : x.numel() / std::max<int64_t>(K, 1);
        c10::cuda::OptionalCUDAGuard guard(x.device());
        at::Tensor y;
        if (x.dim() == 2) {
            y = empty({rows, L->w.N}, at::kHalf, x);
        } else {
            auto shape = x.sizes().vec();
            shape.back() = L->w.N;
            y = empty(shape, at::kHalf, x);
        }
        if (rows == 0 || L->w.N == 0) return wrap(y);
        at::Tensor au;
        if (xu) {
            if (xu->scalar_type() != at::kHalf || xu->dim() != 2 || xu->size(0) != rows || xu->size(1) != L->w.rank)
                fail("precomputed x@U must be fp16 of shape (B, rank)");
            au = xu->contiguous();
            xu = &au;
        }
        if (signs) {
            need(*signs, "signs", at::kFloat, "torch.float32");
            if (signs->numel() != K) fail("signs must have shape (" + std::to_string(K) + ",)");
        }
        auto& needs = L->needs[4 * rows + (signs ? 1 : 0)];
        if (!needs.first && !needs.second) {
            if (L->needs.size() > 4096) {
                L->needs.clear();
                return py_linear(nullptr, a, n);
            }
            needs.first = 1 + (signs ? api.glq_linear_rht_workspace_bytes(L->fmt, L->gs, &L->w, (int)rows)
                                     : api.glq_linear_workspace_bytes(L->fmt, L->gs, &L->w, (int)rows));
            needs.second = api.glq_linear_counters(L->fmt, L->gs, &L->w, (int)rows);
        }
        const int dev = x.get_device();
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
        const Scratch s = scratch(dev, st, needs.first, needs.second);
        void* ws = s.ws.mutable_data_ptr();
        auto* ctr = static_cast<int32_t*>(s.ctr.mutable_data_ptr());
        launch(st, signs ? "linear_rht_forward" : "linear_forward", [&] {
            return signs ? api.glq_linear_rht_forward(L->fmt, L->gs, &L->w, ptr(ut), static_cast<const float*>(signs->const_data_ptr()),
                                                      x.const_data_ptr(), K, ptr(xu), y.mutable_data_ptr(), L->w.N, (int)rows, ws,
                                                      (size_t)s.ws.numel(), ctr, (size_t)s.ctr.numel(), st)
                         : api.glq_linear_forward(L->fmt, L->gs, &L->w, ptr(ut), x.const_data_ptr(), K, ptr(xu), y.mutable_data_ptr(),
                                                  L->w.N, (int)rows, ws, (size_t)s.ws.numel(), ctr, (size_t)s.ctr.numel(), st);
        });
        return wrap(y);
    });
}

// ---- several layers of one shape on the same rows ---------------------------------------------------------------
struct Group {
    int fmt, gs, P, N, K, rank;
    const glq_weight_t *table, *ut_table;      // device arrays, kept alive by the Python object
    std::unordered_map<int64_t, at::Tensor> rows;   // rows 0..B-1, P times (a captured graph reads it: never dropped)
};
PyObject* py_group(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        nargs_are(n, 8);
        auto* G = new Group{(int)integer(a[0]), (int)integer(a[1]), (int)integer(a[2]), (int)integer(a[3]), (int)integer(a[4]),
                            (int)integer(a[5]), reinterpret_cast<const glq_weight_t*>(PyLong_AsVoidPtr(a[6])),
                            reinterpret_cast<const glq_weight_t*>(PyLong_AsVoidPtr(a[7])), {}};
        return PyCapsule_New(G, "glq.group", free_capsule<Group>);
    });
}

// group, x (B, K) fp16 -> (P, B, N): x.U of all layers, then the quantized products with the low-rank term
PyObject* py_grouped_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 2);
        Group* G = capsule<Group>(args[0], "glq.group");
        const at::Tensor& x = tensor(args[1], "x");
        if (x.dim() == 2) need_rows(x, "x", G->K);
        if (x.scalar_type() != at::kHalf || x.dim() != 2 || !x.is_cuda() || x.stride(1) != 1) fail("x must be fp16 CUDA rows");
        c10::cuda::OptionalCUDAGuard guard(x.device());
        const int64_t B = x.size(0);
        const int dev = x.get_device();
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
        at::Tensor& rows = G->rows[B];
        if (!rows.defined()) rows = at::arange(B, x.options().dtype(at::kInt)).repeat({G->P});
        at::Tensor y = empty({G->P, B, G->N}, at::kHalf, x), a;
        auto args = [&](int fmt, int gs, const glq_weight_t* table, int N, int rank, at::Tensor& out, const at::Tensor* xu) {
            glq_mm_args_t m;
            std::memset(&m, 0, sizeof(m));
            m.fmt = fmt;
            m.group_size = gs;
            m.n_problems = G->P;
            m.max_rows = m.rows_stride = (int32_t)B;
            m.N = N;
            m.K = G->K;
            m.rank = rank;
            m.total_rows = (int32_t)(G->P * B);
            m.w_table = table;
            m.entry_row = static_cast<const int32_t*>(rows.const_data_ptr());
            m.x = x.const_data_ptr();
            m.ldx = x.stride(0);
            if (xu) {
                // x.U was launched directly before; the tables came by copies, the weights in them were packed
                m.flags = GLQ_MM_A_FROM_PREVIOUS_LAUNCH | GLQ_MM_WEIGHTS_SETTLED;
                m.a0 = xu->const_data_ptr();
                m.lda = xu->size(2);
            }
            m.y = out.mutable_data_ptr();
            m.ldy = N;
            return m;
        };
        const bool low_rank = G->ut_table && G->rank > 0;
        if (low_rank) a = empty({G->P, B, G->rank}, at::kHalf, x);
        // both products are launched under one lock: nothing of another thread may come between them
        glq_mm_args_t mm[2];
        int n_mm = 0;
        if (low_rank) mm[n_mm++] = args(GLQ_FMT_F16, 0, G->ut_table, G->rank, 0, a, nullptr);
        mm[n_mm++] = args(G->fmt, G->gs, G->table, G->N, low_rank ? G->rank : 0, y, low_rank ? &a : nullptr);
        size_t nbytes = 0, nctr = 0;
        for (int i = 0; i < n_mm; ++i) {
            nbytes = std::max(nbytes, api.glq_mm_workspace_bytes(&mm[i]));
            nctr = std::max(nctr, api.glq_mm_counters(&mm[i]) + 2);       // (and the two of a pair)
        }
        const Scratch s = scratch(dev, st, nbytes, nctr);
        for (int i = 0; i < n_mm; ++i) {
            mm[i].workspace = s.ws.mutable_data_ptr();
            mm[i].workspace_bytes = (size_t)s.ws.numel();
            mm[i].counters = static_cast<int32_t*>(s.ctr.mutable_data_ptr());
            mm[i].n_counters = (size_t)s.ctr.numel();
        }
        launch(st, "grouped_matmul", [&] {
            return low_rank ? api.glq_grouped_matmul_pair(&mm[0], &mm[1], st) : api.glq_grouped_matmul(&mm[0], st);
        });
        return wrap(y);
    });
}

// ---- drop-ins of the reference's native modules --------------------------------------------------------------
PyObject* py_turbo_matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 4);
        const at::Tensor &x = tensor(a[0], "x_rot"), &q = tensor(a[1], "packed_indices"), &nrm = tensor(a[2], "norms"), &cen = tensor(a[3], "centroids");
        need(x, "x_rot", at::kHalf, "torch.float16");
        need(q, "packed_indices", at::kByte, "torch.uint8");
        need(nrm, "norms", at::kFloat, "torch.float32");
        need(cen, "centroids", at::kFloat, "torch.float32");
        if (cen.numel() != 4) fail("centroids must have 4 elements");
        if (x.dim() != 2 || q.dim() != 2) fail("x_rot and packed_indices must be matrices");
        const int64_t B = x.size(0), K = x.size(1), N = q.size(0);
        if (K % 4 != 0) fail("K must be divisible by 4 for 2-bit packing");
        if (q.size(1) != K / 4) fail("packed_indices shape mismatch: expected (N, K/4)");
        if (nrm.size(0) != N) fail("norms shape mismatch");
        c10::cuda::OptionalCUDAGuard guard(x.device());
        at::Tensor y = empty({B, N}, at::kHalf, x);
        if (B == 0 || N == 0) return wrap(y);
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
        launch(st, "turbo_dequant_matmul", [&] {
            return api.glq_turbo_dequant_matmul(x.const_data_ptr(), static_cast<const uint8_t*>(q.const_data_ptr()), static_cast<const float*>(nrm.const_data_ptr()),
                                                static_cast<const float*>(cen.const_data_ptr()), y.mutable_data_ptr(), (int)B, (int)N, (int)K, st);
        });
        return wrap(y);
    });
}

PyObject* py_turbo_grouped_gemv(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 5);
        const at::Tensor &x = tensor(a[0], "x_grouped"), &q = tensor(a[1], "packed_cat"), &nrm = tensor(a[2], "norms_cat"), &cen = tensor(a[3], "centroids");
        const int64_t N = integer(a[4]);
        need(x, "x_grouped", at::kHalf, "torch.float16");
        need(q, "packed_cat", at::kByte, "torch.uint8");
        need(nrm, "norms_cat", at::kFloat, "torch.float32");
        need(cen, "centroids", at::kFloat, "torch.float32");
        if (x.dim() != 2 || q.dim() != 2) fail("x_grouped and packed_cat must be matrices");
        const int64_t E = x.size(0), K = x.size(1);
        if (q.size(0) != E * N) fail("packed_cat first dim must be E * N_out");
        if (K % 4 != 0 || q.size(1) != K / 4) fail("packed_cat col dim must be K/4");
        if (nrm.size(0) != E * N) fail("norms_cat size mismatch");
        c10::cuda::OptionalCUDAGuard guard(x.device());
        at::Tensor y = empty({E * N}, at::kHalf, x);
        if (E == 0 || N == 0) return wrap(y);
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
        launch(st, "turbo_dequant_grouped_gemv", [&] {
            return api.glq_turbo_dequant_grouped_gemv(x.const_data_ptr(), static_cast<const uint8_t*>(q.const_data_ptr()), static_cast<const float*>(nrm.const_data_ptr()),
                                                      static_cast<const float*>(cen.const_data_ptr()), y.mutable_data_ptr(), (int)E, (int)N, (int)K, st);
        });
        return wrap(y);
    });
}

PyObject* py_gptq_matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 7);
        const at::Tensor &x = tensor(a[0], "x"), &q = tensor(a[1], "qweight_i8"), &s = tensor(a[2], "scales"), &z = tensor(a[3], "zeros");
        const at::Tensor* lo = tensor_or_none(a[6], "lora_out");
        need(x, "x", at::kFloat, "torch.float32");
        need(q, "qweight_i8", at::kChar, "torch.int8");
        need(s, "scales", at::kHalf, "torch.float16");
        need(z, "zeros", at::kHalf, "torch.float16");
        if (x.dim() != 2 || q.dim() != 2 || s.dim() != 2 || z.dim() != 2) fail("x, qweight_i8, scales and zeros must be matrices");
        const int64_t B = x.size(0), K = x.size(1), N = q.size(0), G = s.size(1);
        if (q.size(1) != K) fail("qweight_i8 shape mismatch: expected (N, K)");
        if (s.size(0) != N || z.size(0) != N || z.size(1) != G) fail("scales / zeros shape mismatch");
        if (lo && lo->numel() == 0) lo = nullptr;
        if (lo) {
            need(*lo, "lora_out", at::kFloat, "torch.float32");
            if (lo->dim() != 2 || lo->size(0) != B || lo->size(1) != N) fail("lora_out shape mismatch");
        }
        c10::cuda::OptionalCUDAGuard guard(x.device());
        at::Tensor y = empty({B, N}, at::kFloat, x);
        if (B == 0 || N == 0) return wrap(y);
        const int gs = (int)integer(a[4]), sym = PyObject_IsTrue(a[5]);
        if (sym < 0) throw Error{};
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
        launch(st, "gptq_dequant_matmul", [&] {
            return api.glq_gptq_dequant_matmul(static_cast<const float*>(x.const_data_ptr()), static_cast<const int8_t*>(q.const_data_ptr()), s.const_data_ptr(), z.const_data_ptr(),
                                               static_cast<const float*>(ptr(lo)), static_cast<float*>(y.mutable_data_ptr()), (int)B, (int)N, (int)K, gs, (int)G, sym, st);
        });
        return wrap(y);
    });
}

// ---- MoE block ------------------------------------------------------------------------------------------------
struct Block {
    const glq_moe_desc_t* d;                  // owned by the Python object
    int device;
    cudaStream_t side;                        // the shared expert's branch (null: none)
    cudaEvent_t fork, join;
    std::unordered_map<int64_t, Scratch> scratch;   // one per token count (see py_moe)
    std::unordered_map<int64_t, std::pair<size_t, size_t>> needs;
};
PyObject* py_block(PyObject*, PyObject* const* a, Py_ssize_t n) {   // descriptor address, device, stream, two events (0: none)
    return guarded([&]() -> PyObject* {
        nargs_are(n, 5);
        auto* B = new Block{};
        B->d = static_cast<const glq_moe_desc_t*>(PyLong_AsVoidPtr(a[0]));
        B->device = (int)integer(a[1]);
        B->side = static_cast<cudaStream_t>(PyLong_AsVoidPtr(a[2]));
        B->fork = static_cast<cudaEvent_t>(PyLong_AsVoidPtr(a[3]));
        B->join = static_cast<cudaEvent_t>(PyLong_AsVoidPtr(a[4]));
        return PyCapsule_New(B, "glq.block", free_capsule<Block>);
    });
}

// scratch and counters of a call on n tokens.  A block's calls run one after another (it is not re-entrant across
// streams), and a workspace made by the warm-up call must be the one a later capture finds: an allocation inside a
// capture would put its zero fill into the graph, once per replay.
Scratch& block_scratch(Block* B, int64_t n, cudaStream_t st) {
    auto& nd = B->needs[n];
    if (!nd.first) nd = {api.glq_moe_workspace_bytes(B->d, (int)n) + 256, std::max<size_t>(api.glq_moe_counters(B->d, (int)n), 1)};
    const bool big = nd.first > kSharedScratchFrom && !capturing(st);
    Scratch& s = big ? g_big[{B->device, st}] : B->scratch[n];
    const auto opt = at::TensorOptions().device(at::kCUDA, B->device);
    if (!s.ws.defined() || (size_t)s.ws.numel() < nd.first) {
        s.ws = at::Tensor();
        s.ws = at::empty({(int64_t)nd.first}, opt.dtype(at::kByte));
    }
    if (!s.ctr.defined() || (size_t)s.ctr.numel() < nd.second) s.ctr = at::zeros({(int64_t)nd.second}, opt.dtype(at::kInt));
    return s;
}
PyObject* py_block_scratch(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 2);
        Block* B = capsule<Block>(a[0], "glq.block");
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)B->device);
        Scratch& s = block_scratch(B, integer(a[1]), c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)B->device).stream());
        return Py_BuildValue("NN", wrap(s.ws), wrap(s.ctr));
    });
}

// block, hidden (B, S, H) fp16, residual or None, norm weight or None, eps or None (no following norm), routing (n, k)
// int32 or None, routing weights (n, k) fp16 or None -> (out, logits or None, selected, weights, normed or None)
PyObject* py_moe(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    return guarded([&] {
        nargs_are(n_args, 7);
        Block* B = capsule<Block>(a[0], "glq.block");
        const glq_moe_desc_t* d = B->d;
        const at::Tensor& x = tensor(a[1], "hidden_states");
        const at::Tensor *res = tensor_or_none(a[2], "residual"), *nw = tensor_or_none(a[3], "norm weight");
        const bool norm = a[4] != Py_None;
        const at::Tensor *sel_in = tensor_or_none(a[5], "top_k_index"), *wts_in = tensor_or_none(a[6], "top_k_weights");
        const int64_t H = d->H;
        need_rows(x, "hidden_states", H);
        need(x, "hidden_states", at::kHalf, "torch.float16");
        const int64_t n = x.numel() / H;
        if (norm && res && res->numel() != x.numel()) fail("the residual must have the shape of hidden_states");
        if (norm && nw && nw->numel() != H) fail("the norm weight must have " + std::to_string(H) + " values");
        c10::cuda::OptionalCUDAGuard guard(x.device());
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
        at::Tensor out = empty(x.sizes(), at::kHalf, x), logits, normed;
        if (!sel_in) logits = empty({n, d->E}, at::kHalf, x);
        at::Tensor sel = empty({n, d->top_k}, at::kInt, x), wts = empty({n, d->top_k}, at::kHalf, x);
        if (norm) normed = empty(x.sizes(), at::kHalf, x);
        if (n > 0) {
            const Scratch s = block_scratch(B, n, st);
            char* ws = static_cast<char*>(s.ws.mutable_data_ptr());
            char* base = reinterpret_cast<char*>(up256(reinterpret_cast<size_t>(ws)));
            glq_moe_ep_t ep;
            std::memset(&ep, 0, sizeof(ep));
            ep.world = 1;
            ep.phase = GLQ_MOE_PHASE_ALL;
            if (sel_in) {
                ep.sel_in = static_cast<decltype(ep.sel_in)>(sel_in->const_data_ptr());
                ep.weight_in = static_cast<decltype(ep.weight_in)>(ptr(wts_in));
            }
            if (norm) {
                ep.normed_out = normed.mutable_data_ptr();
                ep.norm_eps = number(a[4]);
                ep.residual = static_cast<decltype(ep.residual)>(ptr(res));
                ep.norm_weight = static_cast<decltype(ep.norm_weight)>(ptr(nw));
            }
            launch(st, "moe_forward", [&] {
                return api.glq_moe_forward_ep(d, x.const_data_ptr(), (int)n, out.mutable_data_ptr(), logits.defined() ? logits.mutable_data_ptr() : nullptr,
                                              static_cast<int32_t*>(sel.mutable_data_ptr()), wts.mutable_data_ptr(), base,
                                              (size_t)s.ws.numel() - (size_t)(base - ws), static_cast<int32_t*>(s.ctr.mutable_data_ptr()),
                                              (size_t)s.ctr.numel(), st, B->side, B->fork, B->join, (sel_in || norm) ? &ep : nullptr);
            });
        }
        auto opt = [](at::Tensor& t) {
            if (t.defined()) return wrap(t);
            Py_INCREF(Py_None);
            return Py_None;
        };
        return Py_BuildValue("NNNNN", wrap(out), opt(logits), wrap(sel), wrap(wts), opt(normed));
    });
}

// x, delta (rows, H) fp16 contiguous, weight, eps -> (x + delta, rms_norm(x + delta) * weight)
PyObject* py_add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        nargs_are(n, 4);
        const at::Tensor &x = tensor(a[0], "x"), &dl = tensor(a[1], "delta"), &w = tensor(a[2], "weight");
        need(x, "x", at::kHalf, "torch.float16");
        need(dl, "delta", at::kHalf, "torch.float16");
        c10::cuda::OptionalCUDAGuard guard(x.device());
        const int64_t H = x.size(-1);
        at::Tensor xo = empty(x.sizes(), at::kHalf, x), ho = empty(x.sizes(), at::kHalf, x);
        const float eps = number(a[3]);
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
        launch(st, "add_rmsnorm", [&] {
            return api.glq_add_rmsnorm(x.const_data_ptr(), dl.const_data_ptr(), w.const_data_ptr(), eps, H > 0 ? (int)(x.numel() / H) : 0, (int)H,
                                       xo.mutable_data_ptr(), ho.mutable_data_ptr(), st);
        });
        return Py_BuildValue("NN", wrap(xo), wrap(ho));
    });
}

PyObject* py_bind(PyObject*, PyObject* d) {   // {entry point: address}
#define GLQ_FN(name)                                                                              \
    if (PyObject* v = PyDict_GetItemString(d, #name)) api.name = reinterpret_cast<decltype(api.name)>(PyLong_AsVoidPtr(v)); \
    else return PyErr_Format(PyExc_RuntimeError, "the library has no entry point %s", #name);
    GLQ_FNS
#undef GLQ_FN
    Py_RETURN_NONE;
}
PyObject* py_names(PyObject*, PyObject*) {
#define GLQ_FN(name) #name,
    const char* names[] = {GLQ_FNS};
#undef GLQ_FN
    PyObject* l = PyList_New(0);
    for (const char* s : names) {
        PyObject* u = PyUnicode_FromString(s);
        PyList_Append(l, u);
        Py_DECREF(u);
    }
    return l;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(workspace), FAST(layer), FAST(linear), FAST(group), FAST(grouped_linear), FAST(turbo_matmul),
                         FAST(turbo_grouped_gemv), FAST(gptq_matmul), FAST(block), FAST(block_scratch), FAST(moe), FAST(add_rmsnorm),
                         {"bind", py_bind, METH_O, nullptr}, {"names", py_names, METH_NOARGS, nullptr},
                         {"clear_workspaces", py_clear_workspaces, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "glorcq_b200._native", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }

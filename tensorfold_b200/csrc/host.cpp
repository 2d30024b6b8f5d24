// Python binding of the C ABI (include/tensorfold_b200.h) and the native host path of the single-operator calls.
//
// A single projection at 1..8 rows keeps the GPU busy for 5 to 15 us; the Python and ctypes work around it (argument
// conversion, torch.cuda.device contexts, Stream objects, views, allocations) took 42 us a call, so the host
// bound every small call. Here an entry point is a METH_FASTCALL function generated from its C signature (about 0.3 us
// of conversion for 17 arguments; tensors are passed as tensors), and the matmul calls do their checks,
// allocations and launches in one native call.
//
// The functions take the arguments of the C entry point, in order: a pointer is a CUDA tensor, an address or None. While the
// C call runs the interpreter is released, as under ctypes: a launch that waits for a place in a full queue stops no other thread.

#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "../../include/tensorfold_b200.h"

namespace {

std::atomic<long long> g_launches{0};      // kernels queued by successful calls

struct PyErr {};                           // thrown with a Python error set

struct Released {                          // the interpreter lock given up for a scope; no Python object is touched in it
    PyThreadState* state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
};
[[noreturn]] void fail(PyObject* type, const char* text) {
    PyErr_SetString(type, text);
    throw PyErr{};
}

// ---- one Python object -> one C argument --------------------------------------------------------------
template <class T>
T convert(PyObject* o) {
    if constexpr (std::is_pointer_v<T>) {
        if (o == Py_None) return nullptr;
        if (THPVariable_Check(o)) return reinterpret_cast<T>(THPVariable_Unpack(o).unsafeGetTensorImpl()->mutable_data());
        const unsigned long long v = PyLong_AsUnsignedLongLong(o);
        if (v == ~0ull && PyErr_Occurred()) throw PyErr{};
        return reinterpret_cast<T>(v);
    } else if constexpr (std::is_floating_point_v<T>) {
        const double v = PyFloat_AsDouble(o);
        if (v == -1.0 && PyErr_Occurred()) throw PyErr{};
        return static_cast<T>(v);
    } else if constexpr (sizeof(T) == 8 && std::is_unsigned_v<T>) {
        const unsigned long long v = PyLong_AsUnsignedLongLong(o);
        if (v == ~0ull && PyErr_Occurred()) throw PyErr{};
        return static_cast<T>(v);
    } else {
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) throw PyErr{};
        return static_cast<T>(v);
    }
}

template <class R>
PyObject* to_python(R v) {
    if constexpr (std::is_unsigned_v<R>) return PyLong_FromUnsignedLongLong(v);
    else return PyLong_FromLongLong(v);
}

// LAUNCHES: kernels that a successful call queues (0: a host-only function)
template <auto Fn, int LAUNCHES>
struct Entry;
template <class R, class... A, R (*Fn)(A...), int LAUNCHES>
struct Entry<Fn, LAUNCHES> {
    template <size_t... I>
    static PyObject* apply(PyObject* const* args, std::index_sequence<I...>) {
        std::tuple<A...> v{convert<A>(args[I])...};
        if constexpr (std::is_void_v<R>) {
            {
                const Released unlocked;
                Fn(std::get<I>(v)...);
            }
            Py_RETURN_NONE;
        } else {
            const R rc = [&] {
                const Released unlocked;
                return Fn(std::get<I>(v)...);
            }();
            if (LAUNCHES > 0 && rc == 0) g_launches.fetch_add(LAUNCHES, std::memory_order_relaxed);
            return to_python(rc);
        }
    }
    // `self` is the entry point through ctypes where bound() made the function: it takes what the conversions here do not
    // (ctypes objects, byref, arrays, sizes to be wrapped), or says why not.
    static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
        const bool bound = self != nullptr && PyCallable_Check(self);
        try {
            if (n == (Py_ssize_t)sizeof...(A)) return apply(args, std::index_sequence_for<A...>{});
            PyErr_Format(PyExc_TypeError, "this entry point takes %d arguments, got %zd", (int)sizeof...(A), n);
            throw PyErr{};
        } catch (const PyErr&) {
            if (!bound || !(PyErr_ExceptionMatches(PyExc_TypeError) || PyErr_ExceptionMatches(PyExc_OverflowError))) return nullptr;
            PyErr_Clear();
            PyObject* result = PyObject_Vectorcall(self, args, (size_t)n, nullptr);
            if (LAUNCHES > 0 && result != nullptr && PyLong_Check(result) && PyLong_AsLong(result) == 0)
                g_launches.fetch_add(LAUNCHES, std::memory_order_relaxed);
            return result;
        } catch (const std::exception& e) {
            PyErr_SetString(PyExc_RuntimeError, e.what());
            return nullptr;
        }
    }
};

// ---- matmul scratch: one buffer a (device, stream), zeroed once, kept while the process runs -----------------
// A stream's launches share it in order; other streams have their own, so calls on different streams may overlap.
std::mutex g_scratch_lock;
std::map<std::pair<int, cudaStream_t>, at::Tensor> g_scratch;

at::Tensor scratch_on(int device, cudaStream_t stream) {
    std::lock_guard<std::mutex> hold(g_scratch_lock);
    at::Tensor& t = g_scratch[{device, stream}];
    if (!t.defined())
        t = at::zeros({(int64_t)tf_qmm_scratch_bytes()}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
    return t;
}

void check_rc(int rc, const char* what) {
    if (rc == TF_OK) return;
    const char* name = rc == TF_EINVAL ? "TF_EINVAL (unsupported shape, size or flag)" : rc == TF_EALIGN ? "TF_EALIGN (misaligned pointer)"
                     : rc == TF_ESCRATCH ? "TF_ESCRATCH (scratch missing or too small)" : "TF_ECUDA (launch refused)";
    PyErr_Format(rc == TF_ECUDA ? PyExc_RuntimeError : PyExc_ValueError, "%s: %s", what, name);
    throw PyErr{};
}

template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject*, PyObject* const* args, Py_ssize_t n) {
    try {
        return F(args, n);
    } catch (const PyErr&) {
        return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// scratch(device index) -> the current stream's matmul scratch
PyObject* scratch_py(PyObject* const* args, Py_ssize_t) {
    const int dev = convert<int>(args[0]);
    return THPVariable_Wrap(scratch_on(dev, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream()));
}

const at::Tensor& tensor(PyObject* o) {
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "expected a tensor");
    return THPVariable_Unpack(o);
}

// rows of a projection's input: (x as [m, k] contiguous rows, m)
at::Tensor rows_of(const at::Tensor& x, int64_t k, const char* who, int64_t n) {
    if (!x.is_cuda()) fail(PyExc_ValueError, "lane kernels take CUDA tensors only (there is no CPU path)");
    if (x.scalar_type() != at::kBFloat16) {
        PyErr_Format(PyExc_ValueError, "%s: x must be bf16", who);
        throw PyErr{};
    }
    if (x.dim() < 1 || x.size(-1) != k) {
        PyErr_Format(PyExc_ValueError, "%s: weight (N=%lld, K=%lld) does not match K=%lld", who, (long long)n, (long long)k,
                     (long long)(x.dim() ? x.size(-1) : 0));
        throw PyErr{};
    }
    at::Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, k});
    if (x2.size(0) < 1) {
        PyErr_Format(PyExc_ValueError, "%s: needs at least one row", who);
        throw PyErr{};
    }
    return x2.is_contiguous() ? x2 : x2.contiguous();
}

at::Tensor output_for(PyObject* given, const at::Tensor& x, int64_t m, int64_t n, bool f32, const char* who) {
    const auto type = f32 ? at::kFloat : at::kBFloat16;
    if (given == Py_None) return at::empty({m, n}, x.options().dtype(type));
    at::Tensor out = tensor(given);
    if (out.dim() != 2 || out.size(0) != m || out.size(1) != n || out.scalar_type() != type || !out.is_contiguous()) {
        PyErr_Format(PyExc_ValueError, "%s: out has the wrong shape or dtype", who);
        throw PyErr{};
    }
    return out;
}

PyObject* shaped(const at::Tensor& out, const at::Tensor& x, int64_t n) {
    if (x.dim() == 2) return THPVariable_Wrap(out);
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = n;
    return THPVariable_Wrap(out.reshape(shape));
}

// lane_matmul(x, tiled, n, k, group, f32, out, next_tiled, next_n, next_k, next_group, status): row-major rows in any
// number, packed and multiplied in launches of up to TF_QMM_MAX_ROWS rows
PyObject* lane_matmul_py(PyObject* const* args, Py_ssize_t) {
    at::AutoDispatchBelowADInplaceOrView no_grad;
    const at::Tensor x = tensor(args[0]), w = tensor(args[1]);       // held: the interpreter lock is given up below
    const int n = convert<int>(args[2]), k = convert<int>(args[3]), group = convert<int>(args[4]);
    const bool f32 = convert<int>(args[5]) != 0;
    const at::Tensor x2 = rows_of(x, k, "lane_matmul", n);
    const int64_t m = x2.size(0);
    const c10::cuda::CUDAGuard on(x.device());
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    const at::Tensor out = output_for(args[6], x, m, n, f32, "lane_matmul");
    const at::Tensor scratch = scratch_on(x.device().index(), stream.stream());
    const void* next_w = convert<const void*>(args[7]);
    const int next_n = convert<int>(args[8]), next_k = convert<int>(args[9]), next_group = convert<int>(args[10]);
    int* status = convert<int*>(args[11]);
    const int64_t most = m < TF_QMM_MAX_ROWS ? m : TF_QMM_MAX_ROWS;
    const at::Tensor packed = at::empty({(int64_t)tf_packed_bytes((int)most, k, group)}, x.options().dtype(at::kByte));
    const size_t out_row = (size_t)n * (f32 ? 4 : 2);
    const char* what = "pack_rows";
    const int rc = [&] {
        const Released unlocked;
        for (int64_t r0 = 0; r0 < m; r0 += TF_QMM_MAX_ROWS) {
            const int rows = (int)std::min<int64_t>(m - r0, TF_QMM_MAX_ROWS);
            const bool last = r0 + rows >= m;
            what = "pack_rows";
            if (const int bad = tf_pack_rows(static_cast<const uint8_t*>(x2.const_data_ptr()) + (size_t)r0 * k * 2, packed.mutable_data_ptr(),
                                             nullptr, rows, k, group, stream.stream())) return bad;
            what = "lane_matmul";
            if (const int bad = tf_qmm_next(packed.const_data_ptr(), w.const_data_ptr(), static_cast<uint8_t*>(out.mutable_data_ptr()) + r0 * out_row,
                                            scratch.mutable_data_ptr(), (size_t)scratch.numel(), rows, n, k, group, f32 ? TF_QMM_F32_OUT : 0,
                                            last ? next_w : w.const_data_ptr(), last ? next_n : n, last ? next_k : k,
                                            last ? next_group : group, status, stream.stream())) return bad;
            g_launches.fetch_add(2, std::memory_order_relaxed);
        }
        return (int)TF_OK;
    }();
    check_rc(rc, what);
    return shaped(out, x, n);
}

// prefill_matmul(x, tiled, n, k, group, f32, out, staging, status): the same on the wide-row kernel
PyObject* prefill_matmul_py(PyObject* const* args, Py_ssize_t) {
    at::AutoDispatchBelowADInplaceOrView no_grad;
    const at::Tensor x = tensor(args[0]), w = tensor(args[1]);       // held: the interpreter lock is given up below
    const int n = convert<int>(args[2]), k = convert<int>(args[3]), group = convert<int>(args[4]);
    const bool f32 = convert<int>(args[5]) != 0;
    const at::Tensor x2 = rows_of(x, k, "prefill_matmul", n);
    const int64_t m = x2.size(0);
    const c10::cuda::CUDAGuard on(x.device());
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    const at::Tensor out = output_for(args[6], x, m, n, f32, "prefill_matmul");
    const at::Tensor scratch = scratch_on(x.device().index(), stream.stream());
    const int64_t most = m < TF_QMM_MAX_ROWS ? m : TF_QMM_MAX_ROWS;
    const size_t need = tf_packed_tc_bytes((int)most, k, group);
    const at::Tensor packed = args[7] == Py_None ? at::empty({(int64_t)need}, x.options().dtype(at::kByte)) : tensor(args[7]);
    if ((size_t)packed.numel() < need) fail(PyExc_ValueError, "prefill_matmul: staging buffer too small");
    int* status = convert<int*>(args[8]);
    const size_t out_row = (size_t)n * (f32 ? 4 : 2);
    const char* what = "prefill pack_rows";
    const int rc = [&] {
        const Released unlocked;
        for (int64_t r0 = 0; r0 < m; r0 += TF_QMM_MAX_ROWS) {
            const int rows = (int)std::min<int64_t>(m - r0, TF_QMM_MAX_ROWS);
            what = "prefill pack_rows";
            if (const int bad = tf_pack_rows_tc(static_cast<const uint8_t*>(x2.const_data_ptr()) + (size_t)r0 * k * 2, packed.mutable_data_ptr(),
                                                nullptr, rows, k, group, stream.stream())) return bad;
            what = "prefill_matmul";
            if (const int bad = tf_qmm_tc(packed.const_data_ptr(), w.const_data_ptr(), static_cast<uint8_t*>(out.mutable_data_ptr()) + r0 * out_row,
                                          scratch.mutable_data_ptr(), (size_t)scratch.numel(), rows, n, k, group, f32 ? TF_QMM_F32_OUT : 0,
                                          status, stream.stream())) return bad;
            g_launches.fetch_add(2, std::memory_order_relaxed);
        }
        return (int)TF_OK;
    }();
    check_rc(rc, what);
    return shaped(out, x, n);
}

// current_stream(device index) -> cudaStream_t as an int; -1: the current device's
PyObject* stream_py(PyObject* const* args, Py_ssize_t n) {
    const int dev = n > 0 ? convert<int>(args[0]) : -1;
    return PyLong_FromVoidPtr(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
}
PyObject* device_py(PyObject* const*, Py_ssize_t) { return PyLong_FromLong(c10::cuda::current_device()); }
PyObject* count_py(PyObject* const*, Py_ssize_t) { return PyLong_FromLongLong(g_launches.load(std::memory_order_relaxed)); }

PyObject* bound_py(PyObject* const* args, Py_ssize_t n);

#define TF_FN(name, launches) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&Entry<&name, launches>::call)), METH_FASTCALL, nullptr}
#define TF_OWN(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&guarded<&fn>)), METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    TF_FN(tf_version, 0), TF_FN(tf_qmm_workers, 0), TF_FN(tf_qmm_scratch_bytes, 0), TF_FN(tf_packed_bytes, 0), TF_FN(tf_qmm, 1),
    TF_FN(tf_qmm_set_trace, 0), TF_FN(tf_qmm_next, 1), TF_FN(tf_qmm_grouped, 1), TF_FN(tf_pack_rows, 1), TF_FN(tf_qmm_tiled_bytes, 0),
    TF_FN(tf_qmm_tile, 1), TF_FN(tf_qmm_untile, 1), TF_FN(tf_packed_tc_bytes, 0), TF_FN(tf_qmm_tc_tiled_bytes, 0), TF_FN(tf_qmm_tc, 1),
    TF_FN(tf_pack_rows_tc, 1), TF_FN(tf_qmm_tc_set_trace, 0), TF_FN(tf_repack_tc, 1), TF_FN(tf_qmm_tc_tile, 1), TF_FN(tf_qmm_tc_untile, 1),
    TF_FN(tf_norm_xs, 1), TF_FN(tf_swiglu, 1), TF_FN(tf_gated_norm, 1), TF_FN(tf_gate_mul, 1), TF_FN(tf_attn_prep, 1), TF_FN(tf_gdn_pre, 1),
    TF_FN(tf_embed, 1), TF_FN(tf_gdn_chain, 1), TF_FN(tf_gdn_fused, 1), TF_FN(tf_gdn_replay, 1), TF_FN(tf_conv_commit, 1),
    TF_FN(tf_attention_scratch_bytes, 0), TF_FN(tf_attention_chunks, 0), TF_FN(tf_lane_attention_paged_gated, 2),
    TF_FN(tf_lane_attention_paged, 2), TF_FN(tf_lane_attention_paged_static, 2), TF_FN(tf_kv_commit, 1), TF_FN(tf_moe_max_problems, 0),
    TF_FN(tf_moe_router, 1), TF_FN(tf_moe_select, 1), TF_FN(tf_moe_group, 1), TF_FN(tf_moe_slot_bytes, 0), TF_FN(tf_moe_push, 1),
    TF_FN(tf_moe_combine_peer, 1), TF_FN(tf_moe_pack, 1), TF_FN(tf_moe_act, 1), TF_FN(tf_moe_combine, 1), TF_FN(tf_peer_slot_bytes, 0),
    TF_FN(tf_peer_exchange, 1), TF_FN(tf_qmm_act, 1), TF_FN(tf_swiglu_tiled, 1), TF_FN(tf_qmm_peer, 1), TF_FN(tf_norm_xs_peer, 1),
    TF_FN(tf_set_poll_limit, 0), TF_FN(tf_topk_scratch_bytes, 0), TF_FN(tf_topk_rows, 2), TF_FN(tf_topk_sample_rows, 2), TF_FN(tf_sample_rows, 1),
    TF_OWN("bound", bound_py), TF_OWN("scratch", scratch_py), TF_OWN("lane_matmul", lane_matmul_py), TF_OWN("prefill_matmul", prefill_matmul_py),
    TF_OWN("current_stream", stream_py), TF_OWN("current_device", device_py), TF_OWN("launch_count", count_py),
    {nullptr, nullptr, 0, nullptr}};

// bound(name, fn): the entry point `name`, with `fn` (the same one through ctypes) for the arguments it does not convert itself
PyObject* bound_py(PyObject* const* args, Py_ssize_t n) {
    const char* name = n == 2 ? PyUnicode_AsUTF8(args[0]) : nullptr;
    if (name == nullptr) fail(PyExc_TypeError, "bound(name, function)");
    for (PyMethodDef* def = methods; def->ml_name != nullptr; ++def)
        if (std::strcmp(def->ml_name, name) == 0) return PyCFunction_NewEx(def, args[1], nullptr);
    fail(PyExc_AttributeError, name);
}

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native binding of libtensorfold_b200.so", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }

// Host path between PyTorch and the C ABI: what happens on the CPU for one call of a quantised linear.
//
// A decode call runs 5 to 10 us on the GPU.  The same argument handling in Python (dispatcher to a Python
// implementation, attribute reads, ctypes) took 30 to 36 us a call and was what an eager decode step ran at; here it
// is one C++ function per call: type and shape checks, one output allocation, one C ABI call.
//
// Two ways in:
//   * the CUDA implementations of torch.ops.binary_kernels.* (schemas: nanoquant_b200/ops.py), for operands in the
//     kernels' tile layout; operands in the reference's layouts go to the Python implementation, which converts them
//     once and keeps the result on the tensor;
//   * plain functions for this package's own modules (no dispatcher).  They return None whenever a call is not the
//     plain case (other types, tensor subclasses, wrappers of transforms, dispatch modes, odd dimensions, a linear that
//     autograd would record); the caller then takes the general route.
#include <Python.h>

#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/core/grad_mode.h>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/as_strided.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>

#include <mutex>
#include <optional>
#include <vector>

#include "nanoquant_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

constexpr int kMaxLinears = 4;
constexpr int kMaxDevices = 64;

// ---------------------------------------------------------------------------------------------------------------
// Python callbacks, set once by nanoquant_b200.ops
// ---------------------------------------------------------------------------------------------------------------
PyObject* g_raise_status = nullptr;    // (status, what): raises
PyObject* g_grow_scratch = nullptr;    // (device index, bytes): makes the scratch hold that many bytes, or raises
PyObject* g_dyn_general = nullptr;     // Python implementations of the operators (reference operand layouts)
PyObject* g_marlin_general = nullptr;

// What module_call compares with: NanoQuantLinear and its forward, nn.Module and its way from a call to forward, the hooks on every module.
struct ModuleClass {
    PyTypeObject *type = nullptr, *base = nullptr;
    PyObject *forward = nullptr, *call = nullptr, *call_impl = nullptr;
    std::vector<PyObject*> global_hooks;
};
ModuleClass g_module_class;

// Calls a Python function with the GIL held and throws its exception.
PyObject* call_python(PyObject* fn, PyObject* args) {
    TORCH_CHECK(fn != nullptr, "nanoquant_b200: the host extension has not been initialised");
    PyObject* r = PyObject_CallObject(fn, args);
    Py_DECREF(args);
    if (!r) {
        python_error err;
        err.persist();
        throw std::move(err);
    }
    return r;
}

[[noreturn]] void fail(int status, const char* what) {
    pybind11::gil_scoped_acquire gil;
    Py_XDECREF(call_python(g_raise_status, Py_BuildValue("(is)", status, what)));
    TORCH_CHECK(false, what, ": nq_status ", status);
}

// ---------------------------------------------------------------------------------------------------------------
// scratch: one buffer per device (owned by nanoquant_b200.ops, which keeps it alive), a thread may override it
// ---------------------------------------------------------------------------------------------------------------
struct Scratch {
    void* ptr = nullptr;
    size_t bytes = 0;
};
Scratch g_scratch[kMaxDevices];
std::mutex g_scratch_mutex;            // pointer and size change together
thread_local Scratch t_override;

Scratch scratch_of(int dev) {
    if (t_override.ptr) return t_override;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    return g_scratch[dev];
}

void grow_scratch(int dev, size_t bytes) {
    pybind11::gil_scoped_acquire gil;
    Py_DECREF(call_python(g_grow_scratch, Py_BuildValue("(in)", dev, (Py_ssize_t)bytes)));
}

// ---------------------------------------------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------------------------------------------
// Makes `dev` current for the C ABI call if it is not (a query and nothing else in the usual case).
struct OnDevice {
    explicit OnDevice(int dev) {
        if (c10::cuda::current_device() != dev) guard.emplace(dev);
    }
    std::optional<c10::cuda::CUDAGuard> guard;
};

int dtype_id(at::ScalarType t) { return t == at::kHalf ? NQ_F16 : NQ_BF16; }
bool is_16bit(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }

// Up to four linears at T tokens: the decode kernel for few tokens and for sizes the tensor-core path does not
// take (columns or ranks that are no multiple of 8), the tensor-core path for the rest.
void launch(nq_linear_desc* d, int n, int64_t T, int dtype, int dev) {
    static const int gemv_max = nq_gemv_max_tokens();
    bool gemv = T <= gemv_max;
    if (!gemv && n == 1 && (d->N % 8 != 0 || d->R % 8 != 0)) gemv = true;
    OnDevice on(dev);
    const nq_stream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    const auto fwd = gemv ? nq_decode_group_fwd : nq_gemm_group_fwd;
    Scratch s = scratch_of(dev);
    int st = s.ptr ? fwd(d, n, (int)T, dtype, s.ptr, s.bytes, stream) : (int)NQ_ERR_SCRATCH;
    if (st == NQ_ERR_SCRATCH) {   // nothing has been launched: the scratch is checked first
        grow_scratch(dev, gemv ? nq_gemv_group_scratch_bytes(d, n, (int)T) : nq_gemm_group_scratch_bytes(d, n, (int)T));
        s = scratch_of(dev);
        st = fwd(d, n, (int)T, dtype, s.ptr, s.bytes, stream);
    }
    if (st < 0) fail(st, gemv ? "nq_decode_group_fwd" : "nq_gemm_group_fwd");
}

// A linear's operands.  `rank` comes from the caller: the tile layout pads it.
struct Linear {
    const Tensor *s_in, *v, *s_mid, *u, *s_out, *bias;
    int64_t rank;
};

void describe(nq_linear_desc& d, const Linear& l, const void* x, int64_t N, int64_t ldx, void* y, int64_t ldy) {
    d = nq_linear_desc{};
    d.x = x;
    d.s_in = l.s_in->const_data_ptr();
    d.v_tiles = l.v->const_data_ptr();
    d.s_mid = l.s_mid ? l.s_mid->const_data_ptr() : nullptr;
    d.u_tiles = l.u->const_data_ptr();
    d.s_out = l.s_out->const_data_ptr();
    d.y = y;
    d.N = (int)N;
    d.R = (int)l.rank;
    d.M = (int)l.s_out->size(0);
    d.ldx = ldx;
    d.ldy = ldy;
    d.bias = l.bias ? l.bias->const_data_ptr() : nullptr;
}

// Without the dispatcher (1.2 us of a call): nothing that could intercept it is active where a plain call is taken, and the kernel
// writes every element.
Tensor new_output(at::IntArrayRef shape, const Tensor& like, at::ScalarType type) {
    return at::detail::empty_cuda(shape, type, like.device(), std::nullopt);
}
Tensor new_output(at::IntArrayRef shape, const Tensor& like) { return new_output(shape, like, like.scalar_type()); }

// y[..., M] for a contiguous x[..., N]
Tensor linear(const Tensor& x, const Linear& l) {
    const int64_t N = x.size(-1), T = N ? x.numel() / N : 0, M = l.s_out->size(0);
    c10::SmallVector<int64_t, 4> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = M;
    Tensor y = new_output(shape, x);
    if (T == 0) return y;
    nq_linear_desc d;
    describe(d, l, x.const_data_ptr(), N, N, y.mutable_data_ptr(), M);
    launch(&d, 1, T, dtype_id(x.scalar_type()), x.get_device());
    return y;
}

// ---------------------------------------------------------------------------------------------------------------
// operators
// ---------------------------------------------------------------------------------------------------------------
void check_operand(const Tensor& t, const char* name, at::ScalarType dtype, const char* dtype_name) {
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
    TORCH_CHECK(t.scalar_type() == dtype, name, " must be ", dtype_name, " tensor");
}

// The reference dispatches its tuning arguments through compile-time lists and raises ValueError on a miss
// (cuda/meta_utils.h:14-38, cuda/gemv_kernel.cu:351-354); the kernels here have no such knobs.
void check_sweep(const char* name, int64_t v, std::initializer_list<int64_t> choices) {
    for (int64_t c : choices)
        if (c == v) return;
    std::string list;
    for (int64_t c : choices) list += (list.empty() ? "" : ", ") + std::to_string(c);
    TORCH_CHECK_VALUE(false, name, " should be one of [", list, "], but ", v, " was given");
}

PyObject* wrap(const OptTensor& t) {
    if (!t) Py_RETURN_NONE;
    return THPVariable_Wrap(*t);
}
Tensor unwrap_result(PyObject* r) {
    Tensor y = THPVariable_Unpack(r);
    Py_DECREF(r);
    return y;
}

Tensor nanoquant_dyn_forward(const Tensor& x, const Tensor& scale_g, const Tensor& Ubits, const OptTensor& scale_l,
                             const Tensor& Vbits, const Tensor& scale_h, int64_t th1, int64_t th2, int64_t rpw1,
                             int64_t rpw2, int64_t acc1, int64_t acc2, int64_t pipe1, int64_t pipe2) {
    if (Ubits.dim() != 3 || Vbits.dim() != 3 || !scale_l) {   // operands to convert, or a rank to look up
        pybind11::gil_scoped_acquire gil;
        return unwrap_result(call_python(g_dyn_general, Py_BuildValue(
            "(NNNNNNLLLLLLLL)", THPVariable_Wrap(x), THPVariable_Wrap(scale_g), THPVariable_Wrap(Ubits), wrap(scale_l),
            THPVariable_Wrap(Vbits), THPVariable_Wrap(scale_h), (long long)th1, (long long)th2, (long long)rpw1,
            (long long)rpw2, (long long)acc1, (long long)acc2, (long long)pipe1, (long long)pipe2)));
    }
    const at::ScalarType dt = x.scalar_type();   // checks in the order of the reference (cuda/gemv_kernel.cu:317-338)
    TORCH_CHECK(is_16bit(dt), "Support only Half or BFloat16");
    const char* name = dt == at::kHalf ? "float16" : "bfloat16";
    check_operand(x, "x", dt, name);
    check_operand(scale_g, "scale_g", dt, name);
    check_operand(scale_h, "scale_h", dt, name);
    check_operand(Ubits, "Ubits", at::kInt, "int32");
    check_operand(Vbits, "Vbits", at::kInt, "int32");
    check_operand(*scale_l, "(*scale_l)", dt, name);
    TORCH_CHECK(scale_g.size(0) == x.size(-1), "scale_g size mismatch");
    check_sweep("n_th1", th1, {64, 128, 256});
    check_sweep("n_rpw1", rpw1, {1, 2, 4, 8});
    check_sweep("n_acc1", acc1, {1, 2});
    check_sweep("n_pipe1", pipe1, {1, 2, 4, 8, 16});
    check_sweep("n_th2", th2, {64, 128, 256});
    check_sweep("n_rpw2", rpw2, {1, 2, 4, 8});
    check_sweep("n_acc2", acc2, {1, 2});
    check_sweep("n_pipe2", pipe2, {1, 2, 4, 8, 16});
    return linear(x, Linear{&scale_g, &Ubits, &*scale_l, &Vbits, &scale_h, nullptr, scale_l->size(0)});
}

// `weight_u` is the FIRST stage (module V), `weight_v` the second (reference cuda/gemm.cpp:112-122)
Tensor marlin_nanoquant_forward(const Tensor& x, const Tensor& weight_u, const Tensor& weight_v, const OptTensor& scale_g,
                                const OptTensor& scale_l, const OptTensor& scale_h, const Tensor& workspace) {
    if (weight_u.dim() == 3 && scale_g && scale_l && scale_h && is_16bit(x.scalar_type()) && x.dim() == 2)
        return linear(x.is_contiguous() ? x : x.contiguous(),
                      Linear{&*scale_g, &weight_u, &*scale_l, &weight_v, &*scale_h, nullptr, scale_l->size(0)});
    pybind11::gil_scoped_acquire gil;
    return unwrap_result(call_python(g_marlin_general, Py_BuildValue(
        "(NNNNNNN)", THPVariable_Wrap(x), THPVariable_Wrap(weight_u), THPVariable_Wrap(weight_v), wrap(scale_g),
        wrap(scale_l), wrap(scale_h), THPVariable_Wrap(workspace))));
}

TORCH_LIBRARY_IMPL(binary_kernels, CUDA, m) {
    m.impl("nanoquant_dyn_forward", nanoquant_dyn_forward);
    m.impl("marlin_nanoquant_forward", marlin_nanoquant_forward);
}

// ---------------------------------------------------------------------------------------------------------------
// plain functions
// ---------------------------------------------------------------------------------------------------------------
// A tensor argument without anything that would have to go through the dispatcher: its keys are those of a strided CUDA tensor and of autograd
// alone.  Not so for the wrappers of transforms (vmap, grad, functionalize), subclasses that dispatch in Python and lazily negated or
// zero tensors, whose memory (if they have any) does not hold their values.
const uint64_t kPlainKeys = c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                                                 c10::DispatchKey::AutocastCUDA}).raw_repr();
const Tensor* plain(PyObject* o) {
    if (!THPVariable_Check(o)) return nullptr;
    const Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && (t.key_set().raw_repr() & ~kPlainKeys) == 0 ? &t : nullptr;
}
bool exact_plain(PyObject* o) { return THPVariable_CheckExact(o) && !c10::impl::dispatch_mode_enabled(); }

// (s_in, v_tiles, s_mid | None, u_tiles, s_out, rank, bias | None) from `a[0..6]`; false: not the plain case.
bool parse_linear(PyObject* const* a, at::ScalarType dt, int64_t N, Linear& l) {
    auto vec = [&](PyObject* o, int64_t n) -> const Tensor* {
        const Tensor* t = plain(o);
        return t && t->scalar_type() == dt && t->dim() == 1 && (n < 0 || t->size(0) == n) && t->is_contiguous() ? t : nullptr;
    };
    auto tiles = [&](PyObject* o) -> const Tensor* {
        const Tensor* t = plain(o);
        return t && t->scalar_type() == at::kInt && t->dim() == 3 && t->is_contiguous() ? t : nullptr;
    };
    l.rank = PyLong_AsLongLong(a[5]);
    if (l.rank <= 0) { PyErr_Clear(); return false; }
    l.s_in = vec(a[0], N);
    l.v = tiles(a[1]);
    l.s_mid = a[2] == Py_None ? nullptr : vec(a[2], l.rank);
    l.u = tiles(a[3]);
    l.s_out = vec(a[4], -1);
    if (!l.s_in || !l.v || !l.u || !l.s_out || (a[2] != Py_None && !l.s_mid)) return false;
    const int64_t M = l.s_out->size(0);
    l.bias = a[6] == Py_None ? nullptr : vec(a[6], M);
    if (a[6] != Py_None && !l.bias) return false;
    // the tiles are what the descriptor's sizes say: 16 rows x 256 columns each
    return l.v->size(0) == (l.rank + 15) / 16 && l.v->size(1) == (N + 255) / 256 && l.u->size(0) == (M + 15) / 16 &&
           l.u->size(1) == (l.rank + 255) / 256;
}

// Autograd would record the operator behind this call (as one without a derivative, which backward then says).  A linear with a bias has
// no operator.
bool recorded(const Tensor& x, const Linear& l) {
    if (l.bias || !at::GradMode::is_enabled()) return false;
    for (const Tensor* t : {&x, l.s_in, l.s_mid, l.s_out})
        if (t && t->requires_grad()) return true;
    return false;
}

// linear_forward(x, s_in, v_tiles, s_mid, u_tiles, s_out, rank, bias) -> y or None
PyObject* py_linear_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 8, "linear_forward takes 8 arguments");
    if (!exact_plain(a[0])) Py_RETURN_NONE;
    const Tensor* x = plain(a[0]);
    Linear l;
    if (!x || !is_16bit(x->scalar_type()) || (x->dim() != 2 && x->dim() != 3) || !x->is_contiguous() ||
        !parse_linear(a + 1, x->scalar_type(), x->size(-1), l) || recorded(*x, l))
        Py_RETURN_NONE;
    Tensor y;
    {
        pybind11::gil_scoped_release no_gil;
        y = linear(*x, l);
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// module_call(module, x) -> y or None: the call of a prepared NanoQuantLinear that nn.Module.__call__ would pass to its forward and forward
// to linear_forward, as one function.  None for everything that nn.Module would not have passed on unchanged and unseen: hooks (the
// module's or global ones), a replaced forward, nn.Module's way of calling replaced (tools do that to see every module's calls), tracing, a
// Python profiler or debugger, a subclass, or not a plain call.
PyObject* py_module_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 2, "module_call takes a module and its argument");
    static PyObject* const key[] = {PyUnicode_InternFromString("_forward_hooks"), PyUnicode_InternFromString("_forward_pre_hooks"),
                                    PyUnicode_InternFromString("_backward_hooks"), PyUnicode_InternFromString("_backward_pre_hooks"),
                                    PyUnicode_InternFromString("_parameters"), PyUnicode_InternFromString("forward"),
                                    PyUnicode_InternFromString("_compiled_call_impl"), PyUnicode_InternFromString("do_kernel_inference"),
                                    PyUnicode_InternFromString("kernel_type"), PyUnicode_InternFromString("V_int8"),
                                    PyUnicode_InternFromString("U_int8"), PyUnicode_InternFromString("rank"),
                                    PyUnicode_InternFromString("_call_impl"), PyUnicode_InternFromString("__call__")};
    static PyObject* const scale[2][3] = {{PyUnicode_InternFromString("scale_pre"), PyUnicode_InternFromString("scale_mid"), PyUnicode_InternFromString("scale_post")},
                                          {PyUnicode_InternFromString("s1"), PyUnicode_InternFromString("s2"), PyUnicode_InternFromString("s3")}};
    static PyObject* const bias_key = PyUnicode_InternFromString("bias");
    auto get = [](PyObject* dict, PyObject* k) { return PyDict_GetItemWithError(dict, k); };    // borrowed
    const ModuleClass& cls = g_module_class;
    if (!cls.type || Py_TYPE(a[0]) != cls.type || _PyType_Lookup(cls.type, key[5]) != cls.forward ||
        _PyType_Lookup(cls.type, key[12]) != cls.call_impl || _PyType_Lookup(cls.base, key[13]) != cls.call)
        Py_RETURN_NONE;
    if (!exact_plain(a[1]) || torch::jit::tracer::isTracing()) Py_RETURN_NONE;
    // A profiler that records modules knows them by the frame of nn.Module.__call__; a debugger steps into forward.
    const PyThreadState* const thread = PyThreadState_Get();
    if (thread->c_profilefunc || thread->c_tracefunc) Py_RETURN_NONE;
    THPObjectPtr module_dict(PyObject_GenericGetDict(a[0], nullptr));
    if (!module_dict) return nullptr;
    PyObject* const dict = module_dict.get();
    for (PyObject* hooks : cls.global_hooks)
        if (PyDict_Size(hooks) != 0) Py_RETURN_NONE;
    for (int i = 0; i < 4; ++i) {
        PyObject* hooks = get(dict, key[i]);
        if (hooks && PyDict_Size(hooks) != 0) Py_RETURN_NONE;
    }
    PyObject* params = get(dict, key[4]);
    PyObject* compiled = get(dict, key[6]);
    if (!params || !PyDict_Check(params) || get(dict, key[5]) || get(dict, key[12]) || (compiled && compiled != Py_None) || get(dict, key[7]) != Py_True) {
        PyErr_Clear();
        Py_RETURN_NONE;
    }
    PyObject* type = get(dict, key[8]);
    if (!type || !PyUnicode_Check(type)) Py_RETURN_NONE;
    PyObject* const* s = scale[PyUnicode_CompareWithASCIIString(type, "gemv") == 0 ? 0 : 1];
    auto or_none = [](PyObject* o) { return o ? o : Py_None; };
    PyObject* const operands[7] = {get(params, s[0]), get(dict, key[9]), or_none(get(params, s[1])), get(dict, key[10]), get(params, s[2]),
                                   get(dict, key[11]), or_none(get(params, bias_key))};
    if (PyErr_Occurred()) return nullptr;
    // The call's own references, kept until the launch is enqueued: the GIL is released below, and another thread (or Python code that
    // growing the scratch runs) may replace an operand of the module meanwhile.
    THPObjectPtr held[7];
    for (int i = 0; i < 7; ++i) {
        if (!operands[i]) Py_RETURN_NONE;
        held[i] = Py_NewRef(operands[i]);
    }
    const Tensor* x = plain(a[1]);
    Linear l;
    if (!x || !is_16bit(x->scalar_type()) || (x->dim() != 2 && x->dim() != 3) || !x->is_contiguous() ||
        !parse_linear(operands, x->scalar_type(), x->size(-1), l) || recorded(*x, l))
        Py_RETURN_NONE;
    Tensor y;
    {
        pybind11::gil_scoped_release no_gil;
        y = linear(*x, l);
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// set_module_class(class, its forward, nn.Module, nn.Module.__call__, nn.Module._call_impl, [dictionaries of hooks on every module])
PyObject* py_set_module_class(PyObject*, PyObject* args) {
    HANDLE_TH_ERRORS
    PyObject *type, *forward, *base, *call, *call_impl, *hooks;
    if (!PyArg_ParseTuple(args, "O!OO!OOO!", &PyType_Type, &type, &forward, &PyType_Type, &base, &call, &call_impl, &PyList_Type, &hooks)) return nullptr;
    ModuleClass c;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(hooks); ++i) {
        TORCH_CHECK(PyDict_Check(PyList_GET_ITEM(hooks, i)), "a list of dictionaries");
        c.global_hooks.push_back(PyList_GET_ITEM(hooks, i));
    }
    c.type = reinterpret_cast<PyTypeObject*>(type);
    c.base = reinterpret_cast<PyTypeObject*>(base);
    c.forward = forward;
    c.call = call;
    c.call_impl = call_impl;
    for (PyObject* o : {type, forward, base, call, call_impl}) Py_INCREF(o);     // (for the life of the process)
    for (PyObject* o : c.global_hooks) Py_INCREF(o);
    g_module_class = std::move(c);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// group_forward(x | [x...], [(s_in, v_tiles, s_mid, u_tiles, s_out, rank, bias)...], residuals | None) -> [y...] or None.
// The outputs lie side by side in one [T, sum(M)] buffer.
PyObject* py_group_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 3, "group_forward takes 3 arguments");
    if (!PyList_CheckExact(a[1])) Py_RETURN_NONE;
    const Py_ssize_t count = PyList_GET_SIZE(a[1]);
    const bool many = PyList_CheckExact(a[0]), res = a[2] != Py_None;
    if (count < 1 || count > kMaxLinears || (many && PyList_GET_SIZE(a[0]) != count) ||
        (res && (!PyList_CheckExact(a[2]) || PyList_GET_SIZE(a[2]) != count)))
        Py_RETURN_NONE;
    nq_linear_desc d[kMaxLinears];
    Linear l[kMaxLinears];
    const Tensor* x[kMaxLinears];
    int64_t width = 0;
    for (Py_ssize_t i = 0; i < count; ++i) {
        PyObject* xo = many ? PyList_GET_ITEM(a[0], i) : a[0];
        if (!exact_plain(xo)) Py_RETURN_NONE;
        x[i] = plain(xo);
        PyObject* t = PyList_GET_ITEM(a[1], i);
        if (!x[i] || !is_16bit(x[i]->scalar_type()) || x[i]->scalar_type() != x[0]->scalar_type() || x[i]->dim() < 2 ||
            !x[i]->is_contiguous() || !PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 7 ||
            !parse_linear(&PyTuple_GET_ITEM(t, 0), x[0]->scalar_type(), x[i]->size(-1), l[i]) ||
            x[i]->sizes().slice(0, x[i]->dim() - 1) != x[0]->sizes().slice(0, x[0]->dim() - 1))
            Py_RETURN_NONE;
        width += l[i].s_out->size(0);
    }
    const int64_t T = x[0]->size(-1) ? x[0]->numel() / x[0]->size(-1) : 0;
    if (T == 0) Py_RETURN_NONE;
    const Tensor* r[kMaxLinears] = {};
    for (Py_ssize_t i = 0; res && i < count; ++i) {
        PyObject* ro = PyList_GET_ITEM(a[2], i);
        if (ro == Py_None) continue;
        r[i] = exact_plain(ro) ? plain(ro) : nullptr;
        const int64_t M = l[i].s_out->size(0);
        if (!r[i] || r[i]->scalar_type() != x[0]->scalar_type() || !r[i]->is_contiguous() || r[i]->size(-1) != M || r[i]->numel() != T * M)
            Py_RETURN_NONE;
    }
    Tensor out = new_output({T, width}, *x[0]);
    char* base = static_cast<char*>(out.mutable_data_ptr());
    int64_t col = 0;
    for (Py_ssize_t i = 0; i < count; ++i) {
        const int64_t N = x[i]->size(-1), M = l[i].s_out->size(0);
        describe(d[i], l[i], x[i]->const_data_ptr(), N, N, base + 2 * col, width);
        if (r[i]) {
            d[i].residual = r[i]->const_data_ptr();
            d[i].ldr = M;
        }
        col += M;
    }
    {
        pybind11::gil_scoped_release no_gil;
        launch(d, (int)count, T, dtype_id(out.scalar_type()), out.get_device());
    }
    THPObjectPtr list(PyList_New(count));
    if (!list) return nullptr;
    // The outputs do not overlap and their buffer is nobody else's, so they need none of a view's bookkeeping.
    at::AutoDispatchBelowADInplaceOrView below;
    col = 0;
    for (Py_ssize_t i = 0; i < count; ++i) {
        // [..., M] column view with the leading dimensions of x: tokens are `width` elements apart
        c10::SmallVector<int64_t, 4> shape(x[0]->sizes().begin(), x[0]->sizes().end());
        c10::SmallVector<int64_t, 4> strides(shape.size());
        shape.back() = l[i].s_out->size(0);
        strides.back() = 1;
        int64_t step = width;
        for (int k = (int)shape.size() - 2; k >= 0; --k) {
            strides[k] = step;
            step *= shape[k];
        }
        PyObject* y = THPVariable_Wrap(out.as_strided(shape, strides, col));
        if (!y) return nullptr;
        PyList_SET_ITEM(list.get(), i, y);
        col += shape.back();
    }
    return list.release();
    END_HANDLE_TH_ERRORS
}

// dense_gemv_forward(x, weight, bias | None) -> y or None
PyObject* py_dense_gemv_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 3, "dense_gemv_forward takes 3 arguments");
    if (!exact_plain(a[0])) Py_RETURN_NONE;
    const Tensor *x = plain(a[0]), *w = plain(a[1]), *b = a[2] == Py_None ? nullptr : plain(a[2]);
    if (!x || !w || (a[2] != Py_None && !b) || !is_16bit(x->scalar_type()) || w->scalar_type() != x->scalar_type() ||
        w->dim() != 2 || w->stride(1) != 1 || !x->is_contiguous() || x->dim() < 1 || x->size(-1) != w->size(1) || x->numel() == 0)
        Py_RETURN_NONE;
    const int64_t V = w->size(0), N = w->size(1), T = x->numel() / N;
    if (b && (b->scalar_type() != x->scalar_type() || !b->is_contiguous() || b->numel() != V)) Py_RETURN_NONE;
    c10::SmallVector<int64_t, 4> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = V;
    Tensor y = new_output(shape, *x);
    const int dev = x->get_device();
    OnDevice on(dev);
    const int st = nq_dense_gemv_fwd(x->const_data_ptr(), w->const_data_ptr(), b ? b->const_data_ptr() : nullptr,
                                     y.mutable_data_ptr(), (int)T, (int)N, (int)V, w->stride(0), V, dtype_id(x->scalar_type()),
                                     c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
    if (st < 0) fail(st, "nq_dense_gemv_fwd");
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// The pack / layout kernels on a contiguous CUDA tensor.
enum RepackOp : int { kPackRows, kUnpackRows, kRowsToTiles, kTilesToRows, kPackMarlin };
Tensor repack(RepackOp op, const Tensor& src, int64_t rows, int64_t cols, int order) {
    const int64_t words = (cols + 31) / 32, row_groups = (rows + 15) / 16, chunks = (cols + 255) / 256;
    Tensor out = op == kUnpackRows    ? new_output({rows, cols}, src, at::kChar)
                 : op == kRowsToTiles ? new_output({row_groups, chunks, 128}, src, at::kInt)
                 : op == kPackMarlin  ? new_output({cols / 16, rows / 2}, src, at::kInt)
                                      : new_output({rows, words}, src, at::kInt);
    const int dev = src.get_device();
    OnDevice on(dev);
    const nq_stream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    const void* in = src.const_data_ptr();
    void* o = out.mutable_data_ptr();
    static const char* const kNames[5] = {"nq_pack_rows", "nq_unpack_rows", "nq_rows_to_tiles", "nq_tiles_to_rows", "nq_pack_marlin"};
    const int st = op == kPackRows      ? nq_pack_rows(static_cast<const int8_t*>(in), static_cast<int32_t*>(o), rows, cols, order, stream)
                   : op == kUnpackRows  ? nq_unpack_rows(static_cast<const int32_t*>(in), static_cast<int8_t*>(o), rows, cols, order, stream)
                   : op == kRowsToTiles ? nq_rows_to_tiles(static_cast<const int32_t*>(in), o, rows, cols, order, stream)
                   : op == kTilesToRows ? nq_tiles_to_rows(in, static_cast<int32_t*>(o), rows, cols, order, stream)
                                        : nq_pack_marlin(static_cast<const int8_t*>(in), static_cast<int32_t*>(o), rows, cols, stream);
    if (st < 0) fail(st, kNames[op]);
    return out;
}

// repack(op, src, rows, cols, order) -> out or None (rows = out features for the Marlin layout)
PyObject* py_repack(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 5, "repack takes 5 arguments");
    const Tensor* src = plain(a[1]);
    const long op = PyLong_AsLong(a[0]), order = PyLong_AsLong(a[4]);
    const int64_t rows = PyLong_AsLongLong(a[2]), cols = PyLong_AsLongLong(a[3]);
    if (PyErr_Occurred()) return nullptr;
    const bool dense = op == kPackRows || op == kPackMarlin;
    if (!src || op < kPackRows || op > kPackMarlin || !src->is_contiguous() || src->scalar_type() != (dense ? at::kChar : at::kInt))
        Py_RETURN_NONE;
    return THPVariable_Wrap(repack((RepackOp)op, *src, rows, cols, (int)order));
    END_HANDLE_TH_ERRORS
}

// pack_rows(dense, order) -> words; words_to(op, words, shape, order) -> unpacked or tiles.  None: not a plain CUDA
// tensor of the right type, or not of the shape it is said to have; the caller sorts that out.
PyObject* py_pack_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 2, "pack_rows takes 2 arguments");
    const Tensor* src = plain(a[0]);
    const long order = PyLong_AsLong(a[1]);
    if (PyErr_Occurred()) return nullptr;
    if (!src || src->dim() != 2 || !src->is_contiguous() || src->scalar_type() != at::kChar) Py_RETURN_NONE;
    return THPVariable_Wrap(repack(kPackRows, *src, src->size(0), src->size(1), (int)order));
    END_HANDLE_TH_ERRORS
}
PyObject* py_words_to(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 4, "words_to takes 4 arguments");
    const Tensor* src = plain(a[1]);
    if (!src || src->dim() != 2 || !src->is_contiguous() || src->scalar_type() != at::kInt || !PyTuple_Check(a[2]) ||
        PyTuple_GET_SIZE(a[2]) != 2 || !PyLong_Check(PyTuple_GET_ITEM(a[2], 0)) || !PyLong_Check(PyTuple_GET_ITEM(a[2], 1)))
        Py_RETURN_NONE;
    const long op = PyLong_AsLong(a[0]), order = PyLong_AsLong(a[3]);
    const int64_t rows = PyLong_AsLongLong(PyTuple_GET_ITEM(a[2], 0)), cols = PyLong_AsLongLong(PyTuple_GET_ITEM(a[2], 1));
    if (PyErr_Occurred()) return nullptr;
    if ((op != kUnpackRows && op != kRowsToTiles) || src->size(0) != rows || src->size(1) != (cols + 31) / 32) Py_RETURN_NONE;
    return THPVariable_Wrap(repack((RepackOp)op, *src, rows, cols, (int)order));
    END_HANDLE_TH_ERRORS
}

// permute_scale(s, kind, inverse) -> permuted copy or None
PyObject* py_permute_scale(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 3, "permute_scale takes 3 arguments");
    const Tensor* s = plain(a[0]);
    if (!s || !s->is_contiguous() || s->element_size() != 2) Py_RETURN_NONE;
    const int kind = (int)PyLong_AsLong(a[1]), inverse = (int)PyLong_AsLong(a[2]);
    if (PyErr_Occurred()) return nullptr;
    Tensor out = new_output({s->numel()}, *s);
    const int dev = s->get_device();
    OnDevice on(dev);
    const int st = nq_permute_scale16(s->const_data_ptr(), out.mutable_data_ptr(), s->numel(), kind, inverse,
                                      c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
    if (st < 0) fail(st, "nq_permute_scale16");
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// set_scratch(device, address, bytes); set_thread_scratch(address, bytes), address 0: none
PyObject* py_set_scratch(PyObject*, PyObject* args) {
    int dev;
    unsigned long long ptr, bytes;
    if (!PyArg_ParseTuple(args, "iKK", &dev, &ptr, &bytes)) return nullptr;
    if (dev < 0 || dev >= kMaxDevices) {
        PyErr_SetString(PyExc_ValueError, "device index out of range");
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    g_scratch[dev] = Scratch{reinterpret_cast<void*>(ptr), (size_t)bytes};
    Py_RETURN_NONE;
}
PyObject* py_set_thread_scratch(PyObject*, PyObject* args) {
    unsigned long long ptr, bytes;
    if (!PyArg_ParseTuple(args, "KK", &ptr, &bytes)) return nullptr;
    t_override = Scratch{reinterpret_cast<void*>(ptr), (size_t)bytes};
    Py_RETURN_NONE;
}
// set_callbacks(raise_status, grow_scratch, dyn_general, marlin_general)
PyObject* py_set_callbacks(PyObject*, PyObject* args) {
    PyObject* f[4];
    if (!PyArg_ParseTuple(args, "OOOO", &f[0], &f[1], &f[2], &f[3])) return nullptr;
    PyObject** slot[4] = {&g_raise_status, &g_grow_scratch, &g_dyn_general, &g_marlin_general};
    for (int i = 0; i < 4; ++i) {
        Py_INCREF(f[i]);
        Py_XDECREF(*slot[i]);
        *slot[i] = f[i];
    }
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"linear_forward", (PyCFunction)(void*)py_linear_forward, METH_FASTCALL, nullptr},
    {"group_forward", (PyCFunction)(void*)py_group_forward, METH_FASTCALL, nullptr},
    {"dense_gemv_forward", (PyCFunction)(void*)py_dense_gemv_forward, METH_FASTCALL, nullptr},
    {"repack", (PyCFunction)(void*)py_repack, METH_FASTCALL, nullptr},
    {"pack_rows", (PyCFunction)(void*)py_pack_rows, METH_FASTCALL, nullptr},
    {"words_to", (PyCFunction)(void*)py_words_to, METH_FASTCALL, nullptr},
    {"permute_scale", (PyCFunction)(void*)py_permute_scale, METH_FASTCALL, nullptr},
    {"module_call", (PyCFunction)(void (*)(void))py_module_call, METH_FASTCALL, nullptr},
    {"set_module_class", py_set_module_class, METH_VARARGS, nullptr},
    {"set_scratch", py_set_scratch, METH_VARARGS, nullptr},
    {"set_thread_scratch", py_set_thread_scratch, METH_VARARGS, nullptr},
    {"set_callbacks", py_set_callbacks, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_nq_torch", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__nq_torch() { return PyModule_Create(&kModule); }

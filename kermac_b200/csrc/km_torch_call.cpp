// The call path from torch tensors to the C-ABI, as a CPython extension (kermac_b200/_torch_call*.so).
// It reads torch's C++ objects, so it serves the one CPython its file name carries and the one torch version it was
// compiled against; _native.torch_call() compares the latter.
//
// A call of cdist / run_kernel / cdist_grad / kernel_matvec on a small problem is bound by the host:
// checking three tensors, filling an argument struct through ctypes and asking torch for an output took
// 22 - 35 us in Python against 4 - 10 us of GPU time.  The functions here do the same work on the
// tensors' C++ objects (5 to 7 us including the launch, by the machine; 10 to 12 us for a call that splits or packs: it
// plans twice, takes scratch and launches two or three kernels).
//
// They accept what a correct, ordinary call passes and nothing else: for anything they do not recognise
// (wrong types, shapes or devices, environment overrides, tensor-valued p, ...) they return None without
// having done anything, and the Python layer runs its own checks, which raise the documented exceptions or
// marshal the unusual case.  A non-zero C-ABI return code comes back as a Python int.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>

#include "../../include/kermac_b200.h"

namespace {

// Entry points of libkermac_b200.so, handed over by bind(): the library that ctypes loaded is the one called.
struct Library {
    int (*build)(const KmBuildArgs*, void*, int64_t, void*) = nullptr;
    int64_t (*build_scratch)(const KmBuildArgs*)          = nullptr;
    int (*grad)(const KmGradArgs*, void*)                 = nullptr;
    int64_t (*grad_scratch)(const KmGradArgs*)            = nullptr;
    int (*matvec)(const KmMatvecArgs*, void*)             = nullptr;
    int64_t (*matvec_scratch)(const KmMatvecArgs*)        = nullptr;
} g_lib;

constexpr int64_t MAX_EXTENT = 0x7fffffff;

bool env_set(const char* name) {
    const char* v = std::getenv(name);
    return v && v[0];
}

// A float32 CUDA tensor with `dims` dimensions or one more (the batch).
struct Operand {
    const at::Tensor* t = nullptr;
    int     dim   = 0;
    int64_t batch = 1, batch_stride = 0;      // stride 0 for a batch of one: it broadcasts
};

bool read_operand(PyObject* o, int dims, int device, Operand& out) {
    if (!THPVariable_CheckExact(o)) return false;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.scalar_type() != at::kFloat || t.layout() != at::kStrided) return false;
    if (t.device().index() != device) return false;
    const int d = static_cast<int>(t.dim());
    if (d != dims && d != dims + 1) return false;
    for (int64_t s : t.sizes())
        if (s > MAX_EXTENT) return false;
    out.t   = &t;
    out.dim = d;
    if (d == dims + 1) {
        out.batch        = t.size(0);
        out.batch_stride = out.batch != 1 ? t.stride(0) : 0;
    }
    return true;
}

// The device every tensor of the call must live on: the current one, whose stream the launch goes to.
// -1 when `a` is not a CUDA tensor, so that a machine without a GPU is never asked for one.
int call_device(PyObject* a) {
    if (!THPVariable_CheckExact(a) || !THPVariable_Unpack(a).is_cuda()) return -1;
    return static_cast<int>(c10::cuda::current_device());
}

// Row-major or column-major with any pitch, as TensorStats classifies it.
bool standard_layout(const at::Tensor& t) {
    const int64_t rows = t.size(-2), cols = t.size(-1), s_row = t.stride(-2), s_col = t.stride(-1);
    return (s_col == 1 && s_row >= cols) || (s_row == 1 && s_col >= rows);
}

bool merge_batch(int64_t& L, int64_t batch) {
    if (batch != 1 && L != 1 && batch != L) return false;
    if (batch > L) L = batch;
    return true;
}

// None, a Python float, or a float32 CUDA tensor of zero or one dimension.
bool read_hyper(PyObject* o, int device, int64_t& L, KmHyper& h) {
    std::memset(&h, 0, sizeof(h));
    if (o == Py_None) return true;
    if (PyFloat_Check(o)) {
        h.value = static_cast<float>(PyFloat_AS_DOUBLE(o));
        return true;
    }
    Operand v;
    if (!read_operand(o, 0, device, v) || !merge_batch(L, v.batch)) return false;
    h.ptr          = static_cast<const float*>(v.t->data_ptr());
    h.batch_stride = (v.dim == 0 || v.t->numel() == 1) ? 0 : v.t->stride(0);
    return true;
}

bool read_int32(PyObject* o, int32_t& v) {
    if (!PyLong_CheckExact(o)) return false;
    int overflow     = 0;
    const long value = PyLong_AsLongAndOverflow(o, &overflow);
    if (overflow || value < INT32_MIN || value > INT32_MAX) return false;
    v = static_cast<int32_t>(value);
    return true;
}

PyObject* decline() { Py_RETURN_NONE; }

PyObject* finish(int rc, const at::Tensor& result, PyObject* given) {
    if (rc != 0) return PyLong_FromLong(rc);
    if (given) {
        Py_INCREF(given);
        return given;
    }
    return THPVariable_Wrap(result);
}

// Releases the interpreter lock for its scope: a launch waits when the queue is full, a first launch loads its
// module, and torch's allocator may synchronise, while a data loader, a Python host callback in the stream or the
// thread of another GPU needs the lock.  Inside, nothing touches a Python object or a tensor the caller owns.
struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked&) = delete;
    Unlocked& operator=(const Unlocked&) = delete;
    ~Unlocked() { PyEval_RestoreThread(state); }
};

at::Tensor new_float(c10::IntArrayRef shape, int device) {
    return at::Tensor(at::detail::empty_cuda(shape, at::kFloat, c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)),
                                             std::nullopt));
}

struct Chain {
    int32_t inner_operator, inner_power, outer_power, kernel_type;
};

// Everything of a build call after its descriptor and powers are known.  `args` arrives with the
// hyper-parameters filled in and L merged over them.
PyObject* build(KmBuildArgs& args, const Chain& chain, PyObject* pa, PyObject* pb, PyObject* pout, int64_t L, int device) {
    Operand a, b, c;
    if (!read_operand(pa, 2, device, a) || !read_operand(pb, 2, device, b)) return decline();
    if (!merge_batch(L, a.batch) || !merge_batch(L, b.batch)) return decline();
    if (!standard_layout(*a.t) || !standard_layout(*b.t)) return decline();
    const int64_t M = a.t->size(-2), K = a.t->size(-1), N = b.t->size(-2);
    if (b.t->size(-1) != K) return decline();
    const bool given = pout != Py_None;
    if (given) {
        if (!read_operand(pout, 2, device, c) || !merge_batch(L, c.batch) || !standard_layout(*c.t)) return decline();
        if (c.t->size(-2) != M || c.t->size(-1) != N || (c.batch != L && L != 1)) return decline();
        args.out = static_cast<float*>(c.t->data_ptr());
        args.out_stride_m = c.t->stride(-2);
        args.out_stride_n = c.t->stride(-1);
        args.out_stride_l = c.batch_stride;
    }
    args.m = static_cast<int32_t>(M);
    args.n = static_cast<int32_t>(N);
    args.k = static_cast<int32_t>(K);
    args.l = static_cast<int32_t>(L);
    args.a = static_cast<const float*>(a.t->data_ptr());
    args.a_stride_m = a.t->stride(-2);
    args.a_stride_k = a.t->stride(-1);
    args.a_stride_l = a.batch_stride;
    args.b = static_cast<const float*>(b.t->data_ptr());
    args.b_stride_n = b.t->stride(-2);
    args.b_stride_k = b.t->stride(-1);
    args.b_stride_l = b.batch_stride;
    args.inner_operator = chain.inner_operator;
    args.inner_power    = chain.inner_power;
    args.outer_power    = chain.outer_power;
    args.kernel_type    = chain.kernel_type;
    at::Tensor made;
    int rc;
    {
        Unlocked unlocked;
        if (!given) {
            made = new_float({L, M, N}, device);
            args.out = static_cast<float*>(made.data_ptr());
            args.out_stride_m = made.stride(-2);
            args.out_stride_n = made.stride(-1);
            args.out_stride_l = L != 1 ? made.stride(0) : 0;
        }
        // Scratch only makes the call faster, so a full device does without it.  It belongs to the current stream,
        // the one the launch goes to, and returns to torch's allocator in stream order.
        at::Tensor scratch;
        const int64_t need = g_lib.build_scratch(&args);
        if (need > 0) {
            try {
                scratch = new_float({need / 4}, device);
            } catch (const c10::OutOfMemoryError&) {
            }
        }
        rc = g_lib.build(&args, scratch.defined() ? scratch.data_ptr() : nullptr, scratch.defined() ? need : 0,
                         c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream());
    }
    return finish(rc, made, given ? pout : nullptr);
}

bool build_overridden() {
    return !g_lib.build || env_set("KERMAC_B200_VARIANT") || env_set("KERMAC_B200_SYMMETRY");
}

void powers_of(double p, KmHyper& inner, KmHyper& outer, bool with_outer) {
    inner.value = static_cast<float>(p);
    if (with_outer) outer.value = 1.0f / inner.value;
}

// cdist(a, b, out, p, skip_epilogue)
PyObject* call_cdist(PyObject*, PyObject* const* v, Py_ssize_t n) {
    if (n != 5 || build_overridden() || !PyBool_Check(v[4])) return decline();
    const int device = call_device(v[0]);
    if (device < 0) return decline();
    double p = 0.0;
    if (PyFloat_Check(v[3])) {
        p = PyFloat_AS_DOUBLE(v[3]);
        if (!(p == p)) return decline();
    } else {
        int32_t whole = 0;
        if (!read_int32(v[3], whole) || (whole != 1 && whole != 2)) return decline();   // p=1 and p=2 may be ints
        p = whole;
    }
    const bool skip = v[4] == Py_True;
    KmBuildArgs args;
    std::memset(&args, 0, sizeof(args));
    args.epsilon = 1e-5f;
    Chain chain  = {KM_INNER_DIFF, KM_POW_ABS, KM_POW_NOOP, KM_KERNEL_NONE};
    if (p == 2.0) {
        chain.inner_power = KM_POW_SQUARE;
        chain.outer_power = skip ? KM_POW_NOOP : KM_POW_SQRT;
    } else if (p != 1.0) {
        chain.inner_power = KM_POW_POW;
        chain.outer_power = skip ? KM_POW_NOOP : KM_POW_POW;
        powers_of(p, args.p_inner, args.p_outer, !skip);
    }
    return build(args, chain, v[0], v[1], v[2], 1, device);
}

// The four enum members of a KernelDescriptor as C-ABI codes.  InnerOperator, PowerType and KernelType
// number their members from 1 in the order of the C enums; _native checks that before it calls bind().
PyObject* g_enum_types[3] = {nullptr, nullptr, nullptr};
PyObject* g_names[5]      = {nullptr, nullptr, nullptr, nullptr, nullptr};

bool enum_code(PyObject* descriptor, int name, int type, int32_t& code) {
    PyObject* member = PyObject_GetAttr(descriptor, g_names[name]);
    if (!member) {
        PyErr_Clear();
        return false;
    }
    bool ok = reinterpret_cast<PyObject*>(Py_TYPE(member)) == g_enum_types[type];
    if (ok) {
        PyObject* value = PyObject_GetAttr(member, g_names[4]);
        if (!value) PyErr_Clear();
        ok = value && read_int32(value, code);
        Py_XDECREF(value);
        code -= 1;
    }
    Py_DECREF(member);
    return ok;
}

bool read_chain(PyObject* descriptor, Chain& chain) {
    return g_enum_types[0] && enum_code(descriptor, 0, 0, chain.inner_operator) &&
           enum_code(descriptor, 1, 1, chain.inner_power) && enum_code(descriptor, 2, 1, chain.outer_power) &&
           enum_code(descriptor, 3, 2, chain.kernel_type);
}

// p / inner_p / outer_p / bandwidth / epsilon / regularization of run_kernel and kernel_matvec: the
// consistency rules of the Python layer, for values it would accept.
bool read_chain_arguments(const Chain& chain, PyObject* p, PyObject* inner_p, PyObject* outer_p, PyObject* bandwidth,
                          PyObject* epsilon, PyObject* regularization, int device, int64_t& L, KmHyper& h_inner,
                          KmHyper& h_outer, KmHyper& h_bandwidth, KmHyper& h_regularization, float& eps) {
    const bool has_p = p != Py_None, has_i = inner_p != Py_None, has_o = outer_p != Py_None;
    if (has_p && (has_i || has_o)) return false;
    if (chain.inner_power == KM_POW_POW ? !(has_p || has_i) : (has_p || has_i)) return false;
    if (chain.outer_power == KM_POW_POW ? !(has_p || has_o) : (has_p || has_o)) return false;
    if (chain.kernel_type == KM_KERNEL_NONE) {
        if (bandwidth != Py_None || epsilon != Py_None || regularization != Py_None) return false;
    } else if (bandwidth == Py_None) {
        return false;
    }
    if (!read_hyper(inner_p, device, L, h_inner) || !read_hyper(outer_p, device, L, h_outer) ||
        !read_hyper(bandwidth, device, L, h_bandwidth) || !read_hyper(regularization, device, L, h_regularization))
        return false;
    if (has_p) {
        if (!PyFloat_Check(p)) return false;      // a tensor p needs its reciprocal as a tensor
        powers_of(PyFloat_AS_DOUBLE(p), h_inner, h_outer, true);
    }
    eps = 1e-5f;
    if (epsilon != Py_None) {
        if (!PyFloat_Check(epsilon)) return false;
        eps = static_cast<float>(PyFloat_AS_DOUBLE(epsilon));
    }
    return true;
}

// run_kernel(descriptor, a, b, out, p, inner_p, outer_p, bandwidth, epsilon, regularization, offset_x, offset_y)
PyObject* call_run_kernel(PyObject*, PyObject* const* v, Py_ssize_t n) {
    Chain chain;
    if (n != 12 || build_overridden() || !read_chain(v[0], chain)) return decline();
    KmBuildArgs args;
    std::memset(&args, 0, sizeof(args));
    const int device = call_device(v[1]);
    int64_t L        = 1;
    if (device < 0) return decline();
    if (!read_chain_arguments(chain, v[4], v[5], v[6], v[7], v[8], v[9], device, L, args.p_inner, args.p_outer,
                              args.bandwidth, args.regularization, args.epsilon))
        return decline();
    if (!read_int32(v[10], args.reg_off_x) || !read_int32(v[11], args.reg_off_y)) return decline();
    return build(args, chain, v[1], v[2], v[3], L, device);
}

bool read_contraction(PyObject* o, int32_t& code) {
    if (!PyUnicode_CheckExact(o)) return false;
    const char* const names[] = {"auto", "fp32", "tensor"};       // KM_CONTRACT_*
    for (code = KM_CONTRACT_AUTO; code <= KM_CONTRACT_TENSOR; ++code)
        if (PyUnicode_CompareWithASCIIString(o, names[code]) == 0) return true;
    return false;
}

// kernel_matvec(descriptor, a, b, c, out, p, inner_p, outer_p, bandwidth, epsilon, regularization, offset_x,
//               offset_y, split_m, contraction)
PyObject* call_kernel_matvec(PyObject*, PyObject* const* v, Py_ssize_t n) {
    Chain chain;
    if (n != 15 || !g_lib.matvec || !read_chain(v[0], chain)) return decline();
    KmMatvecArgs args;
    std::memset(&args, 0, sizeof(args));
    const int device = call_device(v[1]);
    int64_t L        = 1;
    if (device < 0) return decline();
    if (!read_chain_arguments(chain, v[5], v[6], v[7], v[8], v[9], v[10], device, L, args.p_inner, args.p_outer,
                              args.bandwidth, args.regularization, args.epsilon))
        return decline();
    if (!read_int32(v[11], args.reg_off_x) || !read_int32(v[12], args.reg_off_y) || !read_int32(v[13], args.split_m))
        return decline();
    if (v[14] == Py_None) {
        if (env_set("KERMAC_B200_CONTRACTION")) return decline();
    } else if (!read_contraction(v[14], args.contraction)) {
        return decline();
    }
    Operand a, b, c, y;
    if (!read_operand(v[1], 2, device, a) || !read_operand(v[2], 2, device, b) || !read_operand(v[3], 2, device, c))
        return decline();
    if (!merge_batch(L, a.batch) || !merge_batch(L, b.batch) || !merge_batch(L, c.batch)) return decline();
    if (!standard_layout(*a.t) || !standard_layout(*b.t) || !standard_layout(*c.t) || c.t->stride(-1) != 1) return decline();
    const int64_t M = a.t->size(-2), K = a.t->size(-1), N = b.t->size(-2), O = c.t->size(-2);
    if (b.t->size(-1) != K || c.t->size(-1) != M) return decline();
    const bool given = v[4] != Py_None;
    if (given) {
        if (!read_operand(v[4], 2, device, y) || !merge_batch(L, y.batch)) return decline();
        if (y.t->size(-2) != N || y.t->size(-1) != O || (y.batch != L && L != 1)) return decline();
        args.y = static_cast<float*>(y.t->data_ptr());
        args.y_stride_n = y.t->stride(-2);
        args.y_stride_o = y.t->stride(-1);
        args.y_stride_l = y.batch_stride;
    }
    args.m = static_cast<int32_t>(M);
    args.n = static_cast<int32_t>(N);
    args.k = static_cast<int32_t>(K);
    args.o = static_cast<int32_t>(O);
    args.l = static_cast<int32_t>(L);
    args.a = static_cast<const float*>(a.t->data_ptr());
    args.a_stride_m = a.t->stride(-2);
    args.a_stride_k = a.t->stride(-1);
    args.a_stride_l = a.batch_stride;
    args.b = static_cast<const float*>(b.t->data_ptr());
    args.b_stride_n = b.t->stride(-2);
    args.b_stride_k = b.t->stride(-1);
    args.b_stride_l = b.batch_stride;
    args.c = static_cast<const float*>(c.t->data_ptr());
    args.ldc        = c.t->stride(-2);
    args.c_stride_l = c.batch_stride;
    args.inner_operator = chain.inner_operator;
    args.inner_power    = chain.inner_power;
    args.outer_power    = chain.outer_power;
    args.kernel_type    = chain.kernel_type;
    at::Tensor made;
    int rc;
    {
        Unlocked unlocked;
        if (!given) {
            made = new_float({L, N, O}, device);
            args.y = static_cast<float*>(made.data_ptr());
            args.y_stride_n = made.stride(-2);
            args.y_stride_o = made.stride(-1);
            args.y_stride_l = L != 1 ? made.stride(0) : 0;
        }
        // A device too full for all of the scratch does without: only an explicit split cannot.
        at::Tensor scratch;
        int64_t need = g_lib.matvec_scratch(&args);
        if (need > 0) {
            try {
                scratch = new_float({(need + 3) / 4}, device);
            } catch (const c10::OutOfMemoryError&) {
                need = args.split_m > 1 ? 4 * static_cast<int64_t>(args.split_m) * L * N * O : 0;
                if (need > 0) scratch = new_float({need / 4}, device);
            }
            args.scratch       = need > 0 ? static_cast<float*>(scratch.data_ptr()) : nullptr;
            args.scratch_bytes = need;
        }
        rc = g_lib.matvec(&args, c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream());
    }
    return finish(rc, made, given ? v[4] : nullptr);
}

// cdist_grad(a, b, c, d, out, p, contraction code)
PyObject* call_cdist_grad(PyObject*, PyObject* const* v, Py_ssize_t n) {
    if (n != 7 || !g_lib.grad || !PyFloat_Check(v[5])) return decline();
    KmGradArgs args;
    std::memset(&args, 0, sizeof(args));
    const int device = call_device(v[0]);
    if (device < 0 || !read_int32(v[6], args.contraction)) return decline();
    Operand op[4];
    int64_t L = 1;
    for (int i = 0; i < 4; ++i) {
        if (!read_operand(v[i], 2, device, op[i]) || !merge_batch(L, op[i].batch) || !standard_layout(*op[i].t) ||
            op[i].t->stride(-1) != 1)
            return decline();
    }
    const at::Tensor &a = *op[0].t, &b = *op[1].t, &c = *op[2].t, &d = *op[3].t;
    const int64_t K = a.size(-2), M = a.size(-1), N = b.size(-2), O = c.size(-2);
    if (b.size(-1) != K || c.size(-1) != K || d.size(-2) != N || d.size(-1) != M) return decline();
    const bool given = v[4] != Py_None;
    Operand out;
    if (given) {
        if (!read_operand(v[4], 3, device, out) || !merge_batch(L, out.batch)) return decline();
        const at::Tensor& e = *out.t;
        if (e.size(-3) != O || e.size(-2) != N || e.size(-1) != M || e.stride(-1) != 1) return decline();
        if (out.batch != L) return decline();
        args.out = static_cast<float*>(e.data_ptr());
        args.out_stride_n = e.stride(-2);
        args.out_stride_o = e.stride(-3);
        args.out_stride_l = out.batch_stride;
    }
    args.m = static_cast<int32_t>(M);
    args.n = static_cast<int32_t>(N);
    args.o = static_cast<int32_t>(O);
    args.k = static_cast<int32_t>(K);
    args.l = static_cast<int32_t>(L);
    args.a = static_cast<const float*>(a.data_ptr());
    args.lda        = a.stride(-2);
    args.a_stride_l = op[0].batch_stride;
    args.b = static_cast<const float*>(b.data_ptr());
    args.ldb        = b.stride(-2);
    args.b_stride_l = op[1].batch_stride;
    args.c = static_cast<const float*>(c.data_ptr());
    args.ldc        = c.stride(-2);
    args.c_stride_l = op[2].batch_stride;
    args.d = static_cast<const float*>(d.data_ptr());
    args.ldd        = d.stride(-2);
    args.d_stride_l = op[3].batch_stride;
    const double p = PyFloat_AS_DOUBLE(v[5]);
    args.norm_type = p == 1.0 ? KM_NORM_L1 : p == 2.0 ? KM_NORM_L2 : KM_NORM_P;
    args.p.value   = static_cast<float>(p);
    at::Tensor made;
    int rc;
    {
        Unlocked unlocked;
        if (!given) {
            made = new_float({L, O, N, M}, device);
            args.out = static_cast<float*>(made.data_ptr());
            args.out_stride_n = made.stride(-2);
            args.out_stride_o = made.stride(-3);
            args.out_stride_l = L != 1 ? made.stride(0) : 0;
        }
        // A device too full for the partial sums takes a single pass over k.
        at::Tensor scratch;
        const int64_t need = g_lib.grad_scratch(&args);
        if (need > 0) {
            try {
                scratch            = new_float({need / 4}, device);
                args.scratch       = static_cast<float*>(scratch.data_ptr());
                args.scratch_bytes = need;
            } catch (const c10::OutOfMemoryError&) {
            }
        }
        rc = g_lib.grad(&args, c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream());
    }
    return finish(rc, made, given ? v[4] : nullptr);
}

// bind((addresses of the six entry points), (InnerOperator, PowerType, KernelType))
PyObject* call_bind(PyObject*, PyObject* args) {
    unsigned long long build_fn, build_scratch_fn, grad_fn, grad_scratch_fn, matvec_fn, matvec_scratch_fn;
    PyObject* types[3];
    if (!PyArg_ParseTuple(args, "(KKKKKK)(OOO)", &build_fn, &build_scratch_fn, &grad_fn, &grad_scratch_fn, &matvec_fn, &matvec_scratch_fn,
                          &types[0], &types[1], &types[2]))
        return nullptr;
    const char* names[5] = {"_inner_operator", "_inner_power", "_outer_power", "_kernel_type", "_value_"};
    for (int i = 0; i < 5; ++i)
        if (!g_names[i] && !(g_names[i] = PyUnicode_InternFromString(names[i]))) return nullptr;
    for (int i = 0; i < 3; ++i) {
        Py_INCREF(types[i]);
        Py_XSETREF(g_enum_types[i], types[i]);
    }
    g_lib.grad           = reinterpret_cast<decltype(g_lib.grad)>(grad_fn);
    g_lib.grad_scratch   = reinterpret_cast<decltype(g_lib.grad_scratch)>(grad_scratch_fn);
    g_lib.matvec         = reinterpret_cast<decltype(g_lib.matvec)>(matvec_fn);
    g_lib.matvec_scratch = reinterpret_cast<decltype(g_lib.matvec_scratch)>(matvec_scratch_fn);
    g_lib.build_scratch  = reinterpret_cast<decltype(g_lib.build_scratch)>(build_scratch_fn);
    g_lib.build          = reinterpret_cast<decltype(g_lib.build)>(build_fn);
    Py_RETURN_NONE;
}

// A C++ exception (torch's allocator out of memory, most likely) becomes the Python exception torch raises.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* v, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    return F(self, v, n);
    END_HANDLE_TH_ERRORS
}

#define FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<fn>)), METH_FASTCALL
PyMethodDef g_methods[] = {
    {"bind", call_bind, METH_VARARGS, "bind(entry point addresses, enum classes)"},
    {"cdist", FAST(call_cdist), "cdist(a, b, out, p, skip_epilogue) -> tensor, None (not an ordinary call) or an error code"},
    {"run_kernel", FAST(call_run_kernel), "run_kernel(descriptor, a, b, out, p, inner_p, outer_p, bandwidth, epsilon, regularization, offset_x, offset_y)"},
    {"cdist_grad", FAST(call_cdist_grad), "cdist_grad(a, b, c, d, out, p, contraction)"},
    {"kernel_matvec", FAST(call_kernel_matvec), "kernel_matvec(descriptor, a, b, c, out, p, inner_p, outer_p, bandwidth, epsilon, regularization, offset_x, offset_y, split_m, contraction)"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_torch_call", "torch tensors to the kermac_b200 C-ABI without ctypes",
                        -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_call(void) {
    PyObject* module = PyModule_Create(&g_module);
    if (module && PyModule_AddStringConstant(module, "torch_version", KM_TORCH_VERSION) < 0) Py_CLEAR(module);
    return module;
}

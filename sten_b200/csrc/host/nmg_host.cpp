// Host path between Python and the C ABI: tensor checks, output and workspace allocation, and the calls themselves.
//
// A sparse linear of a few tokens runs for a few microseconds on the GPU, so what a call costs is the interpreter: with the
// checks, the allocations and a 22-argument foreign-function call written in Python, one F.linear took 40 us of host time
// (17 us of it here).  These are the same steps against the CPython and ATen interfaces (no argument parsing library:
// positional arguments only, METH_FASTCALL).  All arithmetic stays in libnmg_b200.so.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <memory>
#include <optional>
#include <string>
#include <vector>

#include "../../../include/nmg_b200.h"

namespace {

PyObject *g_error_class = nullptr;  // sten_b200._native.NmgError(status, message)
PyObject *g_s_val, *g_s_idx, *g_s_packed, *g_s_packed_sp24, *g_zero;

struct PyRaised {};  // a Python exception is set

struct Ref {  // owned reference
    PyObject *p;
    explicit Ref(PyObject *o) : p(o) {}
    Ref(const Ref &) = delete;
    ~Ref() { Py_XDECREF(p); }
};

[[noreturn]] void py_raise(PyObject *type, const std::string &msg) {
    PyErr_SetString(type, msg.c_str());
    throw PyRaised();
}

void check(int status) {
    if (status == NMG_OK) return;
    PyObject *args = Py_BuildValue("(is)", status, nmg_last_error());
    if (args) {
        PyErr_SetObject(g_error_class ? g_error_class : PyExc_RuntimeError, args);
        Py_DECREF(args);
    }
    throw PyRaised();
}

int dtype_code(const at::Tensor &t) {
    switch (t.scalar_type()) {
        case at::kFloat: return NMG_F32;
        case at::kHalf: return NMG_F16;
        case at::kBFloat16: return NMG_BF16;
        default: break;
    }
    py_raise(PyExc_TypeError, std::string("grouped n:m kernels support float32, float16 and bfloat16, got ") + c10::toString(t.scalar_type()));
}

const at::Tensor &tensor_arg(PyObject *o) {
    if (!THPVariable_Check(o)) py_raise(PyExc_TypeError, "expected a torch.Tensor");
    return THPVariable_Unpack(o);
}
at::Tensor optional_tensor(PyObject *o) { return o == Py_None ? at::Tensor() : tensor_arg(o); }

int64_t int_arg(PyObject *o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyRaised();
    return v;
}

void require_cuda(const at::Tensor &t, c10::Device &dev, bool &have) {
    if (!t.defined()) return;
    if (!t.is_cuda())
        py_raise(PyExc_RuntimeError, "grouped n:m kernels run on CUDA devices only (there is no CPU fallback); move the tensor with .cuda()");
    if (!have) {
        dev = t.device();
        have = true;
    } else if (t.device() != dev) {
        py_raise(PyExc_RuntimeError, "operands live on different devices: " + dev.str() + " and " + t.device().str());
    }
}
c10::Device device_of(std::initializer_list<const at::Tensor *> ts) {
    c10::Device dev(c10::kCPU);
    bool have = false;
    for (const at::Tensor *t : ts) require_cuda(*t, dev, have);
    return dev;
}

std::string shape_str(c10::IntArrayRef s) {
    std::string r = "(";
    for (size_t i = 0; i < s.size(); i++) r += (i ? ", " : "") + std::to_string(s[i]);
    return r + (s.size() == 1 ? ",)" : ")");
}

// Every kernel reads a bias of `feats` elements.
void check_bias(const at::Tensor &bias, int64_t feats) {
    if (bias.defined() && (bias.numel() != feats || (bias.dim() > 1 && bias.size(-1) != feats)))
        py_raise(PyExc_ValueError, "bias must have one element per output feature (" + std::to_string(feats) + "), got shape " + shape_str(bias.sizes()));
}

// contiguous() with the call skipped where it would return the tensor itself
at::Tensor packed_rows(const at::Tensor &t) { return t.is_contiguous() ? t : t.contiguous(); }

// Rows of a 2-D operand with unit stride along them; the copy is made only where the strides do not allow it.
struct Rows {
    at::Tensor t;
    int64_t rows, cols, ld;
};
Rows row_major_2d(const at::Tensor &t) {
    if (t.dim() != 2) py_raise(PyExc_ValueError, "expected a 2-D tensor");
    Rows r{t, t.size(0), t.size(1), 0};
    if (t.stride(1) != 1 || t.stride(0) < r.cols) r.t = t.contiguous();
    r.ld = r.t.is_contiguous() ? r.cols : r.t.stride(0);
    return r;
}
// The same for an operand whose leading dims all count as rows.
Rows rows_of(const at::Tensor &t, int64_t cols) {
    if (t.dim() == 2) {
        Rows r = row_major_2d(t);
        if (r.cols != cols) py_raise(PyExc_ValueError, "activation shape " + shape_str(t.sizes()) + " does not match K=" + std::to_string(cols));
        return r;
    }
    if (t.dim() < 1 || t.size(-1) != cols) py_raise(PyExc_ValueError, "activation shape " + shape_str(t.sizes()) + " does not match K=" + std::to_string(cols));
    if (!t.is_contiguous()) return row_major_2d(t.reshape({cols ? t.numel() / cols : 0, cols}));
    return Rows{t, cols ? t.numel() / cols : 0, cols, cols};
}

// Uninitialised tensor on the current device, straight from the caching allocator (torch's operator dispatch is half a microsecond)
at::Tensor new_empty(c10::IntArrayRef sizes, at::ScalarType type) {
    return at::detail::empty_generic(sizes, c10::cuda::CUDACachingAllocator::get(), c10::DispatchKeySet(c10::DispatchKey::CUDA), type, std::nullopt);
}

struct Geo {
    int64_t M, K;
    int n, m, g;
    int64_t slots;  // entries of idx; val has n times as many
};
Geo make_geo(int64_t M, int64_t K, int n, int m, int g) {
    const int64_t cc = M > 0 && K > 0 && m > 0 && g > 0 ? nmg_num_patterns(n, m) * g : 0;
    return Geo{M, K, n, m, g, cc > 0 ? (M + m - 1) / m * ((K + cc - 1) / cc) * cc : 0};  // 0: the library says what is wrong
}
// The kernels read `batch` weights' worth of both.
void check_weight(const Geo &geo, const at::Tensor &val, const at::Tensor &idx, int64_t batch = 1) {
    if (idx.scalar_type() != at::kShort) py_raise(PyExc_TypeError, std::string("idx must be int16, got ") + c10::toString(idx.scalar_type()));
    if (val.numel() < batch * geo.slots * geo.n || idx.numel() < batch * geo.slots)
        py_raise(PyExc_ValueError, "val and idx are smaller than a " + std::to_string(geo.n) + ":" + std::to_string(geo.m) + " weight of shape " + shape_str({geo.M, geo.K}) +
                                       " with groups of " + std::to_string(geo.g));
}

void *stream_of(c10::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

// Whether work queued now goes into a CUDA graph.
bool capturing(c10::Device dev) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c10::cuda::getCurrentCUDAStream(dev.index()).stream(), &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return false;
}

struct Epi {
    int act = NMG_EPI_NONE;
    at::Tensor residual;  // rows of the output's shape, contiguous along the last dim
    int64_t ld = 0;
};

bool rows_aligned(const Rows &r) { return reinterpret_cast<uintptr_t>(r.t.const_data_ptr()) % 16 == 0 && r.ld % 8 == 0; }
int given(const at::Tensor &packed, const Rows &rows) { return (packed.defined() ? NMG_GIVEN_PACKED : 0) | (rows_aligned(rows) ? NMG_GIVEN_ALIGNED_ROWS : 0); }

// out[rows_out][ld_out] = activation(product + bias) + residual; every operand has been checked against the others.
void call_spmm(const Geo &geo, int code, c10::Device dev, const at::Tensor &val, const at::Tensor &idx, const at::Tensor &packed, const Rows &act,
               int64_t tokens, const at::Tensor &bias, const Epi &epi, const at::Tensor &out, int64_t ld_out, int layout, int algo) {
    check_weight(geo, val, idx);
    const at::Tensor v = packed_rows(val), i = packed_rows(idx), b = bias.defined() ? packed_rows(bias) : bias;
    const size_t nbytes = nmg_spmm_workspace_bytes(geo.M, geo.K, tokens, geo.n, geo.m, geo.g, code, layout, algo, given(packed, act));
    at::Tensor ws;
    if (nbytes) ws = new_empty({(int64_t)nbytes}, at::kByte);
    void *st = stream_of(dev);
    void *wsp = nbytes ? ws.mutable_data_ptr() : nullptr;
    const void *pk = packed.defined() ? packed.const_data_ptr() : nullptr;
    const void *bp = b.defined() ? b.const_data_ptr() : nullptr;
    const int16_t *ip = static_cast<const int16_t *>(i.const_data_ptr());
    int rc;
    PyThreadState *save = PyEval_SaveThread();
    if (epi.act != NMG_EPI_NONE || epi.residual.defined())
        rc = nmg_spmm_fused(v.const_data_ptr(), ip, pk, geo.M, geo.K, geo.n, geo.m, geo.g, code, act.t.const_data_ptr(), act.ld, tokens, bp, epi.act,
                            epi.residual.defined() ? epi.residual.const_data_ptr() : nullptr, epi.ld, out.mutable_data_ptr(), ld_out, layout, algo, wsp,
                            nbytes, st);
    else
        rc = nmg_spmm(v.const_data_ptr(), ip, pk, geo.M, geo.K, geo.n, geo.m, geo.g, code, act.t.const_data_ptr(), act.ld, tokens, bp,
                      out.mutable_data_ptr(), ld_out, layout, algo, wsp, nbytes, st);
    PyEval_RestoreThread(save);
    check(rc);
}

void call_spmm_t(const Geo &geo, int code, c10::Device dev, const at::Tensor &val, const at::Tensor &idx, const at::Tensor &packed, const at::Tensor &sp24,
                 const Rows &dy, const at::Tensor &dx, int algo) {
    check_weight(geo, val, idx);
    const at::Tensor v = packed_rows(val), i = packed_rows(idx);
    void *st = stream_of(dev);
    at::Tensor ws;
    size_t nbytes = 0;
    if (!sp24.defined()) {
        nbytes = nmg_spmm_t_workspace_bytes(geo.M, geo.K, dy.rows, geo.n, geo.m, geo.g, code, algo, given(packed, dy));
        if (nbytes) ws = new_empty({(int64_t)nbytes}, at::kByte);
    }
    int rc;
    PyThreadState *save = PyEval_SaveThread();
    if (sp24.defined())
        rc = nmg_spmm_t_sp24(sp24.const_data_ptr(), geo.M, geo.K, geo.n, geo.m, geo.g, code, dy.t.const_data_ptr(), dy.ld, dy.rows, dx.mutable_data_ptr(),
                             geo.K, st);
    else
        rc = nmg_spmm_t(v.const_data_ptr(), static_cast<const int16_t *>(i.const_data_ptr()), packed.defined() ? packed.const_data_ptr() : nullptr, geo.M,
                        geo.K, geo.n, geo.m, geo.g, code, dy.t.const_data_ptr(), dy.ld, dy.rows, dx.mutable_data_ptr(), geo.K, algo,
                        nbytes ? ws.mutable_data_ptr() : nullptr, nbytes, st);
    PyEval_RestoreThread(save);
    check(rc);
}

// ------------------------------------------------------------------------------------------------ module functions
#define NMG_PY_BEGIN(nargs_wanted)                                                           \
    HANDLE_TH_ERRORS                                                                         \
    if (nargs != (nargs_wanted)) {                                                           \
        PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", (nargs_wanted), nargs); \
        return nullptr;                                                                      \
    }                                                                                        \
    try {
#define NMG_PY_END                    \
    } catch (const PyRaised &) { return nullptr; } \
    END_HANDLE_TH_ERRORS

Geo geo_args(PyObject *const *a) { return make_geo(int_arg(a[0]), int_arg(a[1]), (int)int_arg(a[2]), (int)int_arg(a[3]), (int)int_arg(a[4])); }

// spmm(val, idx, M, K, n, m, g, act, bias, layout, algo, out, packed, activation, residual) -> out
PyObject *py_spmm(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(15)
    const at::Tensor &val = tensor_arg(a[0]), &idx = tensor_arg(a[1]), &act0 = tensor_arg(a[7]);
    const Geo geo = geo_args(a + 2);
    const at::Tensor bias = optional_tensor(a[8]), out0 = optional_tensor(a[11]), packed = optional_tensor(a[12]), residual = optional_tensor(a[14]);
    const int layout = (int)int_arg(a[9]), algo = (int)int_arg(a[10]);
    const c10::Device dev = device_of({&val, &idx, &act0, &bias, &residual});
    const int code = dtype_code(val);
    if (act0.scalar_type() != val.scalar_type() || (bias.defined() && bias.scalar_type() != val.scalar_type()))
        py_raise(PyExc_TypeError, std::string("activation / bias dtype must match the weight dtype ") + c10::toString(val.scalar_type()));
    check_bias(bias, geo.M);
    const c10::cuda::CUDAGuard guard(dev);
    const Rows act = row_major_2d(act0);
    const bool token_major = layout != NMG_ACT_K_MAJOR, out_tm = layout == NMG_ACT_TOKEN_MAJOR;
    const int64_t tokens = token_major ? act.rows : act.cols;
    if ((token_major ? act.cols : act.rows) != geo.K)
        py_raise(PyExc_ValueError, "activation shape " + shape_str(act0.sizes()) + " does not match K=" + std::to_string(geo.K));
    const int64_t out_rows = out_tm ? tokens : geo.M, out_cols = out_tm ? geo.M : tokens;
    at::Tensor out = out0;
    if (!out.defined()) {
        out = new_empty({out_rows, out_cols}, val.scalar_type());
    } else {
        // the kernel writes out_rows rows of out_cols elements, ld_out apart: anything else would land outside `out`
        if (out.scalar_type() != val.scalar_type() || out.device() != dev)
            py_raise(PyExc_ValueError, std::string("out must be a ") + c10::toString(val.scalar_type()) + " tensor on " + dev.str());
        if (out.dim() != 2 || out.size(0) != out_rows || out.size(1) != out_cols)
            py_raise(PyExc_ValueError, "out must have shape (" + std::to_string(out_rows) + ", " + std::to_string(out_cols) + ") for this layout, got " + shape_str(out.sizes()));
        if (out_cols > 1 && out.stride(1) != 1) py_raise(PyExc_ValueError, "out must have unit stride along its rows (a transposed view cannot be written in place)");
        if (out_rows > 1 && out.stride(0) < out_cols) py_raise(PyExc_ValueError, "out rows overlap: the row stride is smaller than the row length");
    }
    Epi epi;
    epi.act = (int)int_arg(a[13]);
    if (residual.defined()) {
        if (residual.scalar_type() != val.scalar_type() || residual.dim() != 2 || residual.size(0) != out_rows || residual.size(1) != out_cols ||
            (out_cols > 1 && residual.stride(1) != 1))
            py_raise(PyExc_ValueError, "residual must match the output's dtype and shape (" + std::to_string(out_rows) + ", " + std::to_string(out_cols) + "), with contiguous rows");
        epi.residual = residual;
        epi.ld = out_rows > 1 ? residual.stride(0) : out_cols;
    }
    if (tokens > 0) call_spmm(geo, code, dev, val, idx, packed, act, tokens, bias, epi, out, out_rows > 1 ? out.stride(0) : out_cols, layout, algo);
    if (a[11] != Py_None) return Py_NewRef(a[11]);
    return THPVariable_Wrap(out);
    NMG_PY_END
}

// spmm_t(val, idx, M, K, n, m, g, dy, algo, packed, sp24, sp24_min_tokens) -> dx
PyObject *py_spmm_t(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(12)
    const at::Tensor &val = tensor_arg(a[0]), &idx = tensor_arg(a[1]), &dy0 = tensor_arg(a[7]);
    const Geo geo = geo_args(a + 2);
    const int algo = (int)int_arg(a[8]);
    const at::Tensor packed = optional_tensor(a[9]), sp24 = optional_tensor(a[10]);
    const c10::Device dev = device_of({&val, &idx, &dy0});
    const int code = dtype_code(val);
    if (dy0.scalar_type() != val.scalar_type())
        py_raise(PyExc_TypeError, std::string("gradient dtype must match the weight dtype ") + c10::toString(val.scalar_type()));
    const c10::cuda::CUDAGuard guard(dev);
    const Rows dy = row_major_2d(dy0);
    if (dy.cols != geo.M) py_raise(PyExc_ValueError, "gradient shape " + shape_str(dy0.sizes()) + " does not match M=" + std::to_string(geo.M));
    const at::Tensor dx = new_empty({dy.rows, geo.K}, val.scalar_type());
    const bool kept = sp24.defined() && dy.rows >= int_arg(a[11]) && (algo == NMG_ALGO_AUTO || algo == NMG_ALGO_TENSOR) && rows_aligned(dy);
    if (dy.rows > 0) call_spmm_t(geo, code, dev, val, idx, packed, kept ? sp24 : at::Tensor(), dy, dx, algo);
    return THPVariable_Wrap(dx);
    NMG_PY_END
}

// [B, M, K] operand of the conversions: unit stride along K, packed strides where a size-1 dim carries arbitrary ones.
struct Dense3 {
    at::Tensor t;
    int64_t B, M, K, ld, bs;
};
Dense3 dense3_arg(const at::Tensor &t) {
    if (t.dim() != 3) py_raise(PyExc_ValueError, "expected a 3-D tensor");
    Dense3 d{t, t.size(0), t.size(1), t.size(2), 0, 0};
    if (t.stride(2) != 1 || t.stride(1) < d.K || (d.B > 1 && t.stride(0) < d.M * t.stride(1))) d.t = t.contiguous();
    const bool c = d.t.is_contiguous();
    d.ld = c ? d.K : d.t.stride(1);
    d.bs = c ? d.M * d.K : d.t.stride(0);
    return d;
}
struct Tiles { int64_t C, cc, count; };
Tiles tiles_of(int64_t B, int64_t M, int64_t K, int n, int m, int g) {
    const int64_t C = nmg_num_patterns(n, m), cc = C * g;
    if (C < 1 || cc < 1) py_raise(PyExc_ValueError, "need 0 <= n <= m and a positive group size");
    return Tiles{C, cc, B * ((M + m - 1) / m) * ((K + cc - 1) / cc)};
}

// sparsify(dense3, n, m, g) -> (val, idx)
PyObject *py_sparsify(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(4)
    const at::Tensor &w = tensor_arg(a[0]);
    const c10::Device dev = device_of({&w});
    const int code = dtype_code(w), n = (int)int_arg(a[1]), m = (int)int_arg(a[2]), g = (int)int_arg(a[3]);
    const c10::cuda::CUDAGuard guard(dev);
    const Dense3 d = dense3_arg(w);
    const Tiles t = tiles_of(d.B, d.M, d.K, n, m, g);
    const at::Tensor val = new_empty({t.count, t.C, g, n}, w.scalar_type()), idx = new_empty({t.count, t.C, g, 1}, at::kShort);
    void *st = stream_of(dev);
    PyThreadState *save = PyEval_SaveThread();
    const int rc = nmg_sparsify(d.t.const_data_ptr(), d.B, d.M, d.K, d.ld, d.bs, n, m, g, code, val.mutable_data_ptr(),
                                static_cast<int16_t *>(idx.mutable_data_ptr()), st);
    PyEval_RestoreThread(save);
    check(rc);
    PyObject *v = THPVariable_Wrap(val), *i = THPVariable_Wrap(idx);
    PyObject *r = PyTuple_New(2);
    PyTuple_SET_ITEM(r, 0, v);
    PyTuple_SET_ITEM(r, 1, i);
    return r;
    NMG_PY_END
}

PyObject *gather_values(const Dense3 &d, const at::Tensor &idx0, int n, int m, int g, int code, c10::Device dev) {
    const at::Tensor &w = d.t;
    const Tiles t = tiles_of(d.B, d.M, d.K, n, m, g);
    const at::Tensor idx = packed_rows(idx0);
    if (idx.scalar_type() != at::kShort || idx.numel() != t.count * t.cc) py_raise(PyExc_ValueError, "idx does not belong to a layout of this shape");
    const at::Tensor val = new_empty({t.count, t.C, g, n}, w.scalar_type());
    void *st = stream_of(dev);
    PyThreadState *save = PyEval_SaveThread();
    const int rc = nmg_gather(d.t.const_data_ptr(), static_cast<const int16_t *>(idx.const_data_ptr()), d.B, d.M, d.K, d.ld, d.bs, n, m, g, code,
                              val.mutable_data_ptr(), st);
    PyEval_RestoreThread(save);
    check(rc);
    return THPVariable_Wrap(val);
}

// gather(dense3, idx, n, m, g) -> val
PyObject *py_gather(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(5)
    const at::Tensor &w = tensor_arg(a[0]), &idx = tensor_arg(a[1]);
    const c10::Device dev = device_of({&w, &idx});
    const int code = dtype_code(w), n = (int)int_arg(a[2]), m = (int)int_arg(a[3]), g = (int)int_arg(a[4]);
    const c10::cuda::CUDAGuard guard(dev);
    return gather_values(dense3_arg(w), idx, n, m, g, code, dev);
    NMG_PY_END
}

// densify(val, idx, B, M, K, n, m, g) -> dense3
PyObject *py_densify(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(8)
    const at::Tensor &val0 = tensor_arg(a[0]), &idx0 = tensor_arg(a[1]);
    const c10::Device dev = device_of({&val0, &idx0});
    const int code = dtype_code(val0);
    const int64_t B = int_arg(a[2]);
    const Geo geo = geo_args(a + 3);
    check_weight(geo, val0, idx0, B);
    const c10::cuda::CUDAGuard guard(dev);
    const at::Tensor val = packed_rows(val0), idx = packed_rows(idx0);
    const at::Tensor out = new_empty({B, geo.M, geo.K}, val.scalar_type());
    void *st = stream_of(dev);
    PyThreadState *save = PyEval_SaveThread();
    const int rc = nmg_densify(val.const_data_ptr(), static_cast<const int16_t *>(idx.const_data_ptr()), B, geo.M, geo.K, geo.n, geo.m, geo.g, code,
                               out.mutable_data_ptr(), geo.K, geo.M * geo.K, st);
    PyEval_RestoreThread(save);
    check(rc);
    return THPVariable_Wrap(out);
    NMG_PY_END
}

// check_weight(val, idx, M, K, n, m, g): raises unless both hold a weight of this geometry
PyObject *py_check_weight(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(7)
    check_weight(geo_args(a + 2), tensor_arg(a[0]), tensor_arg(a[1]));
    Py_RETURN_NONE;
    NMG_PY_END
}

PyObject *py_set_error_class(PyObject *, PyObject *cls) {
    Py_XSETREF(g_error_class, Py_NewRef(cls));
    Py_RETURN_NONE;
}

// ------------------------------------------------------------------------------------------------ Kept
// One of the tensors a copy was derived from.  An address says nothing by itself: a weight that was replaced twice between two
// calls finds its third tensor where its first one was, at version 0 again.  The weak references keep both objects' addresses
// from being given to others (they do not keep the memory of the values); the storage counts too, since `t.data = other` leaves
// the tensor and its version as they were.
struct Source {
    c10::weak_intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl> tensor;
    c10::weak_intrusive_ptr<c10::StorageImpl> storage;
    const void *data;
    uint32_t version;
    at::ScalarType type;
    explicit Source(const at::Tensor &t)
        : tensor(t.getIntrusivePtr()), storage(t.storage().getWeakStorageImpl()), data(t.const_data_ptr()), version(t._version()), type(t.scalar_type()) {}
    bool is(const at::Tensor &t) const {
        return tensor._unsafe_get_target() == t.unsafeGetTensorImpl() && storage._unsafe_get_target() == t.storage().unsafeGetStorageImpl() &&
               data == t.const_data_ptr() && version == t._version() && type == t.scalar_type();
    }
};
// A copy derived from (val, idx), valid while both are the same tensors at the same version.  It is made on the stream that first
// asks for it; a call on another stream waits for that, and the copy's memory then counts as used there too.
struct KeptCopy {
    Source val, idx;
    at::Tensor copy;  // undefined: there is none for this weight, or none has been made
    bool made = false;
    bool captured = false;  // a CUDA graph reads the copy: it is not given back before the weight
    std::optional<c10::cuda::CUDAStream> stream;
    cudaEvent_t ready = nullptr;  // behind the kernels that make it
    bool complete = false;
    KeptCopy(const at::Tensor &v, const at::Tensor &i) : val(v), idx(i) {}  // before the copy is made: a write meanwhile shows
    KeptCopy(const KeptCopy &) = delete;
    ~KeptCopy() {
        if (ready) cudaEventDestroy(ready);
    }
    void put(const at::Tensor &c) {
        copy = c;
        made = true;
        if (!copy.defined() || !copy.is_cuda()) return;
        const c10::cuda::CUDAGuard guard(copy.device());
        stream = c10::cuda::getCurrentCUDAStream(copy.device().index());
        C10_CUDA_CHECK(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
        C10_CUDA_CHECK(cudaEventRecord(ready, stream->stream()));
    }
    const at::Tensor &use(bool in_graph) {
        if (!ready) return copy;
        captured |= in_graph;
        const c10::cuda::CUDAStream now = c10::cuda::getCurrentCUDAStream(copy.device().index());
        if (now == *stream) return copy;
        if (!complete) {
            // a graph cannot wait for an event from outside it: wait here (relaxed: the event has nothing to do with the capture)
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            C10_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
            cudaError_t e = in_graph ? cudaEventSynchronize(ready) : cudaEventQuery(ready);
            complete = e == cudaSuccess;
            if (e == cudaErrorNotReady) {
                cudaGetLastError();
                e = cudaStreamWaitEvent(now.stream(), ready, 0);
            }
            C10_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
            C10_CUDA_CHECK(e);
        }
        if (!in_graph) c10::cuda::CUDACachingAllocator::recordStream(copy.storage().data_ptr(), now);
        return copy;
    }
    bool from(const at::Tensor &v, const at::Tensor &i) const { return val.is(v) && idx.is(i); }
};

// Kept(val, idx), then put(copy): the same for the caches on the Python side.
extern PyTypeObject kept_type;
struct Kept {
    PyObject_HEAD
    KeptCopy *data;
};
PyObject *kept_new(PyTypeObject *type, PyObject *args, PyObject *) {
    HANDLE_TH_ERRORS
    try {
        if (PyTuple_GET_SIZE(args) != 2) py_raise(PyExc_TypeError, "Kept(val, idx)");
        std::unique_ptr<KeptCopy> data(new KeptCopy(tensor_arg(PyTuple_GET_ITEM(args, 0)), tensor_arg(PyTuple_GET_ITEM(args, 1))));
        Kept *k = reinterpret_cast<Kept *>(type->tp_alloc(type, 0));
        if (k) k->data = data.release();
        return reinterpret_cast<PyObject *>(k);
    } catch (const PyRaised &) { return nullptr; }
    END_HANDLE_TH_ERRORS
}
void kept_dealloc(PyObject *self) {
    delete reinterpret_cast<Kept *>(self)->data;
    Py_TYPE(self)->tp_free(self);
}
// get(val, idx) -> the copy, or None when it was made from other tensors or other contents
PyObject *kept_get(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(2)
    KeptCopy *k = reinterpret_cast<Kept *>(self)->data;
    if (!k->made || !k->from(tensor_arg(a[0]), tensor_arg(a[1]))) Py_RETURN_NONE;
    return THPVariable_Wrap(k->use(k->copy.is_cuda() && capturing(k->copy.device())));
    NMG_PY_END
}
PyObject *kept_put(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(1)
    reinterpret_cast<Kept *>(self)->data->put(tensor_arg(a[0]));
    Py_RETURN_NONE;
    NMG_PY_END
}
// captured() -> whether a CUDA graph reads the copy
PyObject *kept_captured(PyObject *self, PyObject *const *, Py_ssize_t nargs) {
    NMG_PY_BEGIN(0)
    return PyBool_FromLong(reinterpret_cast<Kept *>(self)->data->captured);
    NMG_PY_END
}
// capturing(tensor) -> whether work queued now on the current stream of its device goes into a CUDA graph
PyObject *py_capturing(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(1)
    const at::Tensor &t = tensor_arg(a[0]);
    return PyBool_FromLong(t.is_cuda() && capturing(t.device()));
    NMG_PY_END
}

// ------------------------------------------------------------------------------------------------ Handle
// What the host keeps of one 2-D weight between calls: its geometry and, for the kernels that read them, the derived copies.
// They are asked for at the GroupedNMTensor (packed(), packed_sp24()) when (val, idx) are no longer what they were made from.
extern PyTypeObject handle_type;
struct Handle {
    PyObject_HEAD
    Geo geo;
    KeptCopy *packed, *sp24;
    std::vector<at::Tensor> *held;  // copies of earlier contents that a CUDA graph still reads
};

at::Tensor attr_tensor(PyObject *o, PyObject *name) {
    PyObject *v = PyObject_GetAttr(o, name);
    if (!v) throw PyRaised();
    if (!THPVariable_Check(v)) {
        Py_DECREF(v);
        py_raise(PyExc_TypeError, "val and idx must be tensors");
    }
    at::Tensor t = THPVariable_Unpack(v);
    Py_DECREF(v);
    return t;
}

// when_reused: the first call on these contents goes without the copy.  A weight that is written before every call (a training
// step) then never pays for copies that one call reads: 4096 x 4096 bf16, 1280 tokens 97 us with a copy made every time, 72 without.
// A copy made inside a CUDA graph holds nothing before a replay: it belongs to the graph and is not kept.  Nor is one of tensors
// made under inference mode, which do not count their writes: the call then goes without.
at::Tensor derived(Handle *h, KeptCopy *&kept, PyObject *gnm, PyObject *method, const at::Tensor &val, const at::Tensor &idx, bool in_graph, bool when_reused = false) {
    if (val.is_inference() || idx.is_inference()) return at::Tensor();
    const bool known = kept && kept->from(val, idx);
    if (known && kept->made) return kept->use(in_graph);
    std::unique_ptr<KeptCopy> now(new KeptCopy(val, idx));
    if (known || !when_reused) {
        Ref r(PyObject_CallMethodNoArgs(gnm, method));
        if (!r.p) throw PyRaised();
        const at::Tensor copy = THPVariable_Check(r.p) ? THPVariable_Unpack(r.p) : at::Tensor();
        if (in_graph) return copy;
        now->put(copy);
    }
    if (kept && kept->captured) h->held->push_back(kept->copy);
    delete kept;  // here, not earlier: another thread may have been here while the method ran
    kept = now.release();
    return kept->copy;
}

// A column-ordered copy for this call alone.
at::Tensor pack_once(const Geo &geo, int code, c10::Device dev, const at::Tensor &val, const at::Tensor &idx) {
    check_weight(geo, val, idx);
    const at::Tensor v = packed_rows(val), i = packed_rows(idx);
    const size_t nbytes = nmg_packed_bytes(geo.M, geo.K, geo.n, geo.m, geo.g, code);
    at::Tensor buf = new_empty({(int64_t)nbytes}, at::kByte);
    check(nmg_pack(v.const_data_ptr(), static_cast<const int16_t *>(i.const_data_ptr()), geo.M, geo.K, geo.n, geo.m, geo.g, code, buf.mutable_data_ptr(), nbytes,
                   stream_of(dev)));
    return buf;
}

// The column-ordered copy for a call of `tokens` rows (k_major: columns), where the kernel that serves it reads one.
// In a CUDA graph only the calls of few tokens read the kept copy (a decode step: 9 us against 27 with a copy made in every
// replay), and such a graph has to be captured again when the weight changes.  All others read val / idx in every replay.
at::Tensor packed_for(Handle *h, PyObject *gnm, const at::Tensor &val, const at::Tensor &idx, int64_t tokens, int code, c10::Device dev, bool transposed, bool k_major = false) {
    const Geo &geo = h->geo;
    const int uses = nmg_spmm_uses_packed(geo.M, geo.K, tokens, geo.n, geo.m, geo.g, code, NMG_ACT_TOKEN_MAJOR, NMG_ALGO_AUTO, transposed ? 1 : 0);
    if (!uses) return at::Tensor();
    const bool in_graph = capturing(dev);
    if (in_graph && uses == NMG_PACKED_IF_KEPT) return at::Tensor();
    if (in_graph && ((k_major && tokens < 64) || (code == NMG_F32 && tokens >= 256))) return pack_once(geo, code, dev, val, idx);
    return derived(h, h->packed, gnm, g_s_packed, val, idx, in_graph, uses == NMG_PACKED_IF_KEPT);
}

PyObject *handle_new(PyTypeObject *type, PyObject *args, PyObject *) {
    long long M, K;
    int n, m, g;
    if (!PyArg_ParseTuple(args, "LLiii", &M, &K, &n, &m, &g)) return nullptr;
    Handle *h = reinterpret_cast<Handle *>(type->tp_alloc(type, 0));
    if (!h) return nullptr;
    h->geo = make_geo(M, K, n, m, g);
    h->packed = h->sp24 = nullptr;
    h->held = new std::vector<at::Tensor>();
    return reinterpret_cast<PyObject *>(h);
}
void handle_dealloc(PyObject *self) {
    Handle *h = reinterpret_cast<Handle *>(self);
    delete h->packed;
    delete h->sp24;
    delete h->held;
    Py_TYPE(self)->tp_free(self);
}

// linear(gnm, x, bias, activation, residual): x [..., K] -> [..., M] = activation(x W^T + bias) + residual
PyObject *handle_linear(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(5)
    Handle *h = reinterpret_cast<Handle *>(self);
    const Geo &geo = h->geo;
    const at::Tensor val = attr_tensor(a[0], g_s_val), idx = attr_tensor(a[0], g_s_idx);
    const at::Tensor &x = tensor_arg(a[1]);
    const at::Tensor bias = optional_tensor(a[2]), residual = optional_tensor(a[4]);
    const c10::Device dev = device_of({&val, &idx, &x, &bias, &residual});
    const int code = dtype_code(val);
    if (x.scalar_type() != val.scalar_type() || (bias.defined() && bias.scalar_type() != val.scalar_type()))
        py_raise(PyExc_TypeError, std::string("activation / bias dtype must match the weight dtype ") + c10::toString(val.scalar_type()));
    check_bias(bias, geo.M);
    const c10::cuda::CUDAGuard guard(dev);
    const Rows act = rows_of(x, geo.K);
    c10::DimVector sizes(x.sizes().begin(), x.sizes().end());
    sizes.back() = geo.M;
    const at::Tensor out = new_empty(sizes, val.scalar_type());
    Epi epi;
    epi.act = (int)int_arg(a[3]);
    if (residual.defined()) {
        if (residual.scalar_type() != val.scalar_type() || residual.numel() != act.rows * geo.M || residual.dim() < 1 || residual.size(-1) != geo.M)
            py_raise(PyExc_ValueError, "residual must match the output's dtype and shape, with contiguous rows");
        const Rows r = rows_of(residual, geo.M);
        epi.residual = r.t;
        epi.ld = act.rows > 1 ? r.ld : geo.M;
    }
    if (act.rows > 0) {
        call_spmm(geo, code, dev, val, idx, packed_for(h, a[0], val, idx, act.rows, code, dev, false), act, act.rows, bias, epi, out, geo.M, NMG_ACT_TOKEN_MAJOR,
                  NMG_ALGO_AUTO);
    }
    return THPVariable_Wrap(out);
    NMG_PY_END
}

// mm(gnm, b): b [K, tokens] -> [M, tokens] = W b
PyObject *handle_mm(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(2)
    Handle *h = reinterpret_cast<Handle *>(self);
    const Geo &geo = h->geo;
    const at::Tensor val = attr_tensor(a[0], g_s_val), idx = attr_tensor(a[0], g_s_idx);
    const at::Tensor &b = tensor_arg(a[1]);
    const c10::Device dev = device_of({&val, &idx, &b});
    const int code = dtype_code(val);
    if (b.scalar_type() != val.scalar_type())
        py_raise(PyExc_TypeError, std::string("activation / bias dtype must match the weight dtype ") + c10::toString(val.scalar_type()));
    const c10::cuda::CUDAGuard guard(dev);
    const Rows act = row_major_2d(b);
    if (act.rows != geo.K) py_raise(PyExc_ValueError, "activation shape " + shape_str(b.sizes()) + " does not match K=" + std::to_string(geo.K));
    const at::Tensor out = new_empty({geo.M, act.cols}, val.scalar_type());
    if (act.cols > 0) {
        // a handful of columns runs on the tensor cores when the packed copy is there already: keep one for the token-major call
        call_spmm(geo, code, dev, val, idx, packed_for(h, a[0], val, idx, act.cols, code, dev, false, true), act, act.cols, at::Tensor(), Epi(), out, act.cols,
                  NMG_ACT_K_MAJOR, NMG_ALGO_AUTO);
    }
    return THPVariable_Wrap(out);
    NMG_PY_END
}

// dx = dy W; dy's leading dims all count as rows
at::Tensor input_gradient(Handle *h, PyObject *gnm, const at::Tensor &val, const at::Tensor &idx, const at::Tensor &dy0, const Rows &dy, int64_t sp24_min_tokens,
                          int code, c10::Device dev) {
    const Geo &geo = h->geo;
    c10::DimVector sizes(dy0.sizes().begin(), dy0.sizes().end());
    sizes.back() = geo.K;
    const at::Tensor dx = new_empty(sizes, val.scalar_type());
    if (dy.rows > 0) {
        at::Tensor sp24, packed;
        // the compressed transposed copy serves the large batches of a 16-bit weight inside the 2:4 structure
        if (dy.rows >= sp24_min_tokens) sp24 = derived(h, h->sp24, gnm, g_s_packed_sp24, val, idx, capturing(dev));
        if (!sp24.defined()) packed = packed_for(h, gnm, val, idx, dy.rows, code, dev, true);
        call_spmm_t(geo, code, dev, val, idx, packed, sp24.defined() && rows_aligned(dy) ? sp24 : at::Tensor(), dy, dx, NMG_ALGO_AUTO);
    }
    return dx;
}

// linear_t(gnm, dy, sp24_min_tokens): dy [..., M] -> [..., K] = dy W
PyObject *handle_linear_t(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(3)
    Handle *h = reinterpret_cast<Handle *>(self);
    const at::Tensor val = attr_tensor(a[0], g_s_val), idx = attr_tensor(a[0], g_s_idx);
    const at::Tensor &dy0 = tensor_arg(a[1]);
    const c10::Device dev = device_of({&val, &idx, &dy0});
    const int code = dtype_code(val);
    if (dy0.scalar_type() != val.scalar_type())
        py_raise(PyExc_TypeError, std::string("gradient dtype must match the weight dtype ") + c10::toString(val.scalar_type()));
    const c10::cuda::CUDAGuard guard(dev);
    return THPVariable_Wrap(input_gradient(h, a[0], val, idx, dy0, rows_of(dy0, h->geo.M), int_arg(a[2]), code, dev));
    NMG_PY_END
}

// [rows][ld] -> [cols], the bias gradient
at::Tensor column_sums(const Rows &x, int code, c10::Device dev) {
    const at::Tensor out = new_empty({x.cols}, x.t.scalar_type());
    if (x.rows < 1 || x.cols < 1) return out.zero_();
    const size_t nbytes = nmg_column_sum_workspace_bytes(x.rows, x.cols);
    const at::Tensor ws = new_empty({(int64_t)nbytes}, at::kByte);
    void *st = stream_of(dev);
    PyThreadState *save = PyEval_SaveThread();
    const int rc = nmg_column_sum(x.t.const_data_ptr(), x.rows, x.cols, x.ld, code, out.mutable_data_ptr(), ws.mutable_data_ptr(), nbytes, st);
    PyEval_RestoreThread(save);
    check(rc);
    return out;
}

// column_sum(dy): [..., M] -> [M]
PyObject *py_column_sum(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(1)
    const at::Tensor &x = tensor_arg(a[0]);
    const c10::Device dev = device_of({&x});
    const int code = dtype_code(x);
    const c10::cuda::CUDAGuard guard(dev);
    if (x.dim() < 1) py_raise(PyExc_ValueError, "expected at least one dimension");
    return THPVariable_Wrap(column_sums(rows_of(x, x.size(-1)), code, dev));
    NMG_PY_END
}

// linear_grads(gnm, x, dy, sp24_min_tokens, needs, in_layout) -> (dx, dw, db), None where not needed (needs: bits 0, 1, 2).
// dw is the plain product dy^T x, or with in_layout its values at the weight's kept positions.
PyObject *handle_linear_grads(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(6)
    Handle *h = reinterpret_cast<Handle *>(self);
    const Geo &geo = h->geo;
    const at::Tensor val = attr_tensor(a[0], g_s_val), idx = attr_tensor(a[0], g_s_idx);
    const at::Tensor &x = tensor_arg(a[1]), &dy0 = tensor_arg(a[2]);
    const int64_t needs = int_arg(a[4]);
    const bool in_layout = int_arg(a[5]) != 0;
    const c10::Device dev = device_of({&val, &idx, &x, &dy0});
    const int code = dtype_code(val);
    if (dy0.scalar_type() != val.scalar_type())
        py_raise(PyExc_TypeError, std::string("gradient dtype must match the weight dtype ") + c10::toString(val.scalar_type()));
    const c10::cuda::CUDAGuard guard(dev);
    const Rows dy = rows_of(dy0, geo.M);
    PyObject *r = PyTuple_New(3);
    for (int i = 0; i < 3; i++) PyTuple_SET_ITEM(r, i, Py_NewRef(Py_None));
    Ref owner(r);
    if (needs & 1) PyTuple_SetItem(r, 0, THPVariable_Wrap(input_gradient(h, a[0], val, idx, dy0, dy, int_arg(a[3]), code, dev)));
    if (needs & 2) {
        // dense weight gradient (training of nmg weights is outside the inference hot path): plain GEMM
        const at::Tensor dy2 = dy0.dim() == 2 ? dy0 : dy0.reshape({-1, geo.M}), x2 = x.dim() == 2 ? x : x.reshape({-1, geo.K});
        at::Tensor dw;
        {
            pybind11::gil_scoped_release nogil;
            dw = at::mm(dy2.t(), x2);
        }
        PyTuple_SetItem(r, 1, in_layout ? gather_values(Dense3{dw, 1, geo.M, geo.K, geo.K, geo.M * geo.K}, idx, geo.n, geo.m, geo.g, code, dev) : THPVariable_Wrap(dw));
    }
    if (needs & 4) {
        // a backward pass that is recorded itself (create_graph) needs db's dependence on dy
        const bool recorded = c10::GradMode::is_enabled() && dy0.requires_grad();
        PyTuple_SetItem(r, 2, THPVariable_Wrap(recorded ? dy0.reshape({-1, geo.M}).sum(0) : column_sums(dy, code, dev)));
    }
    return Py_NewRef(r);
    NMG_PY_END
}

// ------------------------------------------------------------------------------------------------ repeated calls
// What a torch function does when one of its operands has resolved it before (dispatch.SparseOp.repeat), without the
// interpreter for the implementations that end in one call of a Handle: an F.linear of one token took 9.0 us of host time, 3.3
// of them between the torch function and the handle, and takes 6.9.
PyObject *g_wrapper_type = nullptr, *g_profiling = nullptr;  // SparseTensorWrapper, [bool]
PyObject *g_s_sparsified_ops, *g_s_sparse_op, *g_s_disp_state, *g_s_fast, *g_s_native, *g_s_repeat, *g_s_container, *g_s_native_handle, *g_s_nm_strides,
    *g_s_kernel, *g_s_expanded;

// set_dispatch(wrapper_type, profiling_switch)
PyObject *py_set_dispatch(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    if (nargs != 2 || !PyType_Check(a[0]) || !PyList_Check(a[1])) {
        PyErr_SetString(PyExc_TypeError, "set_dispatch(wrapper_type, profiling_switch)");
        return nullptr;
    }
    g_wrapper_type = Py_NewRef(a[0]);
    g_profiling = Py_NewRef(a[1]);
    Py_RETURN_NONE;
}

// First item of a wrapper's container (borrowed), or NULL.
PyObject *payload_of(PyObject *wrapper) {
    Ref c(PyObject_GetAttr(wrapper, g_s_container));
    if (!c.p || !PyList_Check(c.p) || PyList_GET_SIZE(c.p) < 1) {
        PyErr_Clear();
        return nullptr;
    }
    return PyList_GET_ITEM(c.p, 0);  // the wrapper keeps the list
}

// The call on the weight's handle: kind "linear" (x, weight[, bias]) or "mm" (weight, b); NotImplemented when the general route has to decide.
PyObject *native_call(PyObject *kind, PyObject *args) {
    const bool mm = PyUnicode_CompareWithASCIIString(kind, "mm") == 0;
    PyObject *gnm = payload_of(PyTuple_GET_ITEM(args, mm ? 0 : 1));
    if (!gnm) Py_RETURN_NOTIMPLEMENTED;
    Ref keep(Py_NewRef(gnm));
    Ref strides(PyObject_GetAttr(gnm, g_s_nm_strides)), handle(PyObject_GetAttr(gnm, g_s_native_handle));
    if (!strides.p || !handle.p || !PyDict_Check(strides.p) || Py_TYPE(handle.p) != &handle_type) {
        PyErr_Clear();
        Py_RETURN_NOTIMPLEMENTED;
    }
    if (mm) {
        PyObject *b = PyTuple_GET_ITEM(args, 1);
        if (THPVariable_Unpack(b).dim() != 2) Py_RETURN_NOTIMPLEMENTED;
        PyObject *call[2] = {gnm, b};
        return handle_mm(handle.p, call, 2);
    }
    PyObject *kernel = PyDict_GetItemWithError(strides.p, g_s_kernel);
    if (kernel && PyUnicode_Check(kernel) && PyUnicode_Compare(kernel, g_s_expanded) == 0) Py_RETURN_NOTIMPLEMENTED;
    PyObject *call[5] = {gnm, PyTuple_GET_ITEM(args, 0), PyTuple_GET_SIZE(args) > 2 ? PyTuple_GET_ITEM(args, 2) : Py_None, g_zero, Py_None};
    return handle_linear(handle.p, call, 5);
}

// repeat_call(func, args) -> result or NotImplemented
PyObject *py_repeat_call(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 2 || !PyTuple_Check(a[1])) Py_RETURN_NOTIMPLEMENTED;
    PyObject *func = a[0], *args = a[1];
    const Py_ssize_t n = PyTuple_GET_SIZE(args);
    for (Py_ssize_t i = 0; i < n; i++) {
        PyObject *t = PyTuple_GET_ITEM(args, i);
        if (!PyType_IsSubtype(Py_TYPE(t), reinterpret_cast<PyTypeObject *>(g_wrapper_type))) continue;
        Ref dict(PyObject_GenericGetDict(t, nullptr));
        PyObject *ops = dict.p ? PyDict_GetItemWithError(dict.p, g_s_sparsified_ops) : nullptr;
        PyObject *op = ops && PyDict_Check(ops) ? PyDict_GetItemWithError(ops, func) : nullptr;
        if (!op) {
            PyErr_Clear();
            continue;
        }
        Ref sparse_op(PyObject_GetAttr(op, g_s_sparse_op));
        if (!sparse_op.p) return nullptr;
        Ref state(PyObject_GetAttr(sparse_op.p, g_s_disp_state));
        if (!state.p) return nullptr;
        PyObject *fast = PyDict_GetItemWithError(state.p, g_s_fast), *native = PyDict_GetItemWithError(state.p, g_s_native);
        if (!fast) Py_RETURN_NOTIMPLEMENTED;
        bool direct = native && PyUnicode_Check(native) && PyTuple_GET_SIZE(fast) == n && PyList_GET_ITEM(g_profiling, 0) == Py_False;
        for (Py_ssize_t j = 0; j < n && direct; j++) {  // same types and formats, nothing that needs a gradient
            PyObject *x = PyTuple_GET_ITEM(args, j), *want = PyTuple_GET_ITEM(fast, j), *fmt = PyTuple_GET_ITEM(want, 1);
            direct = reinterpret_cast<PyObject *>(Py_TYPE(x)) == PyTuple_GET_ITEM(want, 0) && THPVariable_Check(x);
            if (direct && fmt != Py_None) {
                PyObject *payload = payload_of(x);
                direct = payload && reinterpret_cast<PyObject *>(Py_TYPE(payload)) == fmt;
            }
            if (direct && c10::GradMode::is_enabled()) direct = !THPVariable_Unpack(x).requires_grad();
        }
        if (direct) {
            PyObject *r = native_call(native, args);
            if (r != Py_NotImplemented) return r;
            Py_DECREF(r);
        }
        return PyObject_CallMethodOneArg(sparse_op.p, g_s_repeat, args);
    }
    Py_RETURN_NOTIMPLEMENTED;
    END_HANDLE_TH_ERRORS
}

#define NMG_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
// gather(gnm, dense2d) -> the dense tensor's values at the weight's kept positions
PyObject *handle_gather(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
    NMG_PY_BEGIN(2)
    const Geo &geo = reinterpret_cast<Handle *>(self)->geo;
    const at::Tensor idx = attr_tensor(a[0], g_s_idx);
    const at::Tensor &w = tensor_arg(a[1]);
    const c10::Device dev = device_of({&w, &idx});
    const int code = dtype_code(w);
    const c10::cuda::CUDAGuard guard(dev);
    const Rows r = row_major_2d(w);
    if (r.rows != geo.M || r.cols != geo.K) py_raise(PyExc_ValueError, "expected a tensor of the weight's shape, got " + shape_str(w.sizes()));
    return gather_values(Dense3{r.t, 1, geo.M, geo.K, r.ld, geo.M * r.ld}, idx, geo.n, geo.m, geo.g, code, dev);
    NMG_PY_END
}

PyMethodDef handle_methods[] = {
    NMG_METHOD("gather", handle_gather),
    NMG_METHOD("linear", handle_linear),
    NMG_METHOD("mm", handle_mm),
    NMG_METHOD("linear_t", handle_linear_t),
    NMG_METHOD("linear_grads", handle_linear_grads),
    {nullptr, nullptr, 0, nullptr},
};
PyTypeObject handle_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyMethodDef kept_methods[] = {
    NMG_METHOD("get", kept_get),
    NMG_METHOD("put", kept_put),
    NMG_METHOD("captured", kept_captured),
    {nullptr, nullptr, 0, nullptr},
};
PyTypeObject kept_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyMethodDef module_methods[] = {
    NMG_METHOD("spmm", py_spmm),
    NMG_METHOD("spmm_t", py_spmm_t),
    NMG_METHOD("sparsify", py_sparsify),
    NMG_METHOD("gather", py_gather),
    NMG_METHOD("column_sum", py_column_sum),
    NMG_METHOD("densify", py_densify),
    NMG_METHOD("capturing", py_capturing),
    NMG_METHOD("check_weight", py_check_weight),
    NMG_METHOD("set_dispatch", py_set_dispatch),
    NMG_METHOD("repeat_call", py_repeat_call),
    {"set_error_class", py_set_error_class, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_nmg_host", "Host path of the grouped n:m kernels.", -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__nmg_host(void) {
    handle_type.tp_name = "sten_b200._nmg_host.Handle";
    handle_type.tp_basicsize = sizeof(Handle);
    handle_type.tp_flags = Py_TPFLAGS_DEFAULT;
    handle_type.tp_doc = "Geometry and derived copies of one 2-D grouped n:m weight.";
    handle_type.tp_new = handle_new;
    handle_type.tp_dealloc = handle_dealloc;
    handle_type.tp_methods = handle_methods;
    if (PyType_Ready(&handle_type) < 0) return nullptr;
    kept_type.tp_name = "sten_b200._nmg_host.Kept";
    kept_type.tp_basicsize = sizeof(Kept);
    kept_type.tp_flags = Py_TPFLAGS_DEFAULT;
    kept_type.tp_doc = "Copy derived from a weight's (val, idx), valid while both are the same tensors at the same version.";
    kept_type.tp_new = kept_new;
    kept_type.tp_dealloc = kept_dealloc;
    kept_type.tp_methods = kept_methods;
    if (PyType_Ready(&kept_type) < 0) return nullptr;
    g_s_val = PyUnicode_InternFromString("val");
    g_s_idx = PyUnicode_InternFromString("idx");
    g_s_packed = PyUnicode_InternFromString("packed");
    g_s_packed_sp24 = PyUnicode_InternFromString("packed_sp24");
    g_s_sparsified_ops = PyUnicode_InternFromString("sparsified_ops");
    g_s_sparse_op = PyUnicode_InternFromString("sparse_op");
    g_s_disp_state = PyUnicode_InternFromString("disp_state");
    g_s_fast = PyUnicode_InternFromString("fast");
    g_s_native = PyUnicode_InternFromString("native");
    g_s_repeat = PyUnicode_InternFromString("repeat");
    g_s_container = PyUnicode_InternFromString("_wrapped_tensor_container");
    g_s_native_handle = PyUnicode_InternFromString("_native");
    g_s_nm_strides = PyUnicode_InternFromString("nm_strides");
    g_s_kernel = PyUnicode_InternFromString("kernel");
    g_s_expanded = PyUnicode_InternFromString("sm100-expanded");
    g_zero = PyLong_FromLong(0);  // NMG_EPI_NONE
    PyObject *mod = PyModule_Create(&module_def);
    if (!mod) return nullptr;
    if (PyModule_AddObjectRef(mod, "Handle", reinterpret_cast<PyObject *>(&handle_type)) < 0 ||
        PyModule_AddObjectRef(mod, "Kept", reinterpret_cast<PyObject *>(&kept_type)) < 0) {
        Py_DECREF(mod);
        return nullptr;
    }
    return mod;
}

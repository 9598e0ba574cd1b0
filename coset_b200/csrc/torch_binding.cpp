// Native entry points for PyTorch callers: argument checks, output allocation and the launch of one C-ABI
// call in a single Python -> C++ step.
//
// What bounds a small call is the host: through ctypes an encode of a few thousand blocks took 25-30 us of
// argument conversion, device context and allocation in Python against 3-9 us on the device.  The functions
// here are plain METH_FASTCALL entry points of a CPython module (no argument parsing library) that read the
// tensors directly; they add nothing to what the C ABI computes.  The library itself (libcoset_b200.so) stays
// free of torch symbols; this module links against both.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/Context.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/coset_b200.h"

namespace {

using at::Tensor;

// ---------------------------------------------------------------- small helpers
// Lets other Python threads run while this one allocates and launches (the first use of the decoder's table also waits for its
// stream), as ctypes and PyTorch's own functions do.  Nothing inside its scope touches a Python object.
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    NoGil() = default;
    NoGil(const NoGil&) = delete;
    ~NoGil() { PyEval_RestoreThread(state); }
};
void* stream_of(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
void* data(const Tensor& t) { return t.defined() && t.numel() > 0 ? t.data_ptr() : nullptr; }
float* fdata(const Tensor& t) { return (float*)data(t); }

void check_rc(int rc, const char* what) {
    TORCH_CHECK(rc == 0, what, " failed with status ", rc, ": ", coset_last_error_string());
}

const Tensor& tensor_arg(PyObject* o, const char* name) {
    TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a torch.Tensor, got ", Py_TYPE(o)->tp_name);
    return THPVariable_Unpack(o);
}
const Tensor& cuda_arg(PyObject* o, const char* name) {
    const Tensor& t = tensor_arg(o, name);
    TORCH_CHECK_VALUE(t.is_cuda(), name, " must live on a CUDA device (coset_b200 has no CPU path); got ", t.device());
    return t;
}
Tensor optional_arg(PyObject* o, const char* name) { return o == Py_None ? Tensor() : tensor_arg(o, name); }
std::optional<Tensor> maybe_arg(PyObject* o, const char* name) { return o == Py_None ? std::nullopt : std::optional<Tensor>(tensor_arg(o, name)); }

int64_t int_arg(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return (int64_t)v;
}
double float_arg(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
}
void nargs_are(Py_ssize_t got, Py_ssize_t want) { TORCH_CHECK_TYPE(got == want, "expected ", want, " arguments, got ", got); }

int dtype_code(const Tensor& t, const char* name) {
    if (t.scalar_type() == at::kFloat) return COSET_DTYPE_F32;
    TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16, name, " must be float32 or bfloat16, got ", t.scalar_type());
    return COSET_DTYPE_BF16;
}
at::ScalarType scalar_type(int code) {
    TORCH_CHECK_TYPE(code == COSET_DTYPE_F32 || code == COSET_DTYPE_BF16, "the result's dtype must be float32 or bfloat16");
    return code == COSET_DTYPE_F32 ? at::kFloat : at::kBFloat16;
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, const Tensor& like) {
    return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}
// The tensor as contiguous float32, itself when it already is.
Tensor as_f32(const Tensor& t) {
    if (!t.defined()) return t;
    Tensor f = t.scalar_type() == at::kFloat ? t : t.to(at::kFloat);
    return f.is_contiguous() ? f : f.contiguous();
}
// A kernel has written through the tensor's pointer: what was saved or made from it has to be seen as out of date.
void written(const Tensor& t) {
    if (!t.is_inference()) t.unsafeGetTensorImpl()->bump_version();
}
Tensor contiguous(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }

// rows of 8: a vector is one row
Tensor as_blocks(PyObject* o, const char* name, bool* squeeze) {
    const Tensor& x = cuda_arg(o, name);
    *squeeze = x.dim() == 1;
    Tensor x2 = *squeeze ? x.unsqueeze(0) : x;
    TORCH_CHECK_VALUE(x2.dim() == 2, name, " must be 1-D or 2-D, got ", x2.dim(), " dimensions");
    TORCH_CHECK_VALUE(x2.size(1) == 8, "Input dimension ", x2.size(1), " doesn't match E8 dimension 8");
    return contiguous(x2);
}
int64_t code_bytes(int64_t q, int64_t M) {
    const int b = coset_e8_code_bytes((int)q, (int)M);
    TORCH_CHECK_VALUE(b != 0, "unsupported (q=", q, ", M=", M, "); the CUDA library handles 2 <= q <= 16, 1 <= M <= 8");
    return b;
}

struct Scale {
    Tensor t;
    int mode = COSET_SCALE_NONE;
    int64_t bpt = 1;
};
Scale scale_arg(PyObject* o, int64_t mode, int64_t n_blocks, int64_t bpt, const Tensor& x) {
    Scale s;
    if (o == Py_None || mode == COSET_SCALE_NONE) return s;
    if (THPVariable_Check(o)) s.t = as_f32(cuda_arg(o, "scale"));
    else {  // filled on the device: no copy from the host
        PyObject* number = PyNumber_Float(o);  // what float(scale) takes
        if (!number) throw python_error();
        const double value = PyFloat_AS_DOUBLE(number);
        Py_DECREF(number);
        s.t = at::full({1}, (double)(float)value, x.options().dtype(at::kFloat));  // beyond float32: an infinity
    }
    if (mode == COSET_SCALE_DIV_SCALAR) {
        TORCH_CHECK_VALUE(s.t.numel() == 1, "the codec (divide) convention takes one scalar beta");
    } else {
        const int64_t tiles = bpt > 0 ? (n_blocks + bpt - 1) / bpt : 0;
        TORCH_CHECK_VALUE(s.t.numel() == tiles, "expected ", tiles, " per-tile scales, got ", s.t.numel());
    }
    s.mode = (int)mode;
    s.bpt = bpt;
    return s;
}

// ---------------------------------------------------------------- codec
// encode_packed(x, q, M, scale, scale_mode, blocks_per_tile, out, sem)
PyObject* encode_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 8);
    bool squeeze;
    const Tensor x = as_blocks(a[0], "x", &squeeze);
    const int64_t q = int_arg(a[1]), M = int_arg(a[2]), nb = x.size(0);
    const int64_t bytes = code_bytes(q, M);
    c10::cuda::CUDAGuard guard(x.device());
    const Scale s = scale_arg(a[3], int_arg(a[4]), nb, int_arg(a[5]), x);
    Tensor out;
    if (a[6] == Py_None) {
        out = empty({nb, bytes}, at::kByte, x);
    } else {
        out = tensor_arg(a[6], "out");
        TORCH_CHECK_VALUE((int64_t)out.nbytes() == nb * bytes && out.is_contiguous() && out.device() == x.device(),
                          "out has the wrong size, layout or device");
    }
    const int sem = (int)int_arg(a[7]);
    {
        NoGil no_gil;
        check_rc(coset_e8_encode(data(x), dtype_code(x, "x"), fdata(s.t), s.mode, nb, s.bpt, (int)q, (int)M, sem, data(out), stream_of(x)), "coset_e8_encode");
    }
    if (a[6] != Py_None) written(out);
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// decode_packed(codes, q, M, scale, scale_mode, blocks_per_tile, dtype_code, out)
PyObject* decode_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 8);
    const Tensor& codes = cuda_arg(a[0], "codes");
    const int64_t q = int_arg(a[1]), M = int_arg(a[2]);
    const int64_t bytes = code_bytes(q, M), total = (int64_t)codes.nbytes();
    TORCH_CHECK_VALUE(total % bytes == 0 && codes.is_contiguous(), "codes is not a contiguous array of packed block codes");
    const int64_t nb = total / bytes;
    c10::cuda::CUDAGuard guard(codes.device());
    const Scale s = scale_arg(a[3], int_arg(a[4]), nb, int_arg(a[5]), codes);
    Tensor out;
    if (a[7] == Py_None) {
        out = empty({nb, 8}, scalar_type((int)int_arg(a[6])), codes);
    } else {
        out = tensor_arg(a[7], "out");
        TORCH_CHECK_VALUE(out.dim() == 2 && out.size(0) == nb && out.size(1) == 8 && out.is_contiguous() && out.device() == codes.device(),
                          "out has the wrong shape, layout or device");
    }
    {
        NoGil no_gil;
        check_rc(coset_e8_decode(data(codes), fdata(s.t), s.mode, nb, s.bpt, (int)q, (int)M, COSET_SEM_CORE, data(out), dtype_code(out, "out"),
                                 stream_of(codes)), "coset_e8_decode");
    }
    if (a[7] != Py_None) written(out);
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// encode_digits(x, q, M, beta) -> float32 digits [N, M, 8]
PyObject* encode_digits(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 4);
    bool squeeze;
    const Tensor x = as_blocks(a[0], "x", &squeeze);
    TORCH_CHECK_TYPE(x.scalar_type() == at::kFloat, "e8_encode expects float32 like the reference; got ", x.scalar_type(),
                     " (use e8_encode_packed for bfloat16 input)");
    const int64_t q = int_arg(a[1]), M = int_arg(a[2]);
    code_bytes(q, M);
    c10::cuda::CUDAGuard guard(x.device());
    const float beta = (float)float_arg(a[3]);
    Tensor digits;
    {
        NoGil no_gil;
        digits = squeeze ? empty({M, 8}, at::kFloat, x) : empty({x.size(0), M, 8}, at::kFloat, x);
        check_rc(coset_e8_encode_digits_f32(fdata(x), beta, x.size(0), (int)q, (int)M, fdata(digits), stream_of(x)), "coset_e8_encode_digits_f32");
    }
    return THPVariable_Wrap(digits);
    END_HANDLE_TH_ERRORS
}

// decode_digits(digits [N, M, 8] or [M, 8], q, beta) -> float32 [N, 8] or [8]
PyObject* decode_digits(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 3);
    const Tensor& b = cuda_arg(a[0], "b");
    const bool squeeze = b.dim() == 2;
    TORCH_CHECK_VALUE((squeeze || b.dim() == 3) && b.size(-1) == 8, "encoding vectors must have shape [N, M, 8] or [M, 8], got ", b.sizes());
    const int64_t q = int_arg(a[1]), M = b.size(-2), nb = squeeze ? 1 : b.size(0);
    code_bytes(q, M);
    c10::cuda::CUDAGuard guard(b.device());
    const float beta = (float)float_arg(a[2]);
    Tensor out;
    {
        NoGil no_gil;
        const Tensor digits = as_f32(b);
        out = squeeze ? empty({8}, at::kFloat, b) : empty({nb, 8}, at::kFloat, b);
        check_rc(coset_e8_decode_digits_f32(fdata(digits), beta, nb, (int)q, (int)M, fdata(out), stream_of(b)), "coset_e8_decode_digits_f32");
    }
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// quantize(x, q): e8_quantize, float32 result
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 2);
    bool squeeze;
    const Tensor x = as_blocks(a[0], "x", &squeeze);
    const int64_t q = int_arg(a[1]);
    code_bytes(q, 2);
    c10::cuda::CUDAGuard guard(x.device());
    Tensor out;
    {
        NoGil no_gil;
        out = squeeze ? empty({8}, at::kFloat, x) : empty({x.size(0), 8}, at::kFloat, x);
        check_rc(coset_e8_quantize(data(x), dtype_code(x, "x"), nullptr, COSET_SCALE_NONE, x.size(0), 1, (int)q, 2, 0.0f, data(out),
                                   COSET_DTYPE_F32, nullptr, stream_of(x)), "coset_e8_quantize");
    }
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- gradient exchange
// grad_encode(blocks [n, 8], scale (1-element tensor), out, sem)
PyObject* grad_encode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 4);
    const Tensor &x = tensor_arg(a[0], "grad"), &s = tensor_arg(a[1], "scale"), &out = tensor_arg(a[2], "out");
    const int64_t nb = x.size(0);
    const int sem = (int)int_arg(a[3]);
    {
        NoGil no_gil;
        c10::cuda::CUDAGuard guard(x.device());
        check_rc(coset_e8_encode(data(x), dtype_code(x, "grad"), fdata(s), COSET_SCALE_MUL_TILE, nb, nb > 0 ? nb : 1, 4, 2, sem, data(out), stream_of(x)),
                 "coset_e8_encode");
    }
    written(out);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// decode_mean(codes [world, stride], world, n_blocks, scale, out)
PyObject* decode_mean(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 5);
    const Tensor &codes = tensor_arg(a[0], "codes"), &out = tensor_arg(a[4], "out");
    const int64_t world = int_arg(a[1]), nb = int_arg(a[2]);
    const float scale = (float)float_arg(a[3]);
    {
        NoGil no_gil;
        c10::cuda::CUDAGuard guard(codes.device());
        check_rc(coset_e8_decode_mean(data(codes), (int)world, nb, codes.size(1), scale, data(out), dtype_code(out, "out"), stream_of(codes)),
                 "coset_e8_decode_mean");
    }
    written(out);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- code-domain product
void check_codes(const Tensor& codes) {
    TORCH_CHECK_VALUE(codes.scalar_type() == at::kInt && codes.dim() == 2 && codes.is_contiguous(),
                      "codes must be a contiguous int32 tensor [n_out, n_in / 8]");
}
// [..., n_in] -> [T, n_in] and the shape of the result
Tensor token_rows(const Tensor& x, int64_t n_in, int64_t n_out, c10::SmallVector<int64_t, 6>* y_shape) {
    for (int64_t i = 0; i + 1 < x.dim(); ++i) y_shape->push_back(x.size(i));
    y_shape->push_back(n_out);
    Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, n_in});
    return contiguous(x2);
}

// vlut_linear(x [..., n_in], codes, beta or None, blocks_per_tile, bias or None, clip, out_dtype_code)
PyObject* vlut_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 7);
    const Tensor &codes = cuda_arg(a[1], "codes"), &x = cuda_arg(a[0], "x");
    check_codes(codes);
    const int64_t n_out = codes.size(0), n_in = codes.size(1) * 8;
    TORCH_CHECK_VALUE(x.dim() >= 1 && x.size(-1) == n_in, "x must be [T, ", n_in, "], got ", x.sizes());
    const Tensor beta_arg = optional_arg(a[2], "beta"), bias_arg = optional_arg(a[4], "bias");
    const int64_t bpt = int_arg(a[3]);
    const float clip = (float)float_arg(a[5]);
    const int y_code = (int)int_arg(a[6]);
    Tensor y;
    {
        NoGil no_gil;
        c10::cuda::CUDAGuard guard(x.device());
        c10::SmallVector<int64_t, 6> shape;
        const Tensor x2 = token_rows(x, n_in, n_out, &shape), beta = as_f32(beta_arg), bias = as_f32(bias_arg);
        y = empty(shape, scalar_type(y_code), x);
        check_rc(coset_e8_vlut_gemv(data(codes), fdata(beta), bpt, (int)n_out, (int)n_in, data(x2), dtype_code(x2, "x"), n_in, (int)x2.size(0), fdata(bias),
                                    data(y), y_code, n_out, clip, stream_of(x)), "coset_e8_vlut_gemv");
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// vlut_layout(codes) -> the decode-ready copy of the weight
PyObject* vlut_layout(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 1);
    const Tensor& codes = cuda_arg(a[0], "codes");
    check_codes(codes);
    const int n_out = (int)codes.size(0), n_in = (int)codes.size(1) * 8;
    c10::cuda::CUDAGuard guard(codes.device());
    Tensor layout;
    {
        NoGil no_gil;
        layout = empty({coset_e8_vlut_layout_bytes(n_out, n_in)}, at::kByte, codes);
        check_rc(coset_e8_vlut_layout(data(codes), n_out, n_in, data(layout), stream_of(codes)), "coset_e8_vlut_layout");
    }
    return THPVariable_Wrap(layout);
    END_HANDLE_TH_ERRORS
}

// The product from a layout; `codes` undefined: the layout is trusted.
Tensor layout_product(const Tensor& x, const Tensor& codes, const Tensor& layout, int64_t n_out, int64_t n_in, const Tensor& beta_arg, int64_t bpt,
                      const Tensor& bias_arg, double clip, int y_code) {
    NoGil no_gil;
    TORCH_CHECK_VALUE(x.dim() >= 1 && x.size(-1) == n_in, "x must be [T, ", n_in, "], got ", x.sizes());
    TORCH_CHECK_VALUE(layout.device() == x.device(), "the weight is on ", layout.device(), ", x on ", x.device());
    TORCH_CHECK_VALUE((int64_t)layout.nbytes() == coset_e8_vlut_layout_bytes((int)n_out, (int)n_in), "the layout is not one of a [", n_out, ", ", n_in, "] weight");
    c10::cuda::CUDAGuard guard(x.device());
    c10::SmallVector<int64_t, 6> shape;
    const Tensor x2 = token_rows(x, n_in, n_out, &shape);
    const Tensor beta = as_f32(beta_arg), bias = as_f32(bias_arg);
    const int x_code = dtype_code(x2, "x");
    Tensor y = empty(shape, scalar_type(y_code), x);
    void* target = data(y);
    if (target && codes.defined())
        check_rc(coset_e8_vlut_product_checked(data(codes), data(layout), fdata(beta), bpt, (int)n_out, (int)n_in, data(x2), x_code, n_in,
                                               (int)x2.size(0), fdata(bias), &target, 1, y_code, n_out, (float)clip, stream_of(x)), "coset_e8_vlut_product_checked");
    else if (target)
        check_rc(coset_e8_vlut_product(data(layout), fdata(beta), bpt, (int)n_out, (int)n_in, data(x2), x_code, n_in,
                                       (int)x2.size(0), fdata(bias), &target, 1, y_code, n_out, (float)clip, stream_of(x)), "coset_e8_vlut_product");
    return y;
}

// vlut_product(x [..., n_in], layout, n_out, n_in, beta or None, blocks_per_tile, bias or None, clip, out_dtype_code)
PyObject* vlut_product(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 9);
    return THPVariable_Wrap(layout_product(cuda_arg(a[0], "x"), Tensor(), tensor_arg(a[1], "layout"), int_arg(a[2]), int_arg(a[3]), optional_arg(a[4], "beta"),
                                           int_arg(a[5]), optional_arg(a[6], "bias"), float_arg(a[7]), (int)int_arg(a[8])));
    END_HANDLE_TH_ERRORS
}

// vlut_product_checked(x [..., n_in], codes, layout, beta or None, blocks_per_tile, bias or None, clip, out_dtype_code)
PyObject* vlut_product_checked(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 8);
    const Tensor &x = cuda_arg(a[0], "x"), &codes = cuda_arg(a[1], "codes");
    check_codes(codes);
    TORCH_CHECK_VALUE(codes.device() == x.device(), "the weight is on ", codes.device(), ", x on ", x.device());
    return THPVariable_Wrap(layout_product(x, codes, tensor_arg(a[2], "layout"), codes.size(0), codes.size(1) * 8, optional_arg(a[3], "beta"),
                                           int_arg(a[4]), optional_arg(a[5], "bias"), float_arg(a[6]), (int)int_arg(a[7])));
    END_HANDLE_TH_ERRORS
}

// decode_gemm(x [..., n_in] bf16, codes, beta or None, blocks_per_tile, bias or None, clip, scratch or None, out_dtype_code, status or None)
// -> (y, status)
PyObject* decode_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 9);
    const Tensor &codes = cuda_arg(a[1], "codes"), &x = cuda_arg(a[0], "x");
    TORCH_CHECK_TYPE(x.scalar_type() == at::kBFloat16, "e8_decode_gemm takes bfloat16 activations");
    check_codes(codes);
    const int64_t n_out = codes.size(0), n_in = codes.size(1) * 8;
    TORCH_CHECK_VALUE(x.dim() >= 1 && x.size(-1) == n_in && n_in % 64 == 0, "x must be [T, ", n_in, "] with n_in a multiple of 64, got ", x.sizes());
    Tensor scratch = optional_arg(a[6], "scratch"), status = optional_arg(a[8], "status"), y;
    const Tensor beta_arg = optional_arg(a[2], "beta"), bias_arg = optional_arg(a[4], "bias");
    const int64_t bpt = int_arg(a[3]);
    const float clip = (float)float_arg(a[5]);
    const int y_code = (int)int_arg(a[7]);
    {
        NoGil no_gil;
        c10::cuda::CUDAGuard guard(x.device());
        c10::SmallVector<int64_t, 6> shape;
        const Tensor x2 = token_rows(x, n_in, n_out, &shape);
        if (!scratch.defined()) scratch = empty({n_out * n_in}, at::kBFloat16, x);
        else
            TORCH_CHECK_VALUE(scratch.scalar_type() == at::kBFloat16 && scratch.numel() >= n_out * n_in && scratch.is_contiguous() && scratch.device() == x.device(),
                              "scratch must be a contiguous bfloat16 tensor of at least ", n_out * n_in, " values on ", x.device());
        y = empty(shape, scalar_type(y_code), x);
        if (!status.defined()) status = at::zeros({1}, x.options().dtype(at::kInt));
        const Tensor beta = as_f32(beta_arg), bias = as_f32(bias_arg);
        check_rc(coset_e8_decode_gemm(data(codes), fdata(beta), bpt, (int)n_out, (int)n_in, data(x2), n_in, (int)x2.size(0), fdata(bias), data(y), y_code, n_out,
                                      clip, data(scratch), (int64_t)scratch.nbytes(), (int*)data(status), stream_of(x)), "coset_e8_decode_gemm");
    }
    return Py_BuildValue("NN", THPVariable_Wrap(y), THPVariable_Wrap(status));
    END_HANDLE_TH_ERRORS
}

// A tensor that is nothing but memory on the GPU: no batch of a transform, no lazy negation, no tangent, not recorded.
bool plain(const Tensor& t) {
    if (!t.defined()) return true;
    static const c10::DispatchKeySet known = c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
                                             c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) | c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA);
    return (t.key_set().raw_repr() & ~known.raw_repr()) == 0 && !(at::GradMode::is_enabled() && t.requires_grad()) && !t._fw_grad(0).defined();
}

// Before torch's product in a capture: a thread's first one makes a cuBLAS handle, whose allocations a capture refuses unless the thread relaxes it.  The eager steps
// before may have been the own kernels' and made none.
void torch_product_in_capture() {
    const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    at::cuda::getCurrentCUDABlasHandle();
}
bool capturing() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }
// The own float32 products multiply in float32: a caller who lets torch's use TF32 gets those.
bool tf32_allowed() { return at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL) == at::Float32Precision::TF32; }
// Whether the library's own kernels may multiply a matrix: contiguous (and in bf16 made of aligned 16-byte chunks), and nobody looks at the torch calls.
bool own_rows(const Tensor& t) {
    const bool f32 = t.scalar_type() == at::kFloat;
    return plain(t) && c10::impl::TorchDispatchModeTLS::stack_len() == 0 && t.dim() == 2 && t.is_contiguous() && t.size(0) > 0 && t.size(0) <= INT32_MAX && t.size(1) > 0 &&
           ((f32 && !tf32_allowed()) || (t.scalar_type() == at::kBFloat16 && t.size(1) % 8 == 0 && (uintptr_t)t.const_data_ptr() % 16 == 0));
}
// Whether they should multiply for a training step: where the host bounds it (110 us with them, 141 with torch's products) and the device, which they cost
// more, does not.  Eager steps of a layer, own / torch, us:
//   bf16   the products take up to 40 % longer, most where rows are wide, and those of a wide input are read or written three times, of a wide
//          output twice: T (n_out + 2 n_in) of 34 M values [8192 x 4096 x 64] 110 / 146, [8192 x 2048 x 1024] 126 / 141; 36 M [4096 x 8192 x 256]
//          120 / 140; 42 M [8192 x 4096 x 512] 142 / 139; 50 M [16384 x 2048 x 512] 150 / 143; 68 M [4096 x 256 x 8192] 180 / 165; 101 M [8192 x 64 x 6144] 174 / 151.
//   float32 up to 61 us of products at 2^28 multiply-adds ([1024 x 512 x 512]; 54 with torch's); tiles count whole ([4096 x 10 x 2048] 131 / 141).
// The weight's gradient has few tiles in a narrow layer, and a cluster of eight CTAs at most sums over all tokens of one: bf16 [32768 x 64 x 64] 111 / 142 but
// [262144 x 64 x 64] 442 / 180; float32 [16384 x 16 x 64] 109 / 143, [65536 x 64 x 64] 314 / 255, [2^20 x 8 x 8] 6195 / 993.
// Under capture the host costs nothing, and what is quicker on the device is recorded: torch's in bf16 ([4096 x 3072 x 768] 105 us a replay against 115, [128 x 768 x 768]
// 39 / 43), the own in float32 up to 2^27 ([128 x 768 x 768] 59 with torch's against 54, [4096 x 64 x 64] 78 / 51; beyond, [1024 x 512 x 512] 72 / 74), but for narrow
// layers with many tokens ([16384 x 16 x 64] 55 / 112).
bool own_training_products(at::ScalarType type, int64_t tokens, int64_t n_out, int64_t n_in, bool capturing) {
    if (tokens <= 0 || tokens > 1 << 15 || n_out <= 0 || n_in <= 0 || n_out > ((int64_t)1 << 22) / n_in) return false;
    const auto whole = [](int64_t v, int64_t tile) { return (v + tile - 1) / tile * tile; };
    const int64_t products = tokens * n_out * n_in;
    // Below 32 tokens torch's float32 sums are the more precise ones (f32_product.cu).  A trace of the layer and a torch-function mode see torch's product, with which the
    // own ones agree to the rounding of the type.  Float32 steps below 2^16 keep torch's, though it costs the host 25 us there as anywhere: a step that small is
    // one that is compared to the bit with its trace.
    if (type == at::kFloat) {
        const int64_t of_tiles = whole(tokens, 32) * whole(n_out, 64) * whole(n_in, 64);
        return tokens >= 32 && tokens <= 1 << 14 && products >= 1 << 16 && products <= 1 << 28 && of_tiles <= 1 << 29 &&
               !(capturing && (tokens > 4096 || of_tiles > 1 << 27));
    }
    return type == at::kBFloat16 && !capturing && n_out % 8 == 0 && n_in % 8 == 0 && products <= (int64_t)1 << 34 && tokens * (n_out + 2 * n_in) <= 9 << 22;
}
// The rows of a layer's input where its product is the library's own, undefined where it is torch's (which refuses what does not fit together).
Tensor own_layer_rows(const Tensor& x, const Tensor& w, const Tensor& bias) {
    const int64_t n_out = w.size(0), n_in = w.size(1);
    if (!x.is_contiguous() || x.dim() < 1 || x.size(-1) != n_in || w.numel() == 0 || x.device() != w.device()) return Tensor();
    if (bias.defined() && !(bias.scalar_type() == at::kFloat && bias.is_contiguous() && bias.device() == w.device() && bias.dim() == 1 && bias.numel() == n_out)) return Tensor();
    const Tensor x2 = x.dim() == 2 ? x : x.view({-1, n_in});
    return own_rows(x2) && own_training_products(x.scalar_type(), x2.size(0), n_out, n_in, capturing()) ? x2 : Tensor();
}

// dense_linear(x [T, n_in] bf16, w [n_out, n_in] bf16, bias or None, status or None, own): x w^T + bias as bf16.  `own`: by the library's own
// kernel, which adds the float32 bias to the float32 sums; else, and for whoever looks at the torch call (autograd, autocast, transforms,
// dispatch modes), by torch's product with the bias rounded to bf16 first.
PyObject* dense_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 5);
    const Tensor &x = cuda_arg(a[0], "x"), &w = cuda_arg(a[1], "w");
    const Tensor bias = optional_arg(a[2], "bias"), status = optional_arg(a[3], "status");
    bool own = a[4] == Py_True;
    Tensor y;
    {
        NoGil no_gil;
        c10::cuda::CUDAGuard guard(x.device());
        own = own && x.dim() == 2 && w.dim() == 2 && x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && x.size(1) == w.size(1) && x.size(1) > 0 &&
              x.size(1) % 8 == 0 && plain(x) && plain(w) && plain(bias) && w.is_contiguous() && (uintptr_t)w.const_data_ptr() % 16 == 0 && w.device() == x.device() &&
              (!bias.defined() || (bias.device() == x.device() && bias.dim() == 1 && bias.size(0) == w.size(0))) &&
              !at::autocast::is_autocast_enabled(at::kCUDA) && c10::impl::TorchDispatchModeTLS::stack_len() == 0;
        if (own) {
            const bool rows = x.stride(1) == 1 && x.stride(0) >= x.size(1) && x.stride(0) % 8 == 0 && (uintptr_t)x.const_data_ptr() % 16 == 0;
            const Tensor x2 = rows ? x : x.clone(at::MemoryFormat::Contiguous), b = as_f32(bias);
            y = empty({x.size(0), w.size(0)}, at::kBFloat16, x);
            check_rc(coset_e8_dense_linear(data(w), (int)w.size(0), (int)w.size(1), data(x2), x2.stride(0), (int)x2.size(0), fdata(b), 0, data(y), y.size(1),
                                           (int*)data(status), stream_of(x)), "coset_e8_dense_linear");
        } else {
            Tensor b = bias;
            if (b.defined()) {
                if (b.scalar_type() == at::kFloat && b.device() == x.device() && b.has_storage() && b.is_contiguous() && !b.requires_grad()) {
                    b = empty(bias.sizes(), at::kBFloat16, bias);
                    check_rc(coset_layer_beta_bias(nullptr, nullptr, nullptr, 0, nullptr, fdata(bias), bias.numel(), data(b), stream_of(x)), "coset_layer_beta_bias");
                } else b = bias.to(at::kBFloat16);
            }
            if (capturing()) torch_product_in_capture();
            y = at::linear(x, w, b.defined() ? std::optional<Tensor>(b) : std::nullopt);
        }
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- training layer
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// W_q = clamp(e8_quantize(W beta) / beta, +-clip) with beta = beta_min + sigmoid(theta) range per tile, and the
// straight-through gradients of the reference graph (coset/core/layers.py:62-110, 415-470).
struct FakeQuant : torch::autograd::Function<FakeQuant> {
    // bias16: the bias in bf16, written by the launch that forms the scales, where the caller wants one
    static void launch(const Tensor& w, const Tensor& th, const Tensor& beta_min, const Tensor& beta_range, int64_t bpt, int64_t q, double clip,
                       at::ScalarType out_type, Tensor& wq, Tensor& codes, Tensor& beta, const Tensor& bias = Tensor(), const Tensor& bias16 = Tensor()) {
        const int bytes = coset_e8_code_bytes((int)q, 2);
        TORCH_CHECK_VALUE(bytes != 0, "unsupported q=", q, " for the fused E8 weight quantiser (2 <= q <= 16)");
        TORCH_CHECK(bpt >= 1, "blocks_per_tile must be >= 1");
        const int64_t nb = w.numel() / 8;
        codes = empty({nb, bytes}, at::kByte, w);
        wq = empty(w.sizes(), out_type, w);
        beta = empty({th.numel()}, at::kFloat, w);
        check_rc(coset_layer_beta_bias(fdata(th), fdata(beta_min), fdata(beta_range), (nb + bpt - 1) / bpt, fdata(beta), fdata(bias),
                                       bias16.defined() ? bias.numel() : 0, data(bias16), stream_of(w)), "coset_layer_beta_bias");
        check_rc(coset_e8_quantize(fdata(w), COSET_DTYPE_F32, fdata(beta), COSET_SCALE_MUL_TILE, nb, bpt, (int)q, 2, (float)clip, data(wq),
                                   out_type == at::kFloat ? COSET_DTYPE_F32 : COSET_DTYPE_BF16, data(codes), stream_of(w)), "coset_e8_quantize");
    }
    // dL/dW and dL/dtheta (undefined unless asked for) from dL/dW_q
    static std::pair<Tensor, Tensor> backward_launch(Tensor g, const Tensor& w, const Tensor& theta, const Tensor& beta, const Tensor& codes,
                                                     const Tensor& beta_range, int64_t bpt, int64_t q, double clip, bool need_theta) {
        g = contiguous(g);
        if (g.scalar_type() != at::kFloat && g.scalar_type() != at::kBFloat16) g = g.to(at::kFloat);
        const Tensor th = as_f32(theta);
        Tensor gw = empty(w.sizes(), at::kFloat, w), gt;
        if (need_theta) gt = empty(theta.sizes(), at::kFloat, w);
        check_rc(coset_e8_layer_fake_quant_bwd(data(g), dtype_code(g, "grad"), fdata(w), data(codes), fdata(beta), fdata(th), fdata(beta_range),
                                               w.numel() / 8, bpt, (int)q, (float)clip, fdata(gw), fdata(gt), stream_of(w)),
                 "coset_e8_layer_fake_quant_bwd");
        return {gw, gt};
    }
    static Tensor forward(AutogradContext* ctx, const Tensor& weight, const Tensor& theta, const Tensor& beta_min, const Tensor& beta_range,
                          int64_t bpt, int64_t q, double clip, int64_t out_code) {
        const Tensor w = contiguous(weight);
        Tensor wq, codes, beta;
        launch(w, as_f32(theta), beta_min, beta_range, bpt, q, clip, scalar_type((int)out_code), wq, codes, beta);
        ctx->save_for_backward({w, theta, beta, codes});
        // the bounds are refreshed in place once every stat_update_interval steps (a captured graph keeps reading
        // them), so they are kept outside save_for_backward, whose version check would refuse that
        ctx->saved_data["range"] = beta_range;
        ctx->saved_data["bpt"] = bpt;
        ctx->saved_data["q"] = q;
        ctx->saved_data["clip"] = clip;
        return wq;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        c10::cuda::CUDAGuard guard(saved[0].device());
        auto r = backward_launch(grads[0], saved[0], saved[1], saved[2], saved[3], ctx->saved_data["range"].toTensor(), ctx->saved_data["bpt"].toInt(),
                                 ctx->saved_data["q"].toInt(), ctx->saved_data["clip"].toDouble(), ctx->needs_input_grad(1));
        return {r.first, r.second, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// y = x W_q^T + bias as ONE autograd node: the forward quantises and multiplies, the backward forms dx, dW, dtheta
// and dbias.  An eager step of a small layer is bound by the host; one node instead of five (cast, quantise,
// transpose, product, bias) and native code on both sides took the step of the [3072, 768] layer with 4096
// tokens from 330 to 171 us, 80 of them on the device.
struct QatLinear : torch::autograd::Function<QatLinear> {
    // the bias is optional, not undefined: an undefined tensor is an input of the node like any other and has no device
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& theta, const std::optional<Tensor>& bias,
                          const Tensor& beta_min, const Tensor& beta_range, int64_t bpt, int64_t q, double clip) {
        const Tensor w = contiguous(weight);
        Tensor wq, codes, beta, b = bias ? *bias : Tensor(), b16;
        const Tensor x2 = own_layer_rows(x, w, b);
        const bool own = x2.defined();
        if (b.defined() && x.scalar_type() == at::kBFloat16 && !own) {
            if (b.scalar_type() == at::kFloat && b.is_contiguous() && b.device() == w.device()) b16 = empty(b.sizes(), at::kBFloat16, w);
            else b = b.to(at::kBFloat16);
        }
        FakeQuant::launch(w, as_f32(theta), beta_min, beta_range, bpt, q, clip, x.scalar_type(), wq, codes, beta, b, b16);
        if (b16.defined()) b = b16;
        Tensor y;
        if (own) {
            c10::SmallVector<int64_t, 6> y_shape(x.sizes().begin(), x.sizes().end());
            y_shape.back() = w.size(0);
            y = empty(y_shape, x.scalar_type(), x);
            const int T = (int)x2.size(0), N = (int)w.size(0), K = (int)w.size(1);
            check_rc(x.scalar_type() == at::kFloat ? coset_f32_linear(fdata(x2), fdata(wq), fdata(b), T, N, K, fdata(y), stream_of(x))
                                                   : coset_e8_dense_linear(data(wq), N, K, data(x2), K, T, fdata(b), 1, data(y), N, nullptr, stream_of(x)), "the layer's product");
        } else {
            if (capturing()) torch_product_in_capture();
            y = at::linear(x, wq, b.defined() ? std::optional<Tensor>(b) : std::nullopt);
        }
        // x serves the gradients of the weight and its scale, wq that of x: a frozen layer does not hold on to its input
        const bool weights = weight.requires_grad() || theta.requires_grad();
        ctx->save_for_backward({weights ? x : Tensor(), w, theta, beta, codes, x.requires_grad() ? wq : Tensor()});
        ctx->saved_data["x_type"] = (int64_t)x.scalar_type();
        ctx->saved_data["range"] = beta_range;
        ctx->saved_data["min"] = beta_min;
        ctx->saved_data["bpt"] = bpt;
        ctx->saved_data["q"] = q;
        ctx->saved_data["clip"] = clip;
        if (bias) ctx->saved_data["bias_type"] = (int64_t)bias->scalar_type();
        return y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &x = saved[0], &w = saved[1], &theta = saved[2], &beta = saved[3], &codes = saved[4];
        c10::cuda::CUDAGuard guard(w.device());
        const int64_t bpt = ctx->saved_data["bpt"].toInt(), q = ctx->saved_data["q"].toInt();
        const double clip = ctx->saved_data["clip"].toDouble();
        const Tensor range = ctx->saved_data["range"].toTensor();
        Tensor wq = saved[5];
        // create_graph: the gradient of x has to depend on the weight, so the weight is quantised again under autograd
        if (at::GradMode::is_enabled() && ctx->needs_input_grad(0))
            wq = FakeQuant::apply(w, theta, ctx->saved_data["min"].toTensor(), range, bpt, q, clip,
                                  (int64_t)((at::ScalarType)ctx->saved_data["x_type"].toInt() == at::kFloat ? COSET_DTYPE_F32 : COSET_DTYPE_BF16));
        const Tensor g2 = grads[0].reshape({-1, w.size(0)});
        variable_list out(9);
        const int64_t T = g2.size(0), N = w.size(0), K = w.size(1);
        const at::ScalarType type = g2.scalar_type();
        const bool captured = capturing();
        const auto torchs = [&](const Tensor& a, const Tensor& b) {
            if (captured) torch_product_in_capture();
            return at::mm(a, b);
        };
        const bool own = !at::GradMode::is_enabled() && own_training_products(type, T, N, K, captured) && own_rows(g2) && g2.device() == w.device() &&
                         !at::autocast::is_autocast_enabled(at::kCUDA), f32 = type == at::kFloat;
        if (ctx->needs_input_grad(0)) {
            c10::SmallVector<int64_t, 6> x_shape(grads[0].sizes().begin(), grads[0].sizes().end());
            x_shape.back() = K;
            if (own && own_rows(wq) && wq.scalar_type() == type && wq.device() == w.device()) {
                out[0] = empty(x_shape, type, g2);
                check_rc(f32 ? coset_f32_input_grad(fdata(g2), fdata(wq), (int)T, (int)N, (int)K, fdata(out[0]), stream_of(g2))
                             : coset_dense_input_grad(data(g2), data(wq), (int)T, (int)N, (int)K, data(out[0]), nullptr, stream_of(g2)), "the gradient of the input");
            } else out[0] = torchs(g2, wq).view(x_shape);
        }
        const bool need_theta = ctx->needs_input_grad(2);
        if (ctx->needs_input_grad(1) || need_theta) {
            const Tensor x2 = x.reshape({-1, K});
            Tensor gw;
            if (own && own_rows(x2) && x2.scalar_type() == type && x2.size(0) == T && x2.device() == w.device()) {
                gw = empty({N, K}, type, g2);
                check_rc(f32 ? coset_f32_weight_grad(fdata(g2), fdata(x2), (int)T, (int)N, (int)K, fdata(gw), stream_of(g2))
                             : coset_dense_weight_grad(data(g2), data(x2), (int)T, (int)N, (int)K, data(gw), nullptr, stream_of(g2)), "the gradient of the weight");
            } else gw = torchs(g2.t(), x2);
            auto r = FakeQuant::backward_launch(gw, w, theta, beta, codes, range, bpt, q, clip, need_theta);
            out[1] = r.first;
            out[2] = r.second;
        }
        const auto bias_type = ctx->saved_data.find("bias_type");  // absent with the bias, which then is no input and has no edge
        if (bias_type != ctx->saved_data.end() && ctx->needs_input_grad(3)) {
            const auto type = (at::ScalarType)bias_type->second.toInt();
            const bool own = g2.is_contiguous() && (type == at::kFloat || type == at::kBFloat16) && (g2.scalar_type() == at::kFloat || g2.scalar_type() == at::kBFloat16)
                             && !at::GradMode::is_enabled();
            if (own) {
                out[3] = empty({g2.size(1)}, type, g2);
                check_rc(coset_column_sum(data(g2), dtype_code(g2, "grad"), g2.size(0), g2.size(1), data(out[3]),
                                          type == at::kFloat ? COSET_DTYPE_F32 : COSET_DTYPE_BF16, stream_of(g2)), "coset_column_sum");
            } else out[3] = at::sum(g2, at::IntArrayRef{0}, false, g2.scalar_type() == type ? std::nullopt : std::optional<at::ScalarType>(type));
        }
        return out;
    }
};

void check_weight(const Tensor& w) {
    TORCH_CHECK_TYPE(w.scalar_type() == at::kFloat, "weight must be float32 (the fused weight kernels read float32 rows), got ", w.scalar_type(),
                     "; keep the layer's parameters in float32 and pass low-precision activations instead");
}

// layer_fake_quant(weight, theta, beta_min, beta_range, blocks_per_tile, q, clip, out_dtype_code)
PyObject* layer_fake_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 8);
    const Tensor& w = tensor_arg(a[0], "weight");
    check_weight(w);
    cuda_arg(a[0], "weight");
    const Tensor &theta = tensor_arg(a[1], "theta"), &beta_min = tensor_arg(a[2], "beta_min"), &beta_range = tensor_arg(a[3], "beta_range");
    const int64_t bpt = int_arg(a[4]), q = int_arg(a[5]), out_code = int_arg(a[7]);
    const double clip = float_arg(a[6]);
    Tensor wq;
    {
        NoGil no_gil;
        c10::cuda::CUDAGuard guard(w.device());
        wq = FakeQuant::apply(w, theta, beta_min, beta_range, bpt, q, clip, out_code);
    }
    return THPVariable_Wrap(wq);
    END_HANDLE_TH_ERRORS
}

// qat_linear(x, weight, theta, bias or None, beta_min, beta_range, blocks_per_tile, q, clip)
PyObject* qat_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 9);
    const Tensor &x = tensor_arg(a[0], "x"), &w = tensor_arg(a[1], "weight");
    check_weight(w);
    cuda_arg(a[1], "weight");
    const Tensor &theta = tensor_arg(a[2], "theta"), &beta_min = tensor_arg(a[4], "beta_min"), &beta_range = tensor_arg(a[5], "beta_range");
    const std::optional<Tensor> bias = maybe_arg(a[3], "bias");
    const int64_t bpt = int_arg(a[6]), q = int_arg(a[7]);
    const double clip = float_arg(a[8]);
    Tensor y;
    {
        NoGil no_gil;
        c10::cuda::CUDAGuard guard(w.device());
        y = QatLinear::apply(x, w, theta, bias, beta_min, beta_range, bpt, q, clip);
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// own_product_sizes(dtype_code, tokens, n_out, n_in, capturing) -> whether a training step of these sizes is multiplied by the library's own kernels
PyObject* own_product_sizes(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 5);
    return PyBool_FromLong(own_training_products(scalar_type((int)int_arg(a[0])), int_arg(a[1]), int_arg(a[2]), int_arg(a[3]), a[4] == Py_True));
    END_HANDLE_TH_ERRORS
}

// own_product(x, weight, bias or None) -> whether qat_linear multiplies x by the library's own kernel; launches nothing
PyObject* own_product(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    nargs_are(n, 3);
    const Tensor &x = tensor_arg(a[0], "x"), &w = tensor_arg(a[1], "weight");
    at::AutoGradMode no_grad(false);  // as inside the node
    const c10::cuda::OptionalCUDAGuard guard(x.is_cuda() ? std::optional<c10::Device>(x.device()) : std::nullopt);
    return PyBool_FromLong(own_layer_rows(x, w, optional_arg(a[2], "bias")).defined());
    END_HANDLE_TH_ERRORS
}

#define COSET_METHOD(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    COSET_METHOD(encode_packed), COSET_METHOD(decode_packed), COSET_METHOD(encode_digits), COSET_METHOD(decode_digits), COSET_METHOD(quantize),
    COSET_METHOD(grad_encode), COSET_METHOD(decode_mean), COSET_METHOD(vlut_linear), COSET_METHOD(vlut_layout), COSET_METHOD(vlut_product), COSET_METHOD(vlut_product_checked),
    COSET_METHOD(decode_gemm), COSET_METHOD(dense_linear), COSET_METHOD(layer_fake_quant), COSET_METHOD(qat_linear), COSET_METHOD(own_product), COSET_METHOD(own_product_sizes), {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_coset_torch", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__coset_torch(void) { return PyModule_Create(&kModule); }

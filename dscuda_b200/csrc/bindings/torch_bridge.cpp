// Python extension of the host side (`_dscuda_torch`, loaded by dscuda_b200/library.py): torch tensors in,
// C-ABI calls of include/dscuda_c_api.h out.  dscuda_b200/mla.py holds the documented signatures; its functions
// hand their arguments to the functions here in order.
//
// Why native: a decode or a small training step is two to five kernels of 5-15 us, and the same work written in
// Python (attribute checks, torch.empty, a ctypes call with 15-21 converted arguments) took 17-20 us of host
// time per call, more than the kernels.  METH_FASTCALL functions that unpack the tensors themselves take 4-8 us,
// most of it the launches.  The interpreter lock is released around every C-ABI call, as ctypes does.
#include "dscuda_c_api.h"

#include <ATen/Functions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/version.h>

#include <Python.h>

#include <optional>
#include <stdexcept>
#include <string>

namespace {

using at::Tensor;

constexpr int64_t LATENT = 512;                // width of the latent part of a cache row
constexpr int64_t VALUE = 128;                 // columns of k_nope and v
constexpr int64_t CACHE_WIDTH = 576;           // of a whole row
constexpr int64_t FP8_ROW_BYTES = 656;

// A Python error that is not one of c10's (HANDLE_TH_ERRORS would turn std::exception into RuntimeError).
struct PythonError {
    PyObject* type;
    std::string message;
};

[[noreturn]] void fail(PyObject* type, std::string message) {
    throw PythonError{type, std::move(message)};
}

void expect_arguments(Py_ssize_t given, Py_ssize_t wanted) {
    if (given != wanted) {
        fail(PyExc_TypeError, "expected " + std::to_string(wanted) + " arguments, got " + std::to_string(given));
    }
}

// A CUDA, contiguous tensor.
const Tensor& tensor(PyObject* object) {
    if (!THPVariable_Check(object)) {
        fail(PyExc_TypeError, std::string("expected a torch tensor, got ") + Py_TYPE(object)->tp_name);
    }
    const Tensor& t = THPVariable_Unpack(object);
    if (!t.is_cuda()) {
        fail(PyExc_RuntimeError, "dscuda_b200 runs on CUDA tensors only; there is no CPU path");
    }
    if (!t.is_contiguous()) {
        fail(PyExc_ValueError, "tensors must be contiguous");
    }
    return t;
}

void expect_dims(const Tensor& t, int64_t dims) {
    if (t.dim() != dims) {
        fail(PyExc_ValueError, "expected a tensor of " + std::to_string(dims) + " dimensions, got " + std::to_string(t.dim()));
    }
}

// The same with a given number of dimensions.
const Tensor& tensor(PyObject* object, int64_t dims) {
    const Tensor& t = tensor(object);
    expect_dims(t, dims);
    return t;
}

// The same, or null for None.
const Tensor* optional_tensor(PyObject* object) {
    return object == Py_None ? nullptr : &tensor(object);
}

// Memory the caller brings for a result or as scratch is written through its pointer, so it has to be where the inputs are and
// large enough (it may be larger).
void expect_device(const Tensor& t, const Tensor& like, const char* what) {
    if (t.device() != like.device()) {
        fail(PyExc_ValueError, std::string(what) + " is on another device than the inputs");
    }
}

// An output the caller may bring, of `elements` values of `type`; null for None.
const Tensor* optional_output(PyObject* object, const Tensor& like, at::ScalarType type, int64_t elements, const char* what) {
    const Tensor* t = optional_tensor(object);
    if (t != nullptr) {
        expect_device(*t, like, what);
        if (t->scalar_type() != type) {
            fail(PyExc_ValueError, std::string(what) + " has the wrong dtype");
        }
        if (t->numel() < elements) {
            fail(PyExc_ValueError, std::string(what) + " has " + std::to_string(t->numel()) + " elements, " + std::to_string(elements) + " are written");
        }
    }
    return t;
}

// Scratch the caller may bring, of at least `bytes` bytes and any dtype; null for None.
const Tensor* optional_workspace(PyObject* object, const Tensor& like, size_t bytes) {
    const Tensor* t = optional_tensor(object);
    if (t != nullptr) {
        expect_device(*t, like, "the workspace");
        if (t->nbytes() < bytes) {
            fail(PyExc_ValueError, "the workspace has " + std::to_string(t->nbytes()) + " bytes, " + std::to_string(bytes) + " are needed");
        }
    }
    return t;
}

void* pointer(const Tensor& t) {
    return t.data_ptr();
}

void* pointer(const Tensor* t) {
    return t == nullptr ? nullptr : t->data_ptr();
}

const int* int_pointer(const Tensor* t) {
    return static_cast<const int*>(pointer(t));
}

float number(PyObject* object) {
    const double value = PyFloat_AsDouble(object);
    if (value == -1.0 && PyErr_Occurred()) {
        throw python_error();
    }
    return static_cast<float>(value);
}

long long integer(PyObject* object) {
    const long long value = PyLong_AsLongLong(object);
    if (value == -1 && PyErr_Occurred()) {
        throw python_error();
    }
    return value;
}

// Rows of a tensor whose last `columns` elements make one row.
long long row_count(const Tensor& t, int64_t columns) {
    if (columns == 0) {
        fail(PyExc_ValueError, "tensors must not be empty");
    }
    return t.numel() / columns;
}

// Sizes go through the C ABI as int; what does not fit is cut like a ctypes c_int argument, and the entry points
// refuse sizes that are not positive.
int extent(const Tensor& t, int64_t dim) {
    return static_cast<int>(t.size(dim));
}

void* current_stream() {
    return c10::cuda::getCurrentCUDAStream().stream();
}

Tensor new_tensor(at::IntArrayRef sizes, const Tensor& like, at::ScalarType type) {
    return at::empty(sizes, at::TensorOptions().device(like.device()).dtype(type));
}

Tensor new_like(const Tensor& t) {
    return at::empty(t.sizes(), at::TensorOptions().device(t.device()).dtype(t.scalar_type()));
}

// The interpreter lock is released for the lifetime of this object; taken back when an exception passes too (data_ptr() of a
// tensor without storage throws inside the call).
struct LockReleased {
    PyThreadState* state = PyEval_SaveThread();
    LockReleased() = default;
    LockReleased(const LockReleased&) = delete;
    LockReleased& operator=(const LockReleased&) = delete;
    ~LockReleased() { PyEval_RestoreThread(state); }
};

// Runs one C-ABI call without the interpreter lock; a non-zero status becomes a RuntimeError with the library's message.
template <class Call>
void checked(const char* (*last_error)(), Call&& call) {
    int status;
    {
        const LockReleased released;
        status = call();
    }
    if (status != 0) {
        fail(PyExc_RuntimeError, last_error());
    }
}

// Entry and exit of every function: c10 errors keep torch's Python types, PythonError sets its own.
template <class Body>
PyObject* guarded(Body&& body) {
    HANDLE_TH_ERRORS
    try {
        return body();
    } catch (const PythonError& error) {
        PyErr_SetString(error.type, error.message.c_str());
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyObject* wrap(const Tensor& t) {
    return THPVariable_Wrap(t);
}

template <class... Tensors>
PyObject* tuple(const Tensors&... tensors) {
    PyObject* result = PyTuple_New(sizeof...(tensors));
    if (result == nullptr) {
        throw python_error();
    }
    Py_ssize_t index = 0;
    (PyTuple_SET_ITEM(result, index++, wrap(tensors)), ...);
    return result;
}

#define DSCUDA_FUNCTION(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t count)

// ---- absorbed forward and backward -------------------------------------------
// query, query_rope, latent, key_rope, scale -> output, lse
DSCUDA_FUNCTION(mla_forward) {
    return guarded([&] {
        expect_arguments(count, 5);
        const Tensor &query = tensor(args[0], 4), &query_rope = tensor(args[1]), &latent = tensor(args[2]), &key_rope = tensor(args[3]);
        const float scale = number(args[4]);
        const int b = extent(query, 0), t = extent(query, 1), h = extent(query, 2), c = extent(query, 3), r = extent(query_rope, -1);
        Tensor output = new_like(query);
        Tensor lse = new_tensor({b, h, t}, query, at::kFloat);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] {
            return dscuda_mla_forward(pointer(output), static_cast<float*>(pointer(lse)), pointer(query), pointer(query_rope), pointer(latent),
                                      pointer(key_rope), b, t, h, c, r, scale, stream);
        });
        return tuple(output, lse);
    });
}

// dout, output, lse, query, query_rope, latent, key_rope, scale -> dquery, dquery_rope, dlatent, dkey_rope
DSCUDA_FUNCTION(mla_backward) {
    return guarded([&] {
        expect_arguments(count, 8);
        const Tensor &dout = tensor(args[0]), &output = tensor(args[1]), &lse = tensor(args[2]), &query = tensor(args[3], 4), &query_rope = tensor(args[4]),
                     &latent = tensor(args[5]), &key_rope = tensor(args[6]);
        const float scale = number(args[7]);
        const int b = extent(query, 0), t = extent(query, 1), h = extent(query, 2), c = extent(query, 3), r = extent(query_rope, -1);
        Tensor dquery = new_like(query), dquery_rope = new_like(query_rope), dlatent = new_like(latent), dkey_rope = new_like(key_rope);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] {
            return dscuda_mla_backward(pointer(dquery), pointer(dquery_rope), pointer(dlatent), pointer(dkey_rope), pointer(dout), pointer(output),
                                       static_cast<const float*>(pointer(lse)), pointer(query), pointer(query_rope), pointer(latent), pointer(key_rope), b,
                                       t, h, c, r, scale, stream);
        });
        return tuple(dquery, dquery_rope, dlatent, dkey_rope);
    });
}

// ---- paged decode --------------------------------------------------------------
// query, paged_cache, block_table, lengths, scale, splits, workspace, output, lse, checked_pages -> output, lse
DSCUDA_FUNCTION(mla_decode) {
    return guarded([&] {
        expect_arguments(count, 10);
        const Tensor &query = tensor(args[0], 4), &cache = tensor(args[1]), &table = tensor(args[2]), &lengths = tensor(args[3]);
        const float scale = number(args[4]);
        const int splits = static_cast<int>(integer(args[5]));
        const int pages_checked = PyObject_IsTrue(args[9]);
        if (pages_checked < 0) {
            throw python_error();
        }
        const int b = extent(query, 0), h = extent(query, 2), rope = static_cast<int>(query.size(3) - LATENT), page_size = extent(cache, 1);
        const int pages = extent(table, 1), blocks = extent(cache, 0);
        const int64_t rows = static_cast<int64_t>(b) * h;
        // sizes that are not positive are refused below
        const size_t partials_bytes = splits > 0 ? dscuda_mla_workspace_elements(b, h, splits, static_cast<int>(LATENT)) * sizeof(float) : 0;
        const Tensor* workspace_given = optional_workspace(args[6], query, partials_bytes);
        const Tensor *output_given = optional_output(args[7], query, at::kBFloat16, rows * LATENT, "the output"),
                     *lse_given = optional_output(args[8], query, at::kFloat, rows, "the LSE");
        Tensor workspace =
            workspace_given != nullptr
                ? *workspace_given
                : new_tensor({static_cast<int64_t>(dscuda_mla_workspace_elements(b, h, splits, static_cast<int>(LATENT)))}, query, at::kFloat);
        Tensor output = output_given != nullptr ? *output_given : new_tensor({b, 1, h, LATENT}, query, at::kBFloat16);
        Tensor lse = lse_given != nullptr ? *lse_given : new_tensor({b, h, 1}, query, at::kFloat);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] {
            float* lse_out = static_cast<float*>(pointer(lse));
            float* partials = static_cast<float*>(pointer(workspace));
            if (pages_checked != 0) {
                return dscuda_mla_decode_checked(pointer(output), lse_out, pointer(query), pointer(cache), int_pointer(&table), int_pointer(&lengths),
                                                 partials, b, h, static_cast<int>(LATENT), rope, page_size, pages, blocks, splits, scale, stream);
            }
            return dscuda_mla_decode(pointer(output), lse_out, pointer(query), pointer(cache), int_pointer(&table), int_pointer(&lengths), partials, b,
                                     h, static_cast<int>(LATENT), rope, page_size, pages, splits, scale, stream);
        });
        return tuple(output, lse);
    });
}

// ---- cache -----------------------------------------------------------------------
// paged_cache, kv_latent, key_rope, block_table, start_positions, token_counts; `fp8` picks the format
PyObject* append(PyObject* const* args, Py_ssize_t count, bool fp8) {
    return guarded([&] {
        expect_arguments(count, 6);
        const Tensor &cache = tensor(args[0]), &latent = tensor(args[1], 3), &key_rope = tensor(args[2]), &table = tensor(args[3]);
        const Tensor *start = optional_tensor(args[4]), *counts = optional_tensor(args[5]);
        if (fp8 && (cache.scalar_type() != at::kByte || cache.size(-1) != FP8_ROW_BYTES)) {
            fail(PyExc_ValueError, "the FP8 cache is a uint8 tensor [blocks, page, 656]");
        }
        const int b = extent(latent, 0), t = extent(latent, 1), rank = extent(latent, 2), rope = extent(key_rope, -1), page_size = extent(cache, 1);
        const int pages = extent(table, 1), blocks = extent(cache, 0);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] {
            return (fp8 ? dscuda_mla_cache_append_fp8 : dscuda_mla_cache_append)(pointer(cache), pointer(latent), pointer(key_rope), int_pointer(&table),
                                                                                 int_pointer(start), int_pointer(counts), b, t, rank, rope, page_size,
                                                                                 pages, blocks, stream);
        });
        Py_INCREF(args[0]);
        return args[0];
    });
}

DSCUDA_FUNCTION(cache_append) {
    return append(args, count, false);
}

DSCUDA_FUNCTION(cache_append_fp8) {
    return append(args, count, true);
}

// paged_fp8_cache, paged_cache, first_row, rows -> paged_cache
DSCUDA_FUNCTION(cache_dequantize_fp8) {
    return guarded([&] {
        expect_arguments(count, 4);
        const Tensor& fp8 = tensor(args[0]);
        const long long first = integer(args[2]);
        if (fp8.dim() != 3) {
            fail(PyExc_ValueError, "the FP8 cache is a uint8 tensor [blocks, page, 656]");
        }
        const int64_t blocks = fp8.size(0), page = fp8.size(1);
        const long long rows = args[3] == Py_None ? blocks * page - first : integer(args[3]);
        int64_t elements = 0;
        if (first >= 0 && rows > 0) {                       // what is not is refused below
            if (first > blocks * page || rows > blocks * page - first || fp8.nbytes() < static_cast<size_t>(first + rows) * FP8_ROW_BYTES) {
                fail(PyExc_ValueError, "the rows do not lie inside the FP8 cache");
            }
            elements = (first + rows) * CACHE_WIDTH;
        }
        const Tensor* given = optional_output(args[1], fp8, at::kBFloat16, elements, "the cache");
        Tensor cache = given != nullptr ? *given : new_tensor({blocks, page, 1, CACHE_WIDTH}, fp8, at::kBFloat16);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] { return dscuda_mla_cache_dequantize_fp8(pointer(cache), pointer(fp8), first, rows, stream); });
        return wrap(cache);
    });
}

// ---- rotary embedding ------------------------------------------------------------
// q_pe, k_pe, positions, theta -> q_pe, k_pe
DSCUDA_FUNCTION(rope_apply) {
    return guarded([&] {
        expect_arguments(count, 4);
        const Tensor *q_pe = optional_tensor(args[0]), *k_pe = optional_tensor(args[1]), *positions = optional_tensor(args[2]);
        const float theta = number(args[3]);
        const Tensor* anchor = q_pe != nullptr ? q_pe : k_pe;
        if (anchor == nullptr) {
            fail(PyExc_ValueError, "nothing to rotate");
        }
        const int heads = q_pe != nullptr ? extent(*q_pe, -2) : 1;
        const int width = extent(*anchor, -1);
        const long long rows = row_count(*anchor, anchor->size(-2) * anchor->size(-1));
        if (positions == nullptr && anchor->dim() != 4) {
            fail(PyExc_ValueError, "packed tensors need explicit positions");
        }
        const int sequence = positions == nullptr ? extent(*anchor, 1) : 0;
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] {
            return dscuda_mla_rope_apply(pointer(q_pe), pointer(k_pe), int_pointer(positions), rows, heads, sequence, width, theta, stream);
        });
        return PyTuple_Pack(2, args[0], args[1]);
    });
}

// ---- projections -------------------------------------------------------------------
// kv_latent, w_uk, w_uv, heads -> k_nope, v
DSCUDA_FUNCTION(up_project) {
    return guarded([&] {
        expect_arguments(count, 4);
        const Tensor &latent = tensor(args[0]), &w_uk = tensor(args[1]), &w_uv = tensor(args[2]);
        const int heads = static_cast<int>(integer(args[3]));
        const long long rows = row_count(latent, latent.size(-1));          // size() refuses a tensor without dimensions
        at::DimVector sizes(latent.sizes().begin(), latent.sizes().end() - 1);
        sizes.push_back(heads);
        sizes.push_back(128);
        Tensor k_nope = new_tensor(sizes, latent, at::kBFloat16), v = new_tensor(sizes, latent, at::kBFloat16);
        void* stream = current_stream();
        checked(dscuda_mla_last_error,
                [&] { return dscuda_mla_up_project(pointer(k_nope), pointer(v), pointer(latent), pointer(w_uk), pointer(w_uv), rows, heads, stream); });
        return tuple(k_nope, v);
    });
}

// x [..., H, k], weight -> [..., H, columns]
template <class Call>
PyObject* per_head_projection(PyObject* const* args, Py_ssize_t count, int64_t columns, Call call) {
    return guarded([&] {
        expect_arguments(count, 2);
        const Tensor &x = tensor(args[0]), &weight = tensor(args[1]);
        const int heads = extent(x, -2);
        const long long rows = row_count(x, x.size(-2) * x.size(-1));
        at::DimVector sizes(x.sizes().begin(), x.sizes().end() - 1);
        sizes.push_back(columns);
        Tensor output = new_tensor(sizes, x, at::kBFloat16);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] { return call(pointer(output), pointer(x), pointer(weight), rows, heads, stream); });
        return wrap(output);
    });
}

DSCUDA_FUNCTION(absorb_query) {
    return per_head_projection(args, count, LATENT, dscuda_mla_absorb_query);
}

DSCUDA_FUNCTION(unabsorb_output) {
    return per_head_projection(args, count, 128, dscuda_mla_unabsorb_output);
}

// ---- non-absorbed forward and backward ---------------------------------------------
struct PrefillShape {
    int batch, longest, total, heads;
};

PrefillShape prefill_shape(const Tensor& q_nope, const Tensor* cu_seqlens, PyObject* max_seqlen) {
    if (cu_seqlens == nullptr) {
        expect_dims(q_nope, 4);
        return {extent(q_nope, 0), extent(q_nope, 1), static_cast<int>(q_nope.size(0) * q_nope.size(1)), extent(q_nope, 2)};
    }
    if (max_seqlen == Py_None) {
        fail(PyExc_ValueError, "packed layout needs max_seqlen (an upper bound on the longest sequence)");
    }
    THPObjectPtr longest(PyNumber_Long(max_seqlen));      // int(max_seqlen): a float or a one-element tensor will do
    if (!longest) {
        throw python_error();
    }
    expect_dims(q_nope, 3);
    return {static_cast<int>(cu_seqlens->numel() - 1), static_cast<int>(integer(longest.get())), extent(q_nope, 0), extent(q_nope, 1)};
}

// q_nope, q_pe, k_nope, k_pe, v, scale, cu_seqlens, max_seqlen, output, lse -> output, lse
DSCUDA_FUNCTION(prefill_forward) {
    return guarded([&] {
        expect_arguments(count, 10);
        const Tensor &q_nope = tensor(args[0]), &q_pe = tensor(args[1]), &k_nope = tensor(args[2]), &k_pe = tensor(args[3]), &v = tensor(args[4]);
        const float scale = number(args[5]);
        const Tensor* cu = optional_tensor(args[6]);
        const PrefillShape n = prefill_shape(q_nope, cu, args[7]);
        const int64_t rows = static_cast<int64_t>(n.total) * n.heads;
        const Tensor *output_given = optional_output(args[8], v, at::kBFloat16, rows * VALUE, "the output"),
                     *lse_given = optional_output(args[9], v, at::kFloat, rows, "the LSE");
        Tensor output = output_given != nullptr ? *output_given : new_like(v);
        Tensor lse = lse_given != nullptr ? *lse_given
                     : cu == nullptr      ? new_tensor({n.batch, n.heads, n.longest}, v, at::kFloat)
                                          : new_tensor({n.heads, n.total}, v, at::kFloat);
        const int nope = extent(q_nope, -1), rope = extent(q_pe, -1), value = extent(v, -1);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] {
            return dscuda_mla_prefill_forward(pointer(output), static_cast<float*>(pointer(lse)), pointer(q_nope), pointer(q_pe), pointer(k_nope),
                                              pointer(k_pe), pointer(v), int_pointer(cu), n.batch, n.longest, n.total, n.heads, nope, rope, value, scale,
                                              stream);
        });
        return tuple(output, lse);
    });
}

// dout, output, lse, q_nope, q_pe, k_nope, k_pe, v, scale, cu_seqlens, max_seqlen, workspace, grads -> dq, dk_nope, dk_pe, dv
DSCUDA_FUNCTION(prefill_backward) {
    return guarded([&]() -> PyObject* {
        expect_arguments(count, 13);
        const Tensor &dout = tensor(args[0]), &output = tensor(args[1]), &lse = tensor(args[2]), &q_nope = tensor(args[3]), &q_pe = tensor(args[4]),
                     &k_nope = tensor(args[5]), &k_pe = tensor(args[6]), &v = tensor(args[7]);
        const float scale = number(args[8]);
        const Tensor* cu = optional_tensor(args[9]);
        const PrefillShape n = prefill_shape(q_nope, cu, args[10]);
        const size_t workspace_bytes = dscuda_mla_prefill_backward_workspace_bytes(n.batch, n.longest, n.total, n.heads);
        const Tensor* workspace_given = optional_workspace(args[11], v, workspace_bytes);
        Tensor grads[4];
        if (args[12] == Py_None) {
            at::DimVector sizes(q_nope.sizes().begin(), q_nope.sizes().end() - 1);
            sizes.push_back(192);
            grads[0] = new_tensor(sizes, v, at::kBFloat16);
            grads[1] = new_like(k_nope);
            grads[2] = new_like(k_pe);
            grads[3] = new_like(v);
        } else {
            PyObject* items = PySequence_Fast(args[12], "grads is a sequence of four tensors");
            if (items == nullptr) {
                throw python_error();
            }
            const THPObjectPtr holder(items);
            if (PySequence_Fast_GET_SIZE(items) != 4) {
                fail(PyExc_ValueError, "grads is a sequence of four tensors");
            }
            const int64_t total = n.total, rows = total * n.heads;
            const int64_t elements[4] = {rows * 192, rows * VALUE, total * 64, rows * VALUE};
            const char* names[4] = {"dq", "dk_nope", "dk_pe", "dv"};
            for (int i = 0; i < 4; ++i) {
                const Tensor* grad = optional_output(PySequence_Fast_GET_ITEM(items, i), v, at::kBFloat16, elements[i], names[i]);
                if (grad == nullptr) {
                    fail(PyExc_TypeError, "grads is a sequence of four tensors");
                }
                grads[i] = *grad;
            }
        }
        Tensor workspace = workspace_given != nullptr ? *workspace_given : new_tensor({static_cast<int64_t>(workspace_bytes)}, v, at::kByte);
        const int nope = extent(q_nope, -1), rope = extent(q_pe, -1), value = extent(v, -1);
        void* stream = current_stream();
        checked(dscuda_mla_last_error, [&] {
            return dscuda_mla_prefill_backward_sized(pointer(grads[0]), pointer(grads[1]), pointer(grads[2]), pointer(grads[3]), pointer(dout),
                                                     pointer(output), static_cast<const float*>(pointer(lse)), pointer(q_nope), pointer(q_pe),
                                                     pointer(k_nope), pointer(k_pe), pointer(v), int_pointer(cu), pointer(workspace),
                                                     workspace.nbytes(), n.batch, n.longest, n.total, n.heads, nope, rope, value, scale, stream);
        });
        if (args[12] != Py_None) {
            Py_INCREF(args[12]);
            return args[12];
        }
        return tuple(grads[0], grads[1], grads[2], grads[3]);
    });
}

// query, key, value, scale -> output, lse
DSCUDA_FUNCTION(flash_forward) {
    return guarded([&] {
        expect_arguments(count, 4);
        const Tensor &query = tensor(args[0], 4), &key = tensor(args[1]), &value = tensor(args[2]);
        const float scale = number(args[3]);
        const int b = extent(query, 0), t = extent(query, 1), hq = extent(query, 2), d = extent(query, 3), hkv = extent(key, 2);
        Tensor output = new_like(query);
        Tensor lse = new_tensor({b, hq, t}, query, at::kFloat);
        void* stream = current_stream();
        checked(dscuda_flash_last_error, [&] {
            return dscuda_flash_forward(pointer(output), static_cast<float*>(pointer(lse)), pointer(query), pointer(key), pointer(value), b, t, hq, hkv, d,
                                        scale, stream);
        });
        return tuple(output, lse);
    });
}

#define DSCUDA_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    DSCUDA_METHOD(mla_forward),      DSCUDA_METHOD(mla_backward),     DSCUDA_METHOD(mla_decode),           DSCUDA_METHOD(cache_append),
    DSCUDA_METHOD(cache_append_fp8), DSCUDA_METHOD(rope_apply),       DSCUDA_METHOD(cache_dequantize_fp8), DSCUDA_METHOD(up_project),
    DSCUDA_METHOD(absorb_query),     DSCUDA_METHOD(unabsorb_output),  DSCUDA_METHOD(prefill_forward),      DSCUDA_METHOD(prefill_backward),
    DSCUDA_METHOD(flash_forward),    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_dscuda_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dscuda_torch() {
    // The extension is compiled against one Python and one torch; library.py compares the latter.
    static const std::string python = std::to_string(PY_MAJOR_VERSION) + "." + std::to_string(PY_MINOR_VERSION) + ".";
    if (std::string(Py_GetVersion()).compare(0, python.size(), python) != 0) {
        PyErr_SetString(PyExc_ImportError, ("built for Python " + python + "x").c_str());
        return nullptr;
    }
    PyObject* result = PyModule_Create(&module);
    if (result != nullptr && PyModule_AddStringConstant(result, "torch_version", TORCH_VERSION) != 0) {
        Py_DECREF(result);
        return nullptr;
    }
    return result;
}

// Python wrappers of the short operations, compiled: argument checks, output allocation through torch's allocator, the
// current stream and one call of the native library.
//
// A pass over a small tensor is bound by its host side.  The same steps as Python statements with ctypes took 15.4 us for the
// cross-entropy (two launches among it), 13.2 and 20.4 us for the short attention's two directions, whose kernels run for
// 5 to 8 us.  Each function here keeps the checks, results and error messages of the Python statements that it replaces;
// defaults and option names stay in ops/__init__.py.
//
// The library's entry points arrive as addresses (bind), so this module links to torch only and always calls the library
// that ops/__init__.py has loaded.  The GIL is released around the native calls, as ctypes does.
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "attention_desc.h"
#include "gemm_desc.h"

#include <cmath>
#include <cstring>

namespace {

PyObject* native_error = nullptr;          // ops.NativeError

enum { F32 = 0, BF16 = 1 };

struct Native {
    const char* (*cme_last_error)();
    int (*cme_cross_entropy)(int, const void*, const int*, void*, float*, float*, int, int, long long, float, float, float, int,
                             void*);
    int (*cme_attention_fwd)(const CmeAttn*, int, void*);
    int (*cme_attention_bwd)(const CmeAttn*, int, void*);
    int (*cme_attention_path)(const CmeAttn*, int, int);
    long long (*cme_attention_gemm_ws_bytes)(int, int);
    int (*cme_layernorm_fwd)(int, const void*, const void*, void*, const void*, const void*, void*, float*, float*, int, int,
                             float, void*);
    int (*cme_layernorm_bwd_blocks)(int);
    int (*cme_layernorm_bwd)(int, const void*, const void*, const void*, const float*, const float*, const void*, void*, void*,
                             void*, float*, int, int, int, void*);
    int (*cme_bias_act_residual)(int, const void*, const void*, const void*, void*, void*, long long, int, int, void*);
    int (*cme_colsum_splits)(int, int);
    int (*cme_dact_colsum)(int, const void*, const void*, void*, void*, float*, int, int, int, int, void*);
    int (*cme_embedding_fwd)(int, const int*, const void*, const void*, void*, int, int, int, int, void*);
    int (*cme_embedding_bwd)(int, const int*, const void*, void*, void*, int, int, int, int, int, void*);
} lib;

// ---------------------------------------------------------------------------------------------------------------------
// Arguments and results.  Errors travel as C++ exceptions to the macros around each function.
// ---------------------------------------------------------------------------------------------------------------------
[[noreturn]] void fail(PyObject* type, const std::string& what) {
    PyErr_SetString(type, what.c_str());
    throw python_error();
}

// A CUDA tensor whose elements are contiguous; undefined for None where that is allowed.
at::Tensor tensor(PyObject* o, bool optional = false) {
    if (optional && o == Py_None) return at::Tensor();
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "native ops take tensors");
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.is_contiguous()) fail(native_error, "native ops need contiguous CUDA tensors");
    return t;
}
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

int dtype(const at::Tensor& t) {
    if (t.scalar_type() == at::kFloat) return F32;
    if (t.scalar_type() == at::kBFloat16) return BF16;
    PyObject* s = PyObject_Str(reinterpret_cast<PyObject*>(torch::getTHPDtype(t.scalar_type())));
    const char* name = s ? PyUnicode_AsUTF8(s) : nullptr;
    const std::string what = std::string("unsupported dtype ") + (name ? name : "?");
    Py_XDECREF(s);
    fail(native_error, what);
}
long long whole(PyObject* o) {
    PyObject* i = PyNumber_Index(o);
    if (!i) throw python_error();
    const long long v = PyLong_AsLongLong(i);
    Py_DECREF(i);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
// What the C entry points take as int; sizes beyond it are an error instead of another number.
int int32(long long v) {
    if (v < INT32_MIN || v > INT32_MAX) fail(native_error, "native ops: a size exceeds 32 bits");
    return (int)v;
}
float real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return (float)v;
}
bool truth(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v != 0;
}
at::Tensor like(const at::Tensor& t) { return at::empty(t.sizes(), t.options()); }
at::Tensor floats(long long n, const at::Tensor& t) { return at::empty({n}, t.options().dtype(at::kFloat)); }

PyObject* wrap(const at::Tensor& t) {
    if (!t.defined()) Py_RETURN_NONE;
    PyObject* o = THPVariable_Wrap(t);
    if (!o) throw python_error();
    return o;
}
template <typename... Ts> PyObject* pack(const Ts&... ts) {
    PyObject* out = PyTuple_New(sizeof...(ts));
    if (!out) throw python_error();
    Py_ssize_t i = 0;
    auto put = [&](const at::Tensor& t) {
        PyObject* o = t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None);
        if (!o) { Py_DECREF(out); throw python_error(); }
        PyTuple_SET_ITEM(out, i++, o);
    };
    (put(ts), ...);
    return out;
}

void check(int rc) {
    if (rc == 0) return;
    const char* what = lib.cme_last_error();
    fail(native_error, "native call failed (status " + std::to_string(rc) + "): " + (what ? what : ""));
}
// One native call on the current stream, without the GIL.
template <typename F> void run(F&& call) {
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = call(stream);
    Py_END_ALLOW_THREADS
    check(rc);
}
// Rows and length of the last dimension.
void rows_of(const at::Tensor& t, int& rows, int& cols) {
    if (t.dim() == 0) fail(PyExc_IndexError, "native ops: a tensor without dimensions");
    if (t.size(-1) == 0) fail(PyExc_ZeroDivisionError, "native ops: rows without elements");
    cols = int32(t.size(-1));
    rows = int32(t.numel() / t.size(-1));
}

// ---------------------------------------------------------------------------------------------------------------------
// The operations
// ---------------------------------------------------------------------------------------------------------------------
// (logits, targets, grad_scale | None, prob_eps, inplace)
PyObject* cross_entropy(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor logits = tensor(a[0]), targets = tensor(a[1]);
    if (logits.dim() != 2) fail(PyExc_ValueError, "cross_entropy: logits have to be [rows, classes]");
    const int rows = int32(logits.size(0)), V = int32(logits.size(1)), dt = dtype(logits);
    const float eps = real(a[3]);
    if (a[2] == Py_None && rows == 0) fail(PyExc_ZeroDivisionError, "cross_entropy: no rows");
    const float scale = a[2] == Py_None ? (float)(1.0 / rows) : real(a[2]);
    const at::Tensor grad = truth(a[4]) ? logits : like(logits), losses = floats(rows, logits), loss = floats(1, logits);
    run([&](void* st) {
        return lib.cme_cross_entropy(dt, ptr(logits), (const int*)ptr(targets), ptr(grad), (float*)ptr(losses), (float*)ptr(loss),
                                     rows, V, V, scale, eps, 1.f, 0, st);
    });
    return pack(loss, grad, losses);
    END_HANDLE_TH_ERRORS
}

// The layout of q, [B*T, D], as the native library takes it; `ws` receives the scratch where the batched-product path runs.
struct Attention {
    CmeAttn d;
    long long B, H, T;
    int backend;
    bool offers_ws;
    at::Tensor ws;

    Attention(const at::Tensor& q, PyObject* const* a) {          // a: B, H, T, flat, causal, backend
        B = whole(a[0]); H = whole(a[1]); T = whole(a[2]);
        const bool flat = truth(a[3]);
        if (q.dim() == 0) fail(PyExc_IndexError, "attention: a tensor without dimensions");
        if (H == 0) fail(PyExc_ZeroDivisionError, "attention: no heads");
        const long long D = q.size(-1), HD = D / H;
        if (HD == 0) fail(PyExc_ZeroDivisionError, "attention: heads without elements");
        std::memset(&d, 0, sizeof d);
        d.nb = int32(flat ? B * H : B);
        d.nh = int32(flat ? 1 : H);
        d.T = int32(T);
        d.HD = int32(HD);
        d.sb = flat ? T * HD : T * D;
        d.sh = flat ? 0 : HD;
        d.st = flat ? HD : D;
        d.osb = d.sb; d.osh = d.sh; d.ost = d.st;
        d.causal = truth(a[4]);
        d.scale = (float)(1.0 / std::sqrt((double)HD));
        d.dtype = dtype(q);
        backend = int32(whole(a[5]));
        offers_ws = flat && T <= 512 && d.dtype == BF16;
    }
    // Which kernels the call takes (see cme_attention_path); the batched products get their scratch.
    int path(int bwd, const at::Tensor& q) {
        if (offers_ws) {
            d.ws_bytes = lib.cme_attention_gemm_ws_bytes(int32(B * H), (int)T);
            d.ws = reinterpret_cast<void*>(256);                  // stands for aligned scratch where the path is chosen
        }
        const int p = lib.cme_attention_path(&d, backend, bwd);
        if (p == CME_ATTN_PATH_GEMM) {
            ws = at::empty({d.ws_bytes + 256}, q.options().dtype(at::kByte));
            d.ws = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(ws.data_ptr()) + 255) / 256 * 256);
        }
        return p;                                                 // (no other path touches it)
    }
};

// (q, k, v, B, H, T, flat, causal, backend)
PyObject* attention_fwd(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]);
    Attention at(q, a + 3);
    const at::Tensor out = like(q), lse = floats(at.B * at.H * at.T, q);
    at.d.q = ptr(q); at.d.k = ptr(k); at.d.v = ptr(v); at.d.o = ptr(out);
    at.d.lse = (float*)ptr(lse);
    at.path(0, q);
    run([&](void* st) { return lib.cme_attention_fwd(&at.d, at.backend, st); });
    return pack(out, lse);
    END_HANDLE_TH_ERRORS
}

// (q, k, v, out, lse, dout, B, H, T, flat, causal, backend, dq_mode, scratch accumulator | None, scratch counters | None)
PyObject* attention_bwd(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), out = tensor(a[3]), lse = tensor(a[4]), dout = tensor(a[5]);
    Attention at(q, a + 6);
    const int mode = int32(whole(a[12]));
    const at::Tensor dq = like(q), dk = like(k), dv = like(v), delta = like(lse);
    at.d.q = ptr(q); at.d.k = ptr(k); at.d.v = ptr(v); at.d.o = ptr(out);
    at.d.lse = (float*)ptr(lse);
    at.d.d_o = ptr(dout); at.d.dq = ptr(dq); at.d.dk = ptr(dk); at.d.dv = ptr(dv);
    at.d.delta = (float*)ptr(delta);
    at.d.dq_mode = mode;
    const int path = at.path(1, q);
    at::Tensor acc, sem;
    if (a[13] != Py_None) {
        if (!THPVariable_Check(a[13]) || !THPVariable_Check(a[14])) fail(PyExc_TypeError, "native ops take tensors");
        acc = THPVariable_Unpack(a[13]);
        sem = THPVariable_Unpack(a[14]);
    } else if (path == CME_ATTN_PATH_TC) {
        // mode 0 clears the scratch itself and counts nothing; the other modes start from zeros
        const auto f = q.options().dtype(at::kFloat), i = q.options().dtype(at::kInt);
        acc = mode ? at::zeros({q.numel()}, f) : at::empty({q.numel()}, f);
        if (mode) sem = at::zeros({at.B * at.H * ((at.T + 127) / 128)}, i);
    } else {
        acc = sem = delta;                 // checked for presence and alignment, touched by none of the other paths
    }
    at.d.dq_accum = (float*)ptr(acc);
    at.d.dq_sem = (int*)ptr(sem);
    run([&](void* st) { return lib.cme_attention_bwd(&at.d, at.backend, st); });
    return pack(dq, dk, dv);
    END_HANDLE_TH_ERRORS
}

// (x, gamma, beta, eps, residual | None, save_sum)
PyObject* layernorm_fwd(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor x = tensor(a[0]), gamma = tensor(a[1]), beta = tensor(a[2]), res = tensor(a[4], true);
    int rows, D;
    rows_of(x, rows, D);
    const int dt = dtype(x);
    const float eps = real(a[3]);
    const at::Tensor y = like(x), mean = floats(rows, x), rstd = floats(rows, x);
    const at::Tensor sum = truth(a[5]) && res.defined() ? like(x) : at::Tensor();
    run([&](void* st) {
        return lib.cme_layernorm_fwd(dt, ptr(x), ptr(res), ptr(sum), ptr(gamma), ptr(beta), ptr(y), (float*)ptr(mean),
                                     (float*)ptr(rstd), rows, D, eps, st);
    });
    return pack(y, mean, rstd, sum);
    END_HANDLE_TH_ERRORS
}

// (dy, x, gamma, mean, rstd, dres | None, dgamma | None, dbeta | None, accumulate)
PyObject* layernorm_bwd(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor dy = tensor(a[0]), x = tensor(a[1]), gamma = tensor(a[2]), mean = tensor(a[3]), rstd = tensor(a[4]),
                     dres = tensor(a[5], true);
    at::Tensor dgamma = tensor(a[6], true), dbeta = tensor(a[7], true);
    int rows, D;
    rows_of(x, rows, D);
    const int dt = dtype(x);
    bool accumulate = truth(a[8]);
    const at::Tensor dx = like(x);
    if (!dgamma.defined()) { dgamma = like(gamma); dbeta = like(gamma); accumulate = false; }
    const at::Tensor scratch = floats((long long)lib.cme_layernorm_bwd_blocks(rows) * 2 * D, x);
    run([&](void* st) {
        return lib.cme_layernorm_bwd(dt, ptr(dy), ptr(x), ptr(gamma), (const float*)ptr(mean), (const float*)ptr(rstd), ptr(dres),
                                     ptr(dx), ptr(dgamma), ptr(dbeta), (float*)ptr(scratch), rows, D, accumulate, st);
    });
    return pack(dx, dgamma, dbeta);
    END_HANDLE_TH_ERRORS
}

// (x, bias | None, activation, residual | None, save_pre)
PyObject* bias_act_residual(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor x = tensor(a[0]), bias = tensor(a[1], true), res = tensor(a[3], true);
    const int act = int32(whole(a[2])), dt = dtype(x);
    int rows, cols;
    rows_of(x, rows, cols);
    const at::Tensor out = like(x), pre = truth(a[4]) ? like(x) : at::Tensor();
    run([&](void* st) {
        return lib.cme_bias_act_residual(dt, ptr(x), ptr(bias), ptr(res), ptr(pre), ptr(out), rows, cols, act, st);
    });
    return pack(out, pre);
    END_HANDLE_TH_ERRORS
}

// (dout, pre | None, activation, want_g, dbias | None, accumulate)
PyObject* dact_colsum(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor dout = tensor(a[0]), pre = tensor(a[1], true);
    at::Tensor dbias = tensor(a[4], true);
    const int act = int32(whole(a[2])), dt = dtype(dout);
    bool accumulate = truth(a[5]);
    int rows, cols;
    rows_of(dout, rows, cols);
    const at::Tensor g = truth(a[3]) && pre.defined() ? like(dout) : at::Tensor();
    if (!dbias.defined()) { dbias = at::empty({cols}, dout.options()); accumulate = false; }
    const at::Tensor scratch = floats((long long)lib.cme_colsum_splits(rows, cols) * cols, dout);
    run([&](void* st) {
        return lib.cme_dact_colsum(dt, ptr(dout), ptr(pre), ptr(g), ptr(dbias), (float*)ptr(scratch), rows, cols, act, accumulate,
                                   st);
    });
    return pack(g, dbias);
    END_HANDLE_TH_ERRORS
}

// (tokens, tok, pos)
PyObject* embedding_fwd(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor tokens = tensor(a[0]), tok = tensor(a[1]), pos = tensor(a[2]);
    if (tok.dim() != 2 || pos.dim() == 0) fail(PyExc_ValueError, "embedding: tables have to be [rows, columns]");
    const int BT = int32(tokens.numel()), V = int32(tok.size(0)), D = int32(tok.size(1)), T = int32(pos.size(0)), dt = dtype(tok);
    const at::Tensor out = at::empty({BT, D}, tok.options());
    run([&](void* st) {
        return lib.cme_embedding_fwd(dt, (const int*)ptr(tokens), ptr(tok), ptr(pos), ptr(out), BT, T, D, V, st);
    });
    return wrap(out);
    END_HANDLE_TH_ERRORS
}

// (tokens, dout, V, T, dtok | None, dpos | None, accumulate)
PyObject* embedding_bwd(PyObject*, PyObject* const* a, Py_ssize_t) {
    HANDLE_TH_ERRORS
    const at::Tensor tokens = tensor(a[0]), dout = tensor(a[1]);
    const long long V = whole(a[2]), T = whole(a[3]);
    at::Tensor dtok = tensor(a[4], true), dpos = tensor(a[5], true);
    bool accumulate = truth(a[6]);
    if (dout.dim() != 2) fail(PyExc_ValueError, "embedding: gradients have to be [tokens, columns]");
    const int BT = int32(dout.size(0)), D = int32(dout.size(1)), dt = dtype(dout);
    if (!dtok.defined()) {
        dtok = at::empty({V, D}, dout.options());
        dpos = at::empty({T, D}, dout.options());
        accumulate = false;
    }
    run([&](void* st) {
        return lib.cme_embedding_bwd(dt, (const int*)ptr(tokens), ptr(dout), ptr(dtok), ptr(dpos), BT, int32(T), D, int32(V),
                                     accumulate, st);
    });
    return pack(dtok, dpos);
    END_HANDLE_TH_ERRORS
}

// The steps of ops.gemm before its native call: shapes, the result, column sums and the descriptor, 5 of the 18 us that the call
// took as Python statements.  Returns (out, column sums | None, descriptor in a bytearray, behind which lies the count that
// colsum_slabs points to).
// (a, b, a_trans, b_trans, out | None, out_dtype | None, bias | None, activation, aux_out | None, dact, aux_in | None, residual | None,
//  accumulate, force_bn, force_splits, aux_deriv, dbias | None, allow_tf32, scratch | None)
PyObject* gemm_prepare(PyObject*, PyObject* const* o, Py_ssize_t) {
    HANDLE_TH_ERRORS
    auto any = [](PyObject* t) {
        if (t == Py_None) return at::Tensor();
        if (!THPVariable_Check(t)) fail(PyExc_TypeError, "native ops take tensors");
        return THPVariable_Unpack(t);
    };
    auto number = [](PyObject* v) {                 // int(v)
        PyObject* i = PyNumber_Long(v);
        if (!i) throw python_error();
        const long long n = PyLong_AsLongLong(i);
        Py_DECREF(i);
        if (n == -1 && PyErr_Occurred()) throw python_error();
        return int32(n);
    };
    const at::Tensor a = any(o[0]), b = any(o[1]), bias = any(o[6]), aux_out = any(o[8]), aux_in = any(o[10]), res = any(o[11]),
                     ws = any(o[18]);
    if (!a.defined() || !b.defined()) fail(PyExc_TypeError, "native ops take tensors");
    at::Tensor out = any(o[4]);
    if (a.dim() < 2 || b.dim() < 2) fail(PyExc_IndexError, "gemm: operands have to be matrices");
    // a leading size of 1 is shared by the entries of the other operand, as a matrix is
    const bool a3 = a.dim() == 3, b3 = b.dim() == 3;
    const long long na = a3 ? a.size(0) : 1, nb = b3 ? b.size(0) : 1, batch = na == 1 ? nb : na;
    if (nb != 1 && nb != batch)
        fail(native_error, "gemm: operands of " + std::to_string(na) + " and " + std::to_string(nb) + " matrices");
    const long long a0 = a.size(-2), a1 = a.size(-1), b0 = b.size(-2), b1 = b.size(-1);
    CmeGemm g;
    std::memset(&g, 0, sizeof g);
    g.a_trans = number(o[2]);
    g.b_trans = number(o[3]);
    const long long M = g.a_trans ? a1 : a0, K = g.a_trans ? a0 : a1, Kb = g.b_trans ? b1 : b0, N = g.b_trans ? b0 : b1;
    if (K != Kb) fail(native_error, "gemm: inner dimensions differ (" + std::to_string(K) + " vs " + std::to_string(Kb) + ")");
    if (!out.defined()) {
        auto opt = a.options();
        if (o[5] != Py_None) {
            if (!THPDtype_Check(o[5])) fail(PyExc_TypeError, "gemm: out_dtype has to be a torch.dtype");
            opt = opt.dtype(reinterpret_cast<THPDtype*>(o[5])->scalar_type);
        }
        out = a3 || b3 ? at::empty({batch, M, N}, opt) : at::empty({M, N}, opt);
    }
    g.ab_dtype = dtype(a);
    g.c_dtype = dtype(out);
    g.act = number(o[7]); g.dact = number(o[9]);
    // the kernels take as many elements of these types as the descriptor says, whatever the tensors hold
    auto holds = [](const char* name, const at::Tensor& t, const at::Tensor& typed, const char* whose, long long count) {
        if (!t.defined()) return;
        if (t.scalar_type() != typed.scalar_type()) fail(native_error, std::string("gemm: ") + name + " has to have the type of " + whose);
        if (t.numel() < count)
            fail(native_error, std::string("gemm: ") + name + " has " + std::to_string(t.numel()) + " of " + std::to_string(count) +
                                   " elements");
    };
    const long long elements = batch * M * N;
    holds("b", b, a, "a", 0);
    holds("out", out, out, "out", elements);
    holds("bias", bias, a, "a", N);
    holds("residual", res, out, "out", elements);
    holds("aux_out", aux_out, out, "out", elements);
    if (g.dact && !aux_in.defined()) fail(native_error, "gemm: dact needs aux_in");
    if (g.dact) holds("aux_in", aux_in, out, "out", elements);
    at::Tensor part;
    if (const at::Tensor sums = any(o[16]); sums.defined()) {
        dtype(sums);                                // one of the two types
        holds("dbias", sums, sums, "dbias", N);
        part = at::empty({(M + 31) / 32 * N}, a.options().dtype(at::kFloat));
    }
    g.M = int32(M); g.N = int32(N); g.K = int32(K); g.batch = int32(batch);
    g.A = ptr(a); g.lda = a1; g.strideA = na == batch && a3 ? a0 * a1 : 0;
    g.B = ptr(b); g.ldb = b1; g.strideB = nb == batch && b3 ? b0 * b1 : 0;
    g.C = ptr(out); g.ldc = N; g.strideC = M * N;
    g.bias = ptr(bias);
    g.residual = ptr(res); g.ldres = N;
    g.aux_out = ptr(aux_out); g.aux_in = ptr(aux_in); g.ldaux = N;
    g.accumulate = number(o[12]);
    g.workspace = ptr(ws);
    g.workspace_bytes = ws.defined() ? ws.numel() * 4 : 0;
    g.force_bn = number(o[13]); g.force_splits = number(o[14]);
    g.aux_deriv = number(o[15]);
    g.allow_tf32 = number(o[17]);
    PyObject* desc = PyByteArray_FromStringAndSize(nullptr, sizeof g + sizeof(int));
    if (!desc) throw python_error();
    char* at_desc = PyByteArray_AS_STRING(desc);
    int* slabs = reinterpret_cast<int*>(at_desc + sizeof g);
    *slabs = 0;
    if (part.defined()) { g.colsum = (float*)ptr(part); g.colsum_slabs = slabs; }
    std::memcpy(at_desc, &g, sizeof g);
    PyObject* all = PyTuple_New(3);
    if (!all) { Py_DECREF(desc); throw python_error(); }
    PyTuple_SET_ITEM(all, 2, desc);
    Py_ssize_t i = 0;
    for (const at::Tensor* t : {static_cast<const at::Tensor*>(&out), static_cast<const at::Tensor*>(&part)}) {
        PyObject* v = t->defined() ? THPVariable_Wrap(*t) : Py_NewRef(Py_None);
        if (!v) { Py_DECREF(all); throw python_error(); }
        PyTuple_SET_ITEM(all, i++, v);
    }
    return all;
    END_HANDLE_TH_ERRORS
}

// (NativeError): for the functions that call no entry point
PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t) {
    Py_XSETREF(native_error, Py_NewRef(a[0]));
    Py_RETURN_NONE;
}

// (NativeError, {name: address}): what the functions above raise and call
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2 || !PyDict_Check(a[1])) fail(PyExc_TypeError, "bind(error class, {name: address})");
    Native next;
    auto get = [&](const char* name, auto& fn) {
        PyObject* v = PyDict_GetItemString(a[1], name);
        void* p = v ? PyLong_AsVoidPtr(v) : nullptr;
        if (!p) fail(PyExc_KeyError, name);
        std::memcpy(&fn, &p, sizeof p);
    };
#define GET(name) get(#name, next.name)
    GET(cme_last_error); GET(cme_cross_entropy); GET(cme_attention_fwd); GET(cme_attention_bwd); GET(cme_attention_path);
    GET(cme_attention_gemm_ws_bytes); GET(cme_layernorm_fwd); GET(cme_layernorm_bwd_blocks); GET(cme_layernorm_bwd);
    GET(cme_bias_act_residual); GET(cme_colsum_splits); GET(cme_dact_colsum); GET(cme_embedding_fwd); GET(cme_embedding_bwd);
#undef GET
    lib = next;
    Py_XSETREF(native_error, Py_NewRef(a[0]));
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

#define METHOD(name, nargs) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(counted<name, nargs>)), METH_FASTCALL, nullptr}
// Each function reads its arguments by position: another number of them is refused here.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t), int N>
PyObject* counted(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    if (n != N) return PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
    return F(self, a, n);
}
PyMethodDef methods[] = {METHOD(bind, 2), METHOD(init, 1), METHOD(gemm_prepare, 19), METHOD(cross_entropy, 5), METHOD(attention_fwd, 9), METHOD(attention_bwd, 15),
                         METHOD(layernorm_fwd, 6), METHOD(layernorm_bwd, 9), METHOD(bias_act_residual, 5), METHOD(dact_colsum, 6),
                         METHOD(embedding_fwd, 3), METHOD(embedding_bwd, 7), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_wrappers", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__wrappers() { return PyModule_Create(&module); }

// CPython binding of the C ABI for tensors that torch owns (tscale_b200/_native.so): what tscale_b200/ops.py and infer.py call
// for every entry point a step runs through.
//
// A call of the smallest sizes is bound by the host: building eight or more tsa_ptr2d records from tensor attributes in
// Python, passing them through ctypes by value and asking torch for the stream took 24 of the 30 us a 77-row forward spent on
// the host (the two kernel launches are the rest).  Here the tensors are read through torch's C++ objects (a few tens of
// nanoseconds each), result tensors are allocated in the same call and the library's entry point is called directly.
// The entry points are looked up in the already loaded shared library (bind), so whichever build of it abi.py selected is used.
// Errors: a status other than TSA_OK is returned as the first element and raised by the Python side; a tensor of a wrong shape
// raises AssertionError here, like ops.p2d.
#include <Python.h>
#include <dlfcn.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include "tsa.h"

namespace {

struct TEntries {
    decltype(&tsa_att_fwd) AttFwd;
    decltype(&tsa_att_fwd_workspace_bytes) AttFwdWs;
    decltype(&tsa_att_bwd) AttBwd;
    decltype(&tsa_att_bwd_workspace_bytes) AttBwdWs;
    decltype(&tsa_quant_rows) QuantRows;
    decltype(&tsa_norm_rope_quant) NormRopeQuant;
    decltype(&tsa_matmul_norm_rope_quant) MatmulNormRopeQuant;
    decltype(&tsa_rope_norm_bwd) RopeNormBwd;
    decltype(&tsa_kv_product) KvProduct;
    decltype(&tsa_kv_product_bwd) KvProductBwd;
    decltype(&tsa_calc_dscale) CalcDScale;
    decltype(&tsa_kv_append) KvAppend;
    decltype(&tsa_att_decode) AttDecode;
    decltype(&tsa_att_decode_static) AttDecodeStatic;
    decltype(&tsa_att_decode_workspace_bytes) AttDecodeWs;
    decltype(&tsa_infer_step) InferStep;
} g;

PyObject *g_outOfMemory; // torch.OutOfMemoryError

// thrown with the Python error already set
struct TPyError {};

void Need(bool ok, PyObject *kind, const char *text)
{
    if (!ok) {
        PyErr_SetString(kind, text);
        throw TPyError();
    }
}

const at::Tensor *Tensor(PyObject *o)
{
    if (o == Py_None) {
        return nullptr;
    }
    Need(THPVariable_Check(o), PyExc_TypeError, "expected a tensor or None");
    return &THPVariable_Unpack(o);
}

const at::Tensor &NeedTensor(PyObject *o)
{
    const at::Tensor *t = Tensor(o);
    Need(t != nullptr, PyExc_TypeError, "expected a tensor");
    return *t;
}

tsa_ptr2d P2D(const at::Tensor *t)
{
    tsa_ptr2d p = {nullptr, 0, 0, 0};
    if (t) {
        Need(t->dim() == 2 && t->stride(1) == 1, PyExc_AssertionError, "expected a row-major 2-D tensor");
        p.data = t->data_ptr();
        p.stride_bytes = (int)(t->stride(0) * (int64_t)t->element_size());
        p.xsize = (int)t->size(1);
        p.ysize = (int)t->size(0);
    }
    return p;
}
tsa_ptr2d P2D(PyObject *o) { return P2D(Tensor(o)); }
tsa_ptr2d P2D(const at::Tensor &t) { return P2D(&t); }

void *Ptr(PyObject *o)
{
    const at::Tensor *t = Tensor(o);
    return t ? t->data_ptr() : nullptr;
}

long Int(PyObject *o)
{
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) {
        throw TPyError();
    }
    return v;
}

float Float(PyObject *o)
{
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) {
        throw TPyError();
    }
    return (float)v;
}

// address of a ctypes structure or array (they export their storage as a buffer; it stays valid while the object lives)
template <class T>
T *Struct(PyObject *o)
{
    Py_buffer view;
    if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) {
        throw TPyError();
    }
    T *p = (T *)view.buf;
    const bool big = view.len >= (Py_ssize_t)sizeof(T);
    PyBuffer_Release(&view);
    Need(big, PyExc_TypeError, "ctypes structure of another type");
    return p;
}

tsa_stream_t Stream() { return (tsa_stream_t)c10::cuda::getCurrentCUDAStream().stream(); }

at::ScalarType TorchType(int dt)
{
    switch (dt) {
    case TSA_F16:
        return at::kHalf;
    case TSA_BF16:
        return at::kBFloat16;
    case TSA_F32:
        return at::kFloat;
    }
    return at::kByte;
}

int TsaType(const at::Tensor &t)
{
    switch (t.scalar_type()) {
    case at::kHalf:
        return TSA_F16;
    case at::kBFloat16:
        return TSA_BF16;
    case at::kFloat:
        return TSA_F32;
    default:
        break;
    }
    PyErr_SetString(PyExc_KeyError, "expected a float16, bfloat16 or float32 tensor");
    throw TPyError();
}

at::Tensor Empty(int64_t rows, int64_t cols, at::ScalarType type, const at::Tensor &like)
{
    return at::empty({rows, cols}, at::TensorOptions().dtype(type).device(like.device()));
}

at::Tensor EmptyBytes(size_t bytes, const at::Tensor &like)
{
    return at::empty({(int64_t)(bytes > 0 ? bytes : 1)}, at::TensorOptions().dtype(at::kByte).device(like.device()));
}

// the given tensor, or a new one
at::Tensor OrEmpty(PyObject *o, int64_t rows, int64_t cols, at::ScalarType type, const at::Tensor &like)
{
    const at::Tensor *t = Tensor(o);
    return t ? *t : Empty(rows, cols, type, like);
}

// (status, tensors...)
template <class... T>
PyObject *Result(int rc, const T &...tensors)
{
    PyObject *res = PyTuple_New(1 + sizeof...(T));
    if (!res) {
        throw TPyError();
    }
    PyTuple_SET_ITEM(res, 0, PyLong_FromLong(rc));
    Py_ssize_t i = 1;
    ((PyTuple_SET_ITEM(res, i, THPVariable_Wrap(tensors)), ++i), ...);
    return res;
}

// runs f without the interpreter lock, like a ctypes call
template <class F>
int Unlocked(F f)
{
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = f();
    Py_END_ALLOW_THREADS return rc;
}

template <Py_ssize_t N, class F>
PyObject *Guard(Py_ssize_t n, F f)
{
    try {
        Need(n == N, PyExc_TypeError, "wrong number of arguments");
        return f();
    } catch (const TPyError &) {
    } catch (const c10::OutOfMemoryError &e) {
        PyErr_SetString(g_outOfMemory, e.what_without_backtrace());
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

PyObject *Bind(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<1>(n, [&]() -> PyObject * {
        void *lib = PyLong_AsVoidPtr(a[0]);
        Need(lib != nullptr, PyExc_ValueError, "null library handle");
        auto get = [&](auto &fn, const char *name) {
            fn = (std::remove_reference_t<decltype(fn)>)dlsym(lib, name);
            Need(fn != nullptr, PyExc_ImportError, name);
        };
        PyObject *torch = PyImport_ImportModule("torch");
        Need(torch != nullptr, PyExc_ImportError, "torch");
        g_outOfMemory = PyObject_GetAttrString(torch, "OutOfMemoryError");
        Py_DECREF(torch);
        Need(g_outOfMemory != nullptr, PyExc_ImportError, "torch.OutOfMemoryError");
        get(g.AttFwd, "tsa_att_fwd");
        get(g.AttFwdWs, "tsa_att_fwd_workspace_bytes");
        get(g.AttBwd, "tsa_att_bwd");
        get(g.AttBwdWs, "tsa_att_bwd_workspace_bytes");
        get(g.QuantRows, "tsa_quant_rows");
        get(g.NormRopeQuant, "tsa_norm_rope_quant");
        get(g.MatmulNormRopeQuant, "tsa_matmul_norm_rope_quant");
        get(g.RopeNormBwd, "tsa_rope_norm_bwd");
        get(g.KvProduct, "tsa_kv_product");
        get(g.KvProductBwd, "tsa_kv_product_bwd");
        get(g.CalcDScale, "tsa_calc_dscale");
        get(g.KvAppend, "tsa_kv_append");
        get(g.AttDecode, "tsa_att_decode");
        get(g.AttDecodeStatic, "tsa_att_decode_static");
        get(g.AttDecodeWs, "tsa_att_decode_workspace_bytes");
        get(g.InferStep, "tsa_infer_step");
        Py_RETURN_NONE;
    });
}

// cfg, globalScale, qk, qv, v, qkScale, qvScale, vScale, groups, groupPtr, slope, out, lse, heads, lenAttTiles, workspace, status
PyObject *AttFwd(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<17>(n, [&] {
        const tsa_att_cfg *cfg = Struct<tsa_att_cfg>(a[0]);
        const at::Tensor &qk = NeedTensor(a[2]);
        const int heads = (int)Int(a[13]), rows = (int)qk.size(0);
        const at::Tensor out = OrEmpty(a[11], rows, (int64_t)heads * cfg->head_dim_v, TorchType(cfg->out_dtype), qk);
        const at::Tensor lse = OrEmpty(a[12], heads, rows, at::kFloat, qk);
        const at::Tensor *given = Tensor(a[15]);
        const at::Tensor ws = given ? *given : EmptyBytes(g.AttFwdWs(cfg, heads, rows), qk);
        const tsa_ptr2d q2 = P2D(qk), k2 = P2D(a[3]), v2 = P2D(a[4]), qs = P2D(a[5]), ks = P2D(a[6]), vs = P2D(a[7]), o2 = P2D(out), l2 = P2D(lse);
        const float *gs = (const float *)Ptr(a[1]);
        const tsa_span_group *groups = (const tsa_span_group *)Ptr(a[8]);
        const int *groupPtr = (const int *)Ptr(a[9]);
        const float slope = Float(a[10]);
        const int tiles = (int)Int(a[14]);
        int *status = (int *)Ptr(a[16]);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] {
            return g.AttFwd(cfg, gs, q2, k2, qs, ks, v2, vs, groups, groupPtr, slope, o2, l2, heads, tiles, ws.data_ptr(), (size_t)ws.numel(), status, stream);
        });
        return Result(rc, out, lse);
    });
}

// cfg, globalScale, qk, qv, v, qkScale, qvScale, vScale, dOut, out, dScale, lse, groups, groupPtr, revGroups, revGroupPtr, slope,
// gradMult, heads, lenAttTiles, workspace, status
PyObject *AttBwd(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<22>(n, [&] {
        const tsa_att_cfg *cfg = Struct<tsa_att_cfg>(a[0]);
        const at::Tensor &qk = NeedTensor(a[2]);
        const int heads = (int)Int(a[18]), rows = (int)qk.size(0);
        const at::ScalarType gt = TorchType(cfg->grad_dtype);
        const at::Tensor dq = Empty(rows, (int64_t)heads * cfg->head_dim_qk, gt, qk), dk = Empty(rows, (int64_t)heads * cfg->head_dim_qk, gt, qk);
        const at::Tensor dv = Empty(rows, (int64_t)heads * cfg->head_dim_v, gt, qk);
        const at::Tensor *given = Tensor(a[20]);
        const at::Tensor ws = given ? *given : EmptyBytes(g.AttBwdWs(cfg, heads, rows), qk);
        const tsa_ptr2d q2 = P2D(qk), k2 = P2D(a[3]), v2 = P2D(a[4]), qs = P2D(a[5]), ks = P2D(a[6]), vs = P2D(a[7]);
        const tsa_ptr2d dO = P2D(a[8]), o2 = P2D(a[9]), ds = P2D(a[10]), l2 = P2D(a[11]), dq2 = P2D(dq), dk2 = P2D(dk), dv2 = P2D(dv);
        const float *gs = (const float *)Ptr(a[1]);
        const tsa_span_group *groups = (const tsa_span_group *)Ptr(a[12]), *rev = (const tsa_span_group *)Ptr(a[14]);
        const int *groupPtr = (const int *)Ptr(a[13]), *revPtr = (const int *)Ptr(a[15]);
        const float slope = Float(a[16]), mult = Float(a[17]);
        const int tiles = (int)Int(a[19]);
        int *status = (int *)Ptr(a[21]);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] {
            return g.AttBwd(cfg, gs, q2, k2, qs, ks, v2, vs, dO, o2, ds, l2, groups, groupPtr, rev, revPtr, slope, mult, dq2, dk2, dv2, heads, tiles,
                ws.data_ptr(), (size_t)ws.numel(), status, stream);
        });
        return Result(rc, dq, dk, dv);
    });
}

// kind, src, dstDtype, vecScale, length, tile
PyObject *QuantRows(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<6>(n, [&] {
        const at::Tensor &src = NeedTensor(a[1]);
        const tsa_ptr2d s2 = P2D(src);
        const int kind = (int)Int(a[0]), dst = (int)Int(a[2]), length = (int)Int(a[4]), tile = (int)Int(a[5]), st = TsaType(src);
        const float vec = Float(a[3]);
        const at::Tensor out = Empty(s2.ysize, s2.xsize, at::kByte, src), scale = Empty(tile > 0 ? s2.xsize / tile : 0, s2.ysize, at::kFloat, src);
        const tsa_ptr2d o2 = P2D(out), sc2 = P2D(scale);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] { return g.QuantRows(kind, st, dst, vec, s2, o2, sc2, length, tile, stream); });
        return Result(rc, out, scale);
    });
}

// src, rope, dstDtype, heads, headDim, vecScale, direction, length
PyObject *NormRopeQuant(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<8>(n, [&] {
        const at::Tensor &src = NeedTensor(a[0]);
        const at::Tensor *rope = Tensor(a[1]);
        const tsa_ptr2d s2 = P2D(src), r2 = P2D(rope);
        const int dst = (int)Int(a[2]), heads = (int)Int(a[3]), d = (int)Int(a[4]), length = (int)Int(a[7]), st = TsaType(src);
        const int rt = rope ? TsaType(*rope) : TSA_F32;
        const float vec = Float(a[5]), dir = Float(a[6]);
        const at::Tensor out = Empty(s2.ysize, (int64_t)heads * d, at::kByte, src), scale = Empty(heads, s2.ysize, at::kFloat, src);
        const tsa_ptr2d o2 = P2D(out), sc2 = P2D(scale);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] { return g.NormRopeQuant(st, dst, vec, s2, r2, rt, dir, o2, sc2, heads, d, length, stream); });
        return Result(rc, out, scale);
    });
}

// srcDtype, x, w, rope, dstDtype, heads, headDim, vecScale, srcScale, direction, length, status
PyObject *MatmulNormRopeQuant(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<12>(n, [&] {
        const at::Tensor &x = NeedTensor(a[1]);
        const tsa_ptr2d x2 = P2D(x), w2 = P2D(a[2]), r2 = P2D(a[3]);
        const int st = (int)Int(a[0]), dst = (int)Int(a[4]), heads = (int)Int(a[5]), d = (int)Int(a[6]), length = (int)Int(a[10]);
        const float vec = Float(a[7]), srcScale = Float(a[8]), dir = Float(a[9]);
        const at::Tensor out = Empty(x2.ysize, (int64_t)heads * d, TorchType(dst), x), scale = Empty(heads, x2.ysize, at::kFloat, x);
        const tsa_ptr2d o2 = P2D(out), sc2 = P2D(scale);
        int *status = (int *)Ptr(a[11]);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] { return g.MatmulNormRopeQuant(st, dst, vec, srcScale, x2, w2, r2, dir, o2, sc2, heads, d, length, status, stream); });
        return Result(rc, out, scale);
    });
}

// src, grad, rope, heads, headDim, direction
PyObject *RopeNormBwd(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<6>(n, [&] {
        const at::Tensor &src = NeedTensor(a[0]), &grad = NeedTensor(a[1]);
        const at::Tensor *rope = Tensor(a[2]);
        const at::Tensor out = at::empty_like(grad);
        const tsa_ptr2d s2 = P2D(src), g2 = P2D(grad), r2 = P2D(rope), o2 = P2D(out);
        const int heads = (int)Int(a[3]), d = (int)Int(a[4]), st = TsaType(src), gt = TsaType(grad), rt = rope ? TsaType(*rope) : TSA_F32;
        const float dir = Float(a[5]);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] { return g.RopeNormBwd(st, gt, s2, g2, r2, rt, dir, o2, heads, d, s2.ysize, stream); });
        return Result(rc, out);
    });
}

// k, val, heads, headDim, kvMult, outDtype, out
PyObject *KvProduct(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<7>(n, [&] {
        const at::Tensor &k = NeedTensor(a[0]);
        const int heads = (int)Int(a[2]), d = (int)Int(a[3]), ot = (int)Int(a[5]), st = TsaType(k);
        const float mult = Float(a[4]);
        const at::Tensor out = OrEmpty(a[6], k.size(0), (int64_t)heads * d * 4, TorchType(ot), k);
        const tsa_ptr2d k2 = P2D(k), v2 = P2D(a[1]), o2 = P2D(out);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] { return g.KvProduct(st, ot, k2, v2, mult, o2, heads, d, k2.ysize, stream); });
        return Result(rc, out);
    });
}

// k, val, dkv, heads, headDim
PyObject *KvProductBwd(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<5>(n, [&] {
        const at::Tensor &k = NeedTensor(a[0]), &dkv = NeedTensor(a[2]);
        const int heads = (int)Int(a[3]), d = (int)Int(a[4]), st = TsaType(k), gt = TsaType(dkv);
        const int64_t rows = k.size(0);
        const at::Tensor dk = Empty(rows, (int64_t)heads * d, dkv.scalar_type(), k), dv = Empty(rows, (int64_t)heads * d, dkv.scalar_type(), k);
        const at::Tensor ds = Empty(heads, rows, at::kFloat, k);
        const tsa_ptr2d k2 = P2D(k), v2 = P2D(a[1]), g2 = P2D(dkv), dk2 = P2D(dk), dv2 = P2D(dv), ds2 = P2D(ds);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] { return g.KvProductBwd(st, gt, k2, v2, g2, dk2, dv2, ds2, heads, d, (int)rows, stream); });
        return Result(rc, dk, dv, ds);
    });
}

// out, dOut, heads, headDimV
PyObject *CalcDScale(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<4>(n, [&] {
        const at::Tensor &out = NeedTensor(a[0]), &dOut = NeedTensor(a[1]);
        const int heads = (int)Int(a[2]), d = (int)Int(a[3]), ot = TsaType(out), gt = TsaType(dOut);
        const at::Tensor res = Empty(heads, out.size(0), at::kFloat, out);
        const tsa_ptr2d o2 = P2D(out), g2 = P2D(dOut), r2 = P2D(res);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] { return g.CalcDScale(ot, gt, o2, g2, r2, heads, d, o2.ysize, stream); });
        return Result(rc, res);
    });
}

// cfg, seqs, ctxLens, nSeq, capacity, kNew, kScaleNew, vNew, vScaleNew, heads, status
PyObject *KvAppend(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<11>(n, [&] {
        const tsa_decode_cfg *cfg = Struct<tsa_decode_cfg>(a[0]);
        const tsa_kv_seq *seqs = (const tsa_kv_seq *)Ptr(a[1]);
        int *lens = (int *)Ptr(a[2]), *status = (int *)Ptr(a[10]);
        const int nSeq = (int)Int(a[3]), capacity = (int)Int(a[4]), heads = (int)Int(a[9]);
        const tsa_ptr2d k2 = P2D(a[5]), ks = P2D(a[6]), v2 = P2D(a[7]), vs = P2D(a[8]);
        tsa_stream_t stream = Stream();
        return PyLong_FromLong(Unlocked([&] { return g.KvAppend(cfg, seqs, lens, nSeq, capacity, k2, ks, v2, vs, heads, status, stream); }));
    });
}

// cfg, nSeq, heads, maxCtx
PyObject *AttDecodeWorkspaceBytes(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<4>(n, [&] { return PyLong_FromSize_t(g.AttDecodeWs(Struct<tsa_decode_cfg>(a[0]), (int)Int(a[1]), (int)Int(a[2]), (int)Int(a[3]))); });
}

// cfg, seqs, ctxLens, nSeq, maxCtx, q, qScale, window, slope, out, heads, workspace (None: the library's static scratch), status
PyObject *AttDecode(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<13>(n, [&] {
        const tsa_decode_cfg *cfg = Struct<tsa_decode_cfg>(a[0]);
        const tsa_kv_seq *seqs = (const tsa_kv_seq *)Ptr(a[1]);
        const int *lens = (const int *)Ptr(a[2]);
        const at::Tensor &q = NeedTensor(a[5]);
        const int nSeq = (int)Int(a[3]), maxCtx = (int)Int(a[4]), window = (int)Int(a[7]), heads = (int)Int(a[10]);
        const float slope = Float(a[8]);
        const at::Tensor out = OrEmpty(a[9], nSeq, (int64_t)heads * cfg->head_dim, TorchType(cfg->out_dtype), q);
        const at::Tensor *ws = Tensor(a[11]);
        const tsa_ptr2d q2 = P2D(q), qs = P2D(a[6]), o2 = P2D(out);
        int *status = (int *)Ptr(a[12]);
        tsa_stream_t stream = Stream();
        const int rc = Unlocked([&] {
            return ws ? g.AttDecode(cfg, seqs, lens, nSeq, maxCtx, q2, qs, window, slope, o2, heads, ws->data_ptr(), (size_t)ws->numel(), status, stream)
                      : g.AttDecodeStatic(cfg, seqs, lens, nSeq, maxCtx, q2, qs, window, slope, o2, heads, status, stream);
        });
        return Result(rc, out);
    });
}

// model, layerSeqs, ctxLens, capacity, labels, labelsPerSeq, nSeq, maxCtx, prediction, logits, workspace, status
PyObject *InferStep(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return Guard<12>(n, [&] {
        const tsa_infer_model *model = Struct<tsa_infer_model>(a[0]);
        const tsa_kv_seq *const *layerSeqs = (const tsa_kv_seq *const *)Struct<void *>(a[1]);
        int *lens = (int *)Ptr(a[2]), *status = (int *)Ptr(a[11]);
        const int capacity = (int)Int(a[3]), labelsPerSeq = (int)Int(a[5]), nSeq = (int)Int(a[6]), maxCtx = (int)Int(a[7]);
        const int *labels = (const int *)Ptr(a[4]);
        float *prediction = (float *)Ptr(a[8]), *logits = (float *)Ptr(a[9]);
        const at::Tensor &ws = NeedTensor(a[10]);
        tsa_stream_t stream = Stream();
        return PyLong_FromLong(Unlocked([&] {
            return g.InferStep(model, layerSeqs, lens, capacity, labels, labelsPerSeq, nSeq, maxCtx, prediction, logits, ws.data_ptr(), (size_t)ws.numel(), status,
                stream);
        }));
    });
}

#define FAST(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST("bind", Bind), FAST("att_fwd", AttFwd), FAST("att_bwd", AttBwd), FAST("quant_rows", QuantRows),
    FAST("norm_rope_quant", NormRopeQuant), FAST("matmul_norm_rope_quant", MatmulNormRopeQuant), FAST("rope_norm_bwd", RopeNormBwd),
    FAST("kv_product", KvProduct), FAST("kv_product_bwd", KvProductBwd), FAST("calc_dscale", CalcDScale), FAST("kv_append", KvAppend),
    FAST("att_decode_workspace_bytes", AttDecodeWorkspaceBytes),
    FAST("att_decode", AttDecode), FAST("infer_step", InferStep), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "torch-tensor binding of libtsa_b200.so", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__native(void)
{
    return PyModule_Create(&g_module);
}

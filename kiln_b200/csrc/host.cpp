// Native host path of the Python entry points (kiln_b200/marlin_gemm.py, marlin_proj.py): argument checks, output and
// workspace allocation, device guard, stream lookup and the call through the C ABI of include/kiln_w4a16.h, in one
// extension call per GEMM.
//
// What bounded small calls before was this path in Python, not the GPU: at M = 1 a 2560 -> 512 projection runs 2.5 us on
// the GPU and took 19.6 us per call (attribute reads, torch.empty, two context managers and ctypes marshalling of eleven
// arguments).  The kernels of consecutive calls overlap, so a decode step made of eager calls runs at the host's pace.
//
// Each function takes the arguments as the Python entry point got them and returns
//   a tensor (or list / tuple of tensors)   done;
//   None    the arguments are not the plain case (wrong shape, dtype or device, a tensor that is not contiguous, a tensor
//           subclass, an empty problem ...): nothing was launched, the caller goes on with its Python path, which copies or
//           casts what has to be, and raises the reference's messages;
//   an int  the C ABI's status code, when it is not 0.
// The library is not linked: Python hands over the entry points of the copy that ctypes loaded (bind), so that the process
// holds one instance of it, KILN_W4A16_LIB included.
//
// Workspaces come from torch's caching allocator on every call and go back to it on return.  Reuse is ordered by the
// stream, so calls on several streams or threads never share one, a CUDA graph keeps its own, and none outlives its call.
// (0.3 us per call that needs one; a kept buffer per stream would have to be guarded against all three.)
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

#include "../../include/kiln_w4a16.h"

namespace {

using at::Tensor;

struct Abi {
    decltype(&kiln_w4a16_gemm_bf16) gemm;
    decltype(&kiln_w4a16_scratch_bytes) scratch;
    decltype(&kiln_w4a16_gemm_bf16_ex) gemm_ex;
    decltype(&kiln_w4a16_gemm_bf16_grouped) grouped;
    decltype(&kiln_w4a16_quantize_and_pack_device) pack;
    decltype(&kiln_w4a16_repack_gptq_device) gptq;
} abi;

PyObject *name_b, *name_s, *name_g, *name_k, *name_n;  // attribute names of MarlinPackedProj

// A plain contiguous CUDA tensor of the given type, or nullptr.
const Tensor *plain(PyObject *o, at::ScalarType type) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const Tensor &t = THPVariable_Unpack(o);
    return t.is_cuda() && t.scalar_type() == type && t.layout() == at::kStrided && t.is_contiguous() ? &t : nullptr;
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device &dev) {
    return Tensor(at::detail::empty_cuda(size, type, dev, std::nullopt));
}

// A packed projection whose tensors fit together and live on `dev`.  It owns them until the launch is enqueued: an attribute may be a
// property that makes them on each read (weights kept in host memory, say), or be assigned by another thread while the GIL is free, and
// memory that is given back before the launch is the next tensor's.
struct Proj {
    Tensor b, s;
    long k, n, groupsize;
};

bool weight_ok(Proj &p, const Tensor *b, const Tensor *s, const at::Device &dev) {
    if (!b || !s || b->dim() != 2 || s->dim() != 2 || b->device() != dev || s->device() != dev) return false;
    if (p.groupsize != -1 && p.groupsize != 128) return false;
    if (p.k <= 0 || p.n <= 0 || p.k % 128 || p.n % 256 || p.k > INT32_MAX || p.n > INT32_MAX / 2) return false;
    if (b->size(0) != p.k / 16 || b->size(1) != 2 * p.n) return false;
    if (s->size(0) != (p.groupsize == -1 ? 1 : p.k / 128) || s->size(1) != p.n) return false;
    p.b = *b;
    p.s = *s;
    return true;
}

struct Ref {  // an owned reference, or nullptr
    PyObject *o;
    ~Ref() { Py_XDECREF(o); }
};

bool as_long(PyObject *v, long &out) {  // false: not an int, or beyond a long (PyLong_AsLong says -1 then, which is a group size)
    int overflow = 1;
    if (PyLong_CheckExact(v)) out = PyLong_AsLongAndOverflow(v, &overflow);
    return overflow == 0;
}

bool read_long(PyObject *obj, PyObject *name, long &out) {
    const Ref v{PyObject_GetAttr(obj, name)};
    return v.o && as_long(v.o, out);
}

bool read_proj(PyObject *obj, const at::Device &dev, Proj &p) {
    PyObject *b = PyObject_GetAttr(obj, name_b), *s = b ? PyObject_GetAttr(obj, name_s) : nullptr;
    bool ok = s && read_long(obj, name_g, p.groupsize) && read_long(obj, name_k, p.k) && read_long(obj, name_n, p.n) &&
              weight_ok(p, plain(b, at::kInt), plain(s, at::kHalf), dev);
    Py_XDECREF(b);
    Py_XDECREF(s);
    if (PyErr_Occurred()) PyErr_Clear();
    return ok;
}

// x [m, k], or [b, s, k] where that is allowed: rows of k bf16 values.
bool activations_ok(const Tensor *x, long k, bool allow_rank3, long &m) {
    if (!x || !(x->dim() == 2 || (allow_rank3 && x->dim() == 3)) || k <= 0 || x->size(-1) != k) return false;
    m = x->numel() / k;
    return m > 0 && m <= INT32_MAX;
}

bool out_ok(PyObject *o, Tensor &out, long m, long n, const at::Device &dev) {
    const Tensor *t = plain(o, at::kBFloat16);
    if (!t || t->dim() != 2 || t->size(0) != m || t->size(1) != n || t->device() != dev) return false;
    out = *t;
    return true;
}

Tensor new_output(const Tensor &x, long n) {
    if (x.dim() == 3) return empty({x.size(0), x.size(1), n}, at::kBFloat16, x.device());
    return empty({x.size(0), n}, at::kBFloat16, x.device());
}

PyObject *finish(int status, const Tensor &out) { return status ? PyLong_FromLong(status) : THPVariable_Wrap(out); }

// Frees the GIL for as long as it lives (a launch blocks while the stream's queue is full).  An exception that leaves its scope takes the
// GIL back before anything touches the interpreter.
struct NoGil {
    PyThreadState *state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

template <class F>
PyObject *guarded(F &&f) {  // C++ exceptions become the Python ones that torch's own functions raise (torch.OutOfMemoryError, say)
    try {
        return f();
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

PyObject *run_gemm(const Tensor &x, long m, const Proj &p, Tensor out) {
    const c10::cuda::CUDAGuard guard(x.device());
    if (!out.defined()) out = new_output(x, p.n);
    const size_t need = abi.scratch(static_cast<int>(m), static_cast<int>(p.n), static_cast<int>(p.k), static_cast<int>(p.groupsize), nullptr);
    Tensor ws;
    if (need) ws = empty({static_cast<int64_t>(need)}, at::kByte, x.device());
    void *const wp = need ? ws.mutable_data_ptr() : nullptr, *const stream = c10::cuda::getCurrentCUDAStream().stream();
    const void *xp = x.const_data_ptr(), *bp = p.b.const_data_ptr(), *sp = p.s.const_data_ptr();
    void *op = out.mutable_data_ptr();
    int rc;
    {
        const NoGil free;
        rc = abi.gemm(xp, bp, op, sp, static_cast<int>(m), static_cast<int>(p.n), static_cast<int>(p.k),
                      static_cast<int>(p.groupsize), wp, need, stream);
    }
    return finish(rc, out);
}

// gemm(a, b_packed, scales, groupsize, out)
PyObject *py_gemm(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 5) Py_RETURN_NONE;
        const Tensor *x = plain(args[0], at::kBFloat16), *b = plain(args[1], at::kInt), *s = plain(args[2], at::kHalf);
        if (!x || !b || !s || x->dim() != 2 || s->dim() != 2) Py_RETURN_NONE;
        Proj p{Tensor(), Tensor(), x->size(1), s->size(1), 0};
        if (!as_long(args[3], p.groupsize)) Py_RETURN_NONE;
        long m;
        Tensor out;
        if (!activations_ok(x, p.k, false, m) || !weight_ok(p, b, s, x->device())) Py_RETURN_NONE;
        if (args[4] != Py_None && !out_ok(args[4], out, m, p.n, x->device())) Py_RETURN_NONE;
        return run_gemm(*x, m, p, out);
    });
}

// matmul(x, proj)
PyObject *py_matmul(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 2) Py_RETURN_NONE;
        const Tensor *x = plain(args[0], at::kBFloat16);
        Proj p;
        long m;
        if (!x || !read_proj(args[1], x->device(), p) || !activations_ok(x, p.k, true, m)) Py_RETURN_NONE;
        return run_gemm(*x, m, p, Tensor());
    });
}

// gemm_ex(x, proj, swiglu, lora_a, lora_b, lora_scale, out)
PyObject *py_gemm_ex(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 7) Py_RETURN_NONE;
        const Tensor *x = plain(args[0], at::kBFloat16);
        Proj p;
        long m;
        if (!x || !read_proj(args[1], x->device(), p) || !activations_ok(x, p.k, true, m)) Py_RETURN_NONE;
        kiln_w4a16_epilogue_t ep = {};
        ep.swiglu = PyObject_IsTrue(args[2]) ? 1 : 0;
        if (args[3] != Py_None) {
            const Tensor *a = plain(args[3], at::kBFloat16), *b = plain(args[4], at::kBFloat16);
            if (!a || !b || a->dim() != 2 || b->dim() != 2 || a->device() != x->device() || b->device() != x->device()) Py_RETURN_NONE;
            const int64_t r = a->size(0);
            if (r < 8 || r > 128 || r % 8 || a->size(1) != p.k || b->size(0) != p.n || b->size(1) != r) Py_RETURN_NONE;
            ep.lora_a = a->const_data_ptr();
            ep.lora_b = b->const_data_ptr();
            ep.lora_rank = static_cast<int>(r);
            ep.lora_scale = static_cast<float>(PyFloat_AsDouble(args[5]));
            if (PyErr_Occurred()) return nullptr;
        }
        const long n_out = ep.swiglu ? p.n / 2 : p.n;
        Tensor out;
        if (args[6] != Py_None && !out_ok(args[6], out, m, n_out, x->device())) Py_RETURN_NONE;
        if (args[6] != Py_None && x->dim() == 3) Py_RETURN_NONE;  // (the result is then a reshaped view of `out`)
        const c10::cuda::CUDAGuard guard(x->device());
        if (!out.defined()) out = new_output(*x, n_out);
        const int mi = static_cast<int>(m), ni = static_cast<int>(p.n), ki = static_cast<int>(p.k);
        const size_t need = abi.scratch(mi, ni, ki, static_cast<int>(p.groupsize), &ep);
        Tensor ws;
        if (need) ws = empty({static_cast<int64_t>(need)}, at::kByte, x->device());
        void *const wp = need ? ws.mutable_data_ptr() : nullptr, *const stream = c10::cuda::getCurrentCUDAStream().stream();
        const void *xp = x->const_data_ptr(), *bp = p.b.const_data_ptr(), *sp = p.s.const_data_ptr();
        void *op = out.mutable_data_ptr();
        int rc;
        {
            const NoGil free;
            rc = abi.gemm_ex(xp, bp, op, sp, mi, ni, ki, static_cast<int>(p.groupsize), &ep, wp, need, stream);
        }
        return finish(rc, out);
    });
}

// grouped(xs, projs, outs): lists or tuples of the same length; outs may be None
PyObject *py_grouped(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 3 || !(PyList_CheckExact(args[0]) || PyTuple_CheckExact(args[0])) ||
            !(PyList_CheckExact(args[1]) || PyTuple_CheckExact(args[1])))
            Py_RETURN_NONE;
        const bool given = args[2] != Py_None;
        if (given && !(PyList_CheckExact(args[2]) || PyTuple_CheckExact(args[2]))) Py_RETURN_NONE;
        // (tuples of our own: a list may change while a property of a projection runs, or while the GIL is free)
        const Ref xt{PySequence_Tuple(args[0])}, pt{PySequence_Tuple(args[1])}, ot{given ? PySequence_Tuple(args[2]) : nullptr};
        if (!xt.o || !pt.o || (given && !ot.o)) return nullptr;
        const Py_ssize_t count = PyTuple_GET_SIZE(xt.o);
        if (count < 1 || count > KILN_W4A16_MAX_GROUP || PyTuple_GET_SIZE(pt.o) != count || (given && PyTuple_GET_SIZE(ot.o) != count))
            Py_RETURN_NONE;
        kiln_w4a16_problem_t prob[KILN_W4A16_MAX_GROUP] = {};
        const Tensor *xs[KILN_W4A16_MAX_GROUP];
        Tensor outs[KILN_W4A16_MAX_GROUP];
        Proj projs[KILN_W4A16_MAX_GROUP];
        size_t need = 0;
        for (Py_ssize_t i = 0; i < count; ++i) {
            xs[i] = plain(PyTuple_GET_ITEM(xt.o, i), at::kBFloat16);
            Proj &p = projs[i];
            long m;
            if (!xs[i] || xs[i]->device() != xs[0]->device() || !read_proj(PyTuple_GET_ITEM(pt.o, i), xs[0]->device(), p) ||
                !activations_ok(xs[i], p.k, false, m))
                Py_RETURN_NONE;
            if (given && !out_ok(PyTuple_GET_ITEM(ot.o, i), outs[i], m, p.n, xs[0]->device())) Py_RETURN_NONE;
            prob[i] = {xs[i]->const_data_ptr(), p.b.const_data_ptr(), nullptr, p.s.const_data_ptr(), static_cast<int>(m), static_cast<int>(p.n),
                       static_cast<int>(p.k), static_cast<int>(p.groupsize)};
        }
        const at::Device dev = xs[0]->device();
        const c10::cuda::CUDAGuard guard(dev);
        for (Py_ssize_t i = 0; i < count; ++i) {
            if (!given) outs[i] = new_output(*xs[i], prob[i].n);
            prob[i].C = outs[i].mutable_data_ptr();
            const size_t w = abi.scratch(prob[i].m, prob[i].n, prob[i].k, prob[i].groupsize, nullptr);
            if (w > need) need = w;
        }
        Tensor ws;
        if (need) ws = empty({static_cast<int64_t>(need)}, at::kByte, dev);
        void *const wp = need ? ws.mutable_data_ptr() : nullptr, *const stream = c10::cuda::getCurrentCUDAStream().stream();
        int rc;
        {
            const NoGil free;
            rc = abi.grouped(prob, static_cast<int>(count), wp, need, stream);
        }
        if (rc) return PyLong_FromLong(rc);
        PyObject *list = PyList_New(count);
        if (!list) return nullptr;
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject *o;
            if (given) {
                o = PyTuple_GET_ITEM(ot.o, i);
                Py_INCREF(o);
            } else if (!(o = THPVariable_Wrap(outs[i]))) {
                Py_DECREF(list);
                return nullptr;
            }
            PyList_SET_ITEM(list, i, o);
        }
        return list;
    });
}

// pack(weight, groupsize) -> (b_packed, scales)
PyObject *py_pack(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        long g;
        if (nargs != 2 || !as_long(args[1], g)) Py_RETURN_NONE;
        const Tensor *w = plain(args[0], at::kBFloat16);
        const bool bf16 = w != nullptr;
        if (!w) w = plain(args[0], at::kFloat);
        if (!w || w->dim() != 2 || (g != -1 && g != 128)) Py_RETURN_NONE;
        const int64_t k = w->size(0), n = w->size(1);
        if (k <= 0 || n <= 0 || k % 128 || n % 256 || k > INT32_MAX || n > INT32_MAX / 2) Py_RETURN_NONE;
        const c10::cuda::CUDAGuard guard(w->device());
        const Tensor b = empty({k / 16, 2 * n}, at::kInt, w->device());
        const Tensor s = empty({g == -1 ? 1 : k / g, n}, at::kHalf, w->device());
        void *const stream = c10::cuda::getCurrentCUDAStream().stream();
        const void *wp = w->const_data_ptr();
        int32_t *bp = static_cast<int32_t *>(b.mutable_data_ptr());
        uint16_t *sp = static_cast<uint16_t *>(s.mutable_data_ptr());
        int rc;
        {
            const NoGil free;
            rc = abi.pack(wp, bf16 ? 1 : 0, static_cast<int>(k), static_cast<int>(n), static_cast<int>(g), bp, sp, nullptr, stream);
        }
        if (rc) return PyLong_FromLong(rc);
        PyObject *pb = THPVariable_Wrap(b), *ps = pb ? THPVariable_Wrap(s) : nullptr;
        PyObject *pair = ps ? PyTuple_Pack(2, pb, ps) : nullptr;
        Py_XDECREF(pb);
        Py_XDECREF(ps);
        return pair;
    });
}

// pack_gptq(qweight, qzeros, scales, groupsize) -> (b_packed, scales), or False for an asymmetric checkpoint
PyObject *py_pack_gptq(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        long g;
        if (nargs != 4 || !as_long(args[3], g)) Py_RETURN_NONE;
        const Tensor *qw = plain(args[0], at::kInt), *qz = plain(args[1], at::kInt), *sc = plain(args[2], at::kHalf);
        if (!qw || !qz || !sc || qw->dim() != 2 || qz->dim() != 2 || sc->dim() != 2 || (g != -1 && g != 128)) Py_RETURN_NONE;
        const int64_t k = qw->size(0) * 8, n = qw->size(1);
        if (k <= 0 || n <= 0 || k % 128 || n % 256 || k > INT32_MAX || n > INT32_MAX / 2) Py_RETURN_NONE;
        const int64_t rows = g == -1 ? 1 : k / g;
        if (qz->size(0) != rows || qz->size(1) != n / 8 || sc->size(0) != rows || sc->size(1) != n || qz->device() != qw->device() ||
            sc->device() != qw->device())
            Py_RETURN_NONE;
        const c10::cuda::CUDAGuard guard(qw->device());
        const Tensor b = empty({k / 16, 2 * n}, at::kInt, qw->device()), s = empty({rows, n}, at::kHalf, qw->device());
        const Tensor bad = empty({1}, at::kInt, qw->device());
        void *const stream = c10::cuda::getCurrentCUDAStream().stream();
        int rc, count = 0;
        {
            const NoGil free;
            rc = abi.gptq(qw->const_data_ptr<int32_t>(), qz->const_data_ptr<int32_t>(), static_cast<const uint16_t *>(sc->const_data_ptr()),
                          static_cast<int>(k), static_cast<int>(n), static_cast<int>(g), b.mutable_data_ptr<int32_t>(),
                          static_cast<uint16_t *>(s.mutable_data_ptr()), static_cast<uint32_t *>(bad.mutable_data_ptr()), stream);
            if (!rc) count = bad.item<int>();  // (waits for the device)
        }
        if (rc) return PyLong_FromLong(rc);
        if (count) Py_RETURN_FALSE;
        PyObject *pb = THPVariable_Wrap(b), *ps = pb ? THPVariable_Wrap(s) : nullptr;
        PyObject *pair = ps ? PyTuple_Pack(2, pb, ps) : nullptr;
        Py_XDECREF(pb);
        Py_XDECREF(ps);
        return pair;
    });
}

// bind(gemm, scratch, gemm_ex, grouped, pack, gptq): addresses of the C ABI's entry points
PyObject *py_bind(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    void *p[6];
    if (nargs != 6) {
        PyErr_SetString(PyExc_TypeError, "bind takes six addresses");
        return nullptr;
    }
    for (int i = 0; i < 6; ++i)
        if (!(p[i] = PyLong_AsVoidPtr(args[i]))) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry point");
            return nullptr;
        }
    abi.gemm = reinterpret_cast<decltype(abi.gemm)>(p[0]);
    abi.scratch = reinterpret_cast<decltype(abi.scratch)>(p[1]);
    abi.gemm_ex = reinterpret_cast<decltype(abi.gemm_ex)>(p[2]);
    abi.grouped = reinterpret_cast<decltype(abi.grouped)>(p[3]);
    abi.pack = reinterpret_cast<decltype(abi.pack)>(p[4]);
    abi.gptq = reinterpret_cast<decltype(abi.gptq)>(p[5]);
    Py_RETURN_NONE;
}

template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
PyMethodDef method(const char *name) {
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)), METH_FASTCALL, nullptr};
}

PyMethodDef methods[] = {method<py_bind>("bind"),       method<py_gemm>("gemm"),       method<py_matmul>("matmul"),
                         method<py_gemm_ex>("gemm_ex"), method<py_grouped>("grouped"), method<py_pack>("pack"),
                         method<py_pack_gptq>("pack_gptq"),
                         {nullptr, nullptr, 0, nullptr}};
// (its doc string says what it was compiled for: the build compares it with what is installed)
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", KILN_NATIVE_KEY, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    name_b = PyUnicode_InternFromString("b_packed");
    name_s = PyUnicode_InternFromString("scales");
    name_g = PyUnicode_InternFromString("groupsize");
    name_k = PyUnicode_InternFromString("k");
    name_n = PyUnicode_InternFromString("n");
    return PyModule_Create(&module);
}

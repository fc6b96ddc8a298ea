// tkd_host.cpp: the Python side's launch path in native code (module tkd_host, used by dense_reader/linear.py and
// moe/moe8.py): a call described once is launched again with other tensors.
//
// What bounds a small decode call is not its kernel (about 5 us) but the host: one launch through ctypes, with the
// output allocated by torch.empty and the stream asked from Python, took 29 us for one token through a [4096, 2048]
// bfloat8_b weight. Here the same steps (the output's allocation, the current stream, the descriptor's addresses, the
// launch) are one call into C++ on a copy of the caller's descriptor, so nothing shared between threads is written.
//
// libtkd.so stays free of torch types (include/tkd.h is its whole interface); this module is a client of it.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/tkd.h"

namespace {

// A tensor argument, or null for None.
const at::Tensor* tensor_or_null(PyObject* o) { return o == Py_None ? nullptr : &THPVariable_Unpack(o); }

bool all_tensors(PyObject* const* args, std::initializer_list<int> need, std::initializer_list<int> may) {
    for (int i : need)
        if (!THPVariable_Check(args[i])) return false;
    for (int i : may)
        if (args[i] != Py_None && !THPVariable_Check(args[i])) return false;
    return true;
}

PyObject* type_error(const char* what) {
    PyErr_SetString(PyExc_TypeError, what);
    return nullptr;
}

// The error of libtkd's code `rc` as the Python layer raises it.
PyObject* tkd_error(int rc, const char* what) {
    PyObject* mod = PyImport_ImportModule("dense_reader._tkd");
    if (!mod) return nullptr;
    PyObject* r = PyObject_CallMethod(mod, "check", "is", rc, what);
    Py_XDECREF(r);
    Py_DECREF(mod);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, what);
    return nullptr;
}

// matmul(descriptor's address, x, out or None, residual or None, workspace, row0) -> the output tensor.
// The descriptor (a TkdMatmul kept by the caller) with this call's tensors: rows row0 .. row0 + m of x, out and residual.
// out None: a new [1, 1, m, ldo] tensor of the descriptor's type.
PyObject* host_matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 6 || !all_tensors(args, {1, 4}, {2, 3}))
        return type_error("tkd_host.matmul: descriptor, x, out, residual, workspace, row0");
    const auto* desc = static_cast<const TkdMatmul*>(PyLong_AsVoidPtr(args[0]));
    const int64_t row0 = PyLong_AsLongLong(args[5]);
    if (PyErr_Occurred()) return nullptr;
    try {
        const at::Tensor& x = THPVariable_Unpack(args[1]);
        const at::Tensor *out = tensor_or_null(args[2]), *res = tensor_or_null(args[3]);
        const at::Tensor& ws = THPVariable_Unpack(args[4]);
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != x.get_device()) guard.set_index(x.get_device());
        TkdMatmul a = *desc;
        at::Tensor made;
        const bool f32 = a.out_dtype == TKD_DT_F32;  // (more than 32 rows: tkd_matmul_rows)
        if (!out) {
            const int64_t shape[4] = {1, 1, a.m, a.ldo};
            made = at::detail::empty_cuda(shape, f32 ? at::kFloat : at::kBFloat16, x.device(), std::nullopt);
            out = &made;
        }
        a.x = static_cast<const char*>(x.data_ptr()) + row0 * a.ldx * 2;
        a.out = static_cast<char*>(out->data_ptr()) + row0 * a.ldo * (f32 ? 4 : 2);
        a.residual = res ? static_cast<const char*>(res->data_ptr()) + row0 * a.ldr * (a.residual_dtype == TKD_DT_F32 ? 4 : 2) : nullptr;
        a.workspace = ws.data_ptr();
        a.workspace_bytes = (uint64_t)ws.nbytes();
        void* stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
        int rc;
        Py_BEGIN_ALLOW_THREADS rc = a.m > 32 ? tkd_matmul_rows(&a, stream) : tkd_matmul(&a, stream);
        Py_END_ALLOW_THREADS if (rc) return tkd_error(rc, "tkd_matmul");
        if (made.defined()) return THPVariable_Wrap(std::move(made));
        Py_INCREF(args[2]);
        return args[2];
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// moe(descriptor's address, x, ids, routing weights (gate_up) or None (down), workspace or None) -> the output: bf16
// [1, 1, 1, ldo], or with by_union [1, 1, 32, ldo] (the kernel writes zeros into the rows past the descriptor's).
PyObject* host_moe(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 5 || !all_tensors(args, {1, 2}, {3, 4})) return type_error("tkd_host.moe: descriptor, x, ids, w, workspace");
    const auto* desc = static_cast<const TkdMoe*>(PyLong_AsVoidPtr(args[0]));
    if (PyErr_Occurred()) return nullptr;
    try {
        const at::Tensor &x = THPVariable_Unpack(args[1]), &ids = THPVariable_Unpack(args[2]);
        const at::Tensor *w = tensor_or_null(args[3]), *ws = tensor_or_null(args[4]);
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != x.get_device()) guard.set_index(x.get_device());
        TkdMoe a = *desc;
        const int64_t shape[4] = {1, 1, a.by_union ? 32 : 1, a.ldo};
        at::Tensor out = at::detail::empty_cuda(shape, at::kBFloat16, x.device(), std::nullopt);
        cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
        a.x = x.data_ptr(), a.ldx = x.stride(-2);
        a.ids = ids.data_ptr(), a.ld_ids = ids.stride(-2);
        if (w) a.route_w = w->data_ptr(), a.ld_w = w->stride(-2);
        if (ws) a.workspace = ws->data_ptr(), a.workspace_bytes = (uint64_t)ws->nbytes();
        a.out = out.data_ptr();
        int rc;
        Py_BEGIN_ALLOW_THREADS rc = w ? tkd_moe_gate_up(&a, stream) : tkd_moe_down(&a, stream);
        Py_END_ALLOW_THREADS if (rc) return tkd_error(rc, w ? "tkd_moe_gate_up" : "tkd_moe_down");
        return THPVariable_Wrap(std::move(out));
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// route(logits, ids, w, bias or None, shared or None, (rows, experts, k, kind, scale, norm, groups, groups kept, has slot, slot,
// 32-bit ids)): the router's picks into ids and w (and the shared expert's gate).
PyObject* host_route(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 6 || !all_tensors(args, {0, 1, 2}, {3, 4})) return type_error("tkd_host.route: logits, ids, w, bias, shared, settings");
    int rows, experts, k, kind, norm, ng, tg, has_slot, ids32;
    unsigned slot;
    double scale;
    if (!PyArg_ParseTuple(args[5], "iiiidiiiiIi", &rows, &experts, &k, &kind, &scale, &norm, &ng, &tg, &has_slot, &slot, &ids32)) return nullptr;
    try {
        const at::Tensor &logits = THPVariable_Unpack(args[0]), &ids = THPVariable_Unpack(args[1]), &w = THPVariable_Unpack(args[2]);
        const at::Tensor *bias = tensor_or_null(args[3]), *shared = tensor_or_null(args[4]);
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != logits.get_device()) guard.set_index(logits.get_device());
        void* stream = c10::cuda::getCurrentCUDAStream(logits.get_device()).stream();
        const int64_t ld = logits.stride(-2), ld_ids = ids.stride(-2), ld_w = w.stride(-2), ld_sh = shared ? shared->stride(-2) : 0;
        const float* lp = static_cast<const float*>(logits.data_ptr());
        const float* bp = bias ? static_cast<const float*>(bias->data_ptr()) : nullptr;
        void *ip = ids.data_ptr(), *wp = w.data_ptr(), *sp = shared ? shared->data_ptr() : nullptr;
        int rc;
        Py_BEGIN_ALLOW_THREADS rc = tkd_moe_route(lp, ld, rows, experts, k, kind, bp, scale, norm, ng, tg, has_slot, slot, ip, ids32, ld_ids, wp,
                                                  ld_w, sp, ld_sh, stream);
        Py_END_ALLOW_THREADS if (rc) return tkd_error(rc, "tkd_moe_route");
        Py_RETURN_NONE;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// pick(records, x, head rows, out, ids_out or None, (records, rows, k, top, vocabulary, whether rounded)): tkd_head_pick.
PyObject* host_pick(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 6 || !all_tensors(args, {0, 1, 2, 3}, {4})) return type_error("tkd_host.pick: records, x, head, out, ids_out, settings");
    int nrec, rows, k, top, round;
    unsigned vocab;
    if (!PyArg_ParseTuple(args[5], "iiiiIi", &nrec, &rows, &k, &top, &vocab, &round)) return nullptr;
    try {
        const at::Tensor &rec = THPVariable_Unpack(args[0]), &x = THPVariable_Unpack(args[1]), &head = THPVariable_Unpack(args[2]);
        const at::Tensor &out = THPVariable_Unpack(args[3]), *ids = tensor_or_null(args[4]);
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != x.get_device()) guard.set_index(x.get_device());
        void* stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
        const int64_t dim = x.size(-1), ld_head = head.size(-1);
        const auto* rp = static_cast<const uint32_t*>(rec.data_ptr());
        const void *xp = x.data_ptr(), *hp = head.data_ptr();
        auto* op = static_cast<uint32_t*>(out.data_ptr());
        auto* ip = ids ? static_cast<uint32_t*>(ids->data_ptr()) : nullptr;
        int rc;
        Py_BEGIN_ALLOW_THREADS rc = tkd_head_pick(rp, nrec, rows, k, top, vocab, xp, dim, (int)dim, hp, ld_head, round, op, ip, stream);
        Py_END_ALLOW_THREADS if (rc) return tkd_error(rc, "tkd_head_pick");
        Py_RETURN_NONE;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// hadamard(x [rows, K], sign words) -> x' [1, 1, rows, K] bf16: tkd_hadamard.
PyObject* host_hadamard(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2 || !all_tensors(args, {0, 1}, {})) return type_error("tkd_host.hadamard: x, signs");
    try {
        const at::Tensor &x = THPVariable_Unpack(args[0]), &signs = THPVariable_Unpack(args[1]);
        if (x.dim() != 2 || !x.is_cuda()) return type_error("tkd_host.hadamard: x is [rows, K] on the device");
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != x.get_device()) guard.set_index(x.get_device());
        const int64_t rows = x.size(0), k = x.size(1), shape[4] = {1, 1, rows, k}, ldx = x.stride(0);
        at::Tensor out = at::detail::empty_cuda(shape, at::kBFloat16, x.device(), std::nullopt);
        void* stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
        const void *xp = x.data_ptr(), *sp = signs.data_ptr();
        void* op = out.data_ptr();
        int rc;
        Py_BEGIN_ALLOW_THREADS rc = tkd_hadamard(xp, ldx, static_cast<const uint32_t*>(sp), (int)rows, (int)k, op, k, stream);
        Py_END_ALLOW_THREADS if (rc) return tkd_error(rc, "tkd_hadamard");
        return THPVariable_Wrap(std::move(out));
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// This thread's int in pinned host memory, which a packing kernel sets when its weight is wide: read after the stream has been
// waited for, with nothing copied back.
struct WideWord {
    int* p = nullptr;
    int* get() {
        if (!p && cudaHostAlloc(reinterpret_cast<void**>(&p), sizeof(int), cudaHostAllocPortable) != cudaSuccess) p = nullptr;
        return p;
    }
    ~WideWord() {
        if (p) (void)cudaFreeHost(p);
    }
};

// pack(format, float32 matrix, orientation, divisors or None, scales (0: none, 1: own, 2: ones), stream or None, emax or None) -> (stream, emax or None,
// scales or None, state): tkd_pack_weight into the tensors given or into new ones, waited for (launches read weights ahead of stream order). state 0: done; 1: the weight
// is wide; 2: this K is not taken (then nothing was packed).
PyObject* host_pack(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 7 || !all_tensors(args, {1}, {3, 5, 6})) return type_error("tkd_host.pack: format, matrix, orientation, divisors, scales, stream, emax");
    const int fmt = (int)PyLong_AsLong(args[0]), orient = (int)PyLong_AsLong(args[2]), own = (int)PyLong_AsLong(args[4]);
    if (PyErr_Occurred()) return nullptr;
    static thread_local WideWord word;
    try {
        const at::Tensor& src = THPVariable_Unpack(args[1]);
        const at::Tensor* div = tensor_or_null(args[3]);
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != src.get_device()) guard.set_index(src.get_device());
        const int64_t cols = src.size(orient ? 1 : 0), k = src.size(orient ? 0 : 1);
        int* wide = word.get();
        if (!wide) return tkd_error(TKD_ERR_CUDA + (int)cudaGetLastError(), "cudaHostAlloc");
        *wide = 0;
        auto bytes = [&](int64_t b) { return at::detail::empty_cuda({b}, at::kByte, src.device(), std::nullopt); };
        auto given = [&](int i, int64_t b) -> at::Tensor {
            const at::Tensor* t = tensor_or_null(args[i]);
            if (t && (!t->is_cuda() || t->get_device() != src.get_device() || !t->is_contiguous() || (int64_t)t->nbytes() != b))
                throw std::runtime_error("tkd_host.pack: a tensor given for the result has another size, device or layout");
            return t ? *t : at::Tensor(bytes(b));
        };
        at::Tensor stream = given(5, tkd_packed_bytes(fmt, k, cols)), emax, scales;
        if (fmt != TKD_FMT_BF16) emax = given(6, tkd_padded_cols(cols) / 16);
        if (own) scales = at::detail::empty_cuda({1, 1, 1, cols}, at::kBFloat16, src.device(), std::nullopt);
        cudaStream_t st = c10::cuda::getCurrentCUDAStream(src.get_device()).stream();
        int rc;
        cudaError_t e = cudaSuccess;
        Py_BEGIN_ALLOW_THREADS {
            const auto* sp = static_cast<const float*>(src.data_ptr());
            uint8_t* ep = emax.defined() ? static_cast<uint8_t*>(emax.data_ptr()) : nullptr;
            rc = own == 2 ? tkd_pack_weight_unit(fmt, sp, orient, src.stride(0), k, cols, scales.data_ptr(), stream.data_ptr(), ep, wide, st)
                          : tkd_pack_weight(fmt, sp, orient, src.stride(0), k, cols, div ? static_cast<const float*>(div->data_ptr()) : nullptr,
                                            own ? scales.data_ptr() : nullptr, stream.data_ptr(), ep, wide, st);
        }
        if (!rc) e = cudaStreamSynchronize(st);
        Py_END_ALLOW_THREADS if (rc && rc != TKD_ERR_UNSUPPORTED) return tkd_error(rc, "tkd_pack_weight");
        if (e != cudaSuccess) return tkd_error(TKD_ERR_CUDA + (int)e, "tkd_pack_weight");
        auto wrap = [](at::Tensor& t) -> PyObject* {
            if (t.defined()) return THPVariable_Wrap(std::move(t));
            Py_RETURN_NONE;
        };
        return Py_BuildValue("NNNi", wrap(stream), wrap(emax), wrap(scales), rc ? 2 : *static_cast<volatile int*>(wide) ? 1 : 0);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyMethodDef fast(const char* name) {
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(F)), METH_FASTCALL, nullptr};
}
PyMethodDef methods[] = {
    fast<host_matmul>("matmul"),
    fast<host_moe>("moe"),
    fast<host_route>("route"),
    fast<host_pack>("pack"),
    fast<host_pick>("pick"),
    fast<host_hadamard>("hadamard"),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "tkd_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_tkd_host() {
    PyObject* m = PyModule_Create(&module_def);
    if (m && PyModule_AddStringConstant(m, "built_for", TKD_HOST_FOR) < 0) Py_CLEAR(m);  // (what build.py compiled it against)
    return m;
}

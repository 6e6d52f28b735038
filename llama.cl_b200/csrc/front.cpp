// Native front of the Python ops: argument checks, output allocation, stream and workspace look-up and the call into
// the C-ABI library, in one CPython call per op.
//
// A decode FC of a Llama-7B projection runs 5-10 us on the GPU; the same steps in Python (device context, stream
// object, two ctypes calls, torch.empty) took 21 us of host time per call and were what a loop over small FCs waited
// for.  In C++ they take about 4 us, launch included (fc_Q4A, 512 x 512, one row).  Checks and error texts are those
// the Python functions state: they mirror the ASSERTs of the reference (ops/tensor.hpp:20-36, ops/op_fc.hpp:286-300).
//
// The C-ABI library stays free of torch types; this module is the only part that sees them.  It keeps no state but a
// table (device, stream) -> workspace of references to objects that llmops owns.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cuda_runtime_api.h>

#include <cstring>
#include <exception>
#include <string>
#include <string_view>
#include <vector>

#include "../../include/q4fc_b200.h"

namespace {

using at::Tensor;

// a Python exception is set; unwinds to the entry point
struct PyFailed {};

[[noreturn]] void fail(const std::string& msg) {
    PyErr_SetString(PyExc_RuntimeError, msg.c_str());
    throw PyFailed();
}

std::string str_of(PyObject* o) {
    PyObject* s = PyObject_Str(o);
    if (!s) throw PyFailed();
    const char* c = PyUnicode_AsUTF8(s);
    std::string r = c ? c : "?";
    Py_DECREF(s);
    return r;
}
std::string attr_str(PyObject* o, const char* name) {
    PyObject* a = PyObject_GetAttrString(o, name);
    if (!a) throw PyFailed();
    std::string r = str_of(a);
    Py_DECREF(a);
    return r;
}

const char* dtype_name(at::ScalarType t) {
    return t == at::kFloat ? "float32" : t == at::kChar ? "int8" : "?";
}

const Tensor& tensor(PyObject* o, const char* name, at::ScalarType dtype, int64_t rank) {
    if (!THPVariable_Check(o))
        fail(std::string(name) + ": expected a torch.Tensor, got " + Py_TYPE(o)->tp_name);
    const Tensor& t = THPVariable_Unpack(o);
    if (t.scalar_type() != dtype || t.dim() != rank)
        fail(std::string("assert ") + name + ".is<" + dtype_name(dtype) + ">(" + std::to_string(rank) + ") failed: got dtype " +
             attr_str(o, "dtype") + ", rank " + std::to_string(t.dim()));
    if (!t.is_cuda()) fail(std::string(name) + ": tensor must live on a CUDA device (there is no CPU path)");
    if (!t.is_contiguous()) fail(std::string(name) + ": tensor must be dense row-major (contiguous)");
    return t;
}

std::string shape_text(at::IntArrayRef s) {  // as Python prints a tuple
    std::string r = "(";
    for (size_t i = 0; i < s.size(); i++) r += (i ? ", " : "") + std::to_string(s[i]);
    return r + (s.size() == 1 ? ",)" : ")");
}

void check(int rc, const char* what) {
    if (rc == Q4FC_OK) return;
    fail(std::string(what) + ": " + q4fc_strerror(rc) + " (" + std::to_string(rc) + "): " + q4fc_last_error());
}

// an integer (anything with __index__); nothing else is one
int64_t as_int(PyObject* o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyFailed();
    return v;
}
int as_c_int(PyObject* o) {
    const int64_t v = as_int(o);
    if (v != (int)v) fail("integer out of range: " + std::to_string(v));
    return (int)v;
}
// int(o)
int64_t to_int(PyObject* o) {
    PyObject* l = PyNumber_Long(o);
    if (!l) throw PyFailed();
    const int64_t v = PyLong_AsLongLong(l);
    Py_DECREF(l);
    if (v == -1 && PyErr_Occurred()) throw PyFailed();
    return v;
}
bool truth(PyObject* o) {
    const int t = PyObject_IsTrue(o);
    if (t < 0) throw PyFailed();
    return t != 0;
}

void variant_of(int64_t bs, int* q, int* G) {
    if (q4fc_infer_variant((int)bs, q, G) != Q4FC_OK)
        fail("assert weiq.size(2) == sizeof(q4_block) failed: block size " + std::to_string(bs) +
             " is none of 576 / 640 / 2112 / 2176");
}

Tensor empty_f32(at::IntArrayRef shape, const at::Device& dev) {
    return at::detail::empty_cuda(shape, at::kFloat, dev, std::nullopt);
}

PyObject* new_ref(PyObject* o) {
    Py_INCREF(o);
    return o;
}

// `out` as given (shape checked), or a new tensor; *ret is a new reference either way
float* output(PyObject* out, at::IntArrayRef shape, const at::Device& dev, PyObject** ret) {
    if (out == Py_None) {
        Tensor t = empty_f32(shape, dev);
        float* p = static_cast<float*>(t.data_ptr());
        *ret = THPVariable_Wrap(std::move(t));
        if (!*ret) throw PyFailed();
        return p;
    }
    const Tensor& t = tensor(out, "out", at::kFloat, (int64_t)shape.size());
    if (t.sizes() != shape) fail("out: expected shape " + shape_text(shape) + ", got " + shape_text(t.sizes()));
    *ret = new_ref(out);
    return static_cast<float*>(t.data_ptr());
}

// ---- scratch kept per (device, stream): made and owned by llmops, looked up here -----------------------------------
struct Scratch {
    int dev;
    cudaStream_t stream;
    PyObject* owner;  // keeps the memory alive
    void* ptr;
    size_t bytes;
};
std::vector<Scratch> g_fc_ws, g_q8c_ws;  // accessed with the GIL held

const Scratch& scratch(std::vector<Scratch>& table, int dev, cudaStream_t stream, size_t need, PyObject* maker,
                       PyObject* args) {
    for (Scratch& s : table)
        if (s.dev == dev && s.stream == stream && s.bytes >= need) return s;
    PyObject* got = PyObject_CallObject(maker, args);  // (owner, address, bytes)
    if (!got) throw PyFailed();
    Scratch s{dev, stream, nullptr, nullptr, 0};
    unsigned long long ptr = 0, bytes = 0;
    PyObject* owner = nullptr;
    if (!PyArg_ParseTuple(got, "OKK", &owner, &ptr, &bytes)) {
        Py_DECREF(got);
        throw PyFailed();
    }
    s.owner = new_ref(owner), s.ptr = reinterpret_cast<void*>(ptr), s.bytes = (size_t)bytes;
    Py_DECREF(got);
    for (Scratch& e : table)
        if (e.dev == dev && e.stream == stream) {
            PyObject* old = e.owner;
            e = s;
            Py_DECREF(old);
            return e;
        }
    table.push_back(s);
    return table.back();
}

PyObject* g_make_fc_ws = nullptr;   // llmops: (rows, K, N, qtype, group_k, device index) -> (owner, address, bytes)
PyObject* g_make_q8c_ws = nullptr;  // llmops: (device index, bytes) -> (owner, address, bytes)

template <typename F>
int without_gil(F f) {
    PyThreadState* st = PyEval_SaveThread();
    const int rc = f();
    PyEval_RestoreThread(st);
    return rc;
}

#define FRONT_BEGIN PyObject* ret = nullptr; try {
#define FRONT_END                                        \
    return ret; }                                        \
    catch (const PyFailed&) {}                           \
    catch (...) { torch::translate_exception_to_python(std::current_exception()); } /* as torch's own functions do */ \
    Py_XDECREF(ret);                                     \
    return nullptr;

bool nargs_ok(Py_ssize_t have, Py_ssize_t want) {
    if (have == want) return true;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, have);
    return false;
}

// ---- fc(input, wei_quantized, N, nibble_signed, out, workspace, pdl, path, prequant, addend) -----------------------
PyObject* fc(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 10)) return nullptr;
    FRONT_BEGIN
    const Tensor& x = tensor(a[0], "input", at::kFloat, 3);
    const Tensor& w = tensor(a[1], "wei_quantized", at::kChar, 3);
    if (w.device() != x.device()) fail("input and wei_quantized live on different devices");
    const int64_t B = x.size(0), M = x.size(1), K = x.size(2), Ng = w.size(0), Kg = w.size(1), rows = B * M;
    int q = 0, G = 0;
    variant_of(w.size(2), &q, &G);
    const int64_t N = to_int(a[2]);
    std::string_view pv;
    if (PyUnicode_Check(a[7])) {
        const char* path = PyUnicode_AsUTF8(a[7]);
        if (!path) throw PyFailed();
        pv = path;
    }
    const bool streamk = pv == "streamk", prefill = pv == "prefill";
    if (a[9] == Py_None && !streamk && !prefill && pv != "auto" && pv != "decode") {  // (an addend has one path only)
        PyErr_SetObject(PyExc_KeyError, a[7]);
        throw PyFailed();
    }
    unsigned flags = (truth(a[3]) ? Q4FC_FLAG_NIBBLE_SIGNED : 0u) | (truth(a[6]) ? Q4FC_FLAG_PDL : 0u) |
                     (streamk ? Q4FC_FLAG_STREAMK : 0u) | (truth(a[8]) ? Q4FC_FLAG_PREQUANT : 0u);
    c10::cuda::CUDAGuard guard(x.device());
    const int dev = x.device().index();
    if (N < 0) fail("fc_Q4A: negative N");
    float* y = output(a[4], {B, M, N}, x.device(), &ret);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    void* ws = nullptr;
    size_t ws_bytes = 0;
    if (a[5] != Py_None) {
        PyObject* p = PyObject_GetAttrString(a[5], "ptr");
        PyObject* b = p ? PyObject_GetAttrString(a[5], "nbytes") : nullptr;
        if (b) ws = PyLong_AsVoidPtr(p), ws_bytes = PyLong_AsSize_t(b);
        Py_XDECREF(p), Py_XDECREF(b);
        if (PyErr_Occurred()) throw PyFailed();
    } else {
        // sized for 8 rows whatever a decode call asks for (see llmops.fc_workspace)
        const size_t need = q4fc_fc_workspace_bytes(rows <= 8 ? 8 : rows, K, N, q, G);
        const Scratch* s = nullptr;
        for (const Scratch& e : g_fc_ws)
            if (e.dev == dev && e.stream == stream && e.bytes >= need) s = &e;
        if (!s) {
            PyObject* args = Py_BuildValue("(LLLiii)", rows, K, N, q, G, dev);
            if (!args) throw PyFailed();
            try {
                s = &scratch(g_fc_ws, dev, stream, need, g_make_fc_ws, args);
            } catch (const PyFailed&) {
                Py_DECREF(args);
                throw;
            }
            Py_DECREF(args);
        }
        ws = s->ptr, ws_bytes = s->bytes;
    }
    const float* xp = static_cast<const float*>(x.data_ptr());
    const void* wp = w.data_ptr();
    int rc;
    if (a[9] != Py_None) {
        if (!THPVariable_Check(a[9])) fail(std::string("addend: expected a torch.Tensor, got ") + Py_TYPE(a[9])->tp_name);
        const Tensor& ad = tensor(a[9], "addend", at::kFloat, THPVariable_Unpack(a[9]).dim());
        if (rows > 8 || streamk || prefill)
            fail("addend is folded into the decode kernel only (B*M <= 8, path auto or decode)");
        int64_t ld;
        if (ad.dim() == 1 && ad.size(0) == N) ld = 0;
        else if (ad.dim() == 3 && ad.size(0) == B && ad.size(1) == M && ad.size(2) == N) ld = N;
        else
            fail("addend: expected contiguous shape " + shape_text({N}) + " or " + shape_text({B, M, N}) + ", got " +
                 shape_text(ad.sizes()));
        const float* ap = static_cast<const float*>(ad.data_ptr());
        rc = without_gil([&] {
            return q4fc_fc_decode_add(xp, rows, K, K, wp, Ng, Kg, q, G, N, y, N, ap, ld, ws, ws_bytes, flags, stream);
        });
    } else {
        auto* fn = prefill ? q4fc_fc_prefill : (pv == "auto" ? q4fc_fc : q4fc_fc_decode);
        rc = without_gil([&] { return fn(xp, rows, K, K, wp, Ng, Kg, q, G, N, y, N, ws, ws_bytes, flags, stream); });
    }
    check(rc, "fc_Q4A");
    FRONT_END
}

// ---- pack(wei, qtype, group_k, out) ---------------------------------------------------------------------------------
PyObject* pack(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 4)) return nullptr;
    FRONT_BEGIN
    const int q = as_c_int(a[1]), G = as_c_int(a[2]);
    const Tensor& w = tensor(a[0], "wei", at::kFloat, 2);
    const int bs = q4fc_block_bytes(q, G);
    if (bs < 0) fail("unsupported block type: qtype=" + std::to_string(q) + ", group_k=" + std::to_string(G));
    const int64_t N = w.size(0), K = w.size(1), Ng = (N + 31) / 32, Kg = (K + G - 1) / G;
    c10::cuda::CUDAGuard guard(w.device());
    void* dst;
    if (a[3] == Py_None) {
        Tensor t = at::detail::empty_cuda({Ng, Kg, bs}, at::kChar, w.device(), std::nullopt);
        dst = t.data_ptr();
        ret = THPVariable_Wrap(std::move(t));
        if (!ret) throw PyFailed();
    } else {
        const Tensor& t = tensor(a[3], "out", at::kChar, 3);
        if (t.sizes() != at::IntArrayRef({Ng, Kg, bs}))
            fail("out: expected shape " + shape_text({Ng, Kg, bs}) + ", got " + shape_text(t.sizes()));
        dst = t.data_ptr();
        ret = new_ref(a[3]);
    }
    const float* wp = static_cast<const float*>(w.data_ptr());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(w.device().index()).stream();
    check(without_gil([&] { return q4fc_pack(wp, N, K, q, G, dst, stream); }), "offline_FC_quant_Q4A");
    FRONT_END
}

// ---- q8c_fc(input, wei_quantized, wei_scales, N, out) ---------------------------------------------------------------
PyObject* q8c_fc(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 5)) return nullptr;
    FRONT_BEGIN
    const Tensor& x = tensor(a[0], "input", at::kFloat, 3);
    const Tensor& w = tensor(a[1], "wei_quantized", at::kChar, 3);
    const Tensor& sc = tensor(a[2], "wei_scales", at::kFloat, 1);
    const int64_t B = x.size(0), M = x.size(1), K = x.size(2), Ng = w.size(0), Kg = w.size(1), N = as_int(a[3]);
    if (w.size(2) != 1024)
        fail("assert wei_quantized.size(2) == sizeof(q8_c_block) failed: got " + std::to_string(w.size(2)));
    if (Kg != (K + 31) / 32 || N > Ng * 32 || sc.numel() < N)
        fail("FC_evaluate_Q8C: weights " + shape_text(w.sizes()) + " / scales " + shape_text(sc.sizes()) +
             " do not match K=" + std::to_string(K) + ", N=" + std::to_string(N));
    c10::cuda::CUDAGuard guard(x.device());
    const int dev = x.device().index();
    float* y = output(a[4], {B, M, N}, x.device(), &ret);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    const size_t need = q4fc_q8c_workspace_bytes(B * M, K);
    const Scratch* s = nullptr;
    for (const Scratch& e : g_q8c_ws)
        if (e.dev == dev && e.stream == stream && e.bytes >= need) s = &e;
    if (!s) {
        PyObject* args = Py_BuildValue("(iKK)", dev, (unsigned long long)(uintptr_t)stream, (unsigned long long)need);
        if (!args) throw PyFailed();
        try {
            s = &scratch(g_q8c_ws, dev, stream, need, g_make_q8c_ws, args);
        } catch (const PyFailed&) {
            Py_DECREF(args);
            throw;
        }
        Py_DECREF(args);
    }
    const Scratch ws = *s;
    const float* xp = static_cast<const float*>(x.data_ptr());
    const int8_t* wp = static_cast<const int8_t*>(w.data_ptr());
    const float* sp = static_cast<const float*>(sc.data_ptr());
    check(without_gil([&] {
              return q4fc_q8c_fc(xp, B * M, K, K, wp, sp, Ng, Kg, N, y, N, ws.ptr, ws.bytes, stream);
          }),
          "FC_evaluate_Q8C");
    FRONT_END
}

// ---- embedding(ids, weight, scales, output): output None -> a new tensor --------------------------------------------
PyObject* embedding(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 4)) return nullptr;
    FRONT_BEGIN
    const Tensor& w = tensor(a[1], "weight", at::kChar, 2);
    const Tensor& sc = tensor(a[2], "scales", at::kFloat, 1);
    if (!THPVariable_Check(a[0])) fail("assert input.is<int64_t>() failed: ids must be int32 or int64");
    const Tensor& ids = THPVariable_Unpack(a[0]);
    if (ids.scalar_type() != at::kInt && ids.scalar_type() != at::kLong)
        fail("assert input.is<int64_t>() failed: ids must be int32 or int64");
    if (!ids.is_cuda() || !ids.is_contiguous()) fail("input: must be a contiguous CUDA tensor");
    const int64_t V = w.size(0), E = w.size(1);
    at::DimVector shape(ids.sizes().begin(), ids.sizes().end());
    shape.push_back(E);
    c10::cuda::CUDAGuard guard(w.device());
    float* out;
    if (a[3] == Py_None) {
        out = output(Py_None, shape, w.device(), &ret);
    } else {
        if (!THPVariable_Check(a[3]) || THPVariable_Unpack(a[3]).scalar_type() != at::kFloat)
            fail("assert output.is<float>() failed");
        const Tensor& o = THPVariable_Unpack(a[3]);
        if (o.sizes() != at::IntArrayRef(shape))
            fail("assert infer_shape() == output.shape() failed: " + shape_text(o.sizes()) + " vs " + shape_text(shape));
        if (!o.is_cuda() || !o.is_contiguous()) fail("output: must be a contiguous CUDA tensor");
        out = static_cast<float*>(o.data_ptr());
        ret = new_ref(a[3]);
    }
    const void* ip = ids.data_ptr();
    const int i32 = ids.scalar_type() == at::kInt;
    const int64_t count = ids.numel();
    const int8_t* wp = static_cast<const int8_t*>(w.data_ptr());
    const float* sp = static_cast<const float*>(sc.data_ptr());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(w.device().index()).stream();
    check(without_gil([&] { return q4fc_emb_q8c(ip, i32, count, wp, sp, V, E, out, E, stream); }), "embedding_q8c");
    FRONT_END
}

// ---- prepared argument blocks: fc_batch(address, n, qtype, group_k, flags, device), quant_batch(address, n, group_k,
//      want_isum, flags, device) ------------------------------------------------------------------------------------------
PyObject* fc_batch(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 6)) return nullptr;
    FRONT_BEGIN
    const auto* calls = static_cast<const q4fc_fc_call*>(PyLong_AsVoidPtr(a[0]));
    const int cnt = (int)as_int(a[1]), q = (int)as_int(a[2]), G = (int)as_int(a[3]), dev = (int)as_int(a[5]);
    const unsigned flags = (unsigned)as_int(a[4]);
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    check(without_gil([&] { return q4fc_fc_decode_batch(calls, cnt, q, G, flags, stream); }), "fc_decode_batch");
    ret = new_ref(Py_None);
    FRONT_END
}

PyObject* quant_batch(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 6)) return nullptr;
    FRONT_BEGIN
    const auto* calls = static_cast<const q4fc_xq_call*>(PyLong_AsVoidPtr(a[0]));
    const int cnt = (int)as_int(a[1]), G = (int)as_int(a[2]), isum = (int)as_int(a[3]), dev = (int)as_int(a[5]);
    const unsigned flags = (unsigned)as_int(a[4]);
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    check(without_gil([&] { return q4fc_quant_x_q8_batch(calls, cnt, G, isum, flags, stream); }), "quant_x_q8_batch");
    ret = new_ref(Py_None);
    FRONT_END
}

// ---- graph_step(dst, src, graph_exec, stream, device, sync, result): copy the step's input, replay its graph, wait -----
// Returns a new view of the tensor `result`, made while the graph runs, or True where that is None.
// The graph holds none of torch's random-number kernels (CUDAGraph.replay() would have to advance their state).
// False: `src` is no plain tensor like `dst`, or shares a part of its memory (Tensor.copy_ refuses that); nothing has been
// done.
PyObject* graph_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 7)) return nullptr;
    FRONT_BEGIN
    cudaGraphExec_t exec = static_cast<cudaGraphExec_t>(PyLong_AsVoidPtr(a[2]));
    cudaStream_t stream = static_cast<cudaStream_t>(PyLong_AsVoidPtr(a[3]));
    const auto dev = (c10::DeviceIndex)as_int(a[4]);
    const bool sync = truth(a[5]);
    void* dst = nullptr;
    const void* src = nullptr;
    size_t bytes = 0;
    bool host_copy = false;
    if (a[1] != Py_None) {
        if (!THPVariable_Check(a[0]) || !THPVariable_Check(a[1])) Py_RETURN_FALSE;
        const Tensor &d = THPVariable_Unpack(a[0]), &s = THPVariable_Unpack(a[1]);
        const bool both_host = d.is_cpu() && s.is_cpu(), both_here = d.is_cuda() && s.is_cuda() && d.device() == s.device();
        if ((!both_host && !both_here) || d.scalar_type() != s.scalar_type() || d.sizes() != s.sizes() ||
            !d.is_contiguous() || !s.is_contiguous() || d.is_neg() || s.is_neg())
            Py_RETURN_FALSE;
        dst = d.data_ptr(), src = s.data_ptr(), bytes = d.nbytes(), host_copy = both_host;
        const uintptr_t da = reinterpret_cast<uintptr_t>(dst), sa = reinterpret_cast<uintptr_t>(src);
        if (da != sa && da < sa + bytes && sa < da + bytes) Py_RETURN_FALSE;
    }
    c10::cuda::CUDAGuard guard(dev);
    int rc = without_gil([&] {
        cudaError_t e = cudaSuccess;
        if (src != dst) {
            if (host_copy) memcpy(dst, src, bytes);
            else e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, stream);
        }
        if (e == cudaSuccess) e = cudaGraphLaunch(exec, stream);
        return (int)e;
    });
    if (a[6] == Py_None) {
        ret = new_ref(Py_True);
    } else {
        ret = THPVariable_Wrap(THPVariable_Unpack(a[6]).detach());
        if (!ret) throw PyFailed();
    }
    if (rc == cudaSuccess && sync) rc = without_gil([&] { return (int)cudaStreamSynchronize(stream); });
    if (rc != cudaSuccess) fail(std::string("CUDA error: ") + cudaGetErrorString((cudaError_t)rc));
    FRONT_END
}

// ---- bind(make_fc_workspace, make_q8c_scratch) ----------------------------------------------------------------------
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!nargs_ok(n, 2)) return nullptr;
    Py_XDECREF(g_make_fc_ws), Py_XDECREF(g_make_q8c_ws);
    g_make_fc_ws = new_ref(a[0]), g_make_q8c_ws = new_ref(a[1]);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"fc", reinterpret_cast<PyCFunction>(fc), METH_FASTCALL, nullptr},
    {"pack", reinterpret_cast<PyCFunction>(pack), METH_FASTCALL, nullptr},
    {"q8c_fc", reinterpret_cast<PyCFunction>(q8c_fc), METH_FASTCALL, nullptr},
    {"embedding", reinterpret_cast<PyCFunction>(embedding), METH_FASTCALL, nullptr},
    {"fc_batch", reinterpret_cast<PyCFunction>(fc_batch), METH_FASTCALL, nullptr},
    {"quant_batch", reinterpret_cast<PyCFunction>(quant_batch), METH_FASTCALL, nullptr},
    {"graph_step", reinterpret_cast<PyCFunction>(graph_step), METH_FASTCALL, nullptr},
    {"bind", reinterpret_cast<PyCFunction>(bind), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_q4fc_front", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__q4fc_front(void) { return PyModule_Create(&module); }

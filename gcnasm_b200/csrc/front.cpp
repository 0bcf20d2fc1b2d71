// Python front end of the per-call operators: what api.py's GEMM and activation-quantiser functions do between the
// user's tensors and the C ABI, in native code.  Checks, output allocation, argument block and launch of one call
// cost about 20 us of interpreter and ctypes time in Python -- more than the small GEMMs and the decode layers take on the
// GPU -- and 4 us here, of which the launch is 2 and an allocation 0.4 (256 x 512 x 1024 per-tensor GEMM, back to back: 22.7 us a call
// before, 4.2 now).
//
// The module holds no state but the addresses of the C ABI entries (bind()), which api.py takes from the library that
// _lib.py has loaded, so that both sides use one copy of it.  Functions return the output tensor(s), or the C ABI's
// negative error code as an int; misuse raises the TypeError / ValueError the operators document.
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200gemm.h"

namespace {

using GemmFn = int (*)(const b200_gemm_args*, void*);
GemmFn g_gemm = nullptr, g_gemm_simple = nullptr, g_gemm16 = nullptr;
decltype(&b200_quantize_act_bf16_1x128) g_act_1x128 = nullptr;
decltype(&b200_quantize_act_bf16_mx32) g_act_mx32 = nullptr;
decltype(&b200_mx_sf_bytes) g_mx_sf_bytes = nullptr;

struct TypeErr { const char* what; };
struct ValueErr { const char* what; };
struct DeviceErr { c10::Device a, b; };          // operands on two devices, or (b without an index) not on the current one

[[noreturn]] void type_error(const char* w) { throw TypeErr{w}; }
[[noreturn]] void value_error(const char* w) { throw ValueErr{w}; }

const at::Tensor& tensor(PyObject* o, const char* what) {
    if (!THPVariable_Check(o)) type_error(what);
    return THPVariable_Unpack(o);
}
const at::Tensor* opt_tensor(PyObject* o, const char* what) { return o == Py_None ? nullptr : &tensor(o, what); }
int64_t integer(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}

// every CUDA operand on ONE device, and that device current (the C side takes its device from cudaGetDevice())
struct SameDevice {
    c10::Device dev{c10::DeviceType::CPU};
    void add(const at::Tensor* t) {
        if (!t) return;
        if (!t->is_cuda()) value_error("operands must be CUDA tensors");
        if (dev.is_cpu()) dev = t->device();
        else if (t->device() != dev) throw DeviceErr{dev, t->device()};
    }
    void current() const {
        if (dev.index() != c10::cuda::current_device()) throw DeviceErr{dev, c10::Device(c10::DeviceType::CUDA, -1)};
    }
};

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
// on the current device, which SameDevice has found to be the operands' (empty_cuda asks for it and sets it, three times a layer)
at::Tensor empty(at::IntArrayRef shape, at::ScalarType t) {
    return at::detail::empty_generic(shape, at::cuda::getCUDADeviceAllocator(), c10::DispatchKeySet(c10::DispatchKey::CUDA), t, std::nullopt);
}
at::ScalarType out_type(PyObject* o) {
    const at::ScalarType t = THPDtype_Check(o) ? reinterpret_cast<THPDtype*>(o)->scalar_type : at::ScalarType::Undefined;
    if (t != at::kBFloat16 && t != at::kFloat) type_error("output dtype must be torch.bfloat16 or torch.float32");
    return t;
}
bool is_e4m3(const at::Tensor& t) { return t.scalar_type() == at::kByte || t.scalar_type() == at::ScalarType::Float8_e4m3fn; }

// The C call without the interpreter lock: a launch waits when the stream's queue is full, and other threads go on.
template <class F>
int unlocked(F&& f) {
    PyThreadState* st = PyEval_SaveThread();
    const int rc = f();
    PyEval_RestoreThread(st);
    return rc;
}

template <class F>
PyObject* guarded(F&& body) {
    try {
        return body();
    } catch (const TypeErr& e) {
        PyErr_SetString(PyExc_TypeError, e.what);
    } catch (const ValueErr& e) {
        PyErr_SetString(PyExc_ValueError, e.what);
    } catch (const DeviceErr& e) {
        if (e.b.has_index())
            PyErr_Format(PyExc_ValueError, "operands live on different devices: %s and %s", e.a.str().c_str(), e.b.str().c_str());
        else
            PyErr_Format(PyExc_ValueError, "operands live on %s but the current device is cuda:%d; wrap the call in "
                         "`with torch.cuda.device(tensor.device):`", e.a.str().c_str(), static_cast<int>(c10::cuda::current_device()));
    } catch (python_error& e) {
        e.restore();
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());      // out of memory and torch's other errors
    }
    return nullptr;
}

PyObject* pair(PyObject* x, PyObject* y) {
    PyObject* t = PyTuple_New(2);
    PyTuple_SET_ITEM(t, 0, x);
    PyTuple_SET_ITEM(t, 1, y);
    return t;
}

// size / stride of dimension `d` of a [batch, rows, cols] view of t; a 2-D tensor is one batch
struct View3 {
    int64_t batch, rows, cols, ld, batch_stride, col_stride;
    explicit View3(const at::Tensor& t, const char* what) {
        const int64_t nd = t.dim();
        if (nd != 2 && nd != 3) value_error(what);
        const auto sz = t.sizes(), st = t.strides();
        rows = sz[nd - 2];
        cols = sz[nd - 1];
        ld = st[nd - 2];
        col_stride = st[nd - 1];
        batch = nd == 3 ? sz[0] : 1;
        batch_stride = nd == 3 ? st[0] : rows * ld;
    }
};

void tensor_scale(const at::Tensor* t, const float** slot) {
    if (!t) return;
    if (t->scalar_type() != at::kFloat || !t->is_cuda() || t->numel() != 1) type_error("per-tensor scales are 1-element float32 CUDA tensors");
    *slot = static_cast<const float*>(t->const_data_ptr());
}

// gemm(a, b, out, sfa, sfb, scale_a, scale_b, batch_ready, n, scale_mode, b_layout, out_dtype, tile, flags, epoch, entry)
// entry: 0 b200_gemm_a8w8, 1 b200_gemm_a8w8_simple, 2 b200_gemm_a16w16 (bf16 operands).
PyObject* front_gemm(PyObject*, PyObject* const* v, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 16) type_error("gemm takes 16 arguments");
        const at::Tensor &a = tensor(v[0], "A must be a tensor"), &b = tensor(v[1], "B must be a tensor");
        const int64_t entry = integer(v[15]);
        const bool ab16 = entry == 2;
        if (ab16 ? a.scalar_type() != at::kBFloat16 || b.scalar_type() != at::kBFloat16 : !(is_e4m3(a) && is_e4m3(b)))
            type_error(ab16 ? "A and B must be torch.bfloat16"
                            : "A and B must hold E4M3 bytes: uint8 or float8_e4m3fn (torch.bfloat16 operands: gemm_a16w16)");
        const at::Tensor *out_in = opt_tensor(v[2], "out must be a tensor"), *sfa = opt_tensor(v[3], "SFA must be a tensor"),
                         *sfb = opt_tensor(v[4], "SFB must be a tensor"), *sca = opt_tensor(v[5], "scale_a must be a tensor"),
                         *scb = opt_tensor(v[6], "scale_b must be a tensor"), *ready = opt_tensor(v[7], "batch_ready must be a tensor");
        const bool flat = integer(v[10]) == B200_B_FLAT_16x16;
        const int32_t mode = static_cast<int32_t>(integer(v[9]));
        SameDevice same;
        for (const at::Tensor* t : {&a, &b, sfa, sfb, sca, scb, out_in, ready}) same.add(t);
        same.current();

        const View3 va(a, "A must be [batch, M, K] or [M, K]");
        if (va.col_stride != 1) value_error("A must be K-contiguous");
        const int64_t batch = va.batch, m = va.rows, k = va.cols;
        b200_gemm_args g{};
        g.ptr_a = a.const_data_ptr();
        g.ptr_b = b.const_data_ptr();
        // a 2-D B (or scale tensor) given with a batched A is ONE operand shared by every batch (batch stride 0)
        const bool b_shared = batch > 1 && !flat && !ab16 && b.dim() == 2;
        int64_t n;
        if (!flat) {
            const View3 vb(b, "B must be [batch, N, K] or [N, K]");
            if ((!b_shared && vb.batch != batch) || vb.cols != k || vb.col_stride != 1)
                value_error("B must be [batch, N, K] (or [N, K], shared by all batches), K-contiguous, matching A");
            n = vb.rows;
            g.stride_b = vb.ld;
            g.stride_b_batch = b_shared ? 0 : vb.batch_stride;
        } else {
            if (v[8] == Py_None) value_error("flat B needs n=");
            n = integer(v[8]);
            if (!b.is_contiguous() || b.numel() != batch * n * k) value_error("flat B must be a contiguous image of batch*N*K values");
            g.stride_b = n;                            // as the reference sets it (flatmm_a8w8_gfx950.cc:765)
            g.stride_b_batch = n * k;
        }
        at::Tensor out;
        if (out_in) {
            const View3 vo(*out_in, "out must be [batch, M, N], N-contiguous");
            if (vo.batch != batch || vo.rows != m || vo.cols != n || vo.col_stride != 1) value_error("out must be [batch, M, N], N-contiguous");
            out = *out_in;
            g.stride_c = vo.ld;
            g.stride_c_batch = vo.batch_stride;
        } else {
            const at::ScalarType t = out_type(v[11]);
            out = a.dim() == 2 ? empty({m, n}, t) : empty({batch, m, n}, t);
            g.stride_c = n;
            g.stride_c_batch = m * n;
        }
        if (out.scalar_type() != at::kBFloat16 && out.scalar_type() != at::kFloat) type_error("output dtype must be torch.bfloat16 or torch.float32");
        g.ptr_c = out.mutable_data_ptr();
        g.m = m; g.n = n; g.k = k; g.batch = batch;
        g.stride_a = va.ld;
        g.stride_a_batch = va.batch_stride;
        at::Tensor hold_a, hold_b;                     // contiguous copies of strided MX scales
        if (mode == B200_SCALE_BLOCK) {
            if (!sfa || !sfb || sfa->scalar_type() != at::kFloat || sfb->scalar_type() != at::kFloat) type_error("block scales are float32");
            const char* shape = "SFA must be [batch, K/128, M] and SFB [batch, N/128, K/128] ([N/128, K/128] with a shared B)";
            const View3 fa(*sfa, shape), fb(*sfb, shape);
            if (fa.batch != batch || fa.rows != k / 128 || fa.cols != m || fb.batch != (b_shared ? 1 : batch) || fb.rows != n / 128 ||
                fb.cols != k / 128)
                value_error(shape);
            if (fa.col_stride != 1 || fb.col_stride != 1) value_error("scale tensors must be contiguous in their last dimension");
            g.ptr_sfa = sfa->const_data_ptr();
            g.ptr_sfb = sfb->const_data_ptr();
            g.stride_sfa = fa.ld;
            g.stride_sfb = fb.ld;
            g.stride_sfa_batch = fa.batch_stride;
            g.stride_sfb_batch = b_shared ? 0 : fb.batch_stride;
        } else if (mode == B200_SCALE_MX) {
            if (!sfa || !sfb) type_error("MX scales must be the relayouted atom images (see mx_sf_relayout)");
            hold_a = sfa->contiguous();
            hold_b = sfb->contiguous();
            const int64_t need_a = static_cast<int64_t>(g_mx_sf_bytes(m, k)), need_b = static_cast<int64_t>(g_mx_sf_bytes(n, k));
            if (static_cast<int64_t>(hold_a.nbytes()) != batch * need_a || static_cast<int64_t>(hold_b.nbytes()) != batch * need_b)
                value_error("MX scales must be the relayouted atom images (see mx_sf_relayout)");
            g.ptr_sfa = hold_a.const_data_ptr();
            g.ptr_sfb = hold_b.const_data_ptr();
            g.stride_sfa_batch = need_a;
            g.stride_sfb_batch = need_b;
        } else if (mode == B200_SCALE_TENSOR) {
            tensor_scale(sca, &g.ptr_scale_a);
            tensor_scale(scb, &g.ptr_scale_b);
        }
        g.scale_mode = mode;
        g.b_layout = flat ? B200_B_FLAT_16x16 : B200_B_NK_ROWMAJOR;
        g.out_dtype = out.scalar_type() == at::kBFloat16 ? B200_OUT_BF16 : B200_OUT_F32;
        g.tile_hint = static_cast<int32_t>(integer(v[12]));
        g.flags = static_cast<int32_t>(integer(v[13]));
        if (ready) {
            if (ready->scalar_type() != at::kInt || ready->numel() < batch || !ready->is_contiguous())
                value_error("batch_ready must be a contiguous int32 CUDA tensor with one word per batch");
            g.flags |= B200_GEMM_BATCH_READY;
            g.ptr_batch_ready = static_cast<const int32_t*>(ready->const_data_ptr());
            g.batch_epoch = static_cast<int32_t>(integer(v[14]));
        }
        const GemmFn fn = ab16 ? g_gemm16 : (entry == 1 ? g_gemm_simple : g_gemm);
        void* st = stream();
        const int rc = unlocked([&] { return fn(&g, st); });
        if (rc) return PyLong_FromLong(rc);
        if (a.dim() == 2 && out.dim() == 3) out = out.select(0, 0);       // the result has as many dimensions as A
        else if (a.dim() == 3 && out.dim() == 2) out = out.unsqueeze(0);
        return THPVariable_Wrap(out);
    });
}

const at::Tensor& activations(PyObject* o) {
    const at::Tensor& x = tensor(o, "x must be a 2-D bf16 tensor with unit column stride");
    if (x.scalar_type() != at::kBFloat16 || x.dim() != 2 || x.stride(1) != 1) value_error("x must be a 2-D bf16 tensor with unit column stride");
    return x;
}

// act_quant_1x128(x, q or None, sfa or None) -> (q, sfa)
PyObject* front_act_quant_1x128(PyObject*, PyObject* const* v, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 3) type_error("act_quant_1x128 takes 3 arguments");
        const at::Tensor& x = activations(v[0]);
        const at::Tensor *q_in = opt_tensor(v[1], "q must be a tensor"), *s_in = opt_tensor(v[2], "sfa must be a tensor");
        SameDevice same;
        for (const at::Tensor* t : {&x, q_in, s_in}) same.add(t);
        same.current();
        const int64_t m = x.size(0), k = x.size(1);
        const at::Tensor q = q_in ? *q_in : empty({m, k}, at::kByte);
        const at::Tensor sfa = s_in ? *s_in : empty({k / 128, m}, at::kFloat);
        if (q.dim() != 2 || q.size(0) != m || q.size(1) != k || q.scalar_type() != at::kByte || q.stride(1) != 1)
            value_error("q must be a [M,K] uint8 tensor with unit column stride");
        if (sfa.dim() != 2 || sfa.size(0) != k / 128 || sfa.size(1) != m || sfa.scalar_type() != at::kFloat || sfa.stride(1) != 1)
            value_error("sfa must be a [K/128, M] fp32 tensor with unit column stride");
        const int64_t ldx = x.stride(0), ldq = q.stride(0), lds = k > 128 ? sfa.stride(0) : m;
        const void* xp = x.const_data_ptr();
        void *qp = q.mutable_data_ptr(), *sp = sfa.mutable_data_ptr(), *st = stream();
        const int rc = unlocked([&] { return g_act_1x128(xp, ldx, qp, ldq, static_cast<float*>(sp), lds, m, k, st); });
        if (rc) return PyLong_FromLong(rc);
        return pair(THPVariable_Wrap(q), THPVariable_Wrap(sfa));
    });
}

// act_quant_mx32(x) -> (q, atoms)
PyObject* front_act_quant_mx32(PyObject*, PyObject* const* v, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 1) type_error("act_quant_mx32 takes 1 argument");
        const at::Tensor& x = activations(v[0]);
        SameDevice same;
        same.add(&x);
        same.current();
        const int64_t m = x.size(0), k = x.size(1), ldx = x.stride(0);
        const at::Tensor q = empty({m, k}, at::kByte);
        const at::Tensor atoms = empty({static_cast<int64_t>(g_mx_sf_bytes(m, k))}, at::kByte);
        const void* xp = x.const_data_ptr();
        void *qp = q.mutable_data_ptr(), *ap = atoms.mutable_data_ptr(), *st = stream();
        const int rc = unlocked([&] { return g_act_mx32(xp, ldx, qp, k, ap, m, k, st); });
        if (rc) return PyLong_FromLong(rc);
        return pair(THPVariable_Wrap(q), THPVariable_Wrap(atoms));
    });
}

// bind({name: address}): the C ABI entries of the library that is in use
PyObject* front_bind(PyObject*, PyObject* d) {
    return guarded([&]() -> PyObject* {
        auto address = [&](const char* name) -> void* {
            PyObject* o = PyDict_Check(d) ? PyDict_GetItemString(d, name) : nullptr;
            if (!o) value_error("bind() misses an entry of the C ABI");
            void* p = PyLong_AsVoidPtr(o);
            if (!p) value_error("bind() got a null address");
            return p;
        };
        g_gemm = reinterpret_cast<GemmFn>(address("b200_gemm_a8w8"));
        g_gemm_simple = reinterpret_cast<GemmFn>(address("b200_gemm_a8w8_simple"));
        g_gemm16 = reinterpret_cast<GemmFn>(address("b200_gemm_a16w16"));
        g_act_1x128 = reinterpret_cast<decltype(g_act_1x128)>(address("b200_quantize_act_bf16_1x128"));
        g_act_mx32 = reinterpret_cast<decltype(g_act_mx32)>(address("b200_quantize_act_bf16_mx32"));
        g_mx_sf_bytes = reinterpret_cast<decltype(g_mx_sf_bytes)>(address("b200_mx_sf_bytes"));
        Py_RETURN_NONE;
    });
}

PyMethodDef methods[] = {
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(front_gemm)), METH_FASTCALL, nullptr},
    {"act_quant_1x128", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(front_act_quant_1x128)), METH_FASTCALL, nullptr},
    {"act_quant_mx32", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(front_act_quant_mx32)), METH_FASTCALL, nullptr},
    {"bind", front_bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_front", "native front end of gcnasm_b200.api", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__front() { return PyModule_Create(&module); }

// The call path of flash_attn_forward on torch tensors: checks, output allocation, parameter block, stream and launch in
// one native function.  Successor of the host side of the reference's main() (src/main.cu:109-205) for callers whose memory
// torch owns.  A short call is bound by the host: [1,4,256,256,64] took 15.0 us a call through ctypes (two allocations through
// Python 5, argument handling 5, the library 4) and takes 6.1, of which the kernel is 4.8; a decode step over 1000 keys 16.4 and 6.6, of
// which the kernel is 5.1.  (On buffers seen before: a new one costs a tensor map each.)
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <cmath>
#include <cstring>
#include <optional>
#include "../../include/fa_b200.h"

namespace {

typedef int (*fwd_fn)(const fa_fwd_params*);
typedef size_t (*workspace_fn)(const fa_fwd_params*);

// A Python error is set.
struct python_error_set {};

[[noreturn]] void value_error(const char* what) {
    PyErr_SetString(PyExc_ValueError, what);
    throw python_error_set();
}

// int(x), as the low bits that a C field of that width takes
unsigned long long bits_of(PyObject* x) {
    PyObject* n = PyLong_Check(x) ? Py_NewRef(x) : PyNumber_Long(x);
    if (!n) throw python_error_set();
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(n);
    Py_DECREF(n);
    if (v == static_cast<unsigned long long>(-1) && PyErr_Occurred()) throw python_error_set();
    return v;
}
int int_of(PyObject* x) { return static_cast<int>(bits_of(x)); }
bool truth_of(PyObject* x) {
    const int t = PyObject_IsTrue(x);
    if (t < 0) throw python_error_set();
    return t != 0;
}
double float_of(PyObject* x) {
    if (PyFloat_CheckExact(x)) return PyFloat_AS_DOUBLE(x);
    PyObject* f = PyNumber_Float(x);
    if (!f) throw python_error_set();
    const double v = PyFloat_AS_DOUBLE(f);
    Py_DECREF(f);
    return v;
}
const at::Tensor& tensor_of(PyObject* x, const char* name) {
    if (!THPVariable_Check(x)) {
        PyErr_Format(PyExc_TypeError, "%s must be a tensor", name);
        throw python_error_set();
    }
    return THPVariable_Unpack(x);
}
// FA_DTYPE_* of a tensor that may be an output
int dtype_of(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kHalf: return FA_DTYPE_FP16;
        case at::kBFloat16: return FA_DTYPE_BF16;
        case at::kFloat: return FA_DTYPE_FP32;
        default:
            PyErr_Format(PyExc_KeyError, "no attention output of dtype %s", c10::toString(t.scalar_type()));
            throw python_error_set();
    }
}
bool same(at::IntArrayRef a, at::IntArrayRef b) { return a == b; }

// Kernels follow a pointer as it is, so memory that `device` does not reach is refused here.  A tensor on the device itself costs a
// comparison; pinned and managed host memory and an enabled peer's memory are reached too, which the runtime is asked about.
bool reaches(const c10::Device& device, const void* memory) {
    const c10::cuda::OptionalCUDAGuard guard(device);
    cudaPointerAttributes at;
    const bool known = cudaPointerGetAttributes(&at, memory) == cudaSuccess;
    if (!known) (void)cudaGetLastError();
    return known && at.devicePointer != nullptr;
}
void need_reach(const c10::Device& device, const at::Tensor& t, const char* name) {
    if (t.device() == device || t.numel() == 0 || reaches(device, t.data_ptr())) return;
    PyErr_Format(PyExc_ValueError, "%s must be on q's device, or in memory that this device reaches", name);
    throw python_error_set();
}

enum Arg {
    kFwd, kWorkspaceFn, kQ, kK, kV, kScale, kCausal, kWindow, kSlopes, kDropout, kSeed, kOffset, kSplits, kOut, kOutDtype,
    kReturnLse, kQPos0, kKPos0, kUnit0, kWorkspace, kStatus, kAccum, kAccumFirst, kAccumFinal, kLaunchIndex, kArgs
};

PyObject* forward_impl(PyObject* const* args) {
    const fwd_fn fwd = reinterpret_cast<fwd_fn>(bits_of(args[kFwd]));
    const workspace_fn workspace_bytes = reinterpret_cast<workspace_fn>(bits_of(args[kWorkspaceFn]));
    const at::Tensor &q = tensor_of(args[kQ], "q"), &k = tensor_of(args[kK], "k"), &v = tensor_of(args[kV], "v");
    if (!q.is_cuda()) value_error("flash_attn_forward needs CUDA tensors (use flash_attn_forward_host for host buffers)");
    if (q.dim() != 4) value_error("q must be [batch, heads, seqlen, head_dim]");
    const int64_t B = q.size(0), H = q.size(1), Nq = q.size(2), d = q.size(3);
    const c10::Device device = q.device();
    const bool accum = args[kAccum] != Py_None, accum_final = truth_of(args[kAccumFinal]);
    const bool writes_output = !accum || accum_final;
    at::Tensor out, lse;
    if (writes_output) {
        if (args[kOut] != Py_None) {
            out = tensor_of(args[kOut], "out");
        } else {
            at::ScalarType type = q.scalar_type();
            if (args[kOutDtype] != Py_None) {
                if (!THPDtype_Check(args[kOutDtype])) {
                    PyErr_SetString(PyExc_TypeError, "out_dtype must be a torch.dtype");
                    throw python_error_set();
                }
                type = reinterpret_cast<THPDtype*>(args[kOutDtype])->scalar_type;
            }
            out = at::empty({B, H, Nq, d}, q.options().dtype(type).layout(at::kStrided).requires_grad(false));
        }
        if (truth_of(args[kReturnLse])) lse = at::empty({B, H, Nq}, q.options().dtype(at::kFloat).layout(at::kStrided).requires_grad(false));
    }
    at::Tensor slopes;
    if (args[kSlopes] != Py_None) {
        slopes = tensor_of(args[kSlopes], "alibi_slopes").to(device, at::kFloat).contiguous();
        if (slopes.numel() < H) value_error("alibi_slopes must hold a slope for each head");
    }
    const at::Tensor& o = out.defined() ? out : q;
    if (k.dim() < 3) value_error("k and v must be [batch, heads_k, seqlen_k, head_dim] with heads a multiple of heads_k");
    const int64_t Hk = k.size(1), Nk = k.size(2);
    const int64_t kv[4] = {B, Hk, Nk, d};
    if (!same(k.sizes(), kv) || !same(v.sizes(), kv) || Hk < 1 || H % Hk != 0)
        value_error("k and v must be [batch, heads_k, seqlen_k, head_dim] with heads a multiple of heads_k");
    if (!(q.is_contiguous() && k.is_contiguous() && v.is_contiguous() && o.is_contiguous()))
        value_error("q, k, v, o must be contiguous [batch, heads, seqlen, head_dim]");
    const at::ScalarType type = q.scalar_type();
    if ((type != at::kHalf && type != at::kBFloat16) || k.scalar_type() != type || v.scalar_type() != type)
        value_error("q, k, v must share dtype float16 or bfloat16");
    // (an output of another shape is filled as [batch, heads, seqlen, head_dim] rows one behind the other: it has to hold them)
    if (o.numel() < q.numel()) value_error("out must hold [batch, heads, seqlen, head_dim]");
    need_reach(device, k, "k");
    need_reach(device, v, "v");
    need_reach(device, o, "out");

    fa_fwd_params p;
    std::memset(&p, 0, sizeof p);
    at::Tensor o_acc, lse_acc;
    if (accum) {
        PyObject* pair = PySequence_Fast(args[kAccum], "accum = (fp32 [B,H,Nq,d], fp32 [B,H,Nq]), contiguous");
        if (!pair) throw python_error_set();
        if (PySequence_Fast_GET_SIZE(pair) != 2) {
            Py_DECREF(pair);
            value_error("accum = (fp32 [B,H,Nq,d], fp32 [B,H,Nq]), contiguous");
        }
        PyObject *a = PySequence_Fast_GET_ITEM(pair, 0), *b = PySequence_Fast_GET_ITEM(pair, 1);
        const bool tensors = THPVariable_Check(a) && THPVariable_Check(b);
        if (tensors) {
            o_acc = THPVariable_Unpack(a);
            lse_acc = THPVariable_Unpack(b);
        }
        Py_DECREF(pair);
        const int64_t rows[4] = {B, H, Nq, d};
        if (!tensors || o_acc.scalar_type() != at::kFloat || lse_acc.scalar_type() != at::kFloat || !o_acc.is_contiguous() ||
            !lse_acc.is_contiguous() || !same(o_acc.sizes(), rows) || !same(lse_acc.sizes(), at::IntArrayRef(rows, 3)))
            value_error("accum = (fp32 [B,H,Nq,d], fp32 [B,H,Nq]), contiguous");
        need_reach(device, o_acc, "accum");
        need_reach(device, lse_acc, "accum");
        p.accum_o = static_cast<float*>(o_acc.data_ptr());
        p.accum_lse = static_cast<float*>(lse_acc.data_ptr());
        p.accum_flags = (truth_of(args[kAccumFirst]) ? FA_ACCUM_FIRST : 0) | (accum_final ? FA_ACCUM_FINAL : 0);
    }
    p.q = q.data_ptr();
    p.k = k.data_ptr();
    p.v = v.data_ptr();
    p.o = out.defined() ? out.data_ptr() : nullptr;
    p.lse = lse.defined() ? static_cast<float*>(lse.data_ptr()) : nullptr;
    p.dtype = dtype_of(q);
    p.o_dtype = dtype_of(o);
    p.batch = static_cast<int>(B);
    p.heads = static_cast<int>(H);
    p.heads_k = static_cast<int>(Hk);
    p.seqlen_q = static_cast<int>(Nq);
    p.seqlen_k = static_cast<int>(Nk);
    p.head_dim = static_cast<int>(d);
    if (args[kScale] != Py_None) {
        p.softmax_scale = static_cast<float>(float_of(args[kScale]));
    } else {
        if (d == 0) {
            PyErr_SetString(PyExc_ZeroDivisionError, "float division by zero");
            throw python_error_set();
        }
        p.softmax_scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(d)));
    }
    p.is_causal = truth_of(args[kCausal]) ? 1 : 0;
    for (int i = 0; i < 2; ++i) {
        PyObject* x;
        if (PyTuple_CheckExact(args[kWindow]) && PyTuple_GET_SIZE(args[kWindow]) > i) {
            x = Py_NewRef(PyTuple_GET_ITEM(args[kWindow], i));
        } else {  // window[i] of whatever has items (a tensor is no sequence)
            PyObject* at = PyLong_FromLong(i);
            x = at ? PyObject_GetItem(args[kWindow], at) : nullptr;
            Py_XDECREF(at);
        }
        if (!x) throw python_error_set();
        int w;
        try {
            w = int_of(x);
        } catch (...) {
            Py_DECREF(x);
            throw;
        }
        Py_DECREF(x);
        (i == 0 ? p.window_left : p.window_right) = w;
    }
    p.alibi_slopes = slopes.defined() ? static_cast<const float*>(slopes.data_ptr()) : nullptr;
    p.p_dropout = static_cast<float>(float_of(args[kDropout]));
    p.seed = bits_of(args[kSeed]);
    p.offset = bits_of(args[kOffset]);
    p.unit0 = bits_of(args[kUnit0]);
    p.launch_index = bits_of(args[kLaunchIndex]);
    p.num_splits = int_of(args[kSplits]);
    p.q_pos0 = static_cast<int64_t>(bits_of(args[kQPos0]));
    p.k_pos0 = static_cast<int64_t>(bits_of(args[kKPos0]));
    if (args[kStatus] != Py_None) {
        const at::Tensor& status = tensor_of(args[kStatus], "status");
        if (status.nbytes() < sizeof(int) || reinterpret_cast<uintptr_t>(status.data_ptr()) % sizeof(int) != 0)
            value_error("status must hold an aligned 32-bit word");
        need_reach(device, status, "status");
        p.status = static_cast<int*>(status.data_ptr());
    }

    const c10::cuda::OptionalCUDAGuard guard(device);  // (nothing where the device is the current one)
    at::Tensor workspace;
    if (p.num_splits != 1 || d % 8 != 0) {
        const size_t need = workspace_bytes(&p);
        if (need != 0) {
            if (args[kWorkspace] != Py_None) workspace = tensor_of(args[kWorkspace], "workspace");
            // (of a tensor that is not contiguous the byte count says nothing about the memory behind its first element)
            if (!workspace.defined() || workspace.nbytes() < need || !workspace.is_contiguous())
                workspace = at::empty({static_cast<int64_t>(need)}, at::TensorOptions().device(device).dtype(at::kByte));
            else
                need_reach(device, workspace, "workspace");
            p.workspace = workspace.data_ptr();
            p.workspace_bytes = workspace.nbytes();
        }
    }
    p.stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fwd(&p);
    Py_END_ALLOW_THREADS
    if (rc != FA_OK) return PyLong_FromLong(rc);
    PyObject* first = !out.defined() ? Py_NewRef(Py_None) : args[kOut] != Py_None ? Py_NewRef(args[kOut]) : THPVariable_Wrap(std::move(out));
    PyObject* second = !lse.defined() ? Py_NewRef(Py_None) : THPVariable_Wrap(std::move(lse));
    PyObject* both = first && second ? PyTuple_Pack(2, first, second) : nullptr;
    Py_XDECREF(first);
    Py_XDECREF(second);
    return both;
}

// forward(address of fa_fwd, address of fa_fwd_workspace_bytes, the arguments of flash_attn_forward in order): (out, lse), or
// the library's error code.
PyObject* forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != kArgs) {
        PyErr_Format(PyExc_TypeError, "forward takes %d arguments, got %zd", static_cast<int>(kArgs), n);
        return nullptr;
    }
    try {
        return forward_impl(args);
    } catch (const python_error_set&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__call() {
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "built_for", FA_BUILT_FOR) != 0) {  // (torch's version: other versions have other classes)
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}

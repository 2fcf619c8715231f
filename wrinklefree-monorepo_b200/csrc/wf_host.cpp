// The per-call host path of the two operators that every projection goes through, as a CPython extension over the C ABI:
// argument checks, allocation of results and workspace, the choice of the kernel family, the launches.
//
// What bounds a small call is this path and not the GPU: written in Python over ctypes, a projection of one token took 20 us
// of host time (device guard 1.5, stream look-up 3.2, three allocations, twenty converted arguments) around a kernel of
// five; here it takes about seven, of which the launch itself is three.
#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/version.h>

#include <algorithm>
#include <cmath>

#include "../../include/wf_b200.h"

namespace {

struct PyFailure {};  // a Python exception is set

[[noreturn]] void raise(PyObject* type, const std::string& msg) {
    PyErr_SetString(type, msg.c_str());
    throw PyFailure();
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return WF_F32;
        case at::kHalf: return WF_F16;
        case at::kBFloat16: return WF_BF16;
        case at::kChar: return WF_I8;
        default: raise(PyExc_KeyError, c10::str("unsupported dtype ", t));
    }
}

const at::Tensor* optional_tensor(PyObject* o) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a tensor or None");
    return &THPVariable_Unpack(o);
}
const at::Tensor& tensor(PyObject* o) {
    const at::Tensor* t = optional_tensor(o);
    if (!t) raise(PyExc_TypeError, "expected a tensor, got None");
    return *t;
}
void need_cuda(std::initializer_list<const at::Tensor*> ts) {
    for (const at::Tensor* t : ts)
        if (t && !t->is_cuda()) raise(PyExc_RuntimeError, "wf_b200 operators need CUDA tensors (there is no CPU path)");
}
long long_arg(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyFailure();
    return v;
}
double float_arg(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyFailure();
    return v;
}
bool truth(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PyFailure();
    return v != 0;
}
void check(int rc, const char* what) {
    if (rc) raise(PyExc_RuntimeError, c10::str(what, " failed (code ", rc, "): ", wf_last_error()));
}

// x as [tokens, K] with unit inner stride
at::Tensor as_rows(const at::Tensor& x) {
    if (x.dim() == 0) raise(PyExc_IndexError, "expected a tensor with at least one dimension");
    at::Tensor r = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
    return r.stride(1) == 1 ? r : r.contiguous();
}
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

struct Quantized {
    at::Tensor q, scale, rowsum;
};
Quantized quantize(const at::Tensor& rows, bool per_tensor, double eps, bool want_rowsum, void* stream) {
    const int64_t m = rows.size(0), k = rows.size(1);
    Quantized r;
    r.q = at::empty({m, k}, rows.options().dtype(at::kChar));
    r.scale = at::empty({per_tensor ? 1 : m}, rows.options().dtype(at::kFloat));
    if (want_rowsum) r.rowsum = at::empty({m}, rows.options().dtype(at::kInt));
    const int dt = dtype_code(rows.scalar_type());
    const int64_t ldx = rows.stride(0);
    int rc;
    {
        pybind11::gil_scoped_release nogil;
        rc = wf_act_quant_i8(rows.data_ptr(), dt, m, k, ldx, per_tensor ? WF_ACT_PER_TENSOR : WF_ACT_PER_TOKEN, static_cast<float>(eps),
                             static_cast<int8_t*>(r.q.data_ptr()), static_cast<float*>(r.scale.data_ptr()), static_cast<int32_t*>(ptr(r.rowsum)), stream);
    }
    check(rc, "wf_act_quant_i8");
    return r;
}

// The contraction's workspace, one of the call's own: two streams of a device never write the same tokens.  The form for many
// tokens wants room for one byte per weight; on a card that has none left the call runs the packed form in the smaller one.
at::Tensor contraction_workspace(int64_t m, int64_t n, int64_t k, const at::TensorOptions& bytes) {
    const int64_t most = static_cast<int64_t>(wf_prefill_workspace_bytes_for(m, n, k)), least = static_cast<int64_t>(wf_prefill_workspace_bytes(m, k));
    if (most > least) {
        try {
            return at::empty({most}, bytes);
        } catch (const c10::OutOfMemoryError&) {
        }
    }
    return at::empty({least}, bytes);
}

PyObject* wrap(const at::Tensor& t) {
    PyObject* o = THPVariable_Wrap(t);
    if (!o) throw PyFailure();
    return o;
}
PyObject* wrap_all(std::initializer_list<at::Tensor> ts) {
    PyObject* out = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
    if (!out) throw PyFailure();
    Py_ssize_t i = 0;
    for (const at::Tensor& t : ts) {
        PyObject* o = THPVariable_Wrap(t);
        if (!o) {
            Py_DECREF(out);
            throw PyFailure();
        }
        PyTuple_SET_ITEM(out, i++, o);
    }
    return out;
}

// act_quant_i8(x, per_tensor, eps, want_rowsum) -> (q, scale[, rowsum])
PyObject* act_quant_i8(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
        if (n != 4) raise(PyExc_TypeError, "act_quant_i8 takes 4 arguments");
        const at::Tensor& x = tensor(a[0]);
        need_cuda({&x});
        const at::Tensor rows = as_rows(x);
        c10::cuda::CUDAGuard guard(x.device());
        const Quantized r = quantize(rows, truth(a[1]), float_arg(a[2]), truth(a[3]), c10::cuda::getCurrentCUDAStream().stream());
        const at::Tensor q = x.dim() == 2 ? r.q : r.q.reshape(x.sizes());
        return r.rowsum.defined() ? wrap_all({q, r.scale, r.rowsum}) : wrap_all({q, r.scale});
    } catch (const PyFailure&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// bitlinear(x, codes, w_scale, bias, out_dtype, layout, x_scale, eps, want_acc, flags, path, out, decode_max_tokens,
//           prequant_min_tokens, prequant_min_elems) -> y | (y, acc);   path: 0 auto, 1 decode, 2 prefill
PyObject* bitlinear(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    try {
        if (n_args != 15) raise(PyExc_TypeError, "bitlinear takes 15 arguments");
        const at::Tensor& x = tensor(a[0]);
        at::Tensor codes = tensor(a[1]);
        const at::Tensor* bias = optional_tensor(a[3]);
        const at::Tensor* x_scale = optional_tensor(a[6]);
        const at::Tensor* out = optional_tensor(a[11]);
        need_cuda({&x, &codes, bias, x_scale});
        if (x.dim() == 0) raise(PyExc_IndexError, "bitlinear: x needs at least one dimension");
        const int64_t k = x.size(-1);
        if (codes.scalar_type() != at::kByte || codes.dim() != 2 || codes.size(1) * 4 != k)
            raise(PyExc_ValueError, c10::str("codes must be uint8 [N, K/4] with K=", k, ", got ", codes.sizes(), " ", codes.scalar_type()));
        const int64_t n = codes.size(0);
        at::Tensor rows = as_rows(x);
        const int64_t m = rows.size(0);
        c10::cuda::CUDAGuard guard(x.device());
        at::ScalarType y_type = x.scalar_type() == at::kChar ? at::kFloat : x.scalar_type();
        if (a[4] != Py_None) {
            if (!THPDtype_Check(a[4])) raise(PyExc_TypeError, "out_dtype must be a torch.dtype");
            y_type = reinterpret_cast<THPDtype*>(a[4])->scalar_type;
        }
        const at::Tensor y = out ? *out : at::empty({m, n}, x.options().dtype(y_type));
        at::Tensor acc;
        if (truth(a[8])) acc = at::empty({m, n}, x.options().dtype(at::kInt));
        const float* ws_dev = nullptr;
        float ws_host = 0.f;
        if (THPVariable_Check(a[2])) {
            const at::Tensor& s = THPVariable_Unpack(a[2]);
            if (s.scalar_type() != at::kFloat || !s.is_cuda()) raise(PyExc_ValueError, "w_scale tensor must be float32 on the GPU");
            ws_dev = static_cast<const float*>(s.data_ptr());
        } else {
            ws_host = static_cast<float>(float_arg(a[2]));
        }
        if (!codes.is_contiguous()) codes = codes.contiguous();
        const int layout = static_cast<int>(long_arg(a[5]));
        const double eps = float_arg(a[7]);
        const unsigned flags = static_cast<unsigned>(long_arg(a[9]));
        const long path = long_arg(a[10]);
        void* const stream = c10::cuda::getCurrentCUDAStream().stream();
        const int bias_type = bias ? dtype_code(bias->scalar_type()) : 0;
        const void* const bias_ptr = bias ? bias->data_ptr() : nullptr;
        const float* xs_ptr = x_scale ? static_cast<const float*>(x_scale->data_ptr()) : nullptr;
        // auto: the tensor-core contraction above decode_max_tokens tokens, and from 16 tokens on for matrices of at least 4 Mi
        // weights (measured: 4096 x 4096 at 32 tokens 14 us against 20 us on the decode kernel; small layers the reverse)
        const bool contraction = path == 2 || (path == 0 && (m > long_arg(a[12]) || (m >= 16 && n * k >= (1 << 22))));
        if (m > 0) {
            const int64_t ldy = y.stride(0);
            const int y_code = dtype_code(y.scalar_type());
            int32_t* const acc_ptr = static_cast<int32_t*>(ptr(acc));
            const uint8_t* const codes_ptr = static_cast<const uint8_t*>(codes.data_ptr());
            int rc;
            if (contraction) {
                const at::Tensor ws = contraction_workspace(m, n, k, x.options().dtype(at::kByte));
                const int x_code = dtype_code(rows.scalar_type());
                pybind11::gil_scoped_release nogil;
                rc = wf_bitlinear_prefill(rows.data_ptr(), x_code, rows.stride(0), xs_ptr, codes_ptr, layout, ws_dev, ws_host, bias_ptr, bias_type,
                                          y.data_ptr(), y_code, ldy, acc_ptr, m, n, k, static_cast<float>(eps), ws.data_ptr(),
                                          static_cast<size_t>(ws.numel()), flags, stream);
            } else {
                Quantized pre;  // alive until the launch: its memory goes back to this stream's pool
                if (rows.scalar_type() != at::kChar && (m >= long_arg(a[13]) || m * k >= long_arg(a[14])) && !wf_decode_fuses_quant(m, k, n * k, 1)) {
                    // every CTA of the decode kernel quantizes the tokens of its problem: from this many tokens on one
                    // quantization kernel in front of it is cheaper (same arithmetic, same bits), unless the launch is of
                    // the kind that does it on the way
                    pre = quantize(rows, false, eps, false, stream);
                    rows = pre.q;
                    xs_ptr = static_cast<const float*>(pre.scale.data_ptr());
                }
                const int x_code = dtype_code(rows.scalar_type());
                pybind11::gil_scoped_release nogil;
                rc = wf_bitlinear_decode(rows.data_ptr(), x_code, rows.stride(0), xs_ptr, codes_ptr, layout, ws_dev, ws_host, bias_ptr, bias_type,
                                         y.data_ptr(), y_code, ldy, acc_ptr, m, n, k, static_cast<float>(eps), flags, stream);
            }
            check(rc, contraction ? "wf_bitlinear_prefill" : "wf_bitlinear_decode");
        }
        at::Tensor shaped = y;
        if (x.dim() != 2 || y.dim() != 2 || y.size(0) != m || y.size(1) != n) {
            std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 1);
            shape.push_back(n);
            shaped = y.reshape(shape);
        }
        return acc.defined() ? wrap_all({shaped, acc}) : wrap(shaped);
    } catch (const PyFailure&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// prompt_layers(layers, h, cos, sin, xq, aq, scale, qkv, gu, att, res, ws, B, S, n_q, n_kv, D, mode, eps, decode_max_tokens,
//               prequant_min_tokens, prequant_min_elems)
// The layers of a decoder's prompt pass (bf16, no sub-layer norms, one GPU) on the caller's buffers; `layers`: per layer a tuple of
// (qkv codes, qkv row scales, o codes, o scale, gate/up codes, gate/up row scales, down codes, down scale, norm 1, norm 2, keys, values).
// The same calls as the loop in the decoder makes, thirteen launches per layer; from Python their nine wrappers took about 100 us of
// host time per layer, which is what bounded a short prompt.  `res` holds the last layer's output of down, not yet added to h.
PyObject* prompt_layers(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    try {
        if (n_args != 22) raise(PyExc_TypeError, "prompt_layers takes 22 arguments");
        struct Layer {
            const uint8_t *qkv, *o, *gu, *down;
            const float *qkv_s, *o_s, *gu_s, *down_s;
            const void *n1, *n2;
            void *kc, *vc;
        };
        const at::Tensor &h = tensor(a[1]), &cos = tensor(a[2]), &sin = tensor(a[3]), &xq = tensor(a[4]), &aq = tensor(a[5]), &scale = tensor(a[6]), &qkv = tensor(a[7]),
                         &gu = tensor(a[8]), &att = tensor(a[9]), &res = tensor(a[10]), &ws = tensor(a[11]);
        const int64_t B = long_arg(a[12]), S = long_arg(a[13]);
        const int nq = static_cast<int>(long_arg(a[14])), nkv = static_cast<int>(long_arg(a[15])), D = static_cast<int>(long_arg(a[16]));
        const int mode = static_cast<int>(long_arg(a[17]));
        const float eps = static_cast<float>(float_arg(a[18]));
        const long decode_max = long_arg(a[19]), pre_tokens = long_arg(a[20]), pre_elems = long_arg(a[21]);
        const int64_t M = h.size(0), hidden = h.size(1), qd = static_cast<int64_t>(nq) * D, kvd = static_cast<int64_t>(nkv) * D, inter = aq.size(1);
        const auto rows_of = [&](const at::Tensor& t, int64_t width) { return t.dim() == 2 && t.size(0) == M && t.size(1) == width && t.is_contiguous(); };
        if (h.dim() != 2 || M != B * S || xq.numel() < M * std::max(hidden, qd) || scale.numel() != M || !rows_of(aq, inter) || !rows_of(qkv, qd + 2 * kvd) ||
            !rows_of(gu, 2 * inter) || !rows_of(att, qd) || !rows_of(res, hidden) || !h.is_contiguous())
            raise(PyExc_ValueError, "prompt_layers: a buffer does not have its shape");
        const auto all_of = [](at::ScalarType type, std::initializer_list<const at::Tensor*> ts) {
            return std::all_of(ts.begin(), ts.end(), [&](const at::Tensor* t) { return t->scalar_type() == type && t->is_contiguous(); });
        };
        if (B < 1 || S < 1 || nq < 1 || nkv < 1 || D < 2 || !all_of(at::kBFloat16, {&h, &qkv, &gu, &att, &res}) || !all_of(at::kChar, {&xq, &aq}) ||
            !all_of(at::kFloat, {&cos, &sin, &scale}) || !all_of(at::kByte, {&ws}) || cos.numel() < S * (D / 2) || sin.numel() < S * (D / 2))
            raise(PyExc_ValueError, "prompt_layers: a buffer does not have its type, or the rotary tables are shorter than the prompt");
        if (!PyList_Check(a[0])) raise(PyExc_TypeError, "prompt_layers: layers must be a list");
        std::vector<Layer> layers(static_cast<size_t>(PyList_GET_SIZE(a[0])));
        int64_t T = 0;
        bool together = true;  // on one device
        for (size_t i = 0; i < layers.size(); ++i) {
            PyObject* t = PyList_GET_ITEM(a[0], static_cast<Py_ssize_t>(i));
            if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 12) raise(PyExc_TypeError, "prompt_layers: a layer is a tuple of twelve tensors");
            const at::Tensor* e[12];
            for (int j = 0; j < 12; ++j) e[j] = &tensor(PyTuple_GET_ITEM(t, j));
            if (!all_of(at::kByte, {e[0], e[2], e[4], e[6]}) || !all_of(at::kFloat, {e[1], e[3], e[5], e[7]}) || !all_of(at::kBFloat16, {e[8], e[9], e[10], e[11]}))
                raise(PyExc_ValueError, "prompt_layers: a layer's tensor does not have its type, or is not contiguous");
            if (e[10]->dim() != 4 || (i && e[10]->size(2) != T)) raise(PyExc_ValueError, "prompt_layers: caches are [B, heads, T, D] with one T for all layers");
            T = e[10]->size(2);
            if (e[0]->numel() * 4 != (qd + 2 * kvd) * hidden || e[1]->numel() != qd + 2 * kvd || e[2]->numel() * 4 != hidden * qd || e[3]->numel() < 1 ||
                e[4]->numel() * 4 != 2 * inter * hidden || e[5]->numel() != 2 * inter || e[6]->numel() * 4 != hidden * inter || e[7]->numel() < 1 ||
                e[8]->numel() != hidden || e[9]->numel() != hidden || e[10]->numel() != B * T * kvd || e[11]->numel() != B * T * kvd || S > T)
                raise(PyExc_ValueError, "prompt_layers: a layer's tensor does not have its shape");
            for (const at::Tensor* one : e) together = together && one->device() == h.device();
            layers[i] = {static_cast<const uint8_t*>(e[0]->data_ptr()), static_cast<const uint8_t*>(e[2]->data_ptr()), static_cast<const uint8_t*>(e[4]->data_ptr()),
                         static_cast<const uint8_t*>(e[6]->data_ptr()), e[1]->data_ptr<float>(), e[3]->data_ptr<float>(), e[5]->data_ptr<float>(), e[7]->data_ptr<float>(),
                         e[8]->data_ptr(), e[9]->data_ptr(), e[10]->data_ptr(), e[11]->data_ptr()};
        }
        for (const at::Tensor* one : {&cos, &sin, &xq, &aq, &scale, &qkv, &gu, &att, &res, &ws}) together = together && one->device() == h.device();
        need_cuda({&h});
        if (!together) raise(PyExc_ValueError, "prompt_layers: tensors on different devices");
        c10::cuda::CUDAGuard guard(h.device());
        void* const stream = c10::cuda::getCurrentCUDAStream().stream();
        int8_t* const q8 = xq.data_ptr<int8_t>();
        int8_t* const a8 = aq.data_ptr<int8_t>();
        float* const xs = scale.data_ptr<float>();
        const auto bytes = h.options().dtype(at::kByte);
        const char* what = "";
        int rc = 0;
        // one projection of the tokens, by the rule of bitlinear(); from bf16 (x_scale null) or int8
        const auto project = [&](const void* x, int type, const float* x_scale, const uint8_t* codes, const float* w_scale, int64_t k) {
            if (M > decode_max || (M >= 16 && hidden * k >= (1 << 22))) {
                const at::Tensor own = contraction_workspace(M, hidden, k, bytes);
                what = "wf_bitlinear_prefill";
                return wf_bitlinear_prefill(x, type, k, x_scale, codes, WF_LAYOUT_WF16, w_scale, 0.f, nullptr, 0, res.data_ptr(), WF_BF16, hidden, nullptr, M, hidden, k, 1e-5f,
                                            own.data_ptr(), static_cast<size_t>(own.numel()), 0, stream);
            }
            if (type != WF_I8 && (M >= pre_tokens || M * k >= pre_elems) && !wf_decode_fuses_quant(M, k, hidden * k, 1)) {
                what = "wf_act_quant_i8";
                if (const int e = wf_act_quant_i8(x, type, M, k, k, WF_ACT_PER_TOKEN, 1e-5f, q8, xs, nullptr, stream)) return e;
                x = q8;
                type = WF_I8;
                x_scale = xs;
            }
            what = "wf_bitlinear_decode";
            return wf_bitlinear_decode(x, type, k, x_scale, codes, WF_LAYOUT_WF16, w_scale, 0.f, nullptr, 0, res.data_ptr(), WF_BF16, hidden, nullptr, M, hidden, k, 1e-5f, 0, stream);
        };
        {
            pybind11::gil_scoped_release nogil;
            const auto step = [&](int e, const char* name) {
                what = name;
                return e;
            };
            char* const qkv_p = static_cast<char*>(qkv.data_ptr());
            char* const gu_p = static_cast<char*>(gu.data_ptr());
            const size_t ws_bytes = static_cast<size_t>(ws.numel());
            bool first = true;
            for (const Layer& L : layers) {
                if ((rc = step(wf_add_rmsnorm_quant_bf16(h.data_ptr(), first ? nullptr : res.data_ptr(), L.n1, nullptr, q8, xs, M, hidden, eps, 1e-5f, first ? 0 : WF_FLAG_PDL, stream), "wf_add_rmsnorm_quant_bf16"))) break;
                first = false;
                if ((rc = step(wf_bitlinear_prefill_rows(q8, hidden, xs, L.qkv, L.qkv_s, qkv_p, WF_BF16, qd + 2 * kvd, M, qd + 2 * kvd, hidden, ws.data_ptr(), ws_bytes, stream), "wf_bitlinear_prefill_rows"))) break;
                if ((rc = step(wf_rope_kv_prompt_ld_bf16(qkv_p, qd + 2 * kvd, qkv_p + 2 * qd, qkv_p + 2 * (qd + kvd), qd + 2 * kvd, cos.data_ptr<float>(), sin.data_ptr<float>(), L.kc, L.vc, B, S, nq,
                                                         nkv, D, T, WF_FLAG_PDL, stream), "wf_rope_kv_prompt_bf16"))) break;
                if ((rc = step(wf_attn_prompt_bf16(qkv_p, qd + 2 * kvd, L.kc, L.vc, att.data_ptr(), B, S, nq, nkv, D, T, static_cast<float>(std::pow(static_cast<double>(D), -0.5)), WF_FLAG_PDL, stream), "wf_attn_prompt_bf16"))) break;
                if ((rc = project(att.data_ptr(), WF_BF16, nullptr, L.o, L.o_s, qd))) break;
                if ((rc = step(wf_add_rmsnorm_quant_bf16(h.data_ptr(), res.data_ptr(), L.n2, nullptr, q8, xs, M, hidden, eps, 1e-5f, WF_FLAG_PDL, stream), "wf_add_rmsnorm_quant_bf16"))) break;
                if ((rc = step(wf_bitlinear_prefill_rows(q8, hidden, xs, L.gu, L.gu_s, gu_p, WF_BF16, 2 * inter, M, 2 * inter, hidden, ws.data_ptr(), ws_bytes, stream), "wf_bitlinear_prefill_rows"))) break;
                if ((rc = step(wf_act_mul_quant_ld_bf16(gu_p, gu_p + 2 * inter, 2 * inter, nullptr, a8, xs, M, inter, mode, 1e-5f, WF_FLAG_PDL, stream), "wf_act_mul_quant_bf16"))) break;
                if ((rc = project(a8, WF_I8, xs, L.down, L.down_s, inter))) break;
            }
        }
        check(rc, what);
        Py_RETURN_NONE;
    } catch (const PyFailure&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"prompt_layers", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(prompt_layers)), METH_FASTCALL, nullptr},
    {"act_quant_i8", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(act_quant_i8)), METH_FASTCALL, nullptr},
    {"bitlinear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bitlinear)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "wf_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_wf_host() {
    PyObject* m = PyModule_Create(&module);
    // the tensors it takes and returns are torch's C++ objects: the loader compares this with the torch that is running
    if (m && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) Py_CLEAR(m);
    return m;
}

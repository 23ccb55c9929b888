// The call site of one ternary linear as a CPython extension type.
//
// An eager call of a small layer costs a few microseconds on the GPU; done in
// Python - shape checks, torch.empty, the current stream, fifteen ctypes
// arguments, the quantiser as eight torch operators - its host side took 18 us
// (int8 input) to 85 us (bf16 input).  `Layer` does all of it in one native call.
//
// A Layer also keeps the module's weights in the two-bit layout of w2_small.cuh, laid out
// from the packed checkpoint tensors.  Nothing on a tensor tells whether its values have
// changed: an address can come back with other values, and a version counter misses
// writes through .data, by collectives, through raw pointers and of inference mode.  So
// the copy is used only while nothing outside of the module can write to the packed
// tensors.  The module keeps its parameters in a dict (linear.py, _OwnedParameters) that
// invalidates the copy whenever it hands one out; the next call lays the weights out
// again once the module alone holds every parameter and its storage, and reads the
// packed tensors until then (and during a capture, where nothing is laid out).
//
// Every method returns None where the native path does not apply (other devices,
// types or sizes); the caller then takes the general path in linear.py.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <limits.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "ternaspmm.h"

namespace {

PyObject* g_keys[5];                   // interned parameter names, in the order of Weights
PyObject* g_layer;                     // interned name of the owning dict's attribute

struct Weights {
    const at::Tensor *signs, *tile_offsets, *quarter_offsets, *bitmap, *scale;
};

struct Layer {
    PyObject_HEAD
    int in_features, out_features, ws_num, seg[3];
    bool valid;                        // w2 holds the weights, and nothing outside of the module can change them
    bool replaced;                     // w2 holds weights that calls in flight on other streams may still read
    at::Tensor* w2;
};

bool get_weights(PyObject* params, Weights& w) {
    const at::Tensor** dst[5] = {&w.signs, &w.tile_offsets, &w.quarter_offsets, &w.bitmap, &w.scale};
    for (int i = 0; i < 5; ++i) {
        PyObject* o = PyDict_GetItem(params, g_keys[i]);   // borrowed
        if (!o || !THPVariable_Check(o)) return false;
        *dst[i] = &THPVariable_Unpack(o);
        if (!(*dst[i])->is_cuda() || !(*dst[i])->is_contiguous() || (*dst[i])->device() != w.signs->device()) return false;
    }
    return w.scale->scalar_type() == at::kBFloat16 && w.scale->numel() >= 4;
}

bool capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone;
}

// Whether `params` is the dict that reports to this layer what it hands out (and not a plain one put in its place).
bool reports(Layer* self, PyObject* params) {
    if (PyDict_CheckExact(params)) return false;
    PyObject* layer = PyObject_GetAttr(params, g_layer);
    const bool same = layer == reinterpret_cast<PyObject*>(self);
    if (!layer) PyErr_Clear();
    Py_XDECREF(layer);
    return same;
}

// Whether the dict holds the only reference to each of the packed tensors, and these the only ones to their storage.
bool exclusive(PyObject* params) {
    for (int i = 0; i < 4; ++i) {
        PyObject* o = PyDict_GetItem(params, g_keys[i]);
        if (!o || !THPVariable_Check(o) || Py_REFCNT(o) != 1) return false;
        const at::Tensor& t = THPVariable_Unpack(o);
        if (t.use_count() != 1 || !t.has_storage()) return false;
        // (a storage that Python has seen keeps its wrapper, which holds the second reference)
        const c10::StorageImpl* storage = t.storage().unsafeGetStorageImpl();
        const size_t refs = t.storage().use_count();
        if (refs != 1 && !(refs == 2 && storage->pyobj_slot()->has_unique_reference())) return false;
    }
    return true;
}

// Writes the two-bit copy.  False where there is none (sizes, a capture under way).
bool lay_out(Layer* self, const Weights& w, cudaStream_t stream) {
    const int64_t N = self->out_features, K = self->in_features, tiles = N * K / 4096;
    if (N < 64 || K < 64 || N % 64 || K % 64 || K >= (1 << 18) || w.bitmap->nbytes() < (size_t)(N * K / 8) ||
        w.tile_offsets->numel() < tiles + 1 || w.quarter_offsets->numel() < 3 * tiles ||
        (reinterpret_cast<uintptr_t>(w.bitmap->data_ptr()) & 15) || capturing(stream))
        return false;
    if (self->replaced) {              // (relaxed: another thread may be capturing)
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        const cudaError_t e = cudaDeviceSynchronize();
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) return false;
        self->replaced = false;
    }
    if (!self->w2->defined() || self->w2->device() != w.bitmap->device())
        *self->w2 = at::empty({ternaspmm_w2_bytes((int)N, (int)K)}, w.bitmap->options().dtype(at::kByte));
    ternaspmm_w2_relayout(static_cast<uint64_t*>(w.bitmap->data_ptr()), static_cast<int*>(w.tile_offsets->data_ptr()),
                          static_cast<uint16_t*>(w.quarter_offsets->data_ptr()), static_cast<uint32_t*>(w.signs->data_ptr()), (int)N,
                          (int)K, self->w2->data_ptr(), stream);
    return cudaStreamSynchronize(stream) == cudaSuccess;   // other streams may use the layer next
}

// The two-bit weights; null where the call reads the packed tensors.
void* two_bit(Layer* self, PyObject* params, const Weights& w, cudaStream_t stream) {
    if (!reports(self, params)) return nullptr;
    if (!self->valid) self->valid = exclusive(params) && lay_out(self, w, stream);
    return self->valid ? self->w2->data_ptr() : nullptr;
}

at::Tensor output_like(const at::Tensor& x, int64_t N) {
    c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = N;
    return at::empty(shape, x.options().dtype(at::kBFloat16));
}

// A contiguous, 16-byte aligned CUDA tensor of this type whose last dimension is K.
bool usable(PyObject* o, at::ScalarType type, int64_t K) {
    if (!THPVariable_Check(o)) return false;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && t.scalar_type() == type && t.dim() >= 1 && t.size(-1) == K && t.numel() > 0 && t.is_contiguous() &&
           !(reinterpret_cast<uintptr_t>(t.data_ptr()) & 15);
}

void run_linear(Layer* self, const Weights& w, void* w2, void* x, int front_end, void* norm_w, float eps, at::Tensor& out, void* s,
                int64_t M, void* residual, cudaStream_t stream) {
    auto* o = static_cast<ternaspmm_bf16*>(out.data_ptr());
    auto* scale = static_cast<ternaspmm_bf16*>(w.scale->data_ptr());
    ternaspmm_w2_linear(x, front_end, static_cast<ternaspmm_bf16*>(norm_w), eps, w2, o, static_cast<ternaspmm_bf16*>(s), scale, self->ws_num,
                        (int)M, self->out_features, self->in_features, self->seg[0], self->seg[1], self->seg[2], -1,
                        static_cast<ternaspmm_bf16*>(residual), stream);
}

void* residual_ptr(PyObject* o, const at::Tensor& x, int64_t M, int64_t N, bool& ok) {   // None, or contiguous bf16 of M*N values
    ok = true;
    if (o == Py_None) return nullptr;
    ok = usable(o, at::kBFloat16, N) && THPVariable_Unpack(o).numel() == M * N && THPVariable_Unpack(o).device() == x.device();
    return ok ? THPVariable_Unpack(o).data_ptr() : nullptr;
}

// int8 rows and scales in one allocation: [M][K] int8, then [M] bf16.
at::Tensor quantised_buffer(const at::Tensor& x, int64_t M, int64_t K) {
    return at::empty({M * K + 2 * M}, x.options().dtype(at::kByte));
}

// front-end + linear of bf16 activations: in one kernel for the smallest calls, else as two launches
PyObject* front_and_linear(Layer* self, PyObject* params, PyObject* xo, int front_end, PyObject* norm_o, float eps, PyObject* res_o) {
    const int64_t K = self->in_features;
    const bool gated = front_end == 3;
    if (!usable(xo, at::kBFloat16, gated ? 2 * K : K)) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(xo);
    const int64_t M = x.numel() / x.size(-1);
    if (M > INT_MAX / 2) Py_RETURN_NONE;
    void* norm_w = nullptr;
    if (norm_o) {
        if (!usable(norm_o, at::kBFloat16, K) || THPVariable_Unpack(norm_o).numel() != K || THPVariable_Unpack(norm_o).device() != x.device())
            Py_RETURN_NONE;
        norm_w = THPVariable_Unpack(norm_o).data_ptr();
    }
    bool ok;
    void* residual = residual_ptr(res_o, x, M, self->out_features, ok);
    Weights w;
    if (!ok || !get_weights(params, w) || w.bitmap->device() != x.device()) Py_RETURN_NONE;
    c10::cuda::OptionalCUDAGuard guard(x.device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    void* w2 = two_bit(self, params, w, stream);
    if (!w2) Py_RETURN_NONE;
    at::Tensor out = output_like(x, self->out_features);
    // The front-end inside the linear's kernel saves a launch of its own, 1.1 us of the stream and as much of the host; every CTA does
    // it, up to four rows at once where a row is one vector per thread (K up to 2560), one after the other above that.  That pays up to 10240
    // values.  us per call, inside / separate: quantiser 2560 x 2560 at 1 / 4 / 8 rows 2.7 / 4.0, 3.2 / 4.3, 5.0 / 4.3, 5120 x 5120 at 2 4.7 / 5.9,
    // 5120 x 4096 at 2 4.2 / 5.9, 2560 x 3072 at 3 4.2 / 4.7 (called eagerly 5.1 / 8.4), 2560 x 6912 at 1 / 3 4.0 / 5.4, 6.0 / 5.9,
    // 10240 x 8192 at 1 / 2 8.9 / 10.8, 12.0 / 11.8, 57344 x 8192 at 1 / 4 37.8 / 34.4, 38.9 / 36.0; norm 2560 x 2560 at 1 3.1 / 4.4, 2560 x 6912 at
    // 1 / 2 (gated) 5.1 / 6.5, 6.8 / 6.8, 10240 x 8192 at 1 12.3 / 11.2.  Norms of 2 to 4 rows gain alone (2560 x 2560 at 4 4.2 / 4.8), but a
    // separate one overlaps the kernel before it: 30-layer model at batch 2 / 4 1043 / 1126 us a token, so 1009 / 1074.
    if (M <= ternaspmm_w2_fused_rows((int)K) && K < 8192 && (M == 1 || (front_end == 1 && M <= 4 && M * K <= 10240))) {
        run_linear(self, w, w2, x.data_ptr(), front_end, norm_w, eps, out, nullptr, M, residual, stream);
        return THPVariable_Wrap(std::move(out));
    }
    if (K > 56 * 1024) Py_RETURN_NONE;
    at::Tensor buf = quantised_buffer(x, M, K);
    int8_t* q = static_cast<int8_t*>(buf.data_ptr());
    ternaspmm_bf16* s = reinterpret_cast<ternaspmm_bf16*>(q + M * K);
    ternaspmm_bf16* xp = static_cast<ternaspmm_bf16*>(x.data_ptr());
    if (front_end == 1) ternaspmm_quant(xp, (int)M, (int)K, q, s, stream);
    else if (gated) ternaspmm_relu2_gate_rmsnorm_quant(xp, static_cast<ternaspmm_bf16*>(norm_w), eps, (int)M, (int)K, q, s, stream);
    else ternaspmm_rmsnorm_quant(xp, static_cast<ternaspmm_bf16*>(norm_w), eps, (int)M, (int)K, q, s, stream);
    run_linear(self, w, w2, q, 0, nullptr, 0.f, out, s, M, residual, stream);
    return THPVariable_Wrap(std::move(out));
}

// forward(params, x): per-token int8 quantiser, then the linear
PyObject* layer_forward(PyObject* o, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2) return PyErr_Format(PyExc_TypeError, "forward(params, x)");
    return front_and_linear(reinterpret_cast<Layer*>(o), args[0], args[1], 1, nullptr, 0.f, Py_None);
    END_HANDLE_TH_ERRORS
}

// forward_normed(params, x, norm_weight, eps, gated, residual): (gate,) RMSNorm, quantiser, linear, residual add
PyObject* layer_forward_normed(PyObject* o, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 6) return PyErr_Format(PyExc_TypeError, "forward_normed(params, x, norm_weight, eps, gated, residual)");
    const double eps = PyFloat_AsDouble(args[3]);
    if (PyErr_Occurred()) return nullptr;
    return front_and_linear(reinterpret_cast<Layer*>(o), args[0], args[1], PyObject_IsTrue(args[4]) ? 3 : 2, args[2], (float)eps, args[5]);
    END_HANDLE_TH_ERRORS
}

// forward_quantized(params, x_q, s, residual): int8 activations and their scales in hand
PyObject* layer_forward_quantized(PyObject* o, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) return PyErr_Format(PyExc_TypeError, "forward_quantized(params, x_q, s, residual)");
    Layer* self = reinterpret_cast<Layer*>(o);
    const int64_t K = self->in_features;
    if (!usable(args[1], at::kChar, K) || !THPVariable_Check(args[2])) Py_RETURN_NONE;
    const at::Tensor &x = THPVariable_Unpack(args[1]), &s = THPVariable_Unpack(args[2]);
    const int64_t M = x.numel() / K;
    if (M > INT_MAX / 2 || s.scalar_type() != at::kBFloat16 || !s.is_contiguous() || s.numel() != M || s.device() != x.device())
        Py_RETURN_NONE;
    bool ok;
    void* residual = residual_ptr(args[3], x, M, self->out_features, ok);
    Weights w;
    if (!ok || !get_weights(args[0], w) || w.bitmap->device() != x.device()) Py_RETURN_NONE;
    c10::cuda::OptionalCUDAGuard guard(x.device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    void* w2 = two_bit(self, args[0], w, stream);
    if (!w2) Py_RETURN_NONE;
    at::Tensor out = output_like(x, self->out_features);
    run_linear(self, w, w2, x.data_ptr(), 0, nullptr, 0.f, out, s.data_ptr(), M, residual, stream);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// prepare(params): lay the weights out now instead of in the first call; without GPU tensors, give the copy back.
// The address of the copy that calls use, 0 where they read the packed tensors.
PyObject* layer_prepare(PyObject* o, PyObject* params) {
    HANDLE_TH_ERRORS
    Layer* self = reinterpret_cast<Layer*>(o);
    Weights w;
    if (!get_weights(params, w)) {
        self->valid = self->replaced = false;
        *self->w2 = at::Tensor();
        return PyLong_FromLong(0);
    }
    c10::cuda::OptionalCUDAGuard guard(w.bitmap->device());
    return PyLong_FromVoidPtr(two_bit(self, params, w, c10::cuda::getCurrentCUDAStream().stream()));
    END_HANDLE_TH_ERRORS
}

// relayout(params): write the copy again from the packed tensors, in place, whoever holds them - captured graphs read it.
// False where there is none.
PyObject* layer_relayout(PyObject* o, PyObject* params) {
    HANDLE_TH_ERRORS
    Layer* self = reinterpret_cast<Layer*>(o);
    Weights w;
    self->valid = false;
    if (!reports(self, params) || !get_weights(params, w)) Py_RETURN_FALSE;
    c10::cuda::OptionalCUDAGuard guard(w.bitmap->device());
    if (!lay_out(self, w, c10::cuda::getCurrentCUDAStream().stream())) Py_RETURN_FALSE;
    self->valid = exclusive(params);
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// invalidate(): a parameter has been handed out
PyObject* layer_invalidate(PyObject* o, PyObject*) {
    reinterpret_cast<Layer*>(o)->valid = false;
    Py_RETURN_NONE;
}

// replace(): a parameter has been replaced; the copy follows in the same memory, for the sake of captured graphs
PyObject* layer_replace(PyObject* o, PyObject*) {
    reinterpret_cast<Layer*>(o)->valid = false;
    reinterpret_cast<Layer*>(o)->replaced = true;
    Py_RETURN_NONE;
}

// exclusive(params): what the copy depends on
PyObject* layer_exclusive(PyObject* o, PyObject* params) {
    HANDLE_TH_ERRORS
    return PyBool_FromLong(PyDict_Check(params) && reports(reinterpret_cast<Layer*>(o), params) && exclusive(params));
    END_HANDLE_TH_ERRORS
}

PyObject* layer_new(PyTypeObject* type, PyObject* args, PyObject*) {
    Layer* self = reinterpret_cast<Layer*>(type->tp_alloc(type, 0));
    if (!self) return nullptr;
    self->w2 = new at::Tensor();
    self->valid = self->replaced = false;
    if (!PyArg_ParseTuple(args, "iiiiii", &self->in_features, &self->out_features, &self->ws_num, &self->seg[0], &self->seg[1], &self->seg[2])) {
        Py_DECREF(self);
        return nullptr;
    }
    return reinterpret_cast<PyObject*>(self);
}

void layer_dealloc(PyObject* o) {
    delete reinterpret_cast<Layer*>(o)->w2;
    Py_TYPE(o)->tp_free(o);
}

// pack(weight): the four packed tensors of a contiguous, 16-byte aligned int8 CUDA tensor [N][K] whose sizes are multiples of 64.
PyObject* pack_weight(PyObject*, PyObject* o) {
    HANDLE_TH_ERRORS
    if (!THPVariable_Check(o)) Py_RETURN_NONE;
    const at::Tensor& w = THPVariable_Unpack(o);
    if (!w.is_cuda() || w.scalar_type() != at::kChar || w.dim() != 2 || !w.is_contiguous() || w.size(0) % 64 || w.size(1) % 64 || !w.numel() ||
        w.size(0) > INT_MAX || w.size(1) > INT_MAX || (reinterpret_cast<uintptr_t>(w.data_ptr()) & 15))
        Py_RETURN_NONE;
    const int64_t N = w.size(0), K = w.size(1), tiles = N / 64 * (K / 64);
    c10::cuda::CUDAGuard guard(w.device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream();
    at::Tensor bitmap = at::empty({tiles * 64}, w.options().dtype(at::kUInt64)), tile_off = at::empty({tiles + 1}, w.options().dtype(at::kInt));
    at::Tensor quarters = at::empty({tiles * 3}, w.options().dtype(at::kUInt16));
    const auto* src = static_cast<const int8_t*>(w.data_ptr());
    auto* offsets = static_cast<int*>(tile_off.data_ptr());
    long long words;
    Py_BEGIN_ALLOW_THREADS
    words = ternaspmm_pack_gpu_layout(src, (int)N, (int)K, static_cast<uint64_t*>(bitmap.data_ptr()), offsets,
                                      static_cast<uint16_t*>(quarters.data_ptr()), stream);
    Py_END_ALLOW_THREADS
    TORCH_CHECK(words >= 0, "packing a ", N, " x ", K, " weight on the GPU failed with status ", ternaspmm_last_status());
    at::Tensor signs = at::empty({words + 4}, w.options().dtype(at::kUInt32));   // four zero words behind the last tile's
    ternaspmm_pack_gpu_signs(src, (int)N, (int)K, offsets, static_cast<uint32_t*>(signs.data_ptr()), stream);
    return Py_BuildValue("NNNN", THPVariable_Wrap(signs), THPVariable_Wrap(tile_off), THPVariable_Wrap(quarters), THPVariable_Wrap(bitmap));
    END_HANDLE_TH_ERRORS
}

PyMethodDef module_methods[] = {{"pack", pack_weight, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};

PyMethodDef layer_methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(layer_forward)), METH_FASTCALL, nullptr},
    {"forward_normed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(layer_forward_normed)), METH_FASTCALL, nullptr},
    {"forward_quantized", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(layer_forward_quantized)), METH_FASTCALL, nullptr},
    {"prepare", layer_prepare, METH_O, nullptr},
    {"relayout", layer_relayout, METH_O, nullptr},
    {"invalidate", layer_invalidate, METH_NOARGS, nullptr},
    {"replace", layer_replace, METH_NOARGS, nullptr},
    {"exclusive", layer_exclusive, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject layer_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host_call", "Native call sites: the ternary linears and the packer.", -1, module_methods};

}  // namespace

PyMODINIT_FUNC PyInit__host_call() {
    static const char* const names[5] = {"weight_compressed_val", "weight_TileOffsets_global", "weight_TileOffsets_median", "weight_bitmap",
                                         "weight_scale"};
    for (int i = 0; i < 5; ++i) g_keys[i] = PyUnicode_InternFromString(names[i]);
    g_layer = PyUnicode_InternFromString("layer");
    layer_type.tp_name = "_host_call.Layer";
    layer_type.tp_basicsize = sizeof(Layer);
    layer_type.tp_flags = Py_TPFLAGS_DEFAULT;
    layer_type.tp_new = layer_new;
    layer_type.tp_dealloc = layer_dealloc;
    layer_type.tp_methods = layer_methods;
    if (PyType_Ready(&layer_type) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&layer_type);
    PyModule_AddObject(m, "Layer", reinterpret_cast<PyObject*>(&layer_type));
    return m;
}

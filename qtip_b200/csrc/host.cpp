// Host path of one QTIP linear: BitshiftLinear.forward (lib/codebook/bitshift.py:428-472 upstream) as one native call.
//
// A layer call is two transforms around a decode + product, 8..60 us of GPU work.  Issued from Python - three wrappers,
// each with its own device switch, stream query, argument checks, tensor construction and ctypes conversion - it cost
// 80-93 us of host time per call (measured at every layer shape that runs for less), so the GPU waited for the
// interpreter.  Here the whole call is made from C++: one scratch allocation for the two intermediates, one for the
// result, and the library's launches back to back on the current stream.
//
// Module functions (CPython API, no binding layer):
//   linear_forward(input, trellis, tlut|None, SU, SV, bits_left|None, k_left, bits_right|None, k_right, code, K,
//                  kernel_layout, rcp, tp, workspace|None) -> (output, launches)
//   matvec_workspace(device_index, m, n, bs) -> uint8 tensor    the fused matvec's scratch of (device, current stream)
//   gemm_status(device_index) -> int32 tensor                   the decompress-GEMM's status word of a device
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>

#include <cmath>
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/qtip_b200.h"

namespace {

constexpr int64_t kMaxMatvecBatch = 8, kMaxGemmBatch = 128;
constexpr double kInternalScale = 32.0;    // bitshift.py:373 upstream: keeps the fp16 activation in range

struct Failure {
    std::string what;
};

void check(int status, const char *what) {
    if (status == QTIP_OK) return;
    std::string msg = std::string(what) + ": " + qtip_status_string(status);
    if (status == QTIP_ERR_CUDA) msg += " (cudaError " + std::to_string(qtip_last_cuda_error()) + ")";
    throw Failure{msg};
}

int dtype_id(const at::Tensor &t) {
    if (t.scalar_type() == at::kHalf) return QTIP_F16;
    if (t.scalar_type() == at::kFloat) return QTIP_F32;
    throw Failure{std::string("unsupported dtype ") + c10::toString(t.scalar_type()) + " (fp16 / fp32 only)"};
}

// Per-device / per-stream scratch that outlives a call.  One matvec workspace per (device, stream): calls on one stream
// are ordered, so they can share it; torch hands out a bounded set of streams.  It is zeroed once and the kernels leave
// it zeroed.  Never destroyed at exit (the CUDA context may be gone by then).
// A CUDA graph keeps the addresses it was captured with: a workspace that has to grow is replaced by one of at least twice its
// size and kept (all replaced ones of a stream are smaller together than the one in use), and a capture that finds none gets one
// of its own from the graph's memory, zeroed by the graph (a zeroing recorded into a graph is no zeroing of what others use).
//
// g_mutex is taken with and without the GIL, so nothing that may call into Python (and wait for the GIL) happens under it:
// no allocation or release of a tensor (memory history, allocator hooks) and no copy of a tensor handle (its Python object).
// The maps hold shared pointers; those are what is read and exchanged under the lock.
using TensorPtr = std::shared_ptr<const at::Tensor>;
std::mutex g_mutex;
std::map<std::pair<int, void *>, TensorPtr> &workspaces() {
    static auto *m = new std::map<std::pair<int, void *>, TensorPtr>();
    return *m;
}
std::vector<TensorPtr> &replaced() {
    static auto *v = new std::vector<TensorPtr>();
    return *v;
}
std::map<int, TensorPtr> &status_words() {
    static auto *m = new std::map<int, TensorPtr>();
    return *m;
}

// The entry of `key`, made by `make` when it is missing or `ok` refuses it.  Of two threads that make one at the same time
// the first to store it wins; what the other made is released outside the lock.
template <class Map, class Key, class Ok, class Make>
TensorPtr find_or_make(Map &map, const Key &key, Ok ok, Make make) {
    size_t had = 0;      // bytes of the entry that is too small
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        const auto it = map.find(key);
        if (it != map.end()) {
            if (ok(*it->second)) return it->second;
            had = it->second->nbytes();
        }
    }
    bool keep = true;
    TensorPtr made = std::make_shared<const at::Tensor>(make(had, keep)), got;
    if (!keep) return made;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        TensorPtr &slot = map[key];
        if (!slot || !ok(*slot)) {
            if (slot) replaced().push_back(std::move(slot));
            slot = std::move(made);
        }
        got = slot;
    }
    return got;
}

at::Tensor matvec_workspace(int dev, int64_t m, int64_t n, int64_t bs, void *stream) {
    const size_t need = qtip_matvec_workspace_bytes((int)m, (int)n, (int)bs);
    return *find_or_make(workspaces(), std::make_pair(dev, stream), [&](const at::Tensor &t) { return (size_t)t.numel() >= need; },
                         [&](size_t had, bool &keep) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &capture) != cudaSuccess) throw Failure{"cudaStreamIsCapturing failed"};
        keep = capture == cudaStreamCaptureStatusNone;
        const size_t bytes = keep ? std::max<size_t>({need, 2 * had, (size_t)1 << 20}) : need;
        return at::zeros({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev));
    });
}

at::Tensor gemm_status(int dev) {
    return *find_or_make(status_words(), dev, [](const at::Tensor &) { return true; },
                         [&](size_t, bool &) { return at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, dev)); });
}

struct Layer {
    const at::Tensor &trellis, &SU, &SV;
    at::Tensor tlut, bits_left, bits_right, workspace;   // undefined = absent
    int k_left, k_right, code, K, rcp, tp;
    bool kernel_layout;
};

bool aligned16(const at::Tensor &t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

at::Tensor linear_forward(const at::Tensor &input, Layer &L, int &launches) {
    const int64_t n = L.SU.numel(), m = L.SV.numel();
    for (const at::Tensor *t : {&input, &L.trellis, &L.SU, &L.SV, (const at::Tensor *)&L.tlut, (const at::Tensor *)&L.bits_left,
                                (const at::Tensor *)&L.bits_right})
        if (t->defined() && !t->is_cuda()) throw Failure{"qtip_b200 runs on CUDA tensors only (no CPU fallback)"};
    const int dev = input.get_device();
    c10::cuda::OptionalCUDAGuard guard;
    if (dev != c10::cuda::current_device()) guard.set_index((c10::DeviceIndex)dev);
    void *stream = at::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();

    at::Tensor x = input.is_contiguous() ? input : input.contiguous();
    if (n == 0 || x.numel() % n) throw Failure{"the input's last dimension does not match SU"};
    const int64_t bs = x.numel() / n;
    const auto in_type = input.scalar_type();
    if (in_type != at::kHalf && in_type != at::kFloat) x = x.to(at::kFloat);
    const auto out_type = in_type == at::kHalf ? at::kHalf : at::kFloat;
    const at::Tensor SU = L.SU.is_contiguous() ? L.SU : L.SU.contiguous();
    const at::Tensor SV = L.SV.scalar_type() == at::kFloat && L.SV.is_contiguous() ? L.SV : L.SV.to(at::kFloat).contiguous();
    const at::Tensor trellis = L.trellis.is_contiguous() ? L.trellis : L.trellis.contiguous();
    if (trellis.nbytes() != (size_t)(m * n * L.K / 8))
        throw Failure{"codes hold " + std::to_string(trellis.nbytes()) + " bytes, expected " + std::to_string(m * n * L.K / 8)};
    at::Tensor tlut = L.tlut;
    if (tlut.defined() && (tlut.scalar_type() != at::kHalf || !tlut.is_contiguous())) tlut = tlut.to(at::kHalf).contiguous();
    const uint32_t *bl = L.bits_left.defined() ? static_cast<const uint32_t *>(L.bits_left.data_ptr()) : nullptr;
    const uint32_t *br = L.bits_right.defined() ? static_cast<const uint32_t *>(L.bits_right.data_ptr()) : nullptr;

    const auto opts = at::TensorOptions().device(at::kCUDA, dev);
    std::vector<int64_t> shape(input.sizes().begin(), input.sizes().end());
    shape.back() = m;
    at::Tensor out = at::empty(shape, opts.dtype(out_type));
    if (bs == 0) return in_type == out_type ? out : out.to(in_type);

    const bool v1 = L.code != QTIP_CODE_HYB;
    const bool whole_tiles = m % 128 == 0 && n % 64 == 0;      // what the tensor-core kernel needs
    // compute codes: the tensor-core kernel decodes eight states per 44-bit window and is the faster one at every batch
    // size it takes; HYB: above 8 rows the matvec's single B fragment is full
    const bool gemm = whole_tiles && bs <= kMaxGemmBatch && (v1 || (L.kernel_layout && bs > kMaxMatvecBatch));
    // long prompts: the tensor-core kernel again where it is the faster way, else decoded once and a dense product
    const bool wide = whole_tiles && bs > kMaxGemmBatch && (v1 || L.kernel_layout) && aligned16(trellis) &&
                      qtip_decompress_gemm_f16_faster(L.code, (int)m, (int)n, (int)bs);
    const bool dense = !gemm && !wide && bs > kMaxMatvecBatch;

    // one allocation for both intermediates: the transformed activation (fp16) and, unless the dense product makes its
    // own, the raw result (fp32; fp16 of a long prompt, as from the dense product)
    const int64_t xh_bytes = (bs * n * 2 + 255) / 256 * 256;
    // (straight from the caching allocator, on the current stream: a tensor around it costs half a microsecond)
    const c10::DataPtr scratch = c10::cuda::CUDACachingAllocator::get()->allocate(xh_bytes + (dense ? 0 : bs * m * (wide ? 2 : 4)));
    char *base = static_cast<char *>(scratch.get());
    void *xh = base;
    float *y = reinterpret_cast<float *>(base + xh_bytes);

    // input side: x * SU -> Hadamard^T (per chunk when row-parallel) -> / 32 -> fp16
    const int64_t seg_n = L.rcp == 1 ? n / L.tp : n;
    // rows that the matvec takes in fragment order are written so by the transform
    const bool fragments = !gemm && !wide && !dense && L.kernel_layout && seg_n == n && aligned16(x) && aligned16(SU) &&
                           qtip_matvec_x_fragments(L.K, (int)m, (int)n, (int)bs);
    check(qtip_rht(xh, fragments ? QTIP_F16_FRAGMENTS : QTIP_F16, x.data_ptr(), dtype_id(x), bs * (n / seg_n), (int)seg_n, SU.data_ptr(), dtype_id(SU), nullptr,
                   n, bl, L.k_left, 1, (float)(1.0 / (std::sqrt((double)seg_n) * kInternalScale)), stream),
          "qtip_rht");
    launches = 3;
    at::Tensor dense_y;
    const void *y_in = y;
    int y_type = QTIP_F32;
    if (gemm || wide) {
        // (qtip_rht starts it when the weights, whatever wrote them, are complete)
        y_type = wide ? QTIP_F16 : QTIP_F32;
        check(qtip_decompress_gemm_settled(y, y_type, trellis.data_ptr(), xh, v1 ? nullptr : tlut.data_ptr(), L.code, L.K, (int)m, (int)n, (int)bs,
                                           static_cast<unsigned *>(gemm_status(dev).data_ptr()), stream),
              "qtip_decompress_gemm_settled");
    } else if (!dense) {
        at::Tensor ws = L.workspace.defined() ? L.workspace : matvec_workspace(dev, m, n, bs, stream);
        if (fragments)
            check(qtip_decompress_matvec_fragments(y, trellis.data_ptr(), xh, tlut.data_ptr(), L.K, (int)m, (int)n, (int)bs, ws.data_ptr(),
                                                   (size_t)ws.nbytes(), stream),
                  "qtip_decompress_matvec_fragments");
        else if (L.kernel_layout)
            check(qtip_decompress_matvec(y, trellis.data_ptr(), xh, tlut.data_ptr(), L.K, (int)m, (int)n, (int)bs, ws.data_ptr(),
                                         (size_t)ws.nbytes(), stream),
                  "qtip_decompress_matvec");
        else
            check(qtip_decompress_matvec_plain(y, trellis.data_ptr(), xh, L.code, L.K, (int)m, (int)n, (int)bs, ws.data_ptr(),
                                               (size_t)ws.nbytes(), stream),
                  "qtip_decompress_matvec_plain");
    } else {
        // anything else: decode once, dense fp16 GEMM (BitshiftLinearKernelAG upstream, bitshift.py:476-489); the fp16
        // product goes to the output transform as it is
        at::Tensor W = at::empty({m, n}, opts.dtype(at::kHalf));
        if (L.kernel_layout)
            check(qtip_decode_hyb_settled(W.data_ptr(), trellis.data_ptr(), tlut.data_ptr(), L.K, (int)m, (int)n, stream),
                  "qtip_decode_hyb_settled");
        else
            check(qtip_decode_plain(W.data_ptr(), trellis.data_ptr(), L.code, tlut.defined() ? tlut.data_ptr() : nullptr, L.K, (int)m,
                                    (int)n, stream),
                  "qtip_decode_plain");
        at::Tensor xt = at::from_blob(xh, {bs, n}, opts.dtype(at::kHalf));
        dense_y = at::mm(xt, W.t());
        y_in = dense_y.data_ptr();
        y_type = QTIP_F16;
    }

    // output side: Hadamard (per chunk when column-parallel) -> * SV * 32
    const int64_t seg_m = L.rcp == 2 ? m / L.tp : m;
    check(qtip_rht(out.data_ptr(), dtype_id(out), y_in, y_type, bs * (m / seg_m), (int)seg_m, nullptr, QTIP_F16,
                   static_cast<const float *>(SV.data_ptr()), m, br, L.k_right, 0, (float)(kInternalScale / std::sqrt((double)seg_m)),
                   stream),
          "qtip_rht");
    return in_type == out_type ? out : out.to(in_type);
}

// ---- CPython module ------------------------------------------------------------------------------------------
at::Tensor tensor_arg(PyObject *o, const char *name) {
    if (o == Py_None) return at::Tensor();
    if (!THPVariable_Check(o)) throw Failure{std::string(name) + " must be a tensor"};
    return THPVariable_Unpack(o);
}
long int_arg(PyObject *o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw Failure{""};
    return v;
}

struct WithoutGil {
    PyThreadState *s = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(s); }
};

// Runs `body`, turning failures (the library's and torch's) into RuntimeError as the Python wrappers raise.
template <class F>
PyObject *guarded(F body) {
    try {
        return body();
    } catch (const Failure &f) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, f.what.c_str());
    } catch (const c10::Error &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

PyObject *py_linear_forward(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 15) throw Failure{"linear_forward takes 15 arguments"};
        const at::Tensor input = tensor_arg(a[0], "input"), trellis = tensor_arg(a[1], "trellis"), SU = tensor_arg(a[3], "SU"),
                         SV = tensor_arg(a[4], "SV");
        if (!input.defined() || !trellis.defined() || !SU.defined() || !SV.defined()) throw Failure{"linear_forward: missing tensor"};
        Layer L{trellis, SU, SV, tensor_arg(a[2], "tlut"), tensor_arg(a[5], "bits_left"), tensor_arg(a[7], "bits_right"),
                tensor_arg(a[14], "workspace"), (int)int_arg(a[6]), (int)int_arg(a[8]), (int)int_arg(a[9]), (int)int_arg(a[10]),
                (int)int_arg(a[12]), (int)int_arg(a[13]), int_arg(a[11]) != 0};
        if (L.code == QTIP_CODE_HYB && !L.tlut.defined()) throw Failure{"the HYB code needs its table"};
        int launches = 0;
        at::Tensor out;
        {
            c10::NoGradGuard no_grad;       // raw launches: nothing here can be differentiated through
            WithoutGil nogil;
            out = linear_forward(input, L, launches);
        }
        return Py_BuildValue("(Ni)", THPVariable_Wrap(std::move(out)), launches);
    });
}

PyObject *py_matvec_workspace(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 4) throw Failure{"matvec_workspace takes 4 arguments"};
        const int dev = (int)int_arg(a[0]);
        const long m = int_arg(a[1]), n = int_arg(a[2]), bs = int_arg(a[3]);
        void *stream = at::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
        return THPVariable_Wrap(matvec_workspace(dev, m, n, bs, stream));
    });
}

PyObject *py_gemm_status(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject * {
        if (nargs != 1) throw Failure{"gemm_status takes 1 argument"};
        return THPVariable_Wrap(gemm_status((int)int_arg(a[0])));
    });
}

PyMethodDef kMethods[] = {
    {"linear_forward", (PyCFunction)(void *)py_linear_forward, METH_FASTCALL, "one QTIP linear on the current stream"},
    {"matvec_workspace", (PyCFunction)(void *)py_matvec_workspace, METH_FASTCALL, "scratch of the fused matvec"},
    {"gemm_status", (PyCFunction)(void *)py_gemm_status, METH_FASTCALL, "status word of the decompress-GEMM"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "native host path of qtip_b200", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&kModule); }

// The torch extension module `int4matmul`: the operator surface of the reference's int4matmul.cpp
// (same eleven functions, argument order, in-place convention, docstrings) over the C ABI of
// libint4matmul_b200.so.  Host code only: it validates tensors, picks the current CUDA stream, keeps one
// zero-initialised scratch buffer per (device, stream) and turns non-zero statuses into exceptions.
//
// Differences from the reference, all on the side of failing earlier and louder:
//   * every precondition the reference checks with assert() (process abort) or not at all (dtype, device,
//     contiguity; matmul_kernel.cu:404-416, 446-451) raises here;
//   * sparse int3 / int2 and non-fp16 activations raise instead of trapping the device (matmul.cuh:188, 331);
//   * launches go to torch's current stream (the reference uses the legacy default stream, which is the same
//     stream unless the caller switched streams);
//   * weight_matrix_packing raises ValueError when a 32-block does not keep exactly 16 weights (the reference
//     device-asserts, utils_kernel.cu:41); for that it waits for the pack kernel to finish.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "../../include/int4matmul_b200.h"

namespace {

using torch::Tensor;

#define I4_TENSOR_MULT_ARGS                                                                            \
    Tensor outs, Tensor matrix, Tensor multiplier, Tensor scales, Tensor zeros, int64_t group_size,    \
        c10::optional<Tensor> sparse_mask
#define I4_TENSOR_MULT_PASS outs, matrix, multiplier, scales, zeros, group_size, sparse_mask

struct Workspace {
    Tensor buffer;
    cudaStream_t stream;
};
std::mutex g_ws_mutex;
std::map<std::pair<int, int64_t>, Workspace> g_workspaces;

Tensor workspace_for(const c10::Device& dev, const c10::cuda::CUDAStream& stream) {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    const auto key = std::make_pair((int)dev.index(), (int64_t)stream.id());
    auto it = g_workspaces.find(key);
    if (it != g_workspaces.end()) return it->second.buffer;
    Tensor ws = torch::zeros({(int64_t)i4mm_workspace_bytes()}, torch::dtype(torch::kUInt8).device(dev));
    g_workspaces.emplace(key, Workspace{ws, stream.stream()});
    return ws;
}

void check_status(int status, const char* what) {
    if (status == I4MM_OK) return;
    std::string msg = std::string(what) + ": " + i4mm_status_string(status);
    if (status == I4MM_ERR_LAUNCH) msg += " (cudaError " + std::to_string(i4mm_last_cuda_error()) + ")";
    if (status == I4MM_ERR_BITS) throw std::invalid_argument(msg);
    TORCH_CHECK(false, msg);
}

enum class Route { AUTO, MATMUL, MATVEC };

// Not in the reference: the caller's promise that the weight-side tensors are never written by the kernel that
// precedes a multiply in the stream (weights of a loaded model), which lets a launch begin while that kernel finishes.
std::atomic<bool> g_static_weights{false};
void set_static_weights(bool flag) { g_static_weights.store(flag); }

void quant_mult(uint32_t bits, Route route, I4_TENSOR_MULT_ARGS) {
    if (bits != 4 && bits != 3 && bits != 2) {
        // int4matmul.cpp:35, 45
        throw std::invalid_argument(multiplier.dim() == 3 && multiplier.size(1) == 1
                                        ? "Unsupported bit width for matvec"
                                        : "Unsupported bit width for matmul");
    }
    const bool is_sparse = sparse_mask.has_value() && sparse_mask.value().defined();
    TORCH_CHECK(multiplier.is_cuda(), "multiplier must be a CUDA tensor");
    const auto dev = multiplier.device();
    auto on_dev = [&](const Tensor& t, const char* name) {
        TORCH_CHECK(t.is_cuda() && t.device() == dev, name, " must be on the same CUDA device as multiplier");
        TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
    };
    on_dev(outs, "outs"); on_dev(matrix, "matrix"); on_dev(multiplier, "multiplier");
    on_dev(scales, "scales"); on_dev(zeros, "zeros");
    TORCH_CHECK(multiplier.scalar_type() == torch::kHalf, "multiplier must be float16 (the reference implements fp16 only)");
    TORCH_CHECK(outs.scalar_type() == torch::kHalf, "outs must be float16");
    TORCH_CHECK(scales.scalar_type() == torch::kHalf && zeros.scalar_type() == torch::kHalf, "scales and zeros must be float16");
    TORCH_CHECK(matrix.scalar_type() == torch::kInt, "matrix must be int32");
    TORCH_CHECK(multiplier.dim() == 3, "multiplier must be (batch, seq_len, in_size)");
    TORCH_CHECK(outs.dim() == 3, "outs must be (batch, seq_len, out_size)");
    TORCH_CHECK(matrix.dim() == 2 && scales.dim() == 2 && zeros.dim() == 2, "matrix, scales, zeros must be 2-D");
    TORCH_CHECK(!is_sparse || bits == 4, "16:32 sparsity is only implemented for 4-bit weights");

    const int64_t batch = multiplier.size(0), seq_len = multiplier.size(1), in_size = multiplier.size(2);
    const int64_t mtx_in = matrix.size(0), out_size = matrix.size(1);
    if (route == Route::MATVEC) TORCH_CHECK(seq_len == 1, "the _vec entry needs seq_len == 1 (matvec_kernel.cu:323)");
    if (is_sparse) {
        TORCH_CHECK(mtx_in * 32 * 2 / bits == in_size, "sparse matrix rows * 16 must equal in_size");
    } else {
        TORCH_CHECK(mtx_in * 32 / bits == in_size && (mtx_in * 32) % bits == 0, "matrix rows * 32 / bits must equal in_size");
    }
    TORCH_CHECK(outs.size(0) == batch && outs.size(1) == seq_len && outs.size(2) == out_size, "outs must be (batch, seq_len, out_size)");
    TORCH_CHECK(zeros.size(1) == out_size && scales.size(1) == out_size, "scales/zeros must have out_size columns");
    TORCH_CHECK(zeros.size(0) == scales.size(0), "scales and zeros must have the same number of groups");
    TORCH_CHECK(group_size < 0 || (group_size > 0 && group_size % 64 == 0), "group_size must be a positive multiple of 64, or negative");
    const void* mask_ptr = nullptr;
    if (is_sparse) {
        const Tensor& m = sparse_mask.value();
        on_dev(m, "sparse_mask");
        TORCH_CHECK(m.scalar_type() == torch::kInt && m.dim() == 2, "sparse_mask must be 2-D int32");
        TORCH_CHECK(m.size(0) * 2 == mtx_in && m.size(1) == out_size, "sparse_mask must be (matrix rows / 2, out_size)");
        mask_ptr = m.data_ptr();
    }

    const bool matvec = route == Route::MATVEC || (route == Route::AUTO && seq_len == 1);
    c10::cuda::CUDAGuard guard(dev);
    auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
    Tensor ws = workspace_for(dev, stream);
    const int status = i4mm_quant_matmul(
        (int)bits, matvec ? 1 : 0, /*path=*/g_static_weights.load() ? I4MM_PATH_STATIC_WEIGHTS : 0, outs.data_ptr(), matrix.data_ptr(), mask_ptr, multiplier.data_ptr(),
        scales.data_ptr(), zeros.data_ptr(), batch * seq_len, in_size, out_size, scales.size(0), group_size,
        ws.data_ptr(), (size_t)ws.numel(), (void*)stream.stream());
    check_status(status, "int4matmul");
}

void quant_matmul(uint32_t bits, I4_TENSOR_MULT_ARGS) { quant_mult(bits, Route::AUTO, I4_TENSOR_MULT_PASS); }

#define I4_REGISTER_WIDTH(N)                                                                              \
    void spec_mm_int##N(I4_TENSOR_MULT_ARGS) { quant_mult(N, Route::AUTO, I4_TENSOR_MULT_PASS); }         \
    void matmul_int##N(I4_TENSOR_MULT_ARGS) { quant_mult(N, Route::MATMUL, I4_TENSOR_MULT_PASS); }        \
    void matvec_int##N(I4_TENSOR_MULT_ARGS) { quant_mult(N, Route::MATVEC, I4_TENSOR_MULT_PASS); }
I4_REGISTER_WIDTH(4)
I4_REGISTER_WIDTH(3)
I4_REGISTER_WIDTH(2)

void weight_matrix_packing(Tensor wt_outs, Tensor msk_outs, Tensor wt_in, Tensor msk_in) {
    TORCH_CHECK(wt_in.is_cuda(), "wt_in must be a CUDA tensor");
    const auto dev = wt_in.device();
    for (const Tensor* t : {&wt_outs, &msk_outs, &wt_in, &msk_in}) {
        TORCH_CHECK(t->is_cuda() && t->device() == dev && t->is_contiguous() && t->dim() == 2,
                    "all four tensors must be contiguous 2-D CUDA tensors on one device");
    }
    // utils_kernel.cu:74-82
    TORCH_CHECK(wt_in.size(1) == wt_outs.size(0) * 16, "wt_in columns must be 16 x wt_outs rows");
    TORCH_CHECK(msk_in.size(1) == msk_outs.size(0) * 32, "msk_in columns must be 32 x msk_outs rows");
    TORCH_CHECK(wt_in.size(0) == wt_outs.size(1) && msk_in.size(0) == msk_outs.size(1), "row/column counts must match");
    TORCH_CHECK(wt_in.size(0) == msk_in.size(0) && wt_in.size(1) == msk_in.size(1), "wt_in and msk_in must have one shape");
    TORCH_CHECK(wt_outs.scalar_type() == torch::kInt && msk_outs.scalar_type() == torch::kInt, "outputs must be int32");
    TORCH_CHECK(wt_in.scalar_type() == torch::kByte && msk_in.scalar_type() == torch::kByte, "inputs must be uint8");
    TORCH_CHECK(wt_in.size(1) % 32 == 0, "in_size must be a multiple of 32 (utils_kernel.cu:101)");

    c10::cuda::CUDAGuard guard(dev);
    auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
    Tensor violations = torch::zeros({1}, torch::dtype(torch::kInt).device(dev));
    const int status = i4mm_sparse_pack(wt_outs.data_ptr(), msk_outs.data_ptr(), wt_in.data_ptr(), msk_in.data_ptr(),
                                        wt_in.size(0), wt_in.size(1), violations.data_ptr(), (void*)stream.stream());
    check_status(status, "weight_matrix_packing");
    const int bad = violations.item<int>();
    if (bad != 0) {
        throw std::invalid_argument("weight_matrix_packing: " + std::to_string(bad) +
                                    " block(s) of 32 weights do not keep exactly 16 (16:32 sparsity)");
    }
}

// ---- the Python package's own calls (ops.py, quantize.py) -----------------------------------------------------------
// What those modules check and launch, for arguments that pass every check: a decoding step is a chain of small launches,
// and the same work done in Python (17 ctypes arguments, a device context, some thirty tensor properties) takes longer
// than most of them run.  Nothing is diagnosed here: whenever a precondition does not hold (an argument that is no tensor
// or no integer, memory that cannot be had, ...), or the scratch buffer of this stream does not exist yet, the caller is told so
// (-1) and takes its own path, which raises, converts or allocates.  The arguments are therefore plain Python objects: a typed
// signature would raise an error of its own first.
// A launch may block when the stream's queue is full, so the interpreter's lock is given up over it, as ctypes does.

// (an undefined tensor stands for None)
bool as_tensor(const py::object& o, Tensor& t) {
    if (!THPVariable_Check(o.ptr())) return false;
    t = THPVariable_Unpack(o.ptr());
    return true;
}
bool as_optional_tensor(const py::object& o, Tensor& t) { return o.is_none() || as_tensor(o, t); }

bool as_int(const py::object& o, int64_t& v) {
    if (!PyIndex_Check(o.ptr())) return false;
    v = PyNumber_AsSsize_t(o.ptr(), PyExc_OverflowError);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

bool plain(const Tensor& t, const c10::Device& dev, c10::ScalarType type) {
    return t.is_cuda() && t.device() == dev && t.scalar_type() == type && t.is_contiguous();
}

// the weight side of a call, as the caller has it
struct Weights {
    Tensor matrix, scales, zeros, mask;
    int64_t bits = 0, group_size = 0;
    bool read(const py::object& bits_, const py::object& matrix_, const py::object& scales_, const py::object& zeros_,
              const py::object& group_size_, const py::object& mask_) {
        return as_int(bits_, bits) && as_int(group_size_, group_size) && as_tensor(matrix_, matrix) && as_tensor(scales_, scales) &&
               as_tensor(zeros_, zeros) && as_optional_tensor(mask_, mask);
    }
};

// Whether a multiply of fp16 rows of `in_size` on `dev` by w passes the entries' checks
bool valid(const Weights& w, const c10::Device& dev, int64_t in_size) {
    if (w.bits != 4 && w.bits != 3 && w.bits != 2) return false;
    if (!plain(w.matrix, dev, torch::kInt) || !plain(w.scales, dev, torch::kHalf) || !plain(w.zeros, dev, torch::kHalf) ||
        w.matrix.dim() != 2 || w.scales.dim() != 2 || w.zeros.dim() != 2)
        return false;
    const int64_t mtx_in = w.matrix.size(0), out_size = w.matrix.size(1);
    if (w.mask.defined()) {
        if (w.bits != 4 || mtx_in * 16 != in_size || mtx_in % 2 || !plain(w.mask, dev, torch::kInt) || w.mask.dim() != 2 ||
            w.mask.size(0) != mtx_in / 2 || w.mask.size(1) != out_size)
            return false;
    } else if ((mtx_in * 32) % w.bits || mtx_in * 32 / w.bits != in_size) {
        return false;
    }
    if (w.scales.size(1) != out_size || w.zeros.sizes() != w.scales.sizes()) return false;
    return w.group_size != 0 && (w.group_size < 0 || w.group_size % 64 == 0);
}

// the scratch of the current stream of `dev`, from the Python package's dict (device index, raw stream) -> zero-initialised uint8
// tensor; undefined if there is none yet
Tensor scratch(const py::dict& workspaces, const c10::Device& dev, cudaStream_t stream) {
    PyObject* const item = PyDict_GetItem(workspaces.ptr(), py::make_tuple((int)dev.index(), (uint64_t)(uintptr_t)stream).ptr());
    return item ? py::cast<Tensor>(py::handle(item)) : Tensor();
}

int launch(const Weights& w, bool matvec, int64_t path, void* out, const void* x, int64_t rows, int64_t in_size, const Tensor& ws, cudaStream_t stream) {
    return i4mm_quant_matmul((int)w.bits, matvec ? 1 : 0, (int)path, out, w.matrix.data_ptr(), w.mask.defined() ? w.mask.data_ptr() : nullptr,
                             x, w.scales.data_ptr(), w.zeros.data_ptr(), rows, in_size, w.matrix.size(1), w.scales.size(0),
                             w.group_size, ws.data_ptr(), (size_t)ws.numel(), (void*)stream);
}

int launch_checked(const Weights& w, bool matvec, int64_t path, void* out, const Tensor& x, int64_t rows, const py::dict& workspaces) {
    const auto dev = x.device();
    if (!plain(x, dev, torch::kHalf) || !valid(w, dev, x.size(-1))) return -1;
    c10::cuda::OptionalCUDAGuard guard;
    if (c10::cuda::current_device() != dev.index()) guard.set_device(dev);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const Tensor ws = scratch(workspaces, dev, stream);
    if (!ws.defined()) return -1;
    // (every tensor is held by a reference of this call's own)
    py::gil_scoped_release release;
    return launch(w, matvec, path, out, x.data_ptr(), rows, x.size(-1), ws, stream);
}

// ops._mult; route 0: by seq_len, 1: matmul, 2: matvec
int try_mult(const py::object& bits, int64_t route, int64_t path, const py::object& outs_, const py::object& matrix, const py::object& x_,
             const py::object& scales, const py::object& zeros, const py::object& group_size, const py::object& mask,
             const py::dict& workspaces) {
    Weights w;
    Tensor outs, x;
    if (!w.read(bits, matrix, scales, zeros, group_size, mask) || !as_tensor(outs_, outs) || !as_tensor(x_, x)) return -1;
    try {
        if (x.dim() != 3 || outs.dim() != 3 || w.matrix.dim() != 2 || !plain(outs, x.device(), torch::kHalf)) return -1;
        const int64_t batch = x.size(0), seq_len = x.size(1);
        if (route == 2 && seq_len != 1) return -1;
        if (outs.size(0) != batch || outs.size(1) != seq_len || outs.size(2) != w.matrix.size(1)) return -1;
        return launch_checked(w, route == 2 || (route == 0 && seq_len == 1), path, outs.data_ptr(), x, batch * seq_len, workspaces);
    } catch (const c10::Error&) {
        return -1;                                          // (nothing was launched: everything that throws comes before that)
    }
}

// QuantLinear.forward: the new output, or a status / -1
py::object try_linear(const py::object& bits, int64_t path, const py::object& x_, const py::object& in_features_,
                      const py::object& out_features_, const py::object& matrix, const py::object& scales, const py::object& zeros,
                      const py::object& group_size, const py::object& mask, const py::dict& workspaces) {
    Weights w;
    Tensor x;
    int64_t in_features = 0, out_features = 0;
    if (!w.read(bits, matrix, scales, zeros, group_size, mask) || !as_tensor(x_, x) || !as_int(in_features_, in_features) ||
        !as_int(out_features_, out_features))
        return py::int_(-1);
    try {
        if (x.dim() < 1 || x.numel() == 0 || x.size(-1) != in_features || w.matrix.dim() != 2 || w.matrix.size(1) != out_features ||
            !plain(x, x.device(), torch::kHalf))
            return py::int_(-1);
        auto sizes = x.sizes().vec();
        sizes.back() = out_features;
        Tensor out = at::empty(sizes, at::TensorOptions().dtype(torch::kHalf).device(x.device()));
        const int status = launch_checked(w, false, path, out.data_ptr(), x, x.numel() / in_features, workspaces);
        if (status != I4MM_OK) return py::int_(status);
        return py::cast(out);
    } catch (const c10::Error&) {
        return py::int_(-1);
    }
}

// ops.row_norm (mode may carry I4MM_PATH_STATIC_WEIGHTS): the new output, or a status / -1
py::object try_row_norm(int64_t mode, const py::object& a_, const py::object& b, const py::object& c) {
    Tensor a, operands[3];
    if (!as_tensor(a_, a) || !as_optional_tensor(b, operands[1]) || !as_optional_tensor(c, operands[2])) return py::int_(-1);
    operands[0] = a;
    try {
        if (!a.is_cuda() || a.dim() != 2 || c10::cuda::current_device() != a.device().index()) return py::int_(-1);
        const void* ptr[3] = {nullptr, nullptr, nullptr};
        int64_t stride[3] = {0, 0, 0};
        for (int i = 0; i < 3; ++i) {
            const Tensor& t = operands[i];
            if (!t.defined()) continue;
            if (!t.is_cuda() || t.device() != a.device() || t.scalar_type() != torch::kHalf || t.sizes() != a.sizes() || t.stride(1) != 1)
                return py::int_(-1);
            ptr[i] = t.data_ptr();
            stride[i] = t.stride(0);
        }
        const int64_t rows = a.size(0), width = a.size(1);
        const auto options = at::TensorOptions().dtype(torch::kHalf).device(a.device());
        Tensor y = (mode & ~(int64_t)I4MM_PATH_STATIC_WEIGHTS) == 4 ? at::empty({2, rows, width}, options) : at::empty({rows, width}, options);
        const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(a.device().index()).stream();
        int status;
        {
            py::gil_scoped_release release;
            status = i4mm_row_norm((int)mode, y.data_ptr(), ptr[0], ptr[1], ptr[2], rows, width, stride[0], stride[1], stride[2], (void*)stream);
        }
        if (status != I4MM_OK) return py::int_(status);
        return py::cast(y);
    } catch (const c10::Error&) {
        return py::int_(-1);
    }
}

// One layer of sharding.DecoderStack on one GPU: the data flow of its forward(), the same eight launches (`early`:
// I4MM_PATH_STATIC_WEIGHTS or 0).  h, x: the residual stream and its normalised rows; returns h, or the pair of the next layer's h and x,
// a status, or -1 with nothing launched.  A layer of one row is 70 us of work on the GPU; eight calls from Python took longer than that.
py::object try_layer(const py::object& mats, const py::object& h_, const py::object& x_, bool last, int64_t early, const py::dict& workspaces) {
    static const char* const kNames[4] = {"qkv", "o", "gate_up", "down"};
    Tensor h, x;
    Weights w[4];
    int64_t columns[4];
    if (!PyDict_Check(mats.ptr()) || !as_tensor(h_, h) || !as_tensor(x_, x)) return py::int_(-1);
    for (int i = 0; i < 4; ++i) {
        PyObject* const m = PyDict_GetItemString(mats.ptr(), kNames[i]);
        if (!m) return py::int_(-1);
        const py::handle q(m);
        const py::object none = py::none();
        if (!w[i].read(py::getattr(q, "bits", none), py::getattr(q, "matrix", none), py::getattr(q, "scales", none), py::getattr(q, "zeros", none),
                       py::getattr(q, "group_size", none), py::getattr(q, "mask", none)) ||
            !as_int(py::getattr(q, "s", none), columns[i]))
            return py::int_(-1);
    }
    try {
        if (!h.is_cuda()) return py::int_(-1);
        const auto dev = h.device();
        if (h.dim() != 2 || h.size(0) == 0 || !plain(h, dev, torch::kHalf) || !plain(x, dev, torch::kHalf) || x.sizes() != h.sizes() ||
            c10::cuda::current_device() != dev.index())
            return py::int_(-1);
        const int64_t rows = h.size(0), width = h.size(1);
        for (int i = 0; i < 4; ++i)
            if (w[i].matrix.dim() != 2 || w[i].matrix.size(1) != columns[i]) return py::int_(-1);
        const int64_t qkv = w[0].matrix.size(1), gate_up = w[2].matrix.size(1), inner = gate_up / 2;
        if (qkv != 3 * width || w[1].matrix.size(1) != width || gate_up % 2 || inner % 2 || width % 2 || w[3].matrix.size(1) != width ||
            !valid(w[0], dev, width) || !valid(w[1], dev, width) || !valid(w[2], dev, width) || !valid(w[3], dev, inner))
            return py::int_(-1);
        const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        const Tensor ws = scratch(workspaces, dev, stream);
        if (!ws.defined()) return py::int_(-1);
        const auto options = at::TensorOptions().dtype(torch::kHalf).device(dev);
        const Tensor p = at::empty({rows, qkv}, options), t = at::empty({rows, width}, options), o = at::empty({rows, width}, options),
                     h2 = at::empty({rows, width}, options), g = at::empty({rows, gate_up}, options), a = at::empty({rows, inner}, options),
                     d = at::empty({rows, width}, options),
                     y = last ? at::empty({rows, width}, options) : at::empty({2, rows, width}, options);
        int status;
        {
            py::gil_scoped_release release;
            const auto col = [](const Tensor& m, int64_t c) -> const void* { return static_cast<const at::Half*>(m.data_ptr()) + c; };
            const auto norm = [&](int mode, const Tensor& out, const void* a0, const void* b0, const void* c0, int64_t n, int64_t sa, int64_t sb, int64_t sc) {
                return i4mm_row_norm(mode | (int)early, out.data_ptr(), a0, b0, c0, rows, n, sa, sb, sc, (void*)stream);
            };
            const auto mult = [&](int i, const Tensor& out, const Tensor& in) {
                return launch(w[i], false, early, out.data_ptr(), in.data_ptr(), rows, in.size(1), ws, stream);
            };
            status = mult(0, p, x);
            if (status == I4MM_OK) status = norm(1, t, col(p, 0), col(p, width), col(p, 2 * width), width, qkv, qkv, qkv);
            if (status == I4MM_OK) status = mult(1, o, t);
            if (status == I4MM_OK) status = norm(2, h2, h.data_ptr(), o.data_ptr(), nullptr, width, width, width, 0);
            if (status == I4MM_OK) status = mult(2, g, h2);
            if (status == I4MM_OK) status = norm(3, a, col(g, 0), col(g, inner), nullptr, inner, gate_up, gate_up, 0);
            if (status == I4MM_OK) status = mult(3, d, a);
            if (status == I4MM_OK) status = norm(last ? 2 : 4, y, h2.data_ptr(), d.data_ptr(), nullptr, width, width, width, 0);
        }
        if (status != I4MM_OK) return py::int_(status);
        if (last) return py::cast(y);
        return py::make_tuple(y.select(0, 0), y.select(0, 1));
    } catch (const c10::Error&) {
        return py::int_(-1);                               // (an allocation failed; nothing was launched)
    }
}

// Not in the reference (its kernels have no waits): waits for every stream this module has launched on, on the
// current device, and raises if a kernel gave up on one of its bounded device-side waits since the last check.
// The multiply entries do not call it themselves, because it synchronises.
void check_device_status() {
    int dev = 0;
    TORCH_CHECK(cudaGetDevice(&dev) == cudaSuccess, "no current CUDA device");
    std::vector<Workspace> mine;
    {
        std::lock_guard<std::mutex> lock(g_ws_mutex);
        for (auto& kv : g_workspaces)
            if (kv.first.first == dev) mine.push_back(kv.second);
    }
    int worst = I4MM_OK;
    for (auto& w : mine) {
        const int st = i4mm_device_status(w.buffer.data_ptr(), (void*)w.stream);
        if (st == I4MM_ERR_TIMEOUT) {                     // the scratch of a cut-short launch is not all-zero any more
            w.buffer.zero_();
            cudaDeviceSynchronize();
        }
        if (st != I4MM_OK) worst = st;
    }
    check_status(worst, "int4matmul device status");
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("set_static_weights", &set_static_weights,
          "declare that weight-side tensors are never written by the kernel preceding a multiply in the stream");
    m.def("check_device_status", &check_device_status,
          "raise if a kernel launched by this module gave up on a bounded device-side wait (synchronises)");

    m.def("_try_mult", &try_mult, "ops._mult for arguments that pass its checks: status, or -1");
    m.def("_try_linear", &try_linear, "QuantLinear.forward for arguments that pass its checks: output, status or -1");
    m.def("_try_layer", &try_layer, "one layer of sharding.DecoderStack on one GPU: h, or (h, x), a status or -1");
    m.def("_try_row_norm", &try_row_norm, "ops.row_norm for arguments that pass its checks: output, status or -1");

    m.def("weight_matrix_packing", &weight_matrix_packing, "int4_sparse_pack");

    m.def("quant_matmul", &quant_matmul, "intn_fp16_mult");

    m.def("quant_int4_linear_mult", &spec_mm_int4, "int4_fp16_mult");
    m.def("quant_int4_linear_mult_mtx", &matmul_int4, "int4_fp16_mult_mtx");
    m.def("quant_int4_linear_mult_vec", &matvec_int4, "int4_fp16_mult_vec");

    m.def("quant_int3_linear_mult", &spec_mm_int3, "int3_fp16_mult");
    m.def("quant_int3_linear_mult_mtx", &matmul_int3, "int3_fp16_mult_mtx");
    m.def("quant_int3_linear_mult_vec", &matvec_int3, "int3_fp16_mult_vec");

    m.def("quant_int2_linear_mult", &spec_mm_int2, "int2_fp16_mult");
    m.def("quant_int2_linear_mult_mtx", &matmul_int2, "int2_fp16_mult_mtx");
    m.def("quant_int2_linear_mult_vec", &matvec_int2, "int2_fp16_mult_vec");
}

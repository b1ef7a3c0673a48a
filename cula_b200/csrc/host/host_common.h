// Native host path: argument checks, output allocation, autograd and launches of the framework's operators, as a Python
// extension on libtorch. The same calls in Python cost 30 us (decode) to 400 us (a training step of six to nine launches)
// of interpreter time per call, several times what their kernels take at small sizes.
#pragma once
#include <dlfcn.h>
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <optional>
#include <string>

#include "../../../include/cula_kda.h"

namespace cula_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

constexpr int64_t CHUNK = 64, DIM = 128;
enum { GATE_NONE = 0, GATE_SOFTPLUS = 1, GATE_LOWER_BOUND = 2 };

// entry points of libcula_kda.so, resolved once by bind()
#define CULA_KDA_ENTRIES(X)                                                                                          \
    X(cula_kda_tile_pack_bytes) X(cula_kda_fwd_intra) X(cula_kda_fwd_scan) X(cula_kda_cp_transition) X(cula_kda_cp_fold) X(cula_kda_fwd_pieces) \
    X(cula_kda_decode) X(cula_kda_bwd_scratch_floats) X(cula_kda_bwd_grad_scale) X(cula_kda_bwd_scale_and_intra) X(cula_kda_bwd_scan) X(cula_kda_bwd_both_scans) \
    X(cula_kda_bwd_dense) X(cula_kda_bwd_gated_checked) X(cula_kda_clear) X(cula_kda_gate_fwd) X(cula_kda_gate_bwd)                              \
    X(cula_kda_beta_sigmoid_fwd) X(cula_kda_beta_sigmoid_bwd) X(cula_kda_short_conv_fwd) X(cula_kda_short_conv_bwd)    \
    X(cula_kda_rms_norm_gated_fwd) X(cula_kda_rms_norm_gated_bwd) X(cula_kda_strerror)
struct Lib {
#define CULA_KDA_MEMBER(name) decltype(&::name) name = nullptr;
    CULA_KDA_ENTRIES(CULA_KDA_MEMBER)
#undef CULA_KDA_MEMBER
};
extern Lib lib;

inline void check(int code, const char* what) {
    if (code != 0)
        throw std::runtime_error(std::string(what) + " failed with code " + std::to_string(code) + ": " + lib.cula_kda_strerror(code));
}
// the exceptions the Python functions have always raised
inline void require(bool ok, const char* message) {
    if (!ok) {
        PyErr_SetString(PyExc_AssertionError, message);
        throw pybind11::error_already_set();
    }
}
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline void* ptr(const OptTensor& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }
inline float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }
inline float* fptr(const OptTensor& t) { return static_cast<float*>(ptr(t)); }
inline int* iptr(const OptTensor& t) { return static_cast<int*>(ptr(t)); }
inline bool is_f32(const Tensor& t) { return t.scalar_type() == at::kFloat; }
inline bool is_bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
inline Tensor contiguous_f32(const Tensor& t) { return (is_f32(t) ? t : t.to(at::kFloat)).contiguous(); }
inline OptTensor contiguous_f32(const OptTensor& t) { return t.has_value() && t->defined() ? OptTensor(contiguous_f32(*t)) : OptTensor(); }
// Output allocations of the native path, straight from the allocator: through the dispatcher at::empty takes 1.7 us, and at::zeros
// 6 us with a kernel of its own, on a path that allocates up to 16 tensors per call.
inline Tensor device_empty(at::IntArrayRef sizes, const at::TensorOptions& options) { return Tensor(at::detail::empty_cuda(sizes, options)); }
inline Tensor device_zeros(at::IntArrayRef sizes, const at::TensorOptions& options, cudaStream_t stream) {
    Tensor t = device_empty(sizes, options);
    check(lib.cula_kda_clear(t.data_ptr(), (long long)t.nbytes(), stream), "cula_kda_clear");
    return t;
}
// contiguous part of an own buffer as a tensor (narrow and view through the dispatcher take 3 us)
inline Tensor part_of(const Tensor& buffer, int64_t offset, at::IntArrayRef sizes) {
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(buffer.storage()), buffer.key_set(), buffer.dtype());
    t.unsafeGetTensorImpl()->set_storage_offset(offset);
    t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
    return t;
}
// a part in the shape of the parameter that it is the gradient of
inline Tensor shaped_like(const Tensor& part, const Tensor& parameter) {
    if (part.numel() != parameter.numel())
        throw std::runtime_error("a gradient of " + std::to_string(part.numel()) + " elements cannot take the shape of a parameter of " +
                                 std::to_string(parameter.numel()));
    return part_of(part, part.storage_offset(), parameter.sizes());
}
// a dual tensor of forward-mode differentiation: no operator here has a forward derivative, and only the autograd function says so
inline bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }
inline cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// B200 guard (cached per device), and the status word of a device: one int in pinned host memory that the kernels write
// directly in the (rare) case that they have something to report, so that reading it costs neither a copy nor a wait
void assert_blackwell(const Tensor& t);
int* status_word(int device_index);
// status reported by kernels that have already finished: raises like check_status()
void poll_status(int device_index);

// the index tables of a packed batch (utils.VarlenTables)
struct Tables {
    Tensor cu_seqlens, chunk_indices, chunk_offsets, seq_order;
    int64_t n_seqs = 0, num_chunks = 0, total_tokens = 0;
};

void bind_attention(pybind11::module_& m);
void bind_layer_ops(pybind11::module_& m);

}  // namespace cula_host

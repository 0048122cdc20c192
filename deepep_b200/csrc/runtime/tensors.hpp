// Output tensors without the operator dispatcher. A dispatch hands back a dozen tensors, most of them small, and at small
// sizes the host is what bounds a call: an allocation through the dispatcher costs about 2 us with its release, one straight
// from the caching allocator 1 us, a tensor that shares an allocation 0.1 us.
#pragma once

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>

namespace ep {

inline at::Device cuda_device(int device) { return at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(device)); }

inline at::Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType dtype, int device) {
    return at::detail::empty_cuda(sizes, dtype, cuda_device(device), std::nullopt);
}
inline at::Tensor new_strided(at::IntArrayRef sizes, at::IntArrayRef strides, at::ScalarType dtype, int device) {
    return at::detail::empty_strided_cuda(sizes, strides, dtype, cuda_device(device));
}

// The first `n` rows of `t`.
inline at::Tensor first_rows(const at::Tensor& t, int64_t n) {
    if (t.size(0) == n) return t;
    at::Tensor v = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(t.storage()), t.key_set(), t.dtype());
    c10::SmallVector<int64_t, 4> sizes(t.sizes().begin(), t.sizes().end());
    sizes[0] = n;
    v.unsafeGetTensorImpl()->set_sizes_and_strides(sizes, t.strides(), t.storage_offset());
    return v;
}

// Contiguous tensors that share one allocation and are kept together (the routing tensors of a handle).
class TensorPack {
public:
    static int64_t room(int64_t elements, int64_t element_size) { return (elements * element_size + kAlign - 1) / kAlign * kAlign; }
    TensorPack(int64_t bytes, int device) : base_(new_tensor({bytes}, at::kByte, device)) {}
    at::Tensor take(at::IntArrayRef sizes, at::ScalarType dtype) {
        const auto type = c10::scalarTypeToTypeMeta(dtype);
        const int64_t item = static_cast<int64_t>(type.itemsize());
        at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(base_.storage()), base_.key_set(), type);
        t.unsafeGetTensorImpl()->set_storage_offset(used_ / item);
        t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
        used_ += room(t.numel(), item);
        TORCH_INTERNAL_ASSERT(used_ <= base_.numel());
        return t;
    }

private:
    static constexpr int64_t kAlign = 256;
    at::Tensor base_;
    int64_t used_ = 0;
};

}  // namespace ep

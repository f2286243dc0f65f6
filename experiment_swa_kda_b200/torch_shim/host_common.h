// What the two translation units of the operator library share: error translation, allocation, the device status watch.
#pragma once

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "kda_b200.h"

namespace kda_host {

using at::Tensor;
using OptTensor = c10::optional<Tensor>;

inline void must(int rc, const char* what) {
    TORCH_CHECK(rc == 0, what, " failed (", rc, "): ", kda_error_string(rc));
}

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

inline bool has(const OptTensor& t) { return t.has_value() && t->defined(); }
inline const void* ptr(const OptTensor& t) { return has(t) ? t->data_ptr() : nullptr; }

// straight to the caching allocator: the dispatcher's share of an allocation is as long as the allocation itself
inline Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
    return Tensor(at::detail::empty_cuda(sizes, type, like.device(), c10::nullopt));
}
inline Tensor empty_as(const Tensor& t) { return empty(t.sizes(), t.scalar_type(), t); }
// t itself, or a copy where its address would rule out 16-byte accesses (a view at an odd offset of a larger buffer)
inline Tensor aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0 ? t : t.clone(); }
inline Tensor bytes(size_t n, const Tensor& like) { return empty({(int64_t)(n < 256 ? 256 : n)}, at::kByte, like); }

// One allocation cut into 256-byte aligned tensors: a call's temporaries cost one trip to the allocator.
class Slab {
public:
    size_t take(size_t n_bytes) {
        const size_t at = size_;
        size_ += (n_bytes + 255) / 256 * 256;
        return at;
    }
    Tensor make(const Tensor& like) {
        all_ = bytes(size_, like);
        return all_;
    }
    const Tensor& tensor() const { return all_; }
    char* at(size_t offset) const { return static_cast<char*>(all_.data_ptr()) + offset; }
    float* f32(size_t offset) const { return reinterpret_cast<float*>(at(offset)); }

private:
    size_t size_ = 0;
    Tensor all_;
};

inline size_t up256(size_t n) { return (n + 255) / 256 * 256; }

// Device status without a hot-path cost: every device has one page-locked word that the kernels write to only when
// something failed (an expired bounded wait, an inconsistent cu_seqlens).  watch_status registers the word on the first
// call on a device and raises if an earlier call left a code in it; the word is cleared by the report.
void watch_status(int device);

}  // namespace kda_host

// What the dispatcher kernels (aten_ops.cpp) and the direct Python entry points (py_calls.cpp) share.
#pragma once

#include <ATen/ATen.h>

#include <array>

#include "../../include/b200_sdpa.h"

namespace b200_ops {

struct PerDevice {
  at::Tensor status;        // int32[4]: first device-side error seen by a kernel
  at::Tensor philox_seed;   // int32 scalar zeros (dropout is off)
  at::Tensor philox_offset;
};

PerDevice& device_state(int dev);

// Output buffer laid out like the query.
at::Tensor alloc_like_query(const at::Tensor& query, std::array<int64_t, 4> shape);

inline int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return B200_SDPA_F32;
    case at::kHalf: return B200_SDPA_F16;
    case at::kBFloat16: return B200_SDPA_BF16;
    default: return -1;
  }
}

// Scratch for one call: a fresh block from the caching allocator (stream-ordered, so the block can be
// reused by the next call on the same stream as soon as this one has been queued).
inline at::Tensor scratch(int dev, uint64_t bytes) {
  return at::empty({static_cast<int64_t>(bytes < 16 ? 16 : bytes)},
                   at::TensorOptions().device(at::kCUDA, dev).dtype(at::kByte));
}

template <size_t N> void copy_strides(const at::Tensor& t, int64_t (&dst)[N]) {
  for (size_t i = 0; i < N; ++i) dst[i] = t.stride(static_cast<int64_t>(i));
}

}  // namespace b200_ops

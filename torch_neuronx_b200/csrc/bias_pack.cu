// A copy of an additive bias that the tensor-core kernels can read: rows of 16-bit elements, unit stride, on 32-byte
// boundaries.  A bias of another layout (a key count that is no multiple of 8, a slice, a transpose) sent the whole request
// to the CUDA-core kernel, which takes 20 to 30 times as long as one pass over the bias and the tensor-core kernel.
// Bound: the bias read and written once.  Columns beyond the last key are filled with -inf, so that the look for
// hidden key tiles sees nothing in them; the attention kernels mask them by their number in any case.
#include "common.cuh"
#include "tc_common.cuh"

namespace b200 {

namespace {

constexpr uint64_t kMaxPackedBytes = 4ull << 30;   // more than this stays where it is

// One CTA per row, 2048 columns at a time; a thread writes four pairs of neighbouring columns, a warp 128 bytes at a time.
__global__ void __launch_bounds__(256) bias_pack_kernel(const uint16_t* src, uint16_t* dst, const int S, const int sp, const int n_rows,
                                                        const int n_heads, const int64_t s0, const int64_t s1, const int64_t s2,
                                                        const int64_t s3, const uint32_t hidden) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t row = blockIdx.x;
  const int r = static_cast<int>(row % n_rows), h = static_cast<int>(row / n_rows % n_heads);
  const int b = static_cast<int>(row / n_rows / n_heads);
  const uint16_t* in = src + b * s0 + h * s1 + r * s2;
  uint32_t* out = reinterpret_cast<uint32_t*>(dst + row * sp);
  for (int c0 = 0; c0 < sp / 2; c0 += 1024) {
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = 2 * (c0 + i * 256 + static_cast<int>(threadIdx.x));
      const uint32_t lo = c < S ? in[c * s3] : hidden, hi = c + 1 < S ? in[(c + 1) * s3] : hidden;
      v[i] = lo | (hi << 16);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = c0 + i * 256 + static_cast<int>(threadIdx.x);
      if (c < sp / 2) out[c] = v[i];
    }
  }
}

}  // namespace

// `packed` := the request with the bias where the copy will be (at `base`).  False where the bias is not one to copy.
bool bias_pack_geometry(const Problem& p, int dtype, void* base, Problem* packed, uint64_t* bytes) {
  if (p.bias == nullptr || (dtype != B200_SDPA_F16 && dtype != B200_SDPA_BF16) || p.bias_dtype != dtype) return false;
  if (p.L < 1 || p.S < 1 || tc::bias_readable(p, dtype, nullptr)) return false;
  const int64_t sp = (static_cast<int64_t>(p.S) + 15) / 16 * 16;
  const int64_t rows = p.bs[2] != 0 && p.L > 1 ? p.L : 1, heads = p.bs[1] != 0 && p.Hq > 1 ? p.Hq : 1,
                batches = p.bs[0] != 0 && p.B > 1 ? p.B : 1;
  if (batches * heads * rows > 0x7fffffffLL) return false;
  *bytes = static_cast<uint64_t>(batches * heads * rows) * sp * 2;
  *bytes = (*bytes + 255) / 256 * 256;
  if (*bytes > kMaxPackedBytes) return false;
  *packed = p;
  packed->bias = base;
  packed->bias_padded = 1;
  packed->bs[0] = batches > 1 ? heads * rows * sp : 0;
  packed->bs[1] = heads > 1 ? rows * sp : 0;
  packed->bs[2] = rows > 1 ? sp : 0;
  packed->bs[3] = 1;
  return true;
}

// The caller has made `packed` with bias_pack_geometry().
int launch_bias_pack(const Problem& p, const Problem& packed, int dtype, cudaStream_t stream) {
  const int sp = (p.S + 15) / 16 * 16;
  const int rows = packed.bs[2] != 0 ? p.L : 1, heads = packed.bs[1] != 0 ? p.Hq : 1, batches = packed.bs[0] != 0 ? p.B : 1;
  if (!launch_pdl(bias_pack_kernel, dim3(static_cast<unsigned>(static_cast<int64_t>(batches) * heads * rows)), 256, 0, stream,
                  static_cast<const uint16_t*>(p.bias), const_cast<uint16_t*>(static_cast<const uint16_t*>(packed.bias)), p.S, sp,
                  rows, heads, p.bs[0], p.bs[1], p.bs[2], p.bs[3], dtype == B200_SDPA_BF16 ? 0xff80u : 0xfc00u))
    return B200_SDPA_ERR_CUDA;
  return B200_SDPA_OK;
}

}  // namespace b200

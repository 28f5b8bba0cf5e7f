// Pieces shared by the tensor-core backward kernels (bwd_sm100.cu, bwd_wide_sm100.cu).
#pragma once

#include "debug.cuh"
#include "tc_common.cuh"

namespace b200 {

// delta = sum(dO * out) and the log-sum-exp in log2 units of every row, rows padded to whole tiles; with `range` also
// the partial maxima that gradient_scale() needs
int launch_bwd_prep(const BwdProblem& bp, bool bf16, float* lse2, float* delta, float2* range, cudaStream_t stream);

namespace tc {

constexpr int kT = 128;                 // tile edge: query rows, keys, TMEM lanes

inline int padded_rows(const Problem& p) { return (p.L + kT - 1) / kT * kT; }

// K-major operand descriptor of a 128-row tile; k-step kk covers 16 elements of D.
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t tile) { return smem_desc_sw128(tile, 16, 1024); }
__device__ __forceinline__ uint64_t kmajor_step(int kk) {
  return static_cast<uint64_t>(((kk >> 2) * kBoxBytes + (kk & 3) * 32) >> 4);
}
// MN-major B operand descriptor of the same tile (rows are the contraction axis);
// k-step kk covers 16 rows.
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t tile) { return smem_desc_sw128(tile, kBoxBytes, 1024); }
__device__ __forceinline__ uint64_t mnmajor_step(int kk) { return static_cast<uint64_t>(kk * (2048 >> 4)); }

// fp16 has no range to spare: where P and dS go into their second product as hi + lo, an fp32 value keeps its 22 bits
// only between 2^-3 and 2^16, and below 2^-25 nothing of it.  So both are brought there by powers of two that are taken
// out again with the result.  The prep kernel writes a log-sum-exp that makes the rebuilt probabilities 2^12 P; with
// gradient_scale() g, dS becomes 2^12 P (dP - delta) g, where g leaves the bound
//   |dP - delta| <= 2 Dv max |dO| max |V|     (over the rows, keys and heads that meet in one (batch, kv head))
// between 4 and 8.  What is lost of dS then is 2^-22 of its value or 2^-40 of the bound, whichever is larger.
constexpr float kPScale = 4096.f, kPScaleLog2 = 12.f;

// Partial maxima of a (batch, kv head): one CTA of the prep kernel for 1024 16-byte pieces of dO and V (four loads a
// thread), for more where that gives more than about eight CTAs to an SM, and at most 128 parts.
inline int range_parts(const Problem& p) {
  const int64_t pieces = (static_cast<int64_t>(p.group) * p.L + p.S) * (p.Dv / 8), streams = static_cast<int64_t>(p.B) * p.Hkv;
  int64_t n = (pieces + 1023) / 1024;
  const int64_t most = (8 * 148 + streams - 1) / streams;
  n = n > most ? most : n;
  return n < 1 ? 1 : (n > 128 ? 128 : static_cast<int>(n));
}

// g for (batch, kv head) number `stream`; the whole warp calls.  (Read past L1, as the row statistics should be.)
__device__ __forceinline__ float gradient_scale(const float2* range, int n_parts, int stream, int dv, int lane) {
  uint32_t go = 0, v = 0;   // (floats that are not negative order like their bits)
  for (int i = lane; i < n_parts; i += 32) {
    const float2 x = __ldcg(range + static_cast<int64_t>(stream) * n_parts + i);
    go = max(go, __float_as_uint(x.x));
    v = max(v, __float_as_uint(x.y));
  }
  go = __reduce_max_sync(0xffffffffu, go);
  v = __reduce_max_sync(0xffffffffu, v);
  const float bound = 2.f * static_cast<float>(dv) * __uint_as_float(go) * __uint_as_float(v);   // 0, or between 2^-47 and 2^42
  const int e = static_cast<int>(__float_as_uint(bound) >> 23) - 127;
  return bound > 0.f ? __uint_as_float(static_cast<uint32_t>(127 + 2 - e) << 23) : 1.f;
}

// One arrival for a warp whose lanes have all done what the barrier stands for.
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(bar));
}

// 32 columns (chunk c) of one thread's accumulator row (TMEM lane) -> 16-bit -> the 128-byte-swizzled staging tile a
// TMA store expects.
template <bool BF16>
__device__ __forceinline__ void stage_chunk(uint32_t acc_addr, bool have_acc, float mul, uint8_t* stage, int r, int c) {
  uint32_t v[32];
  if (have_acc) {
    tmem_ld_32x32(acc_addr + c * 32, v);
    tmem_ld_wait();
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0u;
  }
  uint32_t pk[16];
#pragma unroll
  for (int i = 0; i < 32; i += 2)
    pk[i >> 1] = pack2<BF16>(__uint_as_float(v[i]) * mul, __uint_as_float(v[i + 1]) * mul);
  uint8_t* box = stage + (c >> 1) * kBoxBytes + r * 128;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int unit = ((c & 1) * 4 + u) ^ (r & 7);
    *reinterpret_cast<uint4*>(box + unit * 16) = make_uint4(pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
  }
}

}  // namespace tc
}  // namespace b200

// Pieces shared by the tensor-core backward kernels (bwd_sm100.cu, bwd_wide_sm100.cu).
#pragma once

#include "debug.cuh"
#include "tc_common.cuh"

namespace b200 {

// delta = sum(dO * out) and the log-sum-exp in log2 units of every row, rows padded to whole tiles
int launch_bwd_prep(const BwdProblem& bp, bool bf16, float* lse2, float* delta, cudaStream_t stream);

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

// One arrival for a warp whose lanes have all done what the barrier stands for.
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(bar));
}

// 32 columns (chunk c) of one thread's accumulator row (TMEM lane) -> 16-bit -> the 128-byte-swizzled staging tile a
// TMA store expects; zeros for a row that is not to be kept (a key beyond kv_lens, whose own dP may be NaN).
template <bool BF16>
__device__ __forceinline__ void stage_chunk(uint32_t acc_addr, bool have_acc, float mul, uint8_t* stage, int r, int c,
                                            bool keep = true) {
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
    pk[i >> 1] = keep ? pack2<BF16>(__uint_as_float(v[i]) * mul, __uint_as_float(v[i + 1]) * mul) : 0u;
  uint8_t* box = stage + (c >> 1) * kBoxBytes + r * 128;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int unit = ((c & 1) * 4 + u) ^ (r & 7);
    *reinterpret_cast<uint4*>(box + unit * 16) = make_uint4(pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
  }
}

}  // namespace tc
}  // namespace b200

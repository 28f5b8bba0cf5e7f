// Tensor-core backward for sm_100a: TMA -> shared memory -> tcgen05 with every
// accumulator and every 16-bit intermediate (P, dS) in tensor memory.
//
// Three launches, no atomics, no [L,S] matrix in HBM:
//   bwd_prep_kernel     delta[b,h,i] = sum_d dO*out and the forward's log-sum-exp in log2
//                       units (rows without a visible key, and pad rows, get +inf so that
//                       their rebuilt probabilities are exactly 0)
//   bwd_dq_tc_kernel    one CTA per 128 query rows of one head; walks the key tiles:
//                         S = Q K^T, dP = dO V^T            (SS MMAs, accumulators in TMEM)
//                         dS = exp2(S*c - lse2) * (dP - delta)   -> 16-bit, over dP in TMEM
//                         dQ += dS K                         (TS MMA: A operand from TMEM)
//   bwd_dkv_tc_kernel   one CTA per 128 keys of one kv head; walks the group's query heads
//                       and their row tiles in the transposed orientation (TMEM lane = key):
//                         S^T = K Q^T, dP^T = V dO^T
//                         P^T -> over S^T, dS^T -> over dP^T (16-bit, in TMEM)
//                         dV += P^T dO, dK += dS^T Q         (TS MMAs)
//                       so the grouped-query sum is part of the accumulation.
// The two main kernels recompute S and dP independently (7 tile products instead of 5);
// in exchange dQ needs neither atomics nor an fp32 scratch tensor, and results are
// deterministic.  Arithmetic: torch_neuronx/_sdpa_math.py:133-176 with P and dS rounded
// to the input dtype before their second product (upstream rounds P the same way in the
// forward, :94).  Roles per CTA (320 threads): warps 0-7 elementwise (two threads per TMEM
// lane, 64 score columns each), warp 8 TMA producer, warp 9 MMA issuer.
//
// The dK/dV kernel's tensor memory is full with one pair of score-shaped accumulators:
//   TMEM columns  [0,128) S^T, P^T over it   [128,256) dP^T, dS^T over it   [256, 256+2D) dV and dK (fp32)
// and still neither role waits for the other for long, because the two halves of a tile's
// arithmetic alternate with two groups of products (in issue order, which is also the order
// in which the MMA pipe touches the shared columns):
//   elementwise  P^T(i) from S^T(i)        dS^T(i) from P^T(i), dP^T(i)
//   MMA          dK(i-1), dP^T(i)          dV(i), S^T(i+1)
// Whole 128-row query tiles: a score product with 64 columns costs the tensor pipe as much as one with 128 (its A
// operand is fetched from shared memory either way).  Measured, 1 x 32/8 x 4096, no mask: 3350 cycles per tile against
// 4024 for two 64-column units, of which the products take 2048 and the exponentials 1024 of the MUFU.
// The dQ kernel has one accumulator less and releases its scores as soon as they are in registers
// (layout and pipeline described at the kernel).
// Every wait is bounded (see tc_common.cuh).
#include "bwd_common.cuh"

#include <type_traits>

namespace b200 {

namespace {

using namespace ptx;
using namespace tc;

constexpr int kEWarps = 8;                // elementwise role: two column halves x four lane quadrants
constexpr int kParts = kEWarps / 4;
constexpr int kQ = kT / kParts;           // score columns of one thread, in chunks of 32
constexpr int kChunks = kQ / 32;
constexpr int kThreads = (kEWarps + 2) * 32;
constexpr uint32_t kColS = 0, kColDP = 128, kColAcc = 256;   // TMEM layout of the dK/dV kernel
constexpr int kProducerWarp = kEWarps;
constexpr int kMmaWarp = kEWarps + 1;
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxStages = 4;

template <int D> struct BCfg {
  static constexpr int kBoxes = D / 64;
  static constexpr int kTileBytes = kT * D * 2;
  static constexpr int kStages = (D == 128) ? 2 : 4;           // ring slots of two tiles each
  static constexpr int kSmemTiles = (2 + 2 * kStages) * kTileBytes;
  static constexpr int kStatBytes = kStages * 2 * kT * 4;       // (lse2, delta) of a query tile per slot
  static constexpr int kSmemBytes = kSmemTiles + kStatBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
};

struct BSync {
  uint64_t fixed_full;
  uint64_t ring_full[kMaxStages];
  uint64_t ring_empty[kMaxStages];
  uint64_t s_full;      // S^T of a tile is complete
  uint64_t dp_full;     // dP^T of a tile is complete
  uint64_t p_ready;     // the elementwise role has written P^T (16-bit, over S^T)
  uint64_t ds_ready;    // ... and dS^T (over dP^T)
  uint64_t acc_done;    // last accumulating MMA has retired
  uint64_t staged;
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
};

static_assert(sizeof(BSync) <= 272, "barrier block must fit its reserve (272 bytes + up to 1008 of alignment <= 1280)");

// ------------------------------------------------------------------ prep --

// (fp16) One part of the maxima that gradient_scale() combines, over dO and the visible rows of V, whose rows start on
// 16 bytes.  Infinities and NaN are left out: what they reach is not finite at any scale.
__device__ __forceinline__ void range_part(const BwdProblem& bp, float2* range, int n_parts, int unit) {
  const Problem& p = bp.f;
  __shared__ uint32_t sm[2][8];
  const int part = unit % n_parts, stream = unit / n_parts;
  const int hk = stream % p.Hkv, b = stream / p.Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const __half* go = reinterpret_cast<const __half*>(bp.dout) + b * bp.dos[0] + hk * p.group * bp.dos[1];
  const __half* vb = reinterpret_cast<const __half*>(p.v) + b * p.vs[0] + hk * p.vs[1];
  // 16-byte pieces of a row and in all (31 bits would end at 32 GB of dO in a kv head; 32 go beyond what a device holds)
  const uint32_t pieces = p.Dv / 8, n_l = p.L, step = n_parts * 256;
  const uint32_t go_pieces = p.group * n_l * pieces, all = go_pieces + valid_keys(p, b) * pieces;
  uint32_t top_go = 0, top_v = 0;   // of pairs of |x|; finite halves order like their bits
  for (uint32_t i0 = part * 256 + threadIdx.x; i0 < all; i0 += 4 * step) {
    uint4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {   // four loads in flight
      const uint32_t i = i0 + u * step;
      x[u] = make_uint4(0u, 0u, 0u, 0u);
      if (i < go_pieces) {
        const uint32_t row = i / pieces;
        x[u] = *reinterpret_cast<const uint4*>(go + row / n_l * bp.dos[1] + row % n_l * bp.dos[2] + i % pieces * 8);
      } else if (i < all) {
        x[u] = *reinterpret_cast<const uint4*>(vb + (i - go_pieces) / pieces * p.vs[2] + (i - go_pieces) % pieces * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t top = 0;
      for (const uint32_t w : {x[u].x, x[u].y, x[u].z, x[u].w}) {
        const uint32_t a = w & 0x7fff7fffu;
        top = __vmaxu2(top, a & __vcmpltu2(a, 0x7c007c00u));
      }
      if (i0 + u * step < go_pieces) top_go = __vmaxu2(top_go, top);
      else top_v = __vmaxu2(top_v, top);
    }
  }
  top_go = __reduce_max_sync(0xffffffffu, __vmaxu2(top_go, top_go >> 16) & 0xffffu);
  top_v = __reduce_max_sync(0xffffffffu, __vmaxu2(top_v, top_v >> 16) & 0xffffu);
  if (lane == 0) {
    sm[0][warp] = top_go;
    sm[1][warp] = top_v;
  }
  __syncthreads();
  if (threadIdx.x == 0 && dbg_range(p.status, DBG_BWD_TC * 100 + 11, unit, 1, static_cast<int64_t>(p.B) * p.Hkv * n_parts)) {
    uint32_t a = 0, c = 0;
    for (int i = 0; i < 8; ++i) {
      a = max(a, sm[0][i]);
      c = max(c, sm[1][i]);
    }
    range[unit] = make_float2(__half2float(__ushort_as_half(static_cast<unsigned short>(a))),
                              __half2float(__ushort_as_half(static_cast<unsigned short>(c))));
  }
}

// Eight lanes per row (four rows per warp) when rows can be read 16 bytes at a time,
// otherwise one warp per row with scalar loads.
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) bwd_prep_kernel(const BwdProblem bp, float* __restrict__ lse2,
                                                        float* __restrict__ delta, const int l_pad, float2* range,
                                                        const int n_parts, const unsigned range_blocks) {
  const Problem& p = bp.f;
  constexpr bool kHalf = std::is_same_v<T, __half>;
  if constexpr (kHalf) {
    if (blockIdx.x < range_blocks) {   // (first: they take longer than the others)
      pdl_wait();
      pdl_launch_dependents();
      range_part(bp, range, n_parts, static_cast<int>(blockIdx.x));
      return;
    }
  }
  constexpr int kLanes = VEC ? 8 : 32;             // lanes cooperating on one row
  constexpr int kRowsPerWarp = 32 / kLanes;
  const long long gwarp = (static_cast<long long>(blockIdx.x - range_blocks) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int sub = lane % kLanes;
  const long long row_id = gwarp * kRowsPerWarp + lane / kLanes;
  const long long total = static_cast<long long>(p.B) * p.Hq * l_pad;
  const bool in_range = row_id < total;
  const int i = in_range ? static_cast<int>(row_id % l_pad) : 0;
  const long long bh = in_range ? row_id / l_pad : 0;
  const int h = static_cast<int>(bh % p.Hq);
  const int b = static_cast<int>(bh / p.Hq);
  float d = 0.f, l2 = CUDART_INF_F;
  const bool live = in_range && i < p.L;
  // between the forward and the dK/dV kernel, both of whose launches this one overlaps
  pdl_wait();
  pdl_launch_dependents();
  if (live) {
    const T* go = reinterpret_cast<const T*>(bp.dout) + b * bp.dos[0] + h * bp.dos[1] + i * bp.dos[2];
    const T* o = reinterpret_cast<const T*>(p.out) + b * p.os[0] + h * p.os[1] + i * p.os[2];
    if (VEC) {
      for (int e = sub * 8; e < p.Dv; e += 64) {
        const uint4 a = *reinterpret_cast<const uint4*>(go + e);
        const uint4 c = *reinterpret_cast<const uint4*>(o + e);
        const T* av = reinterpret_cast<const T*>(&a);
        const T* cv = reinterpret_cast<const T*>(&c);
#pragma unroll
        for (int u = 0; u < 8; ++u) d = fmaf(to_f32<T>(av[u]), to_f32<T>(cv[u]), d);
      }
    } else {
      for (int e = sub; e < p.Dv; e += 32) d = fmaf(to_f32<T>(go[e * bp.dos[3]]), to_f32<T>(o[e * p.os[3]]), d);
    }
  }
#pragma unroll
  for (int off = kLanes / 2; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
  if (live && sub == 0) {
    const float l = p.lse[b * p.ls[0] + h * p.ls[1] + i * p.ls[2]];
    l2 = (l == -CUDART_INF_F) ? CUDART_INF_F : l * kLog2e;
    if (kHalf && range != nullptr) l2 -= kPScaleLog2;
  }
  if (in_range && sub == 0 && dbg_range(p.status, DBG_BWD_TC * 100 + 1, row_id, 1, total)) {
    lse2[row_id] = l2;
    delta[row_id] = live ? d : 0.f;
  }
}

// This thread's score columns to registers; 16-bit operands back, chunk c at + STEP c.
__device__ __forceinline__ void ld_chunks(uint32_t addr, uint32_t (&v)[kQ]) {
#pragma unroll
  for (int c = 0; c < kChunks; ++c) tmem_ld_32x32(addr + c * 32, reinterpret_cast<uint32_t(&)[32]>(v[c * 32]));
}
template <int STEP>
__device__ __forceinline__ void st_chunks(uint32_t addr, const uint32_t (&v)[kQ / 2]) {
#pragma unroll
  for (int c = 0; c < kChunks; ++c) tmem_st_32x16(addr + c * STEP, reinterpret_cast<const uint32_t(&)[16]>(v[c * 16]));
}

// acc[tmem d, 128 x 128] = A[smem tile, K-major] * B[smem tile, K-major]^T over D
// (PAD: only the first `steps` of the D / 16 k-steps, the columns beyond hold zeros)
template <int D, bool PAD>
__device__ __forceinline__ void issue_ss(uint32_t d_tmem, uint32_t a_tile, uint32_t b_tile, uint32_t idesc, int steps) {
  const uint64_t ad = kmajor_desc(a_tile), bd = kmajor_desc(b_tile);
  if (elect_one()) {
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      if (PAD && kk >= steps) break;
      mma_ss(d_tmem, ad + kmajor_step(kk), bd + kmajor_step(kk), idesc, kk > 0 ? 1u : 0u);
    }
  }
}
// acc[tmem d] (+)= A[tmem, 128 x 128] * B[smem tile, MN-major].  The 16-bit A operand sits where the elementwise
// role left it: contraction indices 32 c .. 32 c + 31 packed into columns [32 c, 32 c + 16) of the score-shaped
// buffer they came from.  PAD: the other 16 columns hold the remainders of that rounding (remainder2), a second set of
// products.
template <bool PAD>
__device__ __forceinline__ void issue_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_tile, uint32_t idesc, bool accumulate) {
  const uint64_t bd = mnmajor_desc(b_tile);
  if (elect_one()) {
#pragma unroll
    for (int kk = 0; kk < kT / 16; ++kk) {
      const uint32_t a = a_tmem + static_cast<uint32_t>((kk >> 1) * 32 + (kk & 1) * 8);
      mma_ts(d_tmem, a, bd + mnmajor_step(kk), idesc, (kk > 0 || accumulate) ? 1u : 0u);
      if (PAD) mma_ts(d_tmem, a + 16, bd + mnmajor_step(kk), idesc, 1u);
    }
  }
}

__device__ __forceinline__ void init_common_barriers(BSync* sync) {
  mbar_init(smem_u32(&sync->s_full), 1);
  mbar_init(smem_u32(&sync->dp_full), 1);
  mbar_init(smem_u32(&sync->p_ready), kEWarps);
  mbar_init(smem_u32(&sync->ds_ready), kEWarps);
  mbar_init(smem_u32(&sync->acc_done), 1);
  mbar_init(smem_u32(&sync->staged), kEWarps);
  mbar_init(smem_u32(&sync->drain), 1);
  sync->abort_flag = 0;
  mbar_fence_init();
}

__device__ __forceinline__ void drain_after_abort(BSync* sync, long long wait_limit) {
  // let whatever was issued retire before tensor memory is released
  if (elect_one()) mma_commit(smem_u32(&sync->drain));
  const long long t0 = clock64();
  while (!mbar_try_wait(smem_u32(&sync->drain), 0) && clock64() - t0 < kDrainCycles) {
  }
}

// ------------------------------------------------------------------ dQ kernel --
//
// Whole 128-key tiles per step (a 128-column score product costs the tensor pipe the same
// as a 64-column one).  The elementwise role copies S and dP of a tile into registers and
// releases the two accumulators at once, so the score products of tile j+1 run while it
// computes dS of tile j; dS goes to one of two operand buffers, so dQ += dS K of tile j runs
// while tile j+1 is being computed.  K tiles live until their dQ product, V tiles only until
// their dP product, hence separate rings (3 and 2 slots).
//   TMEM columns: [0,128) S, [128,256) dP, [256,320) [320,384) dS operand buffers, [384, 384+D) dQ

template <int D> struct ACfg {
  static constexpr int kBoxes = D / 64;
  static constexpr int kTileBytes = kT * D * 2;
  static constexpr int kKSlots = 3, kVSlots = 2;
  static constexpr int kSmemTiles = (2 + kKSlots + kVSlots) * kTileBytes;
  static constexpr int kSmemBytes = kSmemTiles + 1024 /*alignment slack*/ + 256 /*barriers*/;
};

struct ASync {
  uint64_t fixed_full;
  uint64_t k_full[3], k_empty[3];
  uint64_t v_full[2], v_empty[2];
  uint64_t sp_full;      // S and dP of a tile are complete
  uint64_t f_free;       // the elementwise role holds them in registers
  uint64_t e_ready[2];   // dS of a tile is in its operand buffer
  uint64_t op_empty[2];  // the product reading an operand buffer has retired
  uint64_t acc_done;
  uint64_t staged;
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
};

// One 16-bit bias element (the query's dtype) as fp32.
template <bool BF16>
__device__ __forceinline__ float bias_to_f32(const uint32_t bits16) {
  if (BF16) return __uint_as_float(bits16 << 16);
  return __half2float(__ushort_as_half(static_cast<unsigned short>(bits16)));
}

static_assert(sizeof(ASync) <= 272, "barrier block must fit its reserve (272 bytes + up to 1008 of alignment <= 1280)");

// PAD: head dimensions E, Dv (multiples of 8) that do not fill the D = 128 tile; the tensor maps carry the real
// extents (loads fill with zeros, stores clip) and the products skip the k-steps and output columns beyond them.
template <int D, bool BF16, bool BIAS, bool PAD>
__global__ void __launch_bounds__(kThreads, 1)
bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                 const __grid_constant__ CUtensorMap tm_dq, const Problem p, const float* lse2,
                 const float* delta, const int l_pad, const int n_qblk, const int streams_per_wave,
                 const long long wait_limit, const float2* range, const int n_parts) {
  using C = ACfg<D>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t tiles = (raw_addr + 1023u) & ~1023u;
  ASync* sync = reinterpret_cast<ASync*>(smem_raw + (tiles - raw_addr) + C::kSmemTiles);
  volatile int* abort_flag = &sync->abort_flag;

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;

  // Latest query blocks (most key tiles under a causal mask) first, within waves of
  // `streams_per_wave` (batch, kv head) key/value streams that fit in L2 together.
  const int n_streams = p.Hkv * p.B;
  const int full_wave_ctas = n_qblk * streams_per_wave * p.group;
  const int wave = static_cast<int>(blockIdx.x / full_wave_ctas);
  const int in_wave = static_cast<int>(blockIdx.x - static_cast<unsigned>(wave) * full_wave_ctas);
  const int first_stream = wave * streams_per_wave;
  const int wave_streams = (n_streams - first_stream) < streams_per_wave ? (n_streams - first_stream) : streams_per_wave;
  const int per_blk = wave_streams * p.group;
  const int qblk = n_qblk - 1 - in_wave / per_blk;
  const int rem = in_wave % per_blk;
  const int kv_stream = first_stream + rem / p.group;
  const int hk = kv_stream % p.Hkv;
  const int b = kv_stream / p.Hkv;
  const int h = hk * p.group + rem % p.group;
  const int row0 = qblk * kT;
  const int kv_limit = valid_keys(p, b);
  long long end = kv_limit, first = kv_limit;
  if (p.causal) {
    const int last_row = (row0 + kT < p.L ? row0 + kT : p.L) - 1;
    const long long e = static_cast<long long>(last_row) + p.causal_shift + 1;
    const long long f = static_cast<long long>(row0) + p.causal_shift + 1;
    end = e < end ? e : end;
    first = f < first ? f : first;
  }
  if (end < 0) end = 0;
  if (first < -1) first = -1;
  const int n_tiles = static_cast<int>((end + kT - 1) / kT);
  const int min_lim = static_cast<int>(first);

  const uint32_t q_tile = tiles, do_tile = tiles + C::kTileBytes;
  const uint32_t k_ring = tiles + 2 * C::kTileBytes;
  const uint32_t v_ring = k_ring + C::kKSlots * C::kTileBytes;

  if (warp == kProducerWarp && lane == 0) {
    mbar_init(smem_u32(&sync->fixed_full), 1);
    for (int s = 0; s < C::kKSlots; ++s) {
      mbar_init(smem_u32(&sync->k_full[s]), 1);
      mbar_init(smem_u32(&sync->k_empty[s]), 1);
    }
    for (int s = 0; s < C::kVSlots; ++s) {
      mbar_init(smem_u32(&sync->v_full[s]), 1);
      mbar_init(smem_u32(&sync->v_empty[s]), 1);
    }
    mbar_fence_init();
    if (n_tiles > 0) {
      const uint32_t bar = smem_u32(&sync->fixed_full);
      mbar_arrive_expect_tx(bar, 2 * C::kTileBytes);
      for (int bx = 0; bx < C::kBoxes; ++bx) {
        tma_load_4d(q_tile + bx * kBoxBytes, &tm_q, bar, bx * 64, row0, h, b);
        tma_load_4d(do_tile + bx * kBoxBytes, &tm_do, bar, bx * 64, row0, h, b);
      }
    }
    prefetch_tmap(&tm_dq);
  }
  if (tid == 0) {
    mbar_init(smem_u32(&sync->sp_full), 1);
    mbar_init(smem_u32(&sync->f_free), kEWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sync->e_ready[i]), kEWarps);
      mbar_init(smem_u32(&sync->op_empty[i]), 1);
    }
    mbar_init(smem_u32(&sync->acc_done), 1);
    mbar_init(smem_u32(&sync->staged), kEWarps);
    mbar_init(smem_u32(&sync->drain), 1);
    sync->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(&sync->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = sync->tmem_base;
  constexpr uint32_t kColS = 0, kColDP = 128, kColOp = 256, kColDQ = 384;
  constexpr bool kScaled = PAD && !BF16;   // see gradient_scale
  constexpr int kBufs = PAD ? 1 : 2;   // dS operand buffers (PAD: the second one holds the remainders, see remainder2)

  if (warp == kProducerWarp) {
    if (lane == 0) {
      for (int j = 0; j < n_tiles; ++j) {
        const int ks = j % C::kKSlots, vs = j % C::kVSlots;
        if (j >= C::kKSlots &&
            !wait_clocked(smem_u32(&sync->k_empty[ks]), (j / C::kKSlots - 1) & 1u, abort_flag, wait_limit)) {
          report(p.status, 11, j, ks);
          break;
        }
        {
          const uint32_t bar = smem_u32(&sync->k_full[ks]);
          mbar_arrive_expect_tx(bar, C::kTileBytes);
          for (int bx = 0; bx < C::kBoxes; ++bx)
            tma_load_4d(k_ring + ks * C::kTileBytes + bx * kBoxBytes, &tm_k, bar, bx * 64, j * kT, hk, b);
        }
        if (j >= C::kVSlots &&
            !wait_clocked(smem_u32(&sync->v_empty[vs]), (j / C::kVSlots - 1) & 1u, abort_flag, wait_limit)) {
          report(p.status, 11, j, 8 + vs);
          break;
        }
        {
          const uint32_t bar = smem_u32(&sync->v_full[vs]);
          mbar_arrive_expect_tx(bar, C::kTileBytes);
          for (int bx = 0; bx < C::kBoxes; ++bx)
            tma_load_4d(v_ring + vs * C::kTileBytes + bx * kBoxBytes, &tm_v, bar, bx * 64, j * kT, hk, b);
        }
      }
      if (*abort_flag != 0) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);   // copies in flight must land before exit
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    constexpr uint32_t idesc_score = make_idesc(BF16, false, kT, kT);
    const uint32_t idesc_acc = make_idesc(BF16, true, kT, PAD ? (p.E + 15) / 16 * 16 : D);
    const int steps_e = PAD ? (p.E + 15) / 16 : D / 16, steps_v = PAD ? (p.Dv + 15) / 16 : D / 16;
    bool alive = n_tiles > 0;
    if (alive) {
      alive = wait_clocked(smem_u32(&sync->fixed_full), 0, abort_flag, wait_limit);
      if (!alive && lane == 0) report(p.status, 12, -1, 0);
    }
    // S_j = Q K_j^T, dP_j = dO V_j^T over whole tiles
    auto issue_scores = [&](int j) -> bool {
      const int ks = j % C::kKSlots, vs = j % C::kVSlots;
      if (!wait_clocked(smem_u32(&sync->k_full[ks]), (j / C::kKSlots) & 1u, abort_flag, wait_limit) ||
          !wait_clocked(smem_u32(&sync->v_full[vs]), (j / C::kVSlots) & 1u, abort_flag, wait_limit)) {
        if (lane == 0) report(p.status, 12, j, ks);
        return false;
      }
      tc_fence_after_sync();
      // (PAD: these shapes came from kernels that leave out what lies beyond kv_lens; P = 0 times a NaN of V or K is NaN)
      if (PAD && kv_limit < p.S && (j + 1) * kT > kv_limit) {
        zero_tile_rows<C::kBoxes, kT>(k_ring + ks * C::kTileBytes, kv_limit - j * kT, lane);
        zero_tile_rows<C::kBoxes, kT>(v_ring + vs * C::kTileBytes, kv_limit - j * kT, lane);
      }
      const uint64_t qd = kmajor_desc(q_tile), kd = kmajor_desc(k_ring + ks * C::kTileBytes);
      const uint64_t od = kmajor_desc(do_tile), vd = kmajor_desc(v_ring + vs * C::kTileBytes);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          if (PAD && kk >= steps_e) break;
          mma_ss(tmem_base + kColS, qd + kmajor_step(kk), kd + kmajor_step(kk), idesc_score, kk > 0 ? 1u : 0u);
        }
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          if (PAD && kk >= steps_v) break;
          mma_ss(tmem_base + kColDP, od + kmajor_step(kk), vd + kmajor_step(kk), idesc_score, kk > 0 ? 1u : 0u);
        }
        mma_commit(smem_u32(&sync->sp_full));
        mma_commit(smem_u32(&sync->v_empty[vs]));   // V_j has no reader after dP_j
      }
      return true;
    };
    if (alive) alive = issue_scores(0);
    for (int j = 0; j < n_tiles && alive; ++j) {
      const int buf = j % kBufs, ks = j % C::kKSlots;
      // S_j and dP_j are in registers: the next tile's score products may overwrite them
      alive = wait_clocked(smem_u32(&sync->f_free), j & 1, abort_flag, wait_limit);
      if (!alive) {
        if (lane == 0) report(p.status, 13, j, 1);
        break;
      }
      tc_fence_after_sync();
      if (j + 1 < n_tiles) {
        alive = issue_scores(j + 1);
        if (!alive) break;
      }
      alive = wait_clocked(smem_u32(&sync->e_ready[buf]), (j / kBufs) & 1, abort_flag, wait_limit);
      if (!alive) {
        if (lane == 0) report(p.status, 13, j, 0);
        break;
      }
      tc_fence_after_sync();
      const uint64_t bd = mnmajor_desc(k_ring + ks * C::kTileBytes);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < kT / 16; ++kk) {   // dQ += dS_j K_j
          const uint32_t a = tmem_base + kColOp + buf * 64 + static_cast<uint32_t>(kk * 8);
          mma_ts(tmem_base + kColDQ, a, bd + mnmajor_step(kk), idesc_acc, (kk > 0 || j > 0) ? 1u : 0u);
          if (PAD) mma_ts(tmem_base + kColDQ, a + 64, bd + mnmajor_step(kk), idesc_acc, 1u);
        }
        mma_commit(smem_u32(&sync->op_empty[buf]));
        mma_commit(smem_u32(&sync->k_empty[ks]));
        if (j + 1 == n_tiles) mma_commit(smem_u32(&sync->acc_done));
      }
    }
    if (*abort_flag != 0) {
      if (elect_one()) mma_commit(smem_u32(&sync->drain));
      const long long t0 = clock64();
      while (!mbar_try_wait(smem_u32(&sync->drain), 0) && clock64() - t0 < kDrainCycles) {
      }
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------- elementwise role
    const int r = tid & (kT - 1);              // query row inside the tile = TMEM lane
    const int part = warp >> 2;                // which 64 of the tile's 128 score columns
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_off + kColS + part * kQ;
    const uint32_t dp_addr = tmem_base + lane_off + kColDP + part * kQ;
    const uint32_t op_addr = tmem_base + lane_off + kColOp + part * (kQ / 2);
    const uint32_t dq_addr = tmem_base + lane_off + kColDQ;
    // checked build: the column ranges of this thread's tensor-memory traffic; a violation drains the CTA
    if (!dbg_tmem(p.status, DBG_BWD_TC * 100 + 2, s_addr, tmem_base, kQ, kTmemCols) || !dbg_tmem(p.status, DBG_BWD_TC * 100 + 3, dp_addr, tmem_base, kQ, kTmemCols) ||
        !dbg_tmem(p.status, DBG_BWD_TC * 100 + 4, op_addr, tmem_base, 64 + kQ / 2, kTmemCols) || !dbg_tmem(p.status, DBG_BWD_TC * 100 + 5, dq_addr, tmem_base, D, kTmemCols))
      *abort_flag = 1;
    const int row_g = row0 + r;
    int lim = kv_limit;
    if (p.causal) {
      const long long c = static_cast<long long>(row_g) + p.causal_shift + 1;
      lim = c < lim ? static_cast<int>(c < 0 ? 0 : c) : lim;
    }
    const long long stat_idx = (static_cast<long long>(b) * p.Hq + h) * l_pad + row_g;
    const bool stat_ok = dbg_range(p.status, DBG_BWD_TC * 100 + 6, stat_idx, 1, static_cast<long long>(p.B) * p.Hq * l_pad);
    // Read past L1.  This grid starts when every CTA of the dK/dV grid is past its wait for the prep kernel, so the
    // statistics are in L2; but no wait of its own orders them before these reads, and they lie at the address where
    // the last call's lay, which an L1 may still hold.
    const float neg_l2 = stat_ok ? -__ldcg(lse2 + stat_idx) : -CUDART_INF_F;   // -inf for rows without a visible key
    const float dl = stat_ok ? __ldcg(delta + stat_idx) : 0.f;
    const float sl2 = p.scale * kLog2e;
    const float gs = kScaled ? gradient_scale(range, n_parts, kv_stream, p.Dv, lane) : 1.f;
    const float undo = kScaled ? 1.f / (gs * kPScale) : 1.f;
    bool alive = true;
    // this row of the forward's additive bias (the query's dtype, unit stride along the keys)
    const uint4* bias_row = nullptr;
    if constexpr (BIAS) {
      if (row_g < p.L)
        bias_row = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.bias) + b * p.bs[0] +
                                                  static_cast<long long>(h) * p.bs[1] +
                                                  static_cast<long long>(row_g) * p.bs[2]);
    }
    const bool bias_wide = BIAS && bias_rows_32b(p);
    for (int j = 0; j < n_tiles; ++j) {
      const int buf = j % kBufs;
      uint4 bv[BIAS ? kQ / 8 : 1];   // this thread's bias elements of the tile, fetched under the wait
      if constexpr (BIAS) load_bias_row(bv, bias_row, j * kT + part * kQ, p.S, bias_wide);
      const uint32_t* bw = reinterpret_cast<const uint32_t*>(bv);
      bool ok = wait_clocked(smem_u32(&sync->sp_full), j & 1, abort_flag, wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) report(p.status, 14, j, warp);
        alive = false;
        break;
      }
      tc_fence_after_sync();
      uint32_t sv[kQ], dv[kQ];
      ld_chunks(s_addr, sv);
      ld_chunks(dp_addr, dv);
      tmem_ld_wait();
      tc_fence_before_sync();
      warp_arrive(&sync->f_free, lane);
      const int col0 = j * kT + part * kQ;
      const bool need_mask = col0 + kQ > min_lim;
      uint32_t pk[kQ / 2], lo[PAD ? kQ / 2 : 1];
      // two columns per instruction (packed fp32 pairs) wherever the arithmetic allows
      const uint64_t sl2_2 = f2_pack(sl2, sl2), neg_dl2 = f2_pack(-dl * gs, -dl * gs), gs2 = f2_pack(gs, gs);
#pragma unroll
      for (int i = 0; i < kQ; i += 2) {
        float off0 = neg_l2, off1 = neg_l2;
        if constexpr (BIAS) {
          off0 = fmaf(bias_to_f32<BF16>(bw[i >> 1] & 0xffffu), kLog2e, neg_l2);
          off1 = fmaf(bias_to_f32<BF16>(bw[i >> 1] >> 16), kLog2e, neg_l2);
        }
        float a0, a1;
        f2_unpack(f2_fma(f2_pack(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sl2_2, f2_pack(off0, off1)), a0, a1);
        float p0 = ex2(a0);
        float p1 = ex2(a1);
        if (need_mask) {
          p0 = (col0 + i < lim) ? p0 : 0.f;
          p1 = (col0 + i + 1 < lim) ? p1 : 0.f;
        }
        float d0, d1;
        const uint64_t dp2 = f2_pack(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1]));
        f2_unpack(f2_mul(f2_pack(p0, p1), kScaled ? f2_fma(dp2, gs2, neg_dl2) : f2_add(dp2, neg_dl2)), d0, d1);
        pk[i >> 1] = pack2<BF16>(d0, d1);
        if constexpr (PAD) lo[i >> 1] = remainder2<BF16>(d0, d1, pk[i >> 1]);
      }
      if (j >= kBufs) {   // the product that read this operand buffer before must have retired
        ok = wait_clocked(smem_u32(&sync->op_empty[buf]), (j / kBufs - 1) & 1, abort_flag, wait_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) report(p.status, 16, j, warp);
          alive = false;
          break;
        }
        tc_fence_after_sync();
      }
      st_chunks<16>(op_addr + buf * 64, pk);
      if constexpr (PAD) st_chunks<16>(op_addr + 64, lo);
      tmem_st_wait();
      tc_fence_before_sync();
      warp_arrive(&sync->e_ready[buf], lane);
    }
    if (alive && n_tiles > 0) {
      bool ok = wait_clocked(smem_u32(&sync->acc_done), 0, abort_flag, wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) report(p.status, 15, 0, warp);
        alive = false;
      }
      tc_fence_after_sync();
    }
    if (alive) {
      uint8_t* stage = smem_raw + (q_tile - raw_addr);   // Q is no longer needed
      for (int c = part; c < D / 32; c += kParts) stage_chunk<BF16>(dq_addr, n_tiles > 0, p.scale * undo, stage, r, c);
      fence_proxy_async_smem();
      warp_arrive(&sync->staged, lane);
      if (tid == 0 && wait_clocked(smem_u32(&sync->staged), 0, abort_flag, wait_limit)) {
        for (int bx = 0; bx < C::kBoxes; ++bx) {
          if (PAD && bx * 64 >= p.E) break;
          tma_store_4d(&tm_dq, q_tile + bx * kBoxBytes, bx * 64, row0, h, b);
        }
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }

  // Launched as a programmatic dependent of the dK/dV kernel, of which it reads nothing.  One CTA -- the last
  // of the grid, which is also the last to be placed -- waits for that grid before it exits, so that this grid
  // cannot complete before it and work queued behind finds both done; the others must not wait (a finished CTA
  // parked on its SM would keep the next one from starting).
  if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// --------------------------------------------------------------- dK/dV kernel --

template <int D, bool BF16, bool BIAS, bool PAD>
__global__ void __launch_bounds__(kThreads, 1)
bwd_dkv_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                  const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                  const Problem p, const float* lse2, const float* delta, const int l_pad,
                  const int n_kblk, const int streams_per_wave, const long long wait_limit, const float2* range,
                  const int n_parts) {
  using C = BCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t tiles = (raw_addr + 1023u) & ~1023u;
  float* stats = reinterpret_cast<float*>(smem_raw + (tiles - raw_addr) + C::kSmemTiles);
  BSync* sync = reinterpret_cast<BSync*>(smem_raw + (tiles - raw_addr) + C::kSmemTiles + C::kStatBytes);
  volatile int* abort_flag = &sync->abort_flag;

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;

  // Earliest key blocks (seen by the most query tiles under a causal mask) first, within waves of
  // `streams_per_wave` (batch, kv head) groups whose query-side operands fit in L2 together.
  const int n_streams = p.Hkv * p.B;
  const int full_wave_ctas = n_kblk * streams_per_wave;
  const int wave = static_cast<int>(blockIdx.x / full_wave_ctas);
  const int in_wave = static_cast<int>(blockIdx.x - static_cast<unsigned>(wave) * full_wave_ctas);
  const int first_stream = wave * streams_per_wave;
  const int wave_streams = (n_streams - first_stream) < streams_per_wave ? (n_streams - first_stream) : streams_per_wave;
  const int kblk = in_wave / wave_streams;
  const int kv_stream = first_stream + in_wave % wave_streams;
  const int hk = kv_stream % p.Hkv;
  const int b = kv_stream / p.Hkv;
  const int j0 = kblk * kT;
  // A programmatic dependent of the prep kernel: its launch overlaps that kernel, nothing of global memory is touched
  // before the wait.  (The dQ kernel, which follows without a wait of its own: see there.)
  pdl_wait();
  pdl_launch_dependents();
  const int n_keys = valid_keys(p, b);
  const int n_qt = (p.L + kT - 1) / kT;
  int i_first = 0;
  if (p.causal) {
    const long long f = static_cast<long long>(j0) - p.causal_shift;   // first row that sees key j0
    i_first = f <= 0 ? 0 : (f >= p.L ? n_qt : static_cast<int>(f / kT));
  }
  const int per_head = (j0 < n_keys && n_qt > i_first) ? n_qt - i_first : 0;
  const int n_items = per_head * p.group;

  const uint32_t k_tile = tiles, v_tile = tiles + C::kTileBytes;
  const uint32_t ring = tiles + 2 * C::kTileBytes;   // slot s: Q at ring + 2 s tile, dO right after

  if (warp == kProducerWarp && lane == 0) {
    mbar_init(smem_u32(&sync->fixed_full), 1);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(smem_u32(&sync->ring_full[s]), 1);
      mbar_init(smem_u32(&sync->ring_empty[s]), 1);
    }
    mbar_fence_init();
    if (n_items > 0) {
      const uint32_t bar = smem_u32(&sync->fixed_full);
      mbar_arrive_expect_tx(bar, 2 * C::kTileBytes);
      for (int bx = 0; bx < C::kBoxes; ++bx) {
        tma_load_4d(k_tile + bx * kBoxBytes, &tm_k, bar, bx * 64, j0, hk, b);
        tma_load_4d(v_tile + bx * kBoxBytes, &tm_v, bar, bx * 64, j0, hk, b);
      }
    }
    prefetch_tmap(&tm_dk);
    prefetch_tmap(&tm_dv);
  }
  if (tid == 0) init_common_barriers(sync);
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(&sync->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = sync->tmem_base;
  constexpr uint32_t kColDV = kColAcc, kColDK = kColAcc + D;
  constexpr bool kScaled = PAD && !BF16;   // see gradient_scale

  if (warp == kProducerWarp) {
    // the whole warp runs the loop: the lanes copy the query tile's row statistics into
    // the slot, lane 0 then arms the barrier (its release makes the copies visible) and
    // starts the tile copies
    bool alive = true;
    // The row statistics of an item are fetched one item ahead, so that their global-memory latency
    // passes during the wait for the slot instead of between the slot's release and the tile copies
    // (measured: 1.2-2.0 k cycles per item on the path that feeds the MMA warp).
    float4 st_l = make_float4(0.f, 0.f, 0.f, 0.f), st_d = st_l;
    auto fetch_stats = [&](int item) {
      const int h_ = hk * p.group + item / per_head;
      const int qrow_ = (i_first + item % per_head) * kT;
      const long long src = (static_cast<long long>(b) * p.Hq + h_) * l_pad + qrow_;
      if (dbg_range(p.status, DBG_BWD_TC * 100 + 10, src, kT, static_cast<long long>(p.B) * p.Hq * l_pad)) {
        st_l = reinterpret_cast<const float4*>(lse2 + src)[lane];
        st_d = reinterpret_cast<const float4*>(delta + src)[lane];
      }
    };
    float gs = 1.f;   // delta is kept times this
    if (n_items > 0) fetch_stats(0);
    for (int it = 0; it < n_items && alive; ++it) {
      const int stage = it % C::kStages;
      const uint32_t round = static_cast<uint32_t>(it / C::kStages);
      if (round > 0) {
        alive = wait_clocked(smem_u32(&sync->ring_empty[stage]), (round - 1) & 1u, abort_flag, wait_limit);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) {
          if (lane == 0) report(p.status, 21, it, stage);
          break;
        }
      }
      const int h = hk * p.group + it / per_head;
      const int qrow0 = (i_first + it % per_head) * kT;
      float4* dst = reinterpret_cast<float4*>(stats + stage * 2 * kT);
      const uint32_t bar = smem_u32(&sync->ring_full[stage]);
      auto copy = [&]() {
        const uint32_t q_dst = ring + stage * 2 * C::kTileBytes;
        for (int bx = 0; bx < C::kBoxes; ++bx) {
          tma_load_4d(q_dst + bx * kBoxBytes, &tm_q, bar, bx * 64, qrow0, h, b);
          tma_load_4d(q_dst + C::kTileBytes + bx * kBoxBytes, &tm_do, bar, bx * 64, qrow0, h, b);
        }
      };
      if constexpr (kScaled) {   // the copies go first: the maxima behind gs take a trip to L2
        if (lane == 0) {
          mbar_expect_tx(bar, 2 * C::kTileBytes);
          copy();
        }
        __syncwarp();
        if (it == 0) gs = gradient_scale(range, n_parts, kv_stream, p.Dv, lane);
        st_d = make_float4(st_d.x * gs, st_d.y * gs, st_d.z * gs, st_d.w * gs);
      }
      dst[lane] = st_l;
      dst[32 + lane] = st_d;
      __syncwarp();
      if (lane == 0) {
        if constexpr (kScaled) {
          mbar_arrive(bar);
        } else {
          mbar_arrive_expect_tx(bar, 2 * C::kTileBytes);
          copy();
        }
      }
      if (it + 1 < n_items) fetch_stats(it + 1);
    }
    if (*abort_flag != 0 && lane == 0) {
      for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    constexpr uint32_t idesc_score = make_idesc(BF16, false, kT, kT);
    const uint32_t idesc_dk = make_idesc(BF16, true, kT, PAD ? (p.E + 15) / 16 * 16 : D);
    const uint32_t idesc_dv = make_idesc(BF16, true, kT, PAD ? (p.Dv + 15) / 16 * 16 : D);
    const int steps_e = PAD ? (p.E + 15) / 16 : D / 16, steps_v = PAD ? (p.Dv + 15) / 16 : D / 16;
    bool alive = n_items > 0;
    if (alive) {
      alive = wait_clocked(smem_u32(&sync->fixed_full), 0, abort_flag, wait_limit);
      if (!alive && lane == 0) report(p.status, 22, -1, 0);
      // (as in the dQ kernel: the keys' own gradients would be 0 x NaN)
      if (PAD && alive && n_keys < p.S && j0 + kT > n_keys) zero_tile_rows<C::kBoxes, kT>(v_tile, n_keys - j0, lane);
    }
    auto q_tile = [&](int it) { return ring + (it % C::kStages) * 2 * C::kTileBytes; };   // dO right behind it
    // S^T_i = K Q_i^T (waits for the query tile); the MMA pipe executes in issue order, so it may be issued right
    // behind the product that reads P^T_{i-1} from the same columns
    auto issue_s = [&](int it) -> bool {
      const uint32_t round = static_cast<uint32_t>(it / C::kStages);
      if (!wait_clocked(smem_u32(&sync->ring_full[it % C::kStages]), round & 1u, abort_flag, wait_limit)) {
        if (lane == 0) report(p.status, 22, it, it % C::kStages);
        return false;
      }
      tc_fence_after_sync();
      issue_ss<D, PAD>(tmem_base + kColS, k_tile, q_tile(it), idesc_score, steps_e);
      if (elect_one()) mma_commit(smem_u32(&sync->s_full));
      return true;
    };
    auto issue_dp = [&](int it) {   // dP^T_i = V dO_i^T
      issue_ss<D, PAD>(tmem_base + kColDP, v_tile, q_tile(it) + C::kTileBytes, idesc_score, steps_v);
      if (elect_one()) mma_commit(smem_u32(&sync->dp_full));
    };
    if (alive) alive = issue_s(0);
    if (alive) issue_dp(0);
    for (int it = 0; it < n_items && alive; ++it) {
      const bool more = it + 1 < n_items;
      alive = wait_clocked(smem_u32(&sync->p_ready), it & 1, abort_flag, wait_limit);
      if (!alive) {
        if (lane == 0) report(p.status, 23, it, 0);
        break;
      }
      tc_fence_after_sync();
      issue_ts<PAD>(tmem_base + kColDV, tmem_base + kColS, q_tile(it) + C::kTileBytes, idesc_dv, it > 0);   // dV += P^T dO
      if (more) {
        alive = issue_s(it + 1);
        if (!alive) break;
      }
      alive = wait_clocked(smem_u32(&sync->ds_ready), it & 1, abort_flag, wait_limit);
      if (!alive) {
        if (lane == 0) report(p.status, 23, it, 1);
        break;
      }
      tc_fence_after_sync();
      issue_ts<PAD>(tmem_base + kColDK, tmem_base + kColDP, q_tile(it), idesc_dk, it > 0);                  // dK += dS^T Q
      if (elect_one()) {
        mma_commit(smem_u32(&sync->ring_empty[it % C::kStages]));
        if (!more) mma_commit(smem_u32(&sync->acc_done));
      }
      if (more) issue_dp(it + 1);
    }
    if (*abort_flag != 0) drain_after_abort(sync, wait_limit);
    __syncwarp();
  } else {
    // -------------------------------------------------------- elementwise role
    const int r = tid & (kT - 1);              // key inside the tile = TMEM lane
    const int part = warp >> 2;                // which 64 of the tile's 128 query columns
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_off + kColS + part * kQ;
    const uint32_t dp_addr = tmem_base + lane_off + kColDP + part * kQ;
    // checked build: the score-shaped buffers and the two accumulators
    if (!dbg_tmem(p.status, DBG_BWD_TC * 100 + 7, s_addr, tmem_base, kQ, kTmemCols) ||
        !dbg_tmem(p.status, DBG_BWD_TC * 100 + 8, dp_addr, tmem_base, kQ, kTmemCols) ||
        !dbg_tmem(p.status, DBG_BWD_TC * 100 + 9, tmem_base + lane_off + kColDK, tmem_base, D, kTmemCols))
      *abort_flag = 1;
    const int key_g = j0 + r;
    // query rows i >= i_min see this key; a padded key is seen by nobody
    int i_min = 0;
    if (p.causal) {
      const long long v = static_cast<long long>(key_g) - p.causal_shift;
      i_min = v < 0 ? 0 : (v > (1 << 30) ? (1 << 30) : static_cast<int>(v));
    }
    if (key_g >= n_keys) i_min = 1 << 30;
    const bool tile_has_padding = j0 + kT > n_keys;
    const float sl2 = p.scale * kLog2e;
    const uint64_t sl2_2 = f2_pack(sl2, sl2);
    const float gs = kScaled ? gradient_scale(range, n_parts, kv_stream, p.Dv, lane) : 1.f;
    const uint64_t gs2 = f2_pack(gs, gs);
    bool alive = true;
    int head = hk * p.group, tile = 0;         // query head and row tile (from i_first) of an item
    for (int it = 0; it < n_items; ++it) {
      const int qrow0 = (i_first + tile) * kT + part * kQ;   // first query row of this thread's columns
      uint32_t bq[BIAS ? kQ / 2 : 1];   // bias of this key under the thread's query rows, fetched under the wait
      if constexpr (BIAS) {
        // neighbouring lanes are neighbouring keys: each load is one 64-byte piece per warp
        const uint16_t* col = static_cast<const uint16_t*>(p.bias) + b * p.bs[0] + static_cast<long long>(head) * p.bs[1] + key_g;
#pragma unroll
        for (int i = 0; i < kQ; i += 2) {
          uint32_t lo = 0u, hi = 0u;
          if (key_g < p.S && qrow0 + i < p.L) lo = __ldg(col + static_cast<long long>(qrow0 + i) * p.bs[2]);
          if (key_g < p.S && qrow0 + i + 1 < p.L) hi = __ldg(col + static_cast<long long>(qrow0 + i + 1) * p.bs[2]);
          bq[i >> 1] = lo | (hi << 16);
        }
      }
      if (++tile == per_head) {
        tile = 0;
        ++head;
      }
      bool ok = wait_clocked(smem_u32(&sync->s_full), it & 1, abort_flag, wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) report(p.status, 24, it, warp);
        alive = false;
        break;
      }
      tc_fence_after_sync();
      const float4* st4 = reinterpret_cast<const float4*>(stats + (it % C::kStages) * 2 * kT) + part * (kQ / 4);
      // some key of this tile hides some row of these columns
      const bool need_mask = tile_has_padding ||
                             (p.causal && static_cast<long long>(qrow0) < static_cast<long long>(j0) + kT - 1 - p.causal_shift);
      float pr[kQ];
      {
        uint32_t sv[kQ], pk[kQ / 2], lo[PAD ? kQ / 2 : 1];
        ld_chunks(s_addr, sv);
        tmem_ld_wait();
#pragma unroll
        for (int q4 = 0; q4 < kQ / 4; ++q4) {
          const float4 l4 = st4[q4];
          const float ls[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {   // two query columns per instruction (packed fp32 pairs)
            const int i = q4 * 4 + e;
            float off0 = -ls[e], off1 = -ls[e + 1];
            if constexpr (BIAS) {
              off0 = fmaf(bias_to_f32<BF16>(bq[i >> 1] & 0xffffu), kLog2e, off0);
              off1 = fmaf(bias_to_f32<BF16>(bq[i >> 1] >> 16), kLog2e, off1);
            }
            float a0, a1;
            f2_unpack(f2_fma(f2_pack(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sl2_2, f2_pack(off0, off1)), a0, a1);
            float p0 = ex2(a0), p1 = ex2(a1);
            if (need_mask) {
              p0 = (qrow0 + i >= i_min) ? p0 : 0.f;
              p1 = (qrow0 + i + 1 >= i_min) ? p1 : 0.f;
            }
            pr[i] = p0;
            pr[i + 1] = p1;
            pk[i >> 1] = pack2<BF16>(p0, p1);
            if constexpr (PAD) lo[i >> 1] = remainder2<BF16>(p0, p1, pk[i >> 1]);
          }
        }
        st_chunks<32>(s_addr, pk);
        if constexpr (PAD) st_chunks<32>(s_addr + 16, lo);
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrive(&sync->p_ready, lane);
      }
      ok = wait_clocked(smem_u32(&sync->dp_full), it & 1, abort_flag, wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) report(p.status, 26, it, warp);
        alive = false;
        break;
      }
      tc_fence_after_sync();
      uint32_t dv[kQ], pk[kQ / 2], lo[PAD ? kQ / 2 : 1];
      ld_chunks(dp_addr, dv);
      tmem_ld_wait();
#pragma unroll
      for (int q4 = 0; q4 < kQ / 4; ++q4) {
        const float4 d4 = st4[kT / 4 + q4];
        const float nd[4] = {-d4.x, -d4.y, -d4.z, -d4.w};
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const int i = q4 * 4 + e;
          float d0, d1;
          const uint64_t dp2 = f2_pack(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1])), nd2 = f2_pack(nd[e], nd[e + 1]);
          f2_unpack(f2_mul(f2_pack(pr[i], pr[i + 1]), kScaled ? f2_fma(dp2, gs2, nd2) : f2_add(dp2, nd2)), d0, d1);
          pk[i >> 1] = pack2<BF16>(d0, d1);
          if constexpr (PAD) lo[i >> 1] = remainder2<BF16>(d0, d1, pk[i >> 1]);
        }
      }
      st_chunks<32>(dp_addr, pk);
      if constexpr (PAD) st_chunks<32>(dp_addr + 16, lo);
      tmem_st_wait();
      tc_fence_before_sync();
      warp_arrive(&sync->ds_ready, lane);
    }
    if (alive && n_items > 0) {
      bool ok = wait_clocked(smem_u32(&sync->acc_done), 0, abort_flag, wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) report(p.status, 25, 0, warp);
        alive = false;
      }
      tc_fence_after_sync();
    }
    if (alive) {
      // ring slot 0 is idle by now: its two tiles stage dK and dV
      uint8_t* stage_k = smem_raw + (ring - raw_addr);
      uint8_t* stage_v = stage_k + C::kTileBytes;
      for (int c = part; c < D / 16; c += kParts) {
        if (c < D / 32) stage_chunk<BF16>(tmem_base + lane_off + kColDK, n_items > 0, p.scale * (kScaled ? 1.f / (gs * kPScale) : 1.f), stage_k, r, c);
        else stage_chunk<BF16>(tmem_base + lane_off + kColDV, n_items > 0, kScaled ? 1.f / kPScale : 1.f, stage_v, r, c - D / 32);
      }
      fence_proxy_async_smem();
      warp_arrive(&sync->staged, lane);
      if (tid == 0 && wait_clocked(smem_u32(&sync->staged), 0, abort_flag, wait_limit)) {
        for (int bx = 0; bx < C::kBoxes; ++bx) {
          if (!PAD || bx * 64 < p.E) tma_store_4d(&tm_dk, ring + bx * kBoxBytes, bx * 64, j0, hk, b);
          if (!PAD || bx * 64 < p.Dv) tma_store_4d(&tm_dv, ring + C::kTileBytes + bx * kBoxBytes, bx * 64, j0, hk, b);
        }
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------ host side --

}  // namespace

int launch_bwd_prep(const BwdProblem& bp, bool bf16, float* lse2, float* delta, float2* range, cudaStream_t stream) {
  const Problem& p = bp.f;
  const int l_pad = padded_rows(p);
  const long long rows = static_cast<long long>(p.B) * p.Hq * l_pad;
  auto rows_aligned = [](const void* base, const int64_t* st) {
    return st[3] == 1 && reinterpret_cast<uintptr_t>(base) % 16 == 0 && st[0] % 8 == 0 && st[1] % 8 == 0 && st[2] % 8 == 0;
  };
  const bool vec = p.Dv % 8 == 0 && rows_aligned(bp.dout, bp.dos) && rows_aligned(p.out, p.os);
  const long long warps = vec ? (rows + 3) / 4 : rows;
  const long long blocks = (warps * 32 + 255) / 256;
  const int n_parts = range_parts(p);
  const long long extra = range != nullptr ? static_cast<long long>(p.B) * p.Hkv * n_parts : 0;
  if (blocks + extra > 0x7fffffffLL) return B200_SDPA_ERR_UNSUPPORTED;
  const unsigned grid = static_cast<unsigned>(blocks + extra);
  auto kern = bf16 ? (vec ? bwd_prep_kernel<__nv_bfloat16, true> : bwd_prep_kernel<__nv_bfloat16, false>)
                   : (vec ? bwd_prep_kernel<__half, true> : bwd_prep_kernel<__half, false>);
  if (!launch_pdl(kern, dim3(grid), 256, 0, stream, bp, lse2, delta, l_pad, range, n_parts, static_cast<unsigned>(extra)))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_BWD_PREP);
  return B200_SDPA_OK;
}

namespace {

template <int D, bool BF16, bool BIAS, bool PAD = false>
int launch_tc(const BwdProblem& bp, float* lse2, float* delta, float2* range, cudaStream_t stream) {
  using C = BCfg<D>;
  const Problem& p = bp.f;
  CUtensorMap tq, tk, tv, tdo, tdq, tdk, tdv;
  if (!make_map(&tq, p.q, BF16, p.E, p.L, p.Hq, p.B, p.qs) || !make_map(&tk, p.k, BF16, p.E, p.S, p.Hkv, p.B, p.ks) ||
      !make_map(&tv, p.v, BF16, p.Dv, p.S, p.Hkv, p.B, p.vs) || !make_map(&tdo, bp.dout, BF16, p.Dv, p.L, p.Hq, p.B, bp.dos) ||
      !make_map(&tdq, bp.dq, BF16, p.E, p.L, p.Hq, p.B, bp.dqs) ||
      !make_map(&tdk, bp.dk, BF16, p.E, p.S, p.Hkv, p.B, bp.dks) ||
      !make_map(&tdv, bp.dv, BF16, p.Dv, p.S, p.Hkv, p.B, bp.dvs))
    return B200_SDPA_ERR_CUDA;
  auto kq = bwd_dq_tc_kernel<D, BF16, BIAS, PAD>;
  auto kkv = bwd_dkv_tc_kernel<D, BF16, BIAS, PAD>;
  if (cudaFuncSetAttribute(kq, cudaFuncAttributeMaxDynamicSharedMemorySize, ACfg<D>::kSmemBytes) != cudaSuccess ||
      cudaFuncSetAttribute(kkv, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) {
    cudaGetLastError();
    return B200_SDPA_ERR_CUDA;
  }
  const int l_pad = padded_rows(p);
  const int prep = launch_bwd_prep(bp, BF16, lse2, delta, range, stream);
  if (prep != B200_SDPA_OK) return prep;
  const int n_qblk = (p.L + kT - 1) / kT, n_kblk = (p.S + kT - 1) / kT;
  const long long grid_q = static_cast<long long>(n_qblk) * p.Hq * p.B;
  const long long grid_kv = static_cast<long long>(n_kblk) * p.Hkv * p.B;
  if (grid_q > 0x7fffffffLL || grid_kv > 0x7fffffffLL) return B200_SDPA_ERR_UNSUPPORTED;
  const long long limit = wait_limit_cycles();
  const long long n_streams = static_cast<long long>(p.Hkv) * p.B;
  // the dQ kernel streams keys and values; the dK/dV kernel the queries, dO and row statistics of a group
  const int wave_q = kv_streams_per_wave(static_cast<long long>(p.S) * (p.E + p.Dv) * 2, n_streams);
  const int wave_kv = kv_streams_per_wave(static_cast<long long>(p.L) * p.group * ((p.E + p.Dv) * 2 + 8), n_streams);
  // The two kernels are independent of each other (both read the row statistics of the kernel before them).
  // The dK/dV kernel, whose CTAs are long, goes first and releases its dependents as soon as its last CTA is
  // resident; the dQ kernel is a programmatic dependent launch, so its CTAs take the SMs the first kernel's
  // tail leaves idle.  It waits for the first kernel's completion only before it exits (stream order for
  // whatever follows).
  const float* c_lse2 = lse2;
  const float* c_delta = delta;
  const float2* c_range = range;
  const int n_parts = range_parts(p);
  if (!launch_pdl(kkv, dim3(static_cast<unsigned>(grid_kv)), kThreads, C::kSmemBytes, stream, tq, tk, tv, tdo, tdk, tdv, p, c_lse2,
                  c_delta, l_pad, n_kblk, wave_kv, limit, c_range, n_parts))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_BWD_DKV);
  if (!launch_pdl(kq, dim3(static_cast<unsigned>(grid_q)), kThreads, ACfg<D>::kSmemBytes, stream, tq, tk, tv, tdo, tdq, p, c_lse2,
                  c_delta, l_pad, n_qblk, wave_q, limit, c_range, n_parts))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_BWD_DQ);
  return B200_SDPA_OK;
}

}  // namespace


namespace {

// What every head dimension needs.
bool operands_eligible(const BwdProblem& bp, int dtype, bool* alignment_only_failure) {
  const Problem& p = bp.f;
  if (dtype != B200_SDPA_F16 && dtype != B200_SDPA_BF16) return false;
  if (bp.dbias != nullptr) return false;   // the logit gradient is written by the CUDA-core kernels only
  if (!(p.scale > 0.f) || !(p.scale < 1e30f)) return false;
  if (p.L < 1 || p.S < 1) return false;
  if (p.bias != nullptr) {
    if (!bias_readable(p, dtype, alignment_only_failure)) return false;   // as in the forward
  }
  const bool ok = strides_ok(p.q, p.qs, p.L, p.Hq, p.B) && strides_ok(p.k, p.ks, p.S, p.Hkv, p.B) &&
                  strides_ok(p.v, p.vs, p.S, p.Hkv, p.B) && strides_ok(bp.dout, bp.dos, p.L, p.Hq, p.B) &&
                  strides_ok(bp.dq, bp.dqs, p.L, p.Hq, p.B) && strides_ok(bp.dk, bp.dks, p.S, p.Hkv, p.B) &&
                  strides_ok(bp.dv, bp.dvs, p.S, p.Hkv, p.B);
  if (!ok && alignment_only_failure) *alignment_only_failure = true;
  return ok;
}

}  // namespace

bool bwd_tc_eligible(const BwdProblem& bp, int dtype, bool* alignment_only_failure) {
  const Problem& p = bp.f;
  if (alignment_only_failure) *alignment_only_failure = false;
  if (!bwd_wide_dims(p) && (p.E != p.Dv || (p.E != 64 && p.E != 128))) return false;
  return operands_eligible(bp, dtype, alignment_only_failure);
}

// Head dimensions between 64 and 128 (multiples of 8) on zero-filled 128-wide tiles, as in the forward.  Fewer
// than 64 rows or keys leave more than half of every tile empty and the CUDA-core kernels, one launch fewer, are
// not slower there.
bool bwd_padded_eligible(const BwdProblem& bp, int dtype) {
  const Problem& p = bp.f;
  if (p.L < 64 || p.S < 64) return false;
  const int hi = p.E > p.Dv ? p.E : p.Dv;
  if (hi <= 64 || hi > 128 || p.E % 8 != 0 || p.Dv % 8 != 0 || (p.E == 128 && p.Dv == 128)) return false;
  return operands_eligible(bp, dtype, nullptr);
}

namespace {

uint64_t statistics_bytes(const BwdProblem& bp) {
  return 2ull * sizeof(float) * static_cast<uint64_t>(bp.f.B) * bp.f.Hq * padded_rows(bp.f);
}
// P and dS as hi + lo fp16 pairs: the shapes whose maxima the prep kernel takes
bool scaled_gradients(const BwdProblem& bp, int dtype) {
  return dtype == B200_SDPA_F16 && (bwd_wide_dims(bp.f) || bwd_padded_eligible(bp, dtype));
}

}  // namespace

uint64_t bwd_tc_workspace_bytes(const BwdProblem& bp, int dtype) {
  return statistics_bytes(bp) +
         (scaled_gradients(bp, dtype) ? sizeof(float2) * static_cast<uint64_t>(bp.f.B) * bp.f.Hkv * range_parts(bp.f) : 0);
}

int plan_bwd_tc(const BwdProblem& bp, int dtype, B200SdpaPlan* plan) {
  const Problem& p = bp.f;
  plan->path = B200_SDPA_PATH_PREFILL;
  plan->block_m = kT;
  plan->block_n = kT;
  plan->grid_x = static_cast<int32_t>(static_cast<long long>((p.L + kT - 1) / kT) * p.Hq * p.B);
  plan->grid_y = static_cast<int32_t>(static_cast<long long>((p.S + kT - 1) / kT) * p.Hkv * p.B);
  plan->grid_z = 1;
  plan->threads = kThreads;
  plan->smem_bytes = p.E == 64 && p.Dv == 64 ? BCfg<64>::kSmemBytes : BCfg<128>::kSmemBytes;
  if (bwd_wide_dims(p)) plan_bwd_wide(p, plan);
  plan->kv_splits = 1;
  plan->launches = 3;
  plan->workspace_bytes = bwd_tc_workspace_bytes(bp, dtype);
  return B200_SDPA_OK;
}

int launch_bwd_tc(const BwdProblem& bp, int dtype, void* workspace, uint64_t workspace_bytes, cudaStream_t stream) {
  const bool padded = bwd_padded_eligible(bp, dtype);
  if (!padded && !bwd_tc_eligible(bp, dtype, nullptr)) return B200_SDPA_ERR_UNSUPPORTED;
  const uint64_t need = bwd_tc_workspace_bytes(bp, dtype);
  if (workspace == nullptr || workspace_bytes < need || reinterpret_cast<uintptr_t>(workspace) % 16)
    return B200_SDPA_ERR_WORKSPACE;
  float* lse2 = reinterpret_cast<float*>(workspace);
  float* delta = lse2 + statistics_bytes(bp) / (2 * sizeof(float));
  float2* range = scaled_gradients(bp, dtype) ? reinterpret_cast<float2*>(lse2 + statistics_bytes(bp) / sizeof(float)) : nullptr;
  const bool bf16 = dtype == B200_SDPA_BF16;
  if (bwd_wide_dims(bp.f)) return launch_bwd_wide(bp, bf16, lse2, delta, range, stream);
  if (padded) {
    if (bp.f.bias != nullptr)
      return bf16 ? launch_tc<128, true, true, true>(bp, lse2, delta, range, stream) : launch_tc<128, false, true, true>(bp, lse2, delta, range, stream);
    return bf16 ? launch_tc<128, true, false, true>(bp, lse2, delta, range, stream) : launch_tc<128, false, false, true>(bp, lse2, delta, range, stream);
  }
  if (bp.f.bias != nullptr) {
    if (bp.f.E == 128)
      return bf16 ? launch_tc<128, true, true>(bp, lse2, delta, range, stream) : launch_tc<128, false, true>(bp, lse2, delta, range, stream);
    return bf16 ? launch_tc<64, true, true>(bp, lse2, delta, range, stream) : launch_tc<64, false, true>(bp, lse2, delta, range, stream);
  }
  if (bp.f.E == 128)
    return bf16 ? launch_tc<128, true, false>(bp, lse2, delta, range, stream) : launch_tc<128, false, false>(bp, lse2, delta, range, stream);
  return bf16 ? launch_tc<64, true, false>(bp, lse2, delta, range, stream) : launch_tc<64, false, false>(bp, lse2, delta, range, stream);
}

}  // namespace b200

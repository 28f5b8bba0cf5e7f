// Tensor-core backward for the head dimensions beyond 128: E = 192 with Dv = 128 (multi-head latent attention,
// tests/python_ops/test_scaled_dot_product_attention.py:46-97 upstream) and E = Dv = 256.
//
// The fp32 accumulators of dK and dV (E + Dv columns of tensor memory) leave no room for score tiles beside them
// at these sizes, so the three gradients are three walks of one shape.  A CTA keeps 128 rows of two operands in
// shared memory and streams tiles of NT rows of two others past them:
//
//   gradient   fixed (128 rows)   streamed        per tile
//   dQ         Q, dO              K, V            S = Q K^T, dP = dO V^T, dQ += dS K
//   dK         K, V               Q, dO           S^T = K Q^T, dP^T = V dO^T, dK += dS^T Q
//   dV         K                  Q, dO           S^T = K Q^T, dV += P^T dO
//
// with dS = P (dP - delta), P = 2^(S c - lse2): 8 tile products for the 5 counted.  The dK and dV walks share one
// launch (neighbouring CTAs, which read the same query tiles), the dQ walk is a programmatic dependent of it.
// Bound: the tensor pipe.  NT = 128 at 192/128; at 256 the fixed operands alone take 128 KB and NT is 64.
// Before, these shapes ran on the CUDA-core kernels.  1 x 24 x 2048, 192/128, causal, forward and backward: 19.8 ms
// then, 0.273 ms with these kernels (0.05 of it the forward).
//
// Roles per CTA (576 threads): warps 0-15 elementwise (four threads per TMEM lane), warp 16 TMA producer, warp 17 MMA
// issuer.  The elementwise warps copy a tile's scores into registers and release the accumulators at once, so the
// score products of the next tile run under their arithmetic; the 16-bit operand they leave in tensor memory has
// columns of its own.  These shapes had fp32 probabilities on the CUDA-core kernels, so P and dS go into their second
// product as hi + lo, two 16-bit operands (remainder2).  The dQ and dK walks at E = 192 have no columns for lo: it
// takes the place of dP (kHold), whose next product then follows the one that reads lo.
// Masks, bounded waits: as in bwd_sm100.cu.
#include "bwd_common.cuh"

namespace b200 {

namespace {

using namespace ptx;
using namespace tc;

constexpr int kEWarps = 16;
constexpr int kThreads = (kEWarps + 2) * 32;
constexpr int kProducerWarp = kEWarps;
constexpr int kMmaWarp = kEWarps + 1;
constexpr uint32_t kTmemCols = 512;

enum Walk { kDQ = 0, kDK = 1, kDV = 2 };

template <int WALK, int E, int DV> struct WCfg {
  static constexpr int kNT = E <= 192 ? 128 : 64;                  // rows of a streamed tile
  static constexpr int kStreamBox = kNT * 128;                     // bytes of one copy box of a streamed tile
  static constexpr int kFixedE = kT * E * 2, kFixedV = WALK == kDV ? 0 : kT * DV * 2;
  // the streamed operand of the accumulating product lives until that product, the other one only until its
  // score product: a ring of two slots for the first, one or two for the second
  static constexpr int kLongW = WALK == kDV ? DV : E, kShortW = WALK == kDV ? E : DV;
  static constexpr int kLongBytes = kNT * kLongW * 2, kShortBytes = kNT * kShortW * 2;
  static constexpr int kLongSlots = 2, kShortSlots = WALK == kDV ? 2 : 1;
  static constexpr int kTiles = kFixedE + kFixedV + kLongSlots * kLongBytes + kShortSlots * kShortBytes;
  static constexpr int kStatBytes = 2 * 2 * kNT * 4;               // (lse2, delta) of a streamed query tile, two slots
  static constexpr int kSmemBytes = kTiles + kStatBytes + 256 /*barriers*/;
  static constexpr int kAccW = WALK == kDV ? DV : E;
  // tensor memory: S, dP, one or two operand buffers (hi, then lo), accumulator
  static constexpr uint32_t kColS = 0, kColDP = kNT;
  static constexpr uint32_t kColOp = WALK == kDV ? kNT : 2 * kNT;
  static constexpr uint32_t kColAcc = 512 - kAccW;
  static constexpr bool kHold = kColOp + kNT > kColAcc;            // room for hi, not for lo
  static constexpr int kOpCols = kHold ? kNT / 2 : kNT;            // columns of an operand buffer
  static constexpr int kOpBufs = kColOp + 2 * kOpCols <= kColAcc ? 2 : 1;
  static_assert(kColOp + kOpBufs * kOpCols <= kColAcc, "tensor memory");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory");
};

struct WSync {
  uint64_t fixed_full;
  uint64_t long_full[2], long_empty[2];
  uint64_t short_full[2], short_empty[2];
  uint64_t sp_full;      // the score-shaped accumulators of a tile are complete
  uint64_t f_free;       // the elementwise role holds them in registers
  uint64_t e_ready[2];   // the 16-bit operand of a tile is in its buffer
  uint64_t op_empty[2];  // the product reading an operand buffer has retired
  uint64_t acc_done;
  uint64_t staged;
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(WSync) <= 256, "barrier block must fit its reserve");

// 32 or 16 consecutive columns of this thread's tensor-memory lane to or from registers.
__device__ __forceinline__ void tmem_ld_row(uint32_t addr, uint32_t (&v)[32]) { tmem_ld_32x32(addr, v); }
__device__ __forceinline__ void tmem_ld_row(uint32_t addr, uint32_t (&v)[16]) { tmem_ld_32x16(addr, v); }
__device__ __forceinline__ void tmem_st_row(uint32_t addr, const uint32_t (&v)[16]) { tmem_st_32x16(addr, v); }
__device__ __forceinline__ void tmem_st_row(uint32_t addr, const uint32_t (&v)[8]) { tmem_st_32x8(addr, v); }

// Where a CTA works, decoded by the kernels below.
struct WWork {
  int b, hk, h;          // batch, kv head, query head (dQ walk)
  int row0;              // first fixed row
  int n_tiles;           // streamed tiles
  int n_keys;            // visible keys of the batch
  int first_tile;        // (dK, dV) first streamed tile of every query head
  int per_head;          // (dK, dV) streamed tiles per query head
  int min_lim;           // (dQ) keys visible to the first row
};

template <int WALK, int E, int DV, bool BF16>
__device__ __forceinline__ void walk(const CUtensorMap* tm_fe, const CUtensorMap* tm_fv, const CUtensorMap* tm_long,
                                     const CUtensorMap* tm_short, const CUtensorMap* tm_out, const Problem& p,
                                     const float* lse2, const float* delta, const int l_pad, const long long wait_limit, const float2* range,
                                     const int n_parts, const WWork w, uint8_t* smem_raw) {
  using C = WCfg<WALK, E, DV>;
  constexpr bool kScaled = !BF16;   // see gradient_scale
  constexpr int NT = C::kNT;
  const uint32_t tiles = smem_u32(smem_raw);
  float* stats = reinterpret_cast<float*>(smem_raw + C::kTiles);
  WSync* sync = reinterpret_cast<WSync*>(smem_raw + C::kTiles + C::kStatBytes);
  volatile int* abort_flag = &sync->abort_flag;
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;

  const uint32_t fe_tile = tiles, fv_tile = tiles + C::kFixedE;
  const uint32_t long_ring = tiles + C::kFixedE + C::kFixedV;
  const uint32_t short_ring = long_ring + C::kLongSlots * C::kLongBytes;

  if (warp == kProducerWarp && lane == 0) {
    mbar_init(smem_u32(&sync->fixed_full), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&sync->long_full[s]), 1);
      mbar_init(smem_u32(&sync->long_empty[s]), 1);
      mbar_init(smem_u32(&sync->short_full[s]), 1);
      mbar_init(smem_u32(&sync->short_empty[s]), 1);
    }
    mbar_fence_init();
    if (w.n_tiles > 0) {
      const int head = WALK == kDQ ? w.h : w.hk;
      const uint32_t bar = smem_u32(&sync->fixed_full);
      mbar_arrive_expect_tx(bar, C::kFixedE + C::kFixedV);
      for (int bx = 0; bx < E / 64; ++bx) tma_load_4d(fe_tile + bx * kBoxBytes, tm_fe, bar, bx * 64, w.row0, head, w.b);
      if (WALK != kDV)
        for (int bx = 0; bx < DV / 64; ++bx) tma_load_4d(fv_tile + bx * kBoxBytes, tm_fv, bar, bx * 64, w.row0, head, w.b);
    }
    prefetch_tmap(tm_out);
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

  // query head and first row of streamed tile j
  auto tile_head = [&](int j) { return WALK == kDQ ? w.hk : w.hk * p.group + j / w.per_head; };
  auto tile_row = [&](int j) { return (WALK == kDQ ? j : w.first_tile + j % w.per_head) * NT; };

  if (warp == kProducerWarp) {
    // The whole warp runs the loop: in the dK and dV walks the lanes leave the streamed query rows' statistics
    // beside the tile (fetched one tile ahead), lane 0 then arms the barrier and starts the copies.
    float4 st_l = make_float4(0.f, 0.f, 0.f, 0.f), st_d = st_l;
    auto fetch_stats = [&](int j) {
      const long long src = (static_cast<long long>(w.b) * p.Hq + tile_head(j)) * l_pad + tile_row(j);
      if (lane < NT / 4 &&
          dbg_range(p.status, DBG_BWD_WIDE * 100 + 1, src, NT, static_cast<long long>(p.B) * p.Hq * l_pad)) {
        st_l = reinterpret_cast<const float4*>(lse2 + src)[lane];
        st_d = reinterpret_cast<const float4*>(delta + src)[lane];
      }
    };
    float gs = 1.f;   // delta is kept times this
    if (WALK != kDQ && w.n_tiles > 0) fetch_stats(0);
    bool alive = true;
    for (int j = 0; j < w.n_tiles && alive; ++j) {
      const int ls = j % C::kLongSlots, ss = j % C::kShortSlots;
      const int head = tile_head(j), row = tile_row(j);
      if (j >= C::kLongSlots) {
        alive = wait_clocked(smem_u32(&sync->long_empty[ls]), (j / C::kLongSlots - 1) & 1u, abort_flag, wait_limit);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) {
          if (lane == 0) report(p.status, 31, j, ls);
          break;
        }
      }
      const uint32_t bar = smem_u32(&sync->long_full[ls]);
      auto copy = [&]() {
        for (int bx = 0; bx < C::kLongW / 64; ++bx)
          tma_load_4d(long_ring + ls * C::kLongBytes + bx * C::kStreamBox, tm_long, bar, bx * 64, row, head, w.b);
      };
      constexpr bool kScaleDelta = kScaled && WALK == kDK;
      if constexpr (kScaleDelta) {   // the copies go first: the maxima behind gs take a trip to L2
        if (lane == 0) {
          mbar_expect_tx(bar, C::kLongBytes);
          copy();
        }
        __syncwarp();
        if (j == 0) gs = gradient_scale(range, n_parts, w.b * p.Hkv + w.hk, DV, lane);
        st_d = make_float4(st_d.x * gs, st_d.y * gs, st_d.z * gs, st_d.w * gs);
      }
      if (WALK != kDQ) {
        if (lane < NT / 4) {
          float4* dst = reinterpret_cast<float4*>(stats + ls * 2 * NT);
          dst[lane] = st_l;
          dst[NT / 4 + lane] = st_d;
        }
        __syncwarp();
      }
      if (lane == 0) {
        if constexpr (kScaleDelta) {
          mbar_arrive(bar);
        } else {
          mbar_arrive_expect_tx(bar, C::kLongBytes);
          copy();
        }
      }
      if (WALK != kDQ && j + 1 < w.n_tiles) fetch_stats(j + 1);
      if (j >= C::kShortSlots) {
        alive = wait_clocked(smem_u32(&sync->short_empty[ss]), (j / C::kShortSlots - 1) & 1u, abort_flag, wait_limit);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) {
          if (lane == 0) report(p.status, 31, j, 8 + ss);
          break;
        }
      }
      if (lane == 0) {
        const uint32_t bar = smem_u32(&sync->short_full[ss]);
        mbar_arrive_expect_tx(bar, C::kShortBytes);
        for (int bx = 0; bx < C::kShortW / 64; ++bx)
          tma_load_4d(short_ring + ss * C::kShortBytes + bx * C::kStreamBox, tm_short, bar, bx * 64, row, head, w.b);
      }
    }
    if (*abort_flag != 0 && lane == 0) {
      for (int i = 0; i < 200; ++i) __nanosleep(1000);   // copies in flight must land before exit
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    constexpr uint32_t idesc_score = make_idesc(BF16, false, kT, NT);
    constexpr uint32_t idesc_acc = make_idesc(BF16, true, kT, C::kAccW);
    bool alive = w.n_tiles > 0;
    if (alive) {
      alive = wait_clocked(smem_u32(&sync->fixed_full), 0, abort_flag, wait_limit);
      if (!alive && lane == 0) report(p.status, 32, -1, 0);
      if (WALK == kDK && alive && w.n_keys < p.S && w.row0 + kT > w.n_keys) zero_tile_rows<DV / 64, kT>(fv_tile, w.n_keys - w.row0, lane);
    }
    // k-step kk (16 elements of the head dimension) of a K-major streamed tile
    auto stream_step = [](int kk) { return static_cast<uint64_t>(((kk >> 2) * C::kStreamBox + (kk & 3) * 32) >> 4); };
    auto wait_long = [&](int j) -> bool {
      const int ls = j % C::kLongSlots;
      const bool ok = wait_clocked(smem_u32(&sync->long_full[ls]), (j / C::kLongSlots) & 1u, abort_flag, wait_limit);
      if (!ok && lane == 0) report(p.status, 32, j, ls);
      return ok;
    };
    auto wait_short = [&](int j) -> bool {
      const int ss = j % C::kShortSlots;
      const bool ok = wait_clocked(smem_u32(&sync->short_full[ss]), (j / C::kShortSlots) & 1u, abort_flag, wait_limit);
      if (!ok && lane == 0) report(p.status, 32, j, 8 + ss);
      return ok;
    };
    auto issue_s = [&](int j) -> bool {
      if (!(WALK == kDV ? wait_short(j) : wait_long(j))) return false;
      tc_fence_after_sync();
      const uint32_t e_tile = WALK == kDV ? short_ring + (j % C::kShortSlots) * C::kShortBytes
                                          : long_ring + (j % C::kLongSlots) * C::kLongBytes;
      // (as in bwd_sm100.cu: keys beyond kv_lens, here and in dP)
      if (WALK == kDQ && w.n_keys < p.S && (j + 1) * NT > w.n_keys) zero_tile_rows<E / 64, NT>(e_tile, w.n_keys - j * NT, lane);
      const uint64_t fd = kmajor_desc(fe_tile), gd = kmajor_desc(e_tile);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < E / 16; ++kk)
          mma_ss(tmem_base + C::kColS, fd + kmajor_step(kk), gd + stream_step(kk), idesc_score, kk > 0 ? 1u : 0u);
      }
      return true;
    };
    auto issue_dp = [&](int j) -> bool {   // ... after which the tile's scores are complete
      if (!(WALK == kDV ? wait_long(j) : wait_short(j))) return false;
      tc_fence_after_sync();
      const int ss = j % C::kShortSlots;
      if (WALK == kDQ && w.n_keys < p.S && (j + 1) * NT > w.n_keys)
        zero_tile_rows<DV / 64, NT>(short_ring + ss * C::kShortBytes, w.n_keys - j * NT, lane);
      const uint64_t fvd = kmajor_desc(fv_tile), gvd = kmajor_desc(short_ring + ss * C::kShortBytes);
      if (elect_one()) {
        if (WALK != kDV) {
#pragma unroll
          for (int kk = 0; kk < DV / 16; ++kk)
            mma_ss(tmem_base + C::kColDP, fvd + kmajor_step(kk), gvd + stream_step(kk), idesc_score, kk > 0 ? 1u : 0u);
        }
        mma_commit(smem_u32(&sync->sp_full));
        mma_commit(smem_u32(&sync->short_empty[ss]));
      }
      return true;
    };
    if (alive) alive = issue_s(0) && issue_dp(0);
    for (int j = 0; j < w.n_tiles && alive; ++j) {
      const int buf = j % C::kOpBufs, ls = j % C::kLongSlots;
      const bool more = j + 1 < w.n_tiles;
      alive = wait_clocked(smem_u32(&sync->f_free), j & 1, abort_flag, wait_limit);
      if (!alive) {
        if (lane == 0) report(p.status, 33, j, 1);
        break;
      }
      tc_fence_after_sync();
      if (more) {
        alive = issue_s(j + 1) && (C::kHold || issue_dp(j + 1));
        if (!alive) break;
      }
      alive = wait_clocked(smem_u32(&sync->e_ready[buf]), (j / C::kOpBufs) & 1, abort_flag, wait_limit);
      if (!alive) {
        if (lane == 0) report(p.status, 33, j, 0);
        break;
      }
      tc_fence_after_sync();
      const uint64_t bd = smem_desc_sw128(long_ring + ls * C::kLongBytes, C::kStreamBox, 1024);   // MN-major B operand
      const uint32_t op = tmem_base + C::kColOp + buf * C::kOpCols;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < NT / 16; ++kk) {   // the remainders
          const uint32_t a = C::kHold ? tmem_base + C::kColDP + static_cast<uint32_t>((kk >> 1) * 32 + (kk & 1) * 8)
                                      : op + NT / 2 + static_cast<uint32_t>(kk * 8);
          mma_ts(tmem_base + C::kColAcc, a, bd + mnmajor_step(kk), idesc_acc, (kk > 0 || j > 0) ? 1u : 0u);
        }
      }
      if (C::kHold && more) {   // in issue order behind the products that read lo from its columns
        alive = issue_dp(j + 1);
        if (!alive) break;
      }
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < NT / 16; ++kk)
          mma_ts(tmem_base + C::kColAcc, op + static_cast<uint32_t>(kk * 8), bd + mnmajor_step(kk), idesc_acc, 1u);
        mma_commit(smem_u32(&sync->op_empty[buf]));
        mma_commit(smem_u32(&sync->long_empty[ls]));
        if (!more) mma_commit(smem_u32(&sync->acc_done));
      }
    }
    if (*abort_flag != 0) {
      if (elect_one()) mma_commit(smem_u32(&sync->drain));
      wait_drain(smem_u32(&sync->drain), 0);
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------- elementwise role
    constexpr int HC = NT / 4;                 // score columns of one thread
    const int r = tid & (kT - 1);              // fixed row = TMEM lane
    const int quarter = warp >> 2;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_off + C::kColS + quarter * HC;
    const uint32_t dp_addr = tmem_base + lane_off + C::kColDP + quarter * HC;
    const uint32_t op_addr = tmem_base + lane_off + C::kColOp + quarter * (HC / 2);
    const uint32_t acc_addr = tmem_base + lane_off + C::kColAcc;
    if (!dbg_tmem(p.status, DBG_BWD_WIDE * 100 + 2, s_addr, tmem_base, HC, kTmemCols) ||
        !dbg_tmem(p.status, DBG_BWD_WIDE * 100 + 3, dp_addr, tmem_base, HC, kTmemCols) ||
        !dbg_tmem(p.status, DBG_BWD_WIDE * 100 + 4, op_addr, tmem_base, (C::kOpBufs - 1) * C::kOpCols + (C::kHold ? 0 : NT / 2) + HC / 2, kTmemCols) ||
        !dbg_tmem(p.status, DBG_BWD_WIDE * 100 + 5, acc_addr, tmem_base, C::kAccW, kTmemCols))
      *abort_flag = 1;
    const int row_g = w.row0 + r;
    // dQ walk: the row sees keys [0, lim); dK and dV walks: query rows i >= i_min see this key
    int lim = w.n_keys, i_min = 0;
    if (WALK == kDQ) {
      if (p.causal) {
        const long long c = static_cast<long long>(row_g) + p.causal_shift + 1;
        lim = c < lim ? static_cast<int>(c < 0 ? 0 : c) : lim;
      }
    } else {
      if (p.causal) {
        const long long v = static_cast<long long>(row_g) - p.causal_shift;
        i_min = v < 0 ? 0 : (v > (1 << 30) ? (1 << 30) : static_cast<int>(v));
      }
      if (row_g >= w.n_keys) i_min = 1 << 30;
    }
    float neg_l2 = 0.f, dl = 0.f;
    if (WALK == kDQ) {
      const long long idx = (static_cast<long long>(w.b) * p.Hq + w.h) * l_pad + row_g;
      const bool ok = dbg_range(p.status, DBG_BWD_WIDE * 100 + 6, idx, 1, static_cast<long long>(p.B) * p.Hq * l_pad);
      neg_l2 = ok ? -__ldcg(lse2 + idx) : -CUDART_INF_F;   // -inf for rows without a visible key (past L1: as in bwd_sm100.cu)
      dl = ok ? __ldcg(delta + idx) : 0.f;
    }
    const float sl2 = p.scale * kLog2e;
    const uint64_t sl2_2 = f2_pack(sl2, sl2);
    const float gs = kScaled && WALK != kDV ? gradient_scale(range, n_parts, w.b * p.Hkv + w.hk, DV, lane) : 1.f;
    const uint64_t gs2 = f2_pack(gs, gs);
    const float neg_dl = -dl * gs;
    bool alive = true;
    for (int j = 0; j < w.n_tiles; ++j) {
      const int buf = j % C::kOpBufs;
      bool ok = wait_clocked(smem_u32(&sync->sp_full), j & 1, abort_flag, wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) report(p.status, 34, j, warp);
        alive = false;
        break;
      }
      tc_fence_after_sync();
      uint32_t sv[HC], dv[WALK == kDV ? 1 : HC];
      tmem_ld_row(s_addr, sv);
      if constexpr (WALK != kDV) tmem_ld_row(dp_addr, dv);
      tmem_ld_wait();
      tc_fence_before_sync();
      warp_arrive(&sync->f_free, lane);
      const int tile0 = tile_row(j);           // first streamed row
      const int col0 = tile0 + quarter * HC;      // ... of this thread's columns
      const bool need_mask = WALK == kDQ ? tile0 + NT > w.min_lim
                                         : (w.row0 + kT > w.n_keys ||
                                            (p.causal && static_cast<long long>(tile0) <
                                                             static_cast<long long>(w.row0) + kT - 1 - p.causal_shift));
      const float4* st4 = reinterpret_cast<const float4*>(stats + (j % C::kLongSlots) * 2 * NT + quarter * HC);
      uint32_t pk[HC / 2], lo[HC / 2];
#pragma unroll
      for (int q4 = 0; q4 < HC / 4; ++q4) {
        float nl[4] = {neg_l2, neg_l2, neg_l2, neg_l2}, nd[4] = {neg_dl, neg_dl, neg_dl, neg_dl};
        if constexpr (WALK != kDQ) {
          const float4 l4 = st4[q4];
          nl[0] = -l4.x; nl[1] = -l4.y; nl[2] = -l4.z; nl[3] = -l4.w;
          if constexpr (WALK == kDK) {
            const float4 d4 = st4[NT / 4 + q4];
            nd[0] = -d4.x; nd[1] = -d4.y; nd[2] = -d4.z; nd[3] = -d4.w;
          }
        }
#pragma unroll
        for (int e = 0; e < 4; e += 2) {   // two columns per instruction (packed fp32 pairs)
          const int i = q4 * 4 + e;
          float a0, a1;
          f2_unpack(f2_fma(f2_pack(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sl2_2, f2_pack(nl[e], nl[e + 1])), a0, a1);
          float p0 = ex2(a0), p1 = ex2(a1);
          if (need_mask) {
            p0 = (WALK == kDQ ? col0 + i < lim : col0 + i >= i_min) ? p0 : 0.f;
            p1 = (WALK == kDQ ? col0 + i + 1 < lim : col0 + i + 1 >= i_min) ? p1 : 0.f;
          }
          if constexpr (WALK != kDV) {
            const uint64_t dp2 = f2_pack(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1])), nd2 = f2_pack(nd[e], nd[e + 1]);
            f2_unpack(f2_mul(f2_pack(p0, p1), kScaled ? f2_fma(dp2, gs2, nd2) : f2_add(dp2, nd2)), p0, p1);
          }
          pk[i >> 1] = pack2<BF16>(p0, p1);
          lo[i >> 1] = remainder2<BF16>(p0, p1, pk[i >> 1]);
        }
      }
      if (j >= C::kOpBufs) {   // the product that read this operand buffer before must have retired
        ok = wait_clocked(smem_u32(&sync->op_empty[buf]), (j / C::kOpBufs - 1) & 1, abort_flag, wait_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) report(p.status, 36, j, warp);
          alive = false;
          break;
        }
        tc_fence_after_sync();
      }
      tmem_st_row(op_addr + buf * C::kOpCols, pk);
      tmem_st_row(C::kHold ? dp_addr : op_addr + buf * C::kOpCols + NT / 2, lo);
      tmem_st_wait();
      tc_fence_before_sync();
      warp_arrive(&sync->e_ready[buf], lane);
    }
    if (alive && w.n_tiles > 0) {
      bool ok = wait_clocked(smem_u32(&sync->acc_done), 0, abort_flag, wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) report(p.status, 35, 0, warp);
        alive = false;
      }
      tc_fence_after_sync();
    }
    if (alive) {
      // the fixed operands are no longer needed: their area stages the gradient
      const float mul = (WALK == kDV ? 1.f : p.scale) * (kScaled ? 1.f / ((WALK == kDV ? 1.f : gs) * kPScale) : 1.f);
      for (int c = quarter; c < C::kAccW / 32; c += 4)
        stage_chunk<BF16>(acc_addr, w.n_tiles > 0, mul, smem_raw, r, c);
      fence_proxy_async_smem();
      warp_arrive(&sync->staged, lane);
      if (tid == 0 && wait_clocked(smem_u32(&sync->staged), 0, abort_flag, wait_limit)) {
        const int head = WALK == kDQ ? w.h : w.hk;
        for (int bx = 0; bx < C::kAccW / 64; ++bx) tma_store_4d(tm_out, tiles + bx * kBoxBytes, bx * 64, w.row0, head, w.b);
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }

  // (dQ walk) one CTA, the last of the grid, waits for the dK / dV grid this one is a programmatic dependent of, so
  // that whatever is queued behind finds both complete; it reads nothing that grid writes
  if (WALK == kDQ && blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// The tile area must be 1024-byte aligned (swizzled copies); nothing has been started when this fails.
__device__ __forceinline__ bool smem_aligned(const uint8_t* smem, const Problem& p) {
  if ((smem_u32(smem) & 1023u) == 0u) return true;
  if (threadIdx.x == 0) report(p.status, 30, 0, static_cast<int>(smem_u32(smem) & 1023u));
  return false;
}

template <int E, int DV, bool BF16>
__global__ void __launch_bounds__(kThreads, 1)
bwd_wide_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const __grid_constant__ CUtensorMap tm_dq, const Problem p, const float* lse2,
                   const float* delta, const int l_pad, const int n_qblk, const int streams_per_wave,
                   const long long wait_limit, const float2* range, const int n_parts) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (!smem_aligned(smem_raw, p)) return;
  constexpr int NT = WCfg<kDQ, E, DV>::kNT;
  // latest query blocks first inside waves of streams that fit in L2 together (as in bwd_sm100.cu)
  const int n_streams = p.Hkv * p.B;
  const int full_wave_ctas = n_qblk * streams_per_wave * p.group;
  const int wave = static_cast<int>(blockIdx.x / full_wave_ctas);
  const int in_wave = static_cast<int>(blockIdx.x - static_cast<unsigned>(wave) * full_wave_ctas);
  const int first_stream = wave * streams_per_wave;
  const int wave_streams = (n_streams - first_stream) < streams_per_wave ? (n_streams - first_stream) : streams_per_wave;
  const int per_blk = wave_streams * p.group;
  const int rem = in_wave % per_blk;
  const int stream = first_stream + rem / p.group;
  WWork w;
  w.hk = stream % p.Hkv;
  w.b = stream / p.Hkv;
  w.h = w.hk * p.group + rem % p.group;
  w.row0 = (n_qblk - 1 - in_wave / per_blk) * kT;
  w.n_keys = valid_keys(p, w.b);
  long long end = w.n_keys, first = w.n_keys;
  if (p.causal) {
    const int last_row = (w.row0 + kT < p.L ? w.row0 + kT : p.L) - 1;
    const long long e = static_cast<long long>(last_row) + p.causal_shift + 1;
    const long long f = static_cast<long long>(w.row0) + p.causal_shift + 1;
    end = e < end ? e : end;
    first = f < first ? f : first;
  }
  if (end < 0) end = 0;
  if (first < -1) first = -1;
  w.n_tiles = static_cast<int>((end + NT - 1) / NT);
  w.min_lim = static_cast<int>(first);
  w.first_tile = 0;
  w.per_head = 1;
  walk<kDQ, E, DV, BF16>(&tm_q, &tm_do, &tm_k, &tm_v, &tm_dq, p, lse2, delta, l_pad, wait_limit, range, n_parts, w, smem_raw);
}

template <int E, int DV, bool BF16>
__global__ void __launch_bounds__(kThreads, 1)
bwd_wide_dkv_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                    const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                    const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                    const Problem p, const float* lse2, const float* delta, const int l_pad,
                    const int n_kblk, const int streams_per_wave, const long long wait_limit, const float2* range, const int n_parts) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  pdl_wait();   // as in bwd_sm100.cu
  pdl_launch_dependents();
  if (!smem_aligned(smem_raw, p)) return;
  constexpr int NT = WCfg<kDK, E, DV>::kNT;
  // Earliest key blocks (seen by the most query tiles under a causal mask) first, within waves of groups whose
  // query-side operands fit in L2 together; neighbouring CTAs do dK and dV of the same keys.
  const int unit = static_cast<int>(blockIdx.x >> 1);
  const int n_streams = p.Hkv * p.B;
  const int full_wave = n_kblk * streams_per_wave;
  const int wave = unit / full_wave;
  const int in_wave = unit - wave * full_wave;
  const int first_stream = wave * streams_per_wave;
  const int wave_streams = (n_streams - first_stream) < streams_per_wave ? (n_streams - first_stream) : streams_per_wave;
  const int stream = first_stream + in_wave % wave_streams;
  WWork w;
  w.hk = stream % p.Hkv;
  w.b = stream / p.Hkv;
  w.h = 0;
  w.row0 = in_wave / wave_streams * kT;
  w.n_keys = valid_keys(p, w.b);
  w.min_lim = 0;
  const int n_qt = (p.L + NT - 1) / NT;
  w.first_tile = 0;
  if (p.causal) {
    const long long f = static_cast<long long>(w.row0) - p.causal_shift;   // first row that sees key row0
    w.first_tile = f <= 0 ? 0 : (f >= p.L ? n_qt : static_cast<int>(f / NT));
  }
  const int per_head = (w.row0 < w.n_keys && n_qt > w.first_tile) ? n_qt - w.first_tile : 0;
  w.n_tiles = per_head * p.group;
  w.per_head = per_head > 0 ? per_head : 1;
  if ((blockIdx.x & 1u) == 0u)
    walk<kDK, E, DV, BF16>(&tm_k, &tm_v, &tm_q, &tm_do, &tm_dk, p, lse2, delta, l_pad, wait_limit, range, n_parts, w, smem_raw);
  else
    walk<kDV, E, DV, BF16>(&tm_k, &tm_v, &tm_do, &tm_q, &tm_dv, p, lse2, delta, l_pad, wait_limit, range, n_parts, w, smem_raw);
}

// ------------------------------------------------------------------ host side --

template <int E, int DV, bool BF16>
int launch_wide(const BwdProblem& bp, float* lse2, float* delta, float2* range, cudaStream_t stream) {
  const Problem& p = bp.f;
  constexpr int NT = WCfg<kDQ, E, DV>::kNT;
  constexpr int kSmemQ = WCfg<kDQ, E, DV>::kSmemBytes;
  constexpr int kSmemKV = WCfg<kDK, E, DV>::kSmemBytes > WCfg<kDV, E, DV>::kSmemBytes ? WCfg<kDK, E, DV>::kSmemBytes
                                                                                      : WCfg<kDV, E, DV>::kSmemBytes;
  // every operand is the fixed one of some walk (boxes of 128 rows) and the streamed one of another (NT rows)
  CUtensorMap q_f, k_f, v_f, do_f, q_s, k_s, v_s, do_s, dq, dk, dv;
  if (!make_map(&q_f, p.q, BF16, E, p.L, p.Hq, p.B, p.qs) || !make_map(&q_s, p.q, BF16, E, p.L, p.Hq, p.B, p.qs, NT) ||
      !make_map(&k_f, p.k, BF16, E, p.S, p.Hkv, p.B, p.ks) || !make_map(&k_s, p.k, BF16, E, p.S, p.Hkv, p.B, p.ks, NT) ||
      !make_map(&v_f, p.v, BF16, DV, p.S, p.Hkv, p.B, p.vs) || !make_map(&v_s, p.v, BF16, DV, p.S, p.Hkv, p.B, p.vs, NT) ||
      !make_map(&do_f, bp.dout, BF16, DV, p.L, p.Hq, p.B, bp.dos) || !make_map(&do_s, bp.dout, BF16, DV, p.L, p.Hq, p.B, bp.dos, NT) ||
      !make_map(&dq, bp.dq, BF16, E, p.L, p.Hq, p.B, bp.dqs) || !make_map(&dk, bp.dk, BF16, E, p.S, p.Hkv, p.B, bp.dks) ||
      !make_map(&dv, bp.dv, BF16, DV, p.S, p.Hkv, p.B, bp.dvs))
    return B200_SDPA_ERR_CUDA;
  auto kq = bwd_wide_dq_kernel<E, DV, BF16>;
  auto kkv = bwd_wide_dkv_kernel<E, DV, BF16>;
  if (cudaFuncSetAttribute(kq, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemQ) != cudaSuccess ||
      cudaFuncSetAttribute(kkv, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemKV) != cudaSuccess) {
    cudaGetLastError();
    return B200_SDPA_ERR_CUDA;
  }
  const int l_pad = padded_rows(p);
  const int n_qblk = (p.L + kT - 1) / kT, n_kblk = (p.S + kT - 1) / kT;
  const long long grid_q = static_cast<long long>(n_qblk) * p.Hq * p.B;
  const long long grid_kv = 2LL * n_kblk * p.Hkv * p.B;
  if (grid_q > 0x7fffffffLL || grid_kv > 0x7fffffffLL) return B200_SDPA_ERR_UNSUPPORTED;
  const int prep = launch_bwd_prep(bp, BF16, lse2, delta, range, stream);
  if (prep != B200_SDPA_OK) return prep;
  const long long limit = wait_limit_cycles();
  const long long n_streams = static_cast<long long>(p.Hkv) * p.B;
  const int wave_q = kv_streams_per_wave(static_cast<long long>(p.S) * (E + DV) * 2, n_streams);
  const int wave_kv = kv_streams_per_wave(static_cast<long long>(p.L) * p.group * ((E + DV) * 2 + 8), n_streams);
  const float* c_lse2 = lse2;
  const float* c_delta = delta;
  const float2* c_range = range;
  const int n_parts = range_parts(p);
  if (!launch_pdl(kkv, dim3(static_cast<unsigned>(grid_kv)), kThreads, kSmemKV, stream, k_f, v_f, q_s, do_s, dk, dv, p, c_lse2, c_delta,
                  l_pad, n_kblk, wave_kv, limit, c_range, n_parts))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_BWD_DKV);
  if (!launch_pdl(kq, dim3(static_cast<unsigned>(grid_q)), kThreads, kSmemQ, stream, q_f, do_f, k_s, v_s, dq, p, c_lse2, c_delta, l_pad,
                  n_qblk, wave_q, limit, c_range, n_parts))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_BWD_DQ);
  return B200_SDPA_OK;
}

}  // namespace

// The caller has checked the strides; an additive bias stays with the CUDA-core kernels at these head dimensions.
bool bwd_wide_dims(const Problem& p) {
  return ((p.E == 192 && p.Dv == 128) || (p.E == 256 && p.Dv == 256)) && p.bias == nullptr;
}

void plan_bwd_wide(const Problem& p, B200SdpaPlan* plan) {
  plan->threads = kThreads;
  plan->grid_y *= 2;   // dK and dV are CTAs of their own
  plan->smem_bytes = p.E == 192 ? WCfg<kDQ, 192, 128>::kSmemBytes : WCfg<kDQ, 256, 256>::kSmemBytes;
}

int launch_bwd_wide(const BwdProblem& bp, bool bf16, float* lse2, float* delta, float2* range, cudaStream_t stream) {
  if (bp.f.E == 192)
    return bf16 ? launch_wide<192, 128, true>(bp, lse2, delta, range, stream) : launch_wide<192, 128, false>(bp, lse2, delta, range, stream);
  return bf16 ? launch_wide<256, 256, true>(bp, lse2, delta, range, stream) : launch_wide<256, 256, false>(bp, lse2, delta, range, stream);
}

}  // namespace b200

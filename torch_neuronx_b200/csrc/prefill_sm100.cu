// FlashAttention-style prefill kernel for sm_100a: TMA -> shared memory ->
// tcgen05 tensor cores with accumulators in tensor memory (TMEM).  One work item per CTA; large
// problems at head dimension 128 run the persistent form of the same kernel
// (prefill_persistent_sm100.cu), which produces the same bits.
//
// One CTA owns 256 query rows of one (batch, query head): two 128-row tiles
// that take turns on the tensor cores while the other one is in its softmax.
// Roles (320 threads):
//   warps 0-3   softmax of tile 0: one thread per query row (= one TMEM lane)
//   warps 4-7   softmax of tile 1
//   warp  8     TMA producer: Q once, then K(j), V(j) tiles through a ring
//   warp  9     MMA issuer: S_t = Q_t K(j)^T and O_t += P_t V(j), one thread
// TMEM columns: [0,128) S0, [128,256) S1, [256,256+D) O0, [256+D,256+2D) O1;
// the probabilities P_t (16-bit, two per column) overwrite the first 64 columns
// of S_t and are fed to the second product straight from TMEM.  With D = 64 there
// are 128 columns to spare: P_t then has columns of its own and the next score
// product does not wait for P V (Cfg::kSplitP).
//
// Online softmax in the exp2 domain on raw scores: p = 2^(s*c - m*c) with
// c = scale*log2(e); the running maximum m is only raised when it grows by more
// than 2^8, so O is rarely rescaled.  All statistics and O stay fp32; P is
// rounded to the input dtype exactly once, as upstream rounds its
// probabilities (torch_neuronx/_sdpa_math.py:94).  Rows without a visible key
// give out = 0, lse = -inf (:85-91).  The causal rule is j <= i + shift with
// shift = q_offset - k_offset (0 reproduces the top-left aligned triangle of
// :20-28); kv_lens masks right padding; key tiles that no row of the CTA can
// see are never loaded.
//
// Every wait is bounded: on expiry the role raises a CTA-wide abort flag, every
// other role drains, tensor memory is freed and the status word reports
// B200_SDPA_ERR_TIMEOUT.
#include "tc_common.cuh"
#include "debug.cuh"

#include <type_traits>

namespace b200 {

namespace {

using namespace ptx;
using namespace tc;

constexpr int kBlockM = 128;   // rows per query tile (= TMEM lanes)
constexpr int kBlockN = 128;   // keys per tile
constexpr int kTilesPerCta = 2;
constexpr int kRowsPerCta = kBlockM * kTilesPerCta;
constexpr int kThreads = 320;
constexpr int kProducerWarp = 8;
constexpr int kMmaWarp = 9;
constexpr uint32_t kTmemCols = 512;
constexpr float kRescaleThreshold = 8.0f;         // in units of log2

template <int D> struct Cfg {
  static constexpr int kBoxes = D / 64;                      // TMA boxes per tile
  static constexpr int kTileBytes = kBlockN * D * 2;
  static constexpr int kStages = (D == 128) ? 4 : 8;         // K/V ring slots
  static constexpr int kSmemTiles = (kTilesPerCta + kStages) * kTileBytes;
  static constexpr int kSmemBytes = kSmemTiles + 1024 /*alignment slack*/ + 256 /*barriers*/;
  // With D = 64 the two O accumulators leave 128 tensor-memory columns free: P_t gets columns of its
  // own ([384,448) / [448,512)) instead of overwriting S_t, so Q_t K(j+1)^T no longer has to wait for
  // P_t(j) V(j) -- it is issued as soon as the softmax warps have copied S_t(j) into registers.
  static constexpr bool kSplitP = (D == 64);
};

struct Sync {
  uint64_t q_full;
  uint64_t kv_full[8];
  uint64_t kv_empty[8];
  uint64_t s_full[2];
  uint64_t p_ready[2][2];  // [tile][half of P]
  uint64_t s_free[2];      // (D = 64) the softmax warps hold S_t(j) in registers
  uint64_t pv_done[2];     // (D = 64) P_t(j) V(j) has retired
  uint64_t o_done[2];
  uint64_t o_staged[2];
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
};

static_assert(sizeof(Sync) <= 272, "barrier block must fit its reserve (272 bytes + up to 1008 of alignment <= 1280)");

// Visible-key geometry of one 128-row tile.
struct TileGeom {
  int row0;       // first query row
  int n_tiles;    // key tiles to process (0: nothing visible, or tile beyond L)
  int min_lim;    // visible-key count of the tile's first row (may be <= 0)
  bool in_range;  // row0 < L
};

__device__ __forceinline__ TileGeom tile_geometry(const Problem& p, int row0, int kv_limit, int rows = kBlockM) {
  TileGeom g;
  g.row0 = row0;
  g.in_range = row0 < p.L;
  long long end = kv_limit, first = kv_limit;
  if (p.causal) {
    const int last_row = (row0 + rows < p.L ? row0 + rows : p.L) - 1;
    const long long e = static_cast<long long>(last_row) + p.causal_shift + 1;
    const long long f = static_cast<long long>(row0) + p.causal_shift + 1;
    end = e < end ? e : end;
    first = f < first ? f : first;
  }
  if (end < 0) end = 0;
  if (first < -1) first = -1;
  g.n_tiles = g.in_range ? static_cast<int>((end + kBlockN - 1) / kBlockN) : 0;
  g.min_lim = static_cast<int>(first);
  return g;
}

// The split form (PACK): few query rows against many keys.  A 128-row tile holds `lb` consecutive rows of every
// query head of one kv head (heads * lb <= 128), so the group reads its keys once; the key axis is cut into
// `n_split` ranges, one CTA each, whose unnormalised fp32 results and (maximum, sum) pairs a second launch merges.
struct PackArgs {
  int lb;               // rows of one head in a tile
  int dual;             // one row tile only: the CTA's two tiles are the same rows against even and odd key tiles
  int n_pairs;          // pairs of row tiles along the queries
  int n_split;
  int split_tiles;      // key tiles of one split
  float* part_o;        // [B][Hq][L][n_split][Dv]
  float* part_ml;       // [B][Hq][L][n_split][2]: maximum in log2 units, sum
};

// PAD: head dimensions E, Dv (multiples of 8) that do not fill the D = 128 tile.  The tensor maps carry the
// real extents, so the copies fill the tile's remaining columns with zeros and the output store clips them;
// the products run over ceil(E / 16) k-steps and ceil(Dv / 16) * 16 output columns only.  These shapes had fp32
// probabilities on the CUDA-core kernel, so P goes into the second product as hi + lo (remainder2), lo in the second
// half of the columns of S.
template <int D, bool BF16, bool BIAS, bool ACC, bool PAD, bool PACK>
__global__ void __launch_bounds__(kThreads, 1)
prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, const Problem p,
               const int n_qblk, const int pair_heads, const int streams_per_wave, const long long wait_limit,
               const PackArgs pack) {
  using C = Cfg<D>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t tiles = (raw_addr + 1023u) & ~1023u;            // 1024-byte aligned tile area
  Sync* sync = reinterpret_cast<Sync*>(smem_raw + (tiles - raw_addr) + C::kSmemTiles);
  volatile int* abort_flag = &sync->abort_flag;

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;

  // Work item: longest (latest) query blocks first, heads of one kv group adjacent.
  // Two layouts of the CTA's two 128-row tiles:
  //   pair_heads == 0: rows [256 q, +128) and [256 q + 128, +128) of one query head;
  //   pair_heads == 1: the same 128 rows of two query heads that share a kv head
  //     (even group size) -- both tiles then see exactly the same keys, so under a
  //     causal mask neither waits for the other's extra diagonal tile.
  // The (batch, kv head) key/value streams are taken `streams_per_wave` at a time, so that what the
  // CTAs in flight read together fits in L2 (all streams at once when they do).
  int hk, b, hq0, key_tile0 = 0;
  const bool dual = PACK && pack.dual != 0;
  int head_of_tile[2];
  int row0_0, row0_1;
  if constexpr (PACK) {
    // neighbouring CTAs: the splits of one pair of row tiles (longest first), then the next (batch, kv head)
    const int n_ranges = dual ? pack.n_split / 2 : pack.n_split;   // CTAs along the keys
    const int split = static_cast<int>(blockIdx.x) % n_ranges;
    const int unit = static_cast<int>(blockIdx.x) / n_ranges;
    const int n_streams = p.Hkv * p.B;
    const int pair = pack.n_pairs - 1 - unit / n_streams;
    const int stream = unit % n_streams;
    hk = stream % p.Hkv;
    b = stream / p.Hkv;
    hq0 = hk * p.group;
    head_of_tile[0] = head_of_tile[1] = hq0;
    key_tile0 = split * pack.split_tiles;
    row0_0 = 2 * pair * pack.lb;
    row0_1 = (2 * pair + 1) * pack.lb;
  } else {
    const int heads_per_cta = pair_heads ? 2 : 1;
    const int ctas_per_stream = p.group / heads_per_cta;            // per query block
    const int n_streams = p.Hkv * p.B;
    const int full_wave_ctas = n_qblk * streams_per_wave * ctas_per_stream;
    const int wave = static_cast<int>(blockIdx.x / full_wave_ctas);
    const int in_wave = static_cast<int>(blockIdx.x - static_cast<unsigned>(wave) * full_wave_ctas);
    const int first_stream = wave * streams_per_wave;
    const int wave_streams = (n_streams - first_stream) < streams_per_wave ? (n_streams - first_stream) : streams_per_wave;
    const int per_blk = wave_streams * ctas_per_stream;
    const int qblk = n_qblk - 1 - in_wave / per_blk;
    const int rem = in_wave % per_blk;
    const int stream = first_stream + rem / ctas_per_stream;
    hk = stream % p.Hkv;
    b = stream / p.Hkv;
    hq0 = hk * p.group + (rem % ctas_per_stream) * heads_per_cta;
    head_of_tile[0] = hq0;
    head_of_tile[1] = pair_heads ? hq0 + 1 : hq0;
    const int rows_per_cta = pair_heads ? kBlockM : kRowsPerCta;
    row0_0 = qblk * rows_per_cta;
    row0_1 = row0_0 + (pair_heads ? 0 : kBlockM);
  }
  // A programmatic dependent of whatever precedes it in the stream: the launch and the divisions above run under that
  // kernel's tail, and nothing of global memory is touched before the wait (which returns when that grid is complete and
  // its writes are visible).  The next kernel may be placed where this grid leaves room.  (Barriers and tensor memory
  // could be set up before the wait too, but the compiler then makes a slower softmax loop: head dimension 64 with a
  // bias, 1 x 16 x 4096, 220 us against 205 in this order; without one, 8 x 12 x 1024, 39.6 against 38.3.)
  pdl_wait();
  pdl_launch_dependents();
  const int kv_limit = valid_keys(p, b);
  TileGeom tg0 = tile_geometry(p, row0_0, kv_limit, PACK ? pack.lb : kBlockM);
  TileGeom tg1 = tile_geometry(p, row0_1, kv_limit, PACK ? pack.lb : kBlockM);
  if constexpr (PACK) {
    auto clip = [&](int n) { n -= key_tile0; return n < 0 ? 0 : (n > pack.split_tiles ? pack.split_tiles : n); };
    tg0.n_tiles = clip(tg0.n_tiles);
    tg1.n_tiles = clip(tg1.n_tiles);
    if (dual) {
      const int n = tg0.n_tiles;
      tg1 = tg0;
      tg0.n_tiles = (n + 1) / 2;
      tg1.n_tiles = n / 2;
    }
  }
  const int n_iter = tg0.n_tiles > tg1.n_tiles ? tg0.n_tiles : tg1.n_tiles;

  // Ring items.  Item i is a K or a V tile; plain order K(0) V(0) K(1) V(1) ..., dual order K(0) K(1) V(0) V(1) K(2)
  // K(3) V(2) V(3) ... (the last odd pair may be missing).
  const int n_ring = dual ? 4 * n_iter : 2 * n_iter;
  auto item_is_v = [&](int i) { return dual ? (i >> 1) & 1 : i & 1; };
  auto item_tile = [&](int i) { return dual ? (i >> 2) * 2 + (i & 1) : i >> 1; };
  auto item_exists = [&](int i) { return !dual || item_tile(i) < tg0.n_tiles + tg1.n_tiles; };

  const uint32_t q_smem[2] = {tiles, tiles + C::kTileBytes};
  const uint32_t kv_smem = tiles + kTilesPerCta * C::kTileBytes;

  // Set-up is spread over the roles so that the first copies are in flight while barriers are initialised and tensor
  // memory is allocated: the producer lane owns the barriers of its own copies and starts Q and the first ring slots at
  // once.
  int items_issued = 0;   // (producer lane) ring items already issued
  bool q_armed = false;   // (producer lane) a copy into the Q slots is in flight or has landed
  if (warp == kProducerWarp && lane == 0) {
    mbar_init(smem_u32(&sync->q_full), 1);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(smem_u32(&sync->kv_full[s]), 1);
      mbar_init(smem_u32(&sync->kv_empty[s]), 1);
    }
    mbar_fence_init();
    // A tile without visible keys never reads its Q: its shared-memory slot is used
    // straight away to stage the all-zero output, so nothing may be in flight into it.
    const uint32_t q_tile_bytes = PACK ? C::kBoxes * 128 * pack.lb * p.group : C::kTileBytes;
    uint32_t q_bytes = 0;
    if (tg0.n_tiles > 0) q_bytes += q_tile_bytes;
    if (tg1.n_tiles > 0 && !dual) q_bytes += q_tile_bytes;
    const uint32_t qbar = smem_u32(&sync->q_full);
    if (q_bytes > 0) mbar_arrive_expect_tx(qbar, q_bytes);
    q_armed = q_bytes > 0;
    for (int t = 0; t < 2; ++t) {
      const TileGeom& tg = t == 0 ? tg0 : tg1;
      if (tg.n_tiles == 0 || (dual && t == 1)) continue;
      for (int bx = 0; bx < C::kBoxes; ++bx)
        tma_load_4d(q_smem[t] + bx * kBoxBytes, &tm_q, qbar, bx * 64, tg.row0, head_of_tile[t], b);
    }
    for (; items_issued < n_ring && items_issued < C::kStages; ++items_issued) {
      if (!item_exists(items_issued)) continue;
      const uint32_t bar = smem_u32(&sync->kv_full[items_issued]);
      mbar_arrive_expect_tx(bar, C::kTileBytes);
      const CUtensorMap* map = item_is_v(items_issued) ? &tm_v : &tm_k;
      for (int bx = 0; bx < C::kBoxes; ++bx)
        tma_load_4d(kv_smem + items_issued * C::kTileBytes + bx * kBoxBytes, map, bar, bx * 64,
                    (key_tile0 + item_tile(items_issued)) * kBlockN, hk, b);
    }
    prefetch_tmap(&tm_o);
  }
  if (tid < 2) {
    const int t = tid;
    mbar_init(smem_u32(&sync->s_full[t]), 1);
    mbar_init(smem_u32(&sync->p_ready[t][0]), kBlockM);
    mbar_init(smem_u32(&sync->p_ready[t][1]), kBlockM);
    mbar_init(smem_u32(&sync->o_done[t]), 1);
    mbar_init(smem_u32(&sync->o_staged[t]), kBlockM);
    mbar_init(smem_u32(&sync->s_free[t]), kBlockM);
    mbar_init(smem_u32(&sync->pv_done[t]), 1);
    if (t == 0) {
      mbar_init(smem_u32(&sync->drain), 1);
      sync->abort_flag = 0;
    }
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

  if (warp == kProducerWarp) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      bool alive = true;
      for (int item = items_issued; item < n_ring && alive; ++item) {
        if (!item_exists(item)) continue;
        const int j = item_tile(item);
        const int stage = item % C::kStages;
        const uint32_t round = static_cast<uint32_t>(item / C::kStages);
        if (round > 0) {
          alive = wait_clocked(smem_u32(&sync->kv_empty[stage]), (round - 1) & 1u, abort_flag, wait_limit);
          if (!alive) {
            report(p.status, 1, item, stage);
            break;
          }
        }
        const uint32_t bar = smem_u32(&sync->kv_full[stage]);
        const uint32_t dst = kv_smem + stage * C::kTileBytes;
        mbar_arrive_expect_tx(bar, C::kTileBytes);
        const CUtensorMap* map = item_is_v(item) ? &tm_v : &tm_k;
        for (int bx = 0; bx < C::kBoxes; ++bx) tma_load_4d(dst + bx * kBoxBytes, map, bar, bx * 64, (key_tile0 + j) * kBlockN, hk, b);
        items_issued = item + 1;
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // -------------------------------------------------------------- MMA issuer
    // The whole warp runs the control flow (waits included) so that addresses and
    // descriptors stay in the uniform datapath; one elected lane issues.  The tile
    // index is a compile-time constant everywhere for the same reason.
    {
      constexpr uint32_t idesc_qk = make_idesc(BF16, false, kBlockM, kBlockN);
      const uint32_t idesc_pv = make_idesc(BF16, true, kBlockM, PAD ? (p.Dv + 15) / 16 * 16 : D);
      const int qk_steps = PAD ? (p.E + 15) / 16 : D / 16;
      bool alive = n_iter > 0;

      // descriptors: fixed fields once, then only the 16-byte-unit start address moves
      const uint64_t q_desc0 = smem_desc_sw128(q_smem[0], 16, 1024), q_desc1 = smem_desc_sw128(q_smem[1], 16, 1024);
      const uint64_t kv_desc_k = smem_desc_sw128(kv_smem, 16, 1024);          // K tile as K-major B operand
      const uint64_t kv_desc_v = smem_desc_sw128(kv_smem, kBoxBytes, 1024);   // V tile as MN-major B operand
      auto issue_qk = [&](auto tile_const, uint32_t stage) {
        constexpr int t = decltype(tile_const)::value;
        const uint64_t qd = t == 0 || dual ? q_desc0 : q_desc1;
        const uint64_t kd = kv_desc_k + static_cast<uint64_t>(stage * (C::kTileBytes >> 4));
        const uint32_t d_addr = tmem_base + static_cast<uint32_t>(t * 128);
        if (elect_one() && dbg_tmem(p.status, DBG_PREFILL * 100 + 1, d_addr, tmem_base, 128, 512)) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            if (PAD && kk >= qk_steps) break;
            const uint64_t off = static_cast<uint64_t>(((kk >> 2) * kBoxBytes + (kk & 3) * 32) >> 4);
            mma_ss(d_addr, qd + off, kd + off, idesc_qk, kk > 0 ? 1u : 0u);
          }
        }
      };
      // O_t (+)= P_t[:, half*64 .. half*64+63] . V[half*64 .. , :]   (four K-steps of 16 keys)
      auto issue_pv_half = [&](auto tile_const, uint32_t stage, int half, bool accumulate) {
        constexpr int t = decltype(tile_const)::value;
        const uint64_t vd = kv_desc_v + static_cast<uint64_t>(stage * (C::kTileBytes >> 4) + half * 4 * (2048 >> 4));
        const uint32_t d_addr = tmem_base + static_cast<uint32_t>(256 + t * D);
        const uint32_t a_addr = tmem_base + static_cast<uint32_t>(C::kSplitP ? 384 + t * 64 + half * 32 : t * 128 + half * 32);
        const uint32_t acc0 = (accumulate || half > 0) ? 1u : 0u;
        if (elect_one() && dbg_tmem(p.status, DBG_PREFILL * 100 + 2, d_addr, tmem_base, D, 512) &&
            dbg_tmem(p.status, DBG_PREFILL * 100 + 3, a_addr, tmem_base, 32, 512)) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            mma_ts(d_addr, a_addr + static_cast<uint32_t>(kk * 8), vd + static_cast<uint64_t>(kk * (2048 >> 4)), idesc_pv,
                   kk > 0 ? 1u : acc0);
            if (PAD)
              mma_ts(d_addr, a_addr + static_cast<uint32_t>(64 + kk * 8), vd + static_cast<uint64_t>(kk * (2048 >> 4)), idesc_pv, 1u);
          }
        }
      };
      auto commit = [&](uint32_t bar) {
        if (elect_one()) mma_commit(bar);
      };
      auto wait_full = [&](int item) -> bool {
        const int stage = item % C::kStages;
        const uint32_t round = static_cast<uint32_t>(item / C::kStages);
        const bool ok = wait_clocked(smem_u32(&sync->kv_full[stage]), round & 1u, abort_flag, wait_limit);
        if (!ok && lane == 0) report(p.status, 2, item, stage);
        return ok;
      };
      auto stage_addr = [&](int item) { return static_cast<uint32_t>(item % C::kStages); };
      auto empty_bar = [&](int item) { return smem_u32(&sync->kv_empty[item % C::kStages]); };
      const std::integral_constant<int, 0> T0{};
      const std::integral_constant<int, 1> T1{};

      if (alive) {
        alive = wait_clocked(smem_u32(&sync->q_full), 0, abort_flag, wait_limit);
        if (!alive && lane == 0) report(p.status, 2, -1, 0);
      }
      if (alive) alive = wait_full(0);
      if (PACK && dual) {
        // Tile t works on key tiles 2 j + t: K at ring item 4 j + t, V at 4 j + 2 + t, each with one reader.
        auto scores = [&](auto tile_const, int j) {
          constexpr int t = decltype(tile_const)::value;
          const int item = 4 * j + t;
          alive = wait_full(item);
          if (!alive) return;
          tc_fence_after_sync();
          issue_qk(tile_const, stage_addr(item));
          commit(smem_u32(&sync->s_full[t]));
          commit(empty_bar(item));
        };
        auto serve = [&](auto tile_const, int j) {
          constexpr int t = decltype(tile_const)::value;
          const int nt = t == 0 ? tg0.n_tiles : tg1.n_tiles;
          if (j >= nt) return;
          if (C::kSplitP && j + 1 < nt) {   // as below: next scores first
            alive = wait_clocked(smem_u32(&sync->s_free[t]), j & 1, abort_flag, wait_limit);
            if (!alive) {
              if (lane == 0) report(p.status, 9, j, t);
              return;
            }
            scores(tile_const, j + 1);
            if (!alive) return;
          }
          alive = wait_full(4 * j + 2 + t);
          if (!alive) return;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            alive = wait_clocked(smem_u32(&sync->p_ready[t][half]), j & 1, abort_flag, wait_limit);
            if (!alive) {
              if (lane == 0) report(p.status, 3, j, t);
              return;
            }
            tc_fence_after_sync();
            issue_pv_half(tile_const, stage_addr(4 * j + 2 + t), half, j > 0);
          }
          commit(empty_bar(4 * j + 2 + t));
          if (C::kSplitP) commit(smem_u32(&sync->pv_done[t]));
          if (j + 1 >= nt) commit(smem_u32(&sync->o_done[t]));
          else if (!C::kSplitP) scores(tile_const, j + 1);
        };
        if (alive && tg0.n_tiles > 0) scores(T0, 0);
        if (alive && tg1.n_tiles > 0) scores(T1, 0);
        for (int j = 0; j < n_iter && alive; ++j) {
          serve(T0, j);
          if (alive) serve(T1, j);
        }
        alive = false;   // done: the loop below is the plain order's
      }
      if (alive) {
        tc_fence_after_sync();
        if (tg0.n_tiles > 0) {
          issue_qk(T0, stage_addr(0));
          commit(smem_u32(&sync->s_full[0]));
        }
        if (tg1.n_tiles > 0) {
          issue_qk(T1, stage_addr(0));
          commit(smem_u32(&sync->s_full[1]));
        }
        commit(empty_bar(0));
      }
      for (int j = 0; j < n_iter && alive; ++j) {
        const int item_v = 2 * j + 1, item_kn = 2 * j + 2;
        const bool has_next = j + 1 < n_iter;
        alive = wait_full(item_v);
        if (!alive) break;
        // (these shapes came from a kernel that never reads a key beyond kv_lens)
        if (PAD && !has_next && kv_limit < p.S && (j + 1) * kBlockN > kv_limit)
          zero_tile_rows<C::kBoxes, kBlockN>(kv_smem + stage_addr(item_v) * C::kTileBytes, kv_limit - j * kBlockN, lane);
        // one tile: P_t(j) V(j) in two halves as the halves of P arrive, then Q_t K(j+1)^T
        auto serve = [&](auto tile_const) {
          constexpr int t = decltype(tile_const)::value;
          const int nt = t == 0 ? tg0.n_tiles : tg1.n_tiles;
          if (C::kSplitP) {
            // next scores first: S_t(j) only has to be out of tensor memory, not consumed
            if (t == 0 && has_next) {
              alive = wait_full(item_kn);
              if (!alive) return;
            }
            if (j + 1 < nt) {
              alive = wait_clocked(smem_u32(&sync->s_free[t]), j & 1, abort_flag, wait_limit);
              if (!alive) {
                if (lane == 0) report(p.status, 9, j, t);
                return;
              }
              tc_fence_after_sync();
              issue_qk(tile_const, stage_addr(item_kn));
              commit(smem_u32(&sync->s_full[t]));
            }
          }
          if (j < nt) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              alive = wait_clocked(smem_u32(&sync->p_ready[t][half]), j & 1, abort_flag, wait_limit);
              if (!alive) {
                if (lane == 0) report(p.status, 3, j, t);
                return;
              }
              tc_fence_after_sync();
              issue_pv_half(tile_const, stage_addr(item_v), half, j > 0);
            }
          }
          if (C::kSplitP) {
            if (j < nt) {
              commit(smem_u32(&sync->pv_done[t]));
              if (j + 1 >= nt) commit(smem_u32(&sync->o_done[t]));
            }
          } else {
            if (t == 0 && has_next) {
              alive = wait_full(item_kn);
              if (!alive) return;
              tc_fence_after_sync();
            }
            if (j + 1 < nt) {
              issue_qk(tile_const, stage_addr(item_kn));
              commit(smem_u32(&sync->s_full[t]));
            } else if (j < nt) {
              commit(smem_u32(&sync->o_done[t]));
            }
          }
        };
        serve(T0);
        if (!alive) break;
        serve(T1);
        if (!alive) break;
        commit(empty_bar(item_v));
        if (has_next) commit(empty_bar(item_kn));
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ softmax roles
    const int t = warp >> 2;                 // which 128-row tile
    const int quad = warp & 3;               // TMEM lane quadrant this warp may touch
    const int r = tid & 127;                 // row inside the tile
    const TileGeom& tg = t == 0 ? tg0 : tg1;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_off + static_cast<uint32_t>(t) * 128u;
    const uint32_t o_addr = tmem_base + lane_off + 256u + static_cast<uint32_t>(t) * D;
    const uint32_t p_addr = C::kSplitP ? tmem_base + lane_off + 384u + static_cast<uint32_t>(t) * 64u : s_addr;
    // checked build: the three column ranges this thread reads and writes; a violation drains the CTA
    if (!dbg_tmem(p.status, DBG_PREFILL * 100 + 4, s_addr, tmem_base, 128, 512) ||
        !dbg_tmem(p.status, DBG_PREFILL * 100 + 5, o_addr, tmem_base, D, 512) ||
        !dbg_tmem(p.status, DBG_PREFILL * 100 + 6, p_addr, tmem_base, 64, 512))
      *abort_flag = 1;
    const int row_g = tg.row0 + (PACK ? r % pack.lb : r);
    // (split form) a tile row that belongs to no query row holds whatever was in shared memory: its lane computes on
    // that, in its own accumulator row, and stores nothing
    const int head_g = PACK ? hq0 + r / pack.lb : head_of_tile[t];
    const bool row_used = !PACK || (r < pack.lb * p.group && row_g < p.L);
    int lim = kv_limit;                      // keys [0, lim) are visible to this row
    if (p.causal) {
      const long long c = static_cast<long long>(row_g) + p.causal_shift + 1;
      lim = c < lim ? static_cast<int>(c < 0 ? 0 : c) : lim;
    }
    // With an additive bias the logits s * scale + bias are formed when the scores are read;
    // everything after that then works on them with scale 1 (log2 e in the exponent).
    const float sl2_in = BIAS ? p.scale : p.scale * kLog2e;
    const float sl2 = BIAS ? kLog2e : sl2_in;
    float m_run = -CUDART_INF_F, l_run = 0.f;
    bool alive = true;
    // accumulating form: the row's running lse is fetched now and used in the epilogue
    float old_lse = -CUDART_INF_F;
    if constexpr (ACC) {
      if (row_g < p.L && p.acc_mode == 2)
        old_lse = p.acc_lse[b * p.als[0] + head_of_tile[t] * p.als[1] + row_g * p.als[2]];
    }
    // this row of the bias, 16-bit elements in the query's dtype, unit stride along the keys
    const uint4* bias_row = nullptr;
    if constexpr (BIAS) {
      if (row_g < p.L)
        bias_row = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.bias) + b * p.bs[0] +
                                                  static_cast<long long>(head_of_tile[t]) * p.bs[1] +
                                                  static_cast<long long>(row_g) * p.bs[2]);
    }

    const bool bias_wide = BIAS && bias_rows_32b(p);

    if (tg.in_range) {
      for (int j = 0; j < tg.n_tiles; ++j) {
        uint4 bv[BIAS ? kBlockN / 8 : 1];
        if constexpr (BIAS) {
          // the bias of this key tile travels while the scores are awaited
          load_bias_row(bv, bias_row, j * kBlockN, p.S, bias_wide);
        }
        bool ok = wait_clocked(smem_u32(&sync->s_full[t]), j & 1, abort_flag, wait_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) report(p.status, 4 + t, j, quad);
          alive = false;
          break;
        }
        tc_fence_after_sync();
        const int col0 = (key_tile0 + (dual ? 2 * j + t : j)) * kBlockN;
        const bool need_mask = col0 + kBlockN > tg.min_lim;

        // S row -> registers in two halves; the second half is in flight while the
        // maximum of the first is taken
        uint32_t sv[kBlockN];
        tmem_ld_32x32(s_addr, reinterpret_cast<uint32_t(&)[32]>(sv[0]));
        tmem_ld_32x32(s_addr + 32, reinterpret_cast<uint32_t(&)[32]>(sv[32]));
        tmem_ld_wait();
        tmem_ld_32x32(s_addr + 64, reinterpret_cast<uint32_t(&)[32]>(sv[64]));
        tmem_ld_32x32(s_addr + 96, reinterpret_cast<uint32_t(&)[32]>(sv[96]));
        float mxa = -CUDART_INF_F, mxb = -CUDART_INF_F;
        if constexpr (BIAS) {
#pragma unroll
          for (int i = 0; i < 8; ++i) add_bias8<BF16>(&sv[8 * i], bv[i], sl2_in);
        }
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 64; ++i) sv[i] = (col0 + i < lim) ? sv[i] : 0xff800000u;  // -inf
        }
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          mxa = max3(mxa, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
          mxb = max3(mxb, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
        }
        tmem_ld_wait();
        if (C::kSplitP) {
          tc_fence_before_sync();
          mbar_arrive(smem_u32(&sync->s_free[t]));
        }
        if constexpr (BIAS) {
#pragma unroll
          for (int i = 8; i < 16; ++i) add_bias8<BF16>(&sv[8 * i], bv[i], sl2_in);
        }
        if (need_mask) {
#pragma unroll
          for (int i = 64; i < kBlockN; ++i) sv[i] = (col0 + i < lim) ? sv[i] : 0xff800000u;
        }
#pragma unroll
        for (int i = 64; i < kBlockN; i += 4) {
          mxa = max3(mxa, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
          mxb = max3(mxb, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
        }
        const float mx = fmaxf(mxa, mxb);
        const float m_new = fmaxf(m_run, mx);
        const bool grow = (m_new - m_run) * sl2 > kRescaleThreshold;  // false for NaN (-inf - -inf)
        float alpha = 1.f;
        if (grow) {
          alpha = ex2((m_run - m_new) * sl2);   // m_run = -inf -> 0
          l_run *= alpha;
          m_run = m_new;
        }
        if (C::kSplitP && j > 0) {
          // here S(j) can be ready before P V of the previous tile has retired, and that product
          // still reads the P columns and writes O_t: wait for it before touching either
          bool pv_ok = wait_clocked(smem_u32(&sync->pv_done[t]), (j - 1) & 1, abort_flag, wait_limit);
          pv_ok = __all_sync(0xffffffffu, pv_ok);
          if (!pv_ok) {
            if (lane == 0) report(p.status, 10, j, t);
            alive = false;
            break;
          }
          tc_fence_after_sync();
        }
        if (j > 0 && __any_sync(0xffffffffu, grow)) {
          // raise the reference maximum: O_t *= alpha (PV(j-1) has retired: without the split its
          // completion is ordered before s_full(j))
#pragma unroll
          for (int c = 0; c < D / 16; ++c) {
            uint32_t v[16];
            tmem_ld_32x16(o_addr + c * 16, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            tmem_st_32x16(o_addr + c * 16, v);
          }
          tmem_st_wait();
        }
        const float nms = (m_run == -CUDART_INF_F) ? 0.f : -m_run * sl2;

        // probabilities, row sum (two packed accumulators), P -> TMEM over the first 64
        // columns of S.  (Measured alternatives that lost: a polynomial exp2 on the FMA
        // pipe for part of the row, and ex2 on packed 16-bit pairs.)
        uint64_t sum2[2] = {0ull, 0ull};           // two packed accumulators = four chains
#pragma unroll
        for (int c = 0; c < kBlockN / 32; ++c) {
          uint32_t pk[16], lo[PAD ? 16 : 1];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = ex2(fmaf(__uint_as_float(sv[c * 32 + i]), sl2, nms));
            const float p1 = ex2(fmaf(__uint_as_float(sv[c * 32 + i + 1]), sl2, nms));
            sum2[(i >> 1) & 1] = f2_add(sum2[(i >> 1) & 1], f2_pack(p0, p1));
            pk[i >> 1] = pack2<BF16>(p0, p1);
            if constexpr (PAD) lo[i >> 1] = remainder2<BF16>(p0, p1, pk[i >> 1]);
          }
          tmem_st_32x16(p_addr + c * 16, pk);
          if constexpr (PAD) tmem_st_32x16(p_addr + 64 + c * 16, lo);
          if (c == 1) {
            // first 64 keys of P are in TMEM: let P V start on them while the rest is computed
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(smem_u32(&sync->p_ready[t][0]));
          }
        }
        float sum4[4];
        f2_unpack(sum2[0], sum4[0], sum4[1]);
        f2_unpack(sum2[1], sum4[2], sum4[3]);
        const float sum = (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
        l_run += sum;
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(smem_u32(&sync->p_ready[t][1]));
      }

      // ------------------------------------------------------------- epilogue
      if (alive && tg.n_tiles > 0) {
        bool ok = wait_clocked(smem_u32(&sync->o_done[t]), 0, abort_flag, wait_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) report(p.status, 6 + t, 0, quad);
          alive = false;
        }
        tc_fence_after_sync();
      }
      if constexpr (PACK) {
        if (alive) {
          const int64_t slot = ((static_cast<int64_t>(b) * p.Hq + head_g) * p.L + row_g) * pack.n_split +
                               (dual ? 2 * (key_tile0 / pack.split_tiles) + t : key_tile0 / pack.split_tiles);
          const bool slot_ok = row_used && dbg_range(p.status, DBG_PREFILL * 100 + 9, slot, 1,
                                                     static_cast<int64_t>(p.B) * p.Hq * p.L * pack.n_split);
          if (slot_ok) *reinterpret_cast<float2*>(pack.part_ml + slot * 2) = make_float2(m_run * sl2, l_run);
          // O: every lane holds a row; 32 columns at a time go through this warp's 4 KB of the (idle) Q slot, so
          // that eight lanes store the 128 bytes of one row
          const int64_t my_row = slot_ok && l_run != 0.f ? slot : -1;   // (a NaN sum is not an empty one)
          uint8_t* buf = smem_raw + (q_smem[t] - raw_addr) + quad * 4096;
          if (tg.n_tiles > 0) {
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
              uint32_t v[32];
              tmem_ld_32x32(o_addr + c * 32, v);
              tmem_ld_wait();
              __syncwarp();
#pragma unroll
              for (int u = 0; u < 8; ++u)
                *reinterpret_cast<uint4*>(buf + lane * 128 + ((u ^ (lane & 7)) << 4)) =
                    make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int row = i * 4 + (lane >> 3), u = lane & 7;
                const int64_t dst = __shfl_sync(0xffffffffu, my_row, row);
                if (dst >= 0)
                  *reinterpret_cast<uint4*>(pack.part_o + dst * D + c * 32 + u * 4) =
                      *reinterpret_cast<const uint4*>(buf + row * 128 + ((u ^ (row & 7)) << 4));
              }
            }
          }
        }
      } else if constexpr (ACC) {
        // Accumulating form (a ring step): fold this block's result into the row's running fp32 pair
        // (acc, acc_lse) in place -- acc = acc * w_acc + O * w_o -- instead of writing out / lse.  Same
        // arithmetic as the persistent kernel's accumulating epilogue.  A tile without a visible key
        // leaves a started accumulator alone.
        if (alive && !(tg.n_tiles == 0 && p.acc_mode == 2)) {
          const bool row_ok = row_g < p.L &&
                              dbg_bhrc(p.status, DBG_PREFILL * 100 + 8, b, p.B, head_of_tile[t], p.Hq, row_g, p.L, 0, D, p.Dv);
          const float lse = l_run > 0.f ? fmaf(m_run, p.scale, lg2(l_run) * kLn2) : -CUDART_INF_F;
          float w_acc = 0.f, w_o = l_run > 0.f ? 1.f / l_run : 0.f;
          const float hi = fmaxf(old_lse, lse);
          float merged = -CUDART_INF_F;
          if (hi != -CUDART_INF_F) {
            const float e_old = ex2((old_lse - hi) * kLog2e), e_new = ex2((lse - hi) * kLog2e);   // -inf -> 0
            merged = hi + lg2(e_old + e_new) * kLn2;
            w_acc = ex2((old_lse - merged) * kLog2e);
            w_o *= ex2((lse - merged) * kLog2e);
          } else {
            w_o = 0.f;
          }
          float* arow = p.acc + b * p.as[0] + static_cast<long long>(head_of_tile[t]) * p.as[1] +
                        static_cast<long long>(row_g) * p.as[2];
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            uint32_t v[32];
            if (tg.n_tiles > 0) {   // (uniform over the warp: tensor-memory loads stay outside per-lane conditions)
              tmem_ld_32x32(o_addr + c * 32, v);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0u;
            }
            if (row_ok) {
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                float4* dst = reinterpret_cast<float4*>(arow + c * 32 + u * 4);
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
                if (p.acc_mode == 2) a = *dst;
                a.x = fmaf(a.x, w_acc, __uint_as_float(v[4 * u]) * w_o);
                a.y = fmaf(a.y, w_acc, __uint_as_float(v[4 * u + 1]) * w_o);
                a.z = fmaf(a.z, w_acc, __uint_as_float(v[4 * u + 2]) * w_o);
                a.w = fmaf(a.w, w_acc, __uint_as_float(v[4 * u + 3]) * w_o);
                *dst = a;
              }
            }
          }
          if (row_ok) p.acc_lse[b * p.als[0] + head_of_tile[t] * p.als[1] + row_g * p.als[2]] = merged;
        }
      } else if (alive) {
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        uint8_t* o_stage = smem_raw + (q_smem[t] - raw_addr);   // the Q tile is no longer needed
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t v[32];
          if (tg.n_tiles > 0) {
            tmem_ld_32x32(o_addr + c * 32, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            pk[i >> 1] = pack2<BF16>(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv);
          // 32 columns = 64 bytes = four 16-byte units of the 128-byte swizzled row
          uint8_t* box = o_stage + (c >> 1) * kBoxBytes + r * 128;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int unit = ((c & 1) * 4 + u) ^ (r & 7);
            *reinterpret_cast<uint4*>(box + unit * 16) = make_uint4(pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
          }
        }
        // Every writer publishes its rows to the async proxy and arrives; only the
        // storing thread waits (bounded), so a role that gave up cannot strand the
        // others at a barrier.
        fence_proxy_async_smem();
        mbar_arrive(smem_u32(&sync->o_staged[t]));
        if (r == 0 && wait_clocked(smem_u32(&sync->o_staged[t]), 0, abort_flag, wait_limit)) {
          for (int bx = 0; bx < C::kBoxes; ++bx) {
            if (PAD && bx * 64 >= p.Dv) break;
            tma_store_4d(&tm_o, q_smem[t] + bx * kBoxBytes, bx * 64, tg.row0, head_of_tile[t], b);
          }
          tma_store_commit();
          tma_store_wait_read();
        }
        if (p.lse != nullptr && row_g < p.L) {
          // one rounding at the magnitude of the maximum: m*scale + ln(l)
          const float lse = l_run > 0.f ? fmaf(m_run, BIAS ? 1.f : p.scale, lg2(l_run) * kLn2) : -CUDART_INF_F;
          if (dbg_bhrc(p.status, DBG_PREFILL * 100 + 7, b, p.B, head_of_tile[t], p.Hq, row_g, p.L, 0, 0, 1))
            p.lse[b * p.ls[0] + head_of_tile[t] * p.ls[1] + row_g * p.ls[2]] = lse;
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (sync->abort_flag != 0) {
    // A role gave up.  Before shared and tensor memory are handed back, whatever this CTA already
    // issued must have finished: the copies into the Q slots and the ring (their barriers complete
    // when the bytes have landed) and every MMA (one more commit, which arrives when all earlier ones
    // have retired).  These waits have their own generous bound, whatever the wait limit.
    if (warp == kProducerWarp && lane == 0) {
      if (q_armed) wait_drain(smem_u32(&sync->q_full), 0);
      for (int s = 0; s < C::kStages && s < items_issued; ++s) {
        const uint32_t last_round = static_cast<uint32_t>((items_issued - 1 - s) / C::kStages);
        wait_drain(smem_u32(&sync->kv_full[s]), last_round & 1u);
      }
    }
    if (warp == kMmaWarp) {
      if (elect_one()) mma_commit(smem_u32(&sync->drain));
      wait_drain(smem_u32(&sync->drain), 0);
    }
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------ host side --

// Pair two query heads of one kv head per CTA when the group size allows it and the
// mask is causal (that is where the row-block layout leaves one tile idle at the end).
int pair_heads_mode(const Problem& p) { return (p.causal && p.group % 2 == 0) ? 1 : 0; }

template <int D, bool BF16, bool BIAS, bool ACC = false, bool PAD = false>
int launch_variant(const Problem& p, cudaStream_t stream) {
  using C = Cfg<D>;
  CUtensorMap tq, tk, tv, to;
  if (!make_map(&tq, p.q, BF16, p.E, p.L, p.Hq, p.B, p.qs) || !make_map(&tk, p.k, BF16, p.E, p.S, p.Hkv, p.B, p.ks) ||
      !make_map(&tv, p.v, BF16, p.Dv, p.S, p.Hkv, p.B, p.vs))
    return B200_SDPA_ERR_CUDA;
  if (ACC) {
    to = tq;   // the accumulating form stores through plain pointers; the map is never used
  } else if (!make_map(&to, p.out, BF16, p.Dv, p.L, p.Hq, p.B, p.os)) {
    return B200_SDPA_ERR_CUDA;
  }
  auto kern = prefill_kernel<D, BF16, BIAS, ACC, PAD, false>;
  // the opt-in to more than 48 KB of dynamic shared memory is a per-device attribute: set on every
  // launch (a cheap host-side call), so a process that drives several GPUs gets it on each of them
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) {
    cudaGetLastError();
    return B200_SDPA_ERR_CUDA;
  }
  const int pair_heads = pair_heads_mode(p);
  const int rows = pair_heads ? kBlockM : kRowsPerCta;
  const int n_qblk = (p.L + rows - 1) / rows;
  const long long grid = static_cast<long long>(n_qblk) * (p.Hq / (pair_heads ? 2 : 1)) * p.B;
  if (grid <= 0 || grid > 0x7fffffffLL) return B200_SDPA_ERR_UNSUPPORTED;
  const int per_wave = kv_streams_per_wave(static_cast<long long>(p.S) * (p.E + p.Dv) * 2, static_cast<long long>(p.Hkv) * p.B);
  if (!launch_pdl(kern, dim3(static_cast<unsigned>(grid)), kThreads, C::kSmemBytes, stream, tq, tk, tv, to, p, n_qblk, pair_heads,
                  per_wave, wait_limit_cycles(), PackArgs{}))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_PREFILL);
  return B200_SDPA_OK;
}

}  // namespace

namespace {

// What every head dimension needs: 16-bit types, a positive finite scale, TMA-legal bases and strides.
bool operands_eligible(const Problem& p, int dtype, bool* alignment_only_failure) {
  if (dtype != B200_SDPA_F16 && dtype != B200_SDPA_BF16) return false;
  if (!(p.scale > 0.f) || !(p.scale < 1e30f)) return false;
  if (p.L < 1 || p.S < 1) return false;
  if (p.bias != nullptr) {
    if (!bias_readable(p, dtype, alignment_only_failure)) return false;
  }
  const bool ok = strides_ok(p.q, p.qs, p.L, p.Hq, p.B) && strides_ok(p.k, p.ks, p.S, p.Hkv, p.B) &&
                  strides_ok(p.v, p.vs, p.S, p.Hkv, p.B) && strides_ok(p.out, p.os, p.L, p.Hq, p.B);
  if (!ok && alignment_only_failure) *alignment_only_failure = true;
  return ok;
}

void plan_per_cta(const Problem& p, long long grid, int rows, B200SdpaPlan* plan) {
  plan->path = B200_SDPA_PATH_PREFILL;
  plan->block_m = rows;
  plan->block_n = kBlockN;
  plan->grid_x = static_cast<int32_t>(grid);
  plan->grid_y = plan->grid_z = 1;
  plan->threads = kThreads;
  plan->smem_bytes = p.E == 64 && p.Dv == 64 ? Cfg<64>::kSmemBytes : Cfg<128>::kSmemBytes;
  plan->kv_splits = 1;
  plan->launches = 1;
  plan->workspace_bytes = 0;
}

// Merge of the split form's partials: one warp per query row, the row's columns spread over the lanes.
template <typename T, int D>
__global__ void __launch_bounds__(256) prefill_combine_kernel(const Problem p, const int n_split,
                                                              const float* __restrict__ part_o,
                                                              const float* __restrict__ part_ml) {
  constexpr int C = D / 32;   // columns per lane
  const int lane = threadIdx.x & 31;
  const int64_t row_id = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  pdl_wait();
  pdl_launch_dependents();
  if (row_id >= static_cast<int64_t>(p.B) * p.Hq * p.L) return;
  const int i = static_cast<int>(row_id % p.L);
  const int h = static_cast<int>((row_id / p.L) % p.Hq);
  const int b = static_cast<int>(row_id / p.L / p.Hq);
  float2 ml = make_float2(-CUDART_INF_F, 0.f);
  if (lane < n_split) ml = *reinterpret_cast<const float2*>(part_ml + (row_id * n_split + lane) * 2);
  float mx = ml.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  // A split without a visible key for this row has a sum of 0 and wrote nothing else.  Everything but 0 counts: NaN in
  // a score must come out as NaN, as it does where one CTA walks all keys.
  const unsigned seen = __ballot_sync(0xffffffffu, ml.y != 0.f);
  const float w = ml.y != 0.f ? ex2(ml.x - mx) : 0.f;
  float lsum = ml.y != 0.f ? w * ml.y : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  float acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = 0.f;
  const float* src = part_o + row_id * n_split * D + lane * C;
#pragma unroll 4
  for (int s = 0; s < n_split; ++s) {
    const float ws = __shfl_sync(0xffffffffu, w, s);
    if ((seen >> s) & 1u) {
      float v[C];
      if constexpr (C == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src + s * D);
      else *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(src + s * D);
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] = fmaf(v[c], ws, acc[c]);
    }
  }
  const float inv = lsum != 0.f ? 1.f / lsum : 0.f;
  if (!dbg_bhrc(p.status, DBG_PREFILL * 100 + 10, b, p.B, h, p.Hq, i, p.L, lane * C, C, p.Dv)) return;
  T* out = reinterpret_cast<T*>(p.out) + b * p.os[0] + static_cast<int64_t>(h) * p.os[1] + static_cast<int64_t>(i) * p.os[2] + lane * C;
  T r[C];
#pragma unroll
  for (int c = 0; c < C; ++c) r[c] = from_f32<T>(acc[c] * inv);
  if constexpr (C == 4) *reinterpret_cast<uint2*>(out) = *reinterpret_cast<const uint2*>(r);
  else *reinterpret_cast<uint32_t*>(out) = *reinterpret_cast<const uint32_t*>(r);
  if (p.lse != nullptr && lane == 0)
    p.lse[b * p.ls[0] + h * p.ls[1] + i * p.ls[2]] = lsum > 0.f ? fmaf(mx, kLn2, lg2(lsum) * kLn2) : -CUDART_INF_F;
}

struct PackGeom {
  int lb, n_pairs, dual, n_split, split_tiles;
  long long grid;
  uint64_t ws_bytes;
};

// Whether the split form serves a request, and how.  The plain form gives every 128 (or 256) rows of a head a CTA
// that walks all its keys: with a handful of rows, or few heads and sequences, that leaves most SMs without work and
// most of every tile without rows.  The rule compares estimates of both, in cycles of one SM:
//   plain   the longest CTA, or all key tiles spread over the SMs, at kPairCycles each, + kCtaCycles per round of CTAs
//   split   the same for the packed tiles, + the fp32 partials written and read once, + a second launch
// neither below the time the keys and values need from HBM, and takes the split form where it saves a twentieth.
// bf16, 32/8 heads: 8 x 8 rows against 4096 keys 72 -> 34 us (HBM floor 21), 1 x 16 rows against 8192 keys 123 -> 20,
// 1 x 128 against 8192 keys 123 -> 29; 8/8 heads, 1024 rows and keys 23.7 -> 17.6.
bool pack_geometry(const Problem& p, PackGeom* best) {
  constexpr long long kSms = 148, kPairCycles = 3400, kPackedCycles = 3600, kCtaCycles = 9000, kLaunchCycles = 6000, kHbmBytesPerCycle = 3400;
  constexpr int kMaxSplit = 32;
  if (p.E != p.Dv || (p.E != 64 && p.E != 128) || p.bias != nullptr || p.acc_mode != 0 || p.group > kBlockM) return false;
  const char* mode = getenv("B200_SDPA_PREFILL");
  const bool forced = mode != nullptr && mode[0] == 's';   // "split"
  if (mode != nullptr && !forced) return false;
  const long long streams = static_cast<long long>(p.Hkv) * p.B;
  const long long tiles = (p.S + kBlockN - 1) / kBlockN;
  if (tiles < 2) return false;
  auto key_tiles = [&](long long last_row) {   // tiles that rows up to last_row see
    long long end = p.S;
    if (p.causal) {
      const long long e = (last_row < p.L ? last_row : p.L - 1) + p.causal_shift + 1;
      end = e < end ? (e < 0 ? 0 : e) : end;
    }
    return (end + kBlockN - 1) / kBlockN;
  };
  const long long hbm = streams * key_tiles(p.L - 1) * kBlockN * (p.E + p.Dv) * 2 / kHbmBytesPerCycle;
  auto estimate = [&](long long total, long long longest, long long ctas, long long per_tile) {
    // equal CTAs run in whole rounds; unequal ones (a causal mask), longest first, spread out
    const long long rounds = (ctas + kSms - 1) / kSms, spread = (total + kSms - 1) / kSms + longest / 2;
    const bool equal = total * 4 > ctas * longest * 3;
    const long long steps = equal ? rounds * longest : (ctas <= kSms || spread < longest ? longest : spread);
    const long long work = steps * per_tile;
    return kLaunchCycles + (work > hbm ? work : hbm) + kCtaCycles * rounds;
  };
  const int pair_heads = pair_heads_mode(p);
  const int rows = pair_heads ? kBlockM : kRowsPerCta;
  const long long blocks = (p.L + rows - 1) / rows, per_block = static_cast<long long>(p.Hq / (pair_heads ? 2 : 1)) * p.B;
  if (!forced && blocks >= 64) return false;   // many rows: the plain form's tiles are full
  long long total = 0, longest = 0;
  for (long long i = 0; i < blocks; ++i) {
    const long long n = key_tiles((i + 1) * rows - 1);
    total += n * per_block;
    longest = n > longest ? n : longest;
  }
  const long long plain = estimate(total, longest, blocks * per_block, kPairCycles);

  PackGeom g;
  g.lb = kBlockM / p.group < p.L ? kBlockM / p.group : p.L;
  const int n_rt = (p.L + g.lb - 1) / g.lb;
  g.n_pairs = (n_rt + 1) / 2;
  g.dual = n_rt == 1 ? 1 : 0;
  total = longest = 0;
  for (long long i = 0; i < g.n_pairs; ++i) {
    const long long n = key_tiles((i + 1) * 2 * g.lb - 1);
    total += n * streams;
    longest = n > longest ? n : longest;
  }
  const long long row_bytes = static_cast<long long>(p.B) * p.Hq * p.L * (p.Dv + 2) * 4;
  long long best_cost = forced ? (1LL << 60) : plain * 19 / 20;
  bool found = false;
  const int per_cta = g.dual ? 2 : 1;   // partials a CTA leaves for a row
  for (int n = 1; n * per_cta <= kMaxSplit && n <= tiles; ++n) {
    g.split_tiles = static_cast<int>((tiles + n - 1) / n);
    if ((tiles + g.split_tiles - 1) / g.split_tiles != n || (forced && n == 1 && !g.dual)) continue;
    g.n_split = n * per_cta;
    g.grid = g.n_pairs * streams * n;
    g.ws_bytes = static_cast<uint64_t>(row_bytes) * g.n_split;
    if (g.grid > 0x7fffffffLL) break;
    const long long part = longest < g.split_tiles ? longest : g.split_tiles;
    // two key tiles in the time of one where both tiles of the CTA are the same rows; partials written and read
    // back at about 6 KB a cycle for the whole chip
    const long long cost = estimate((total + per_cta - 1) / per_cta, (part + per_cta - 1) / per_cta, g.grid, g.dual ? kPairCycles : kPackedCycles) +
                           kLaunchCycles + 2 * row_bytes * g.n_split / 6000;
    if (cost < best_cost) {
      best_cost = cost;
      *best = g;
      found = true;
    }
  }
  return found;
}

template <int D, bool BF16>
int launch_packed(const Problem& p, const PackGeom& g, float* workspace, cudaStream_t stream) {
  using C = Cfg<D>;
  CUtensorMap tq, tk, tv;
  if (!make_map(&tq, p.q, BF16, D, p.L, p.Hq, p.B, p.qs, g.lb, p.group) || !make_map(&tk, p.k, BF16, D, p.S, p.Hkv, p.B, p.ks) ||
      !make_map(&tv, p.v, BF16, D, p.S, p.Hkv, p.B, p.vs))
    return B200_SDPA_ERR_CUDA;
  auto kern = prefill_kernel<D, BF16, false, false, false, true>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) {
    cudaGetLastError();
    return B200_SDPA_ERR_CUDA;
  }
  const long long n_rows = static_cast<long long>(p.B) * p.Hq * p.L;
  PackArgs a;
  a.lb = g.lb;
  a.dual = g.dual;
  a.n_pairs = g.n_pairs;
  a.n_split = g.n_split;
  a.split_tiles = g.split_tiles;
  a.part_o = workspace;
  a.part_ml = workspace + n_rows * g.n_split * D;
  if (!launch_pdl(kern, dim3(static_cast<unsigned>(g.grid)), kThreads, C::kSmemBytes, stream, tq, tk, tv, tq, p, 0, 0, 1,
                  wait_limit_cycles(), a))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_PREFILL);
  using T = std::conditional_t<BF16, __nv_bfloat16, __half>;
  if (!launch_pdl(prefill_combine_kernel<T, D>, dim3(static_cast<unsigned>((n_rows + 7) / 8)), 256, 0, stream, p, g.n_split,
                  a.part_o, a.part_ml))
    return B200_SDPA_ERR_CUDA;
  count_launch(KID_COMBINE);
  return B200_SDPA_OK;
}

}  // namespace

bool prefill_eligible(const Problem& p, int dtype, bool* alignment_only_failure) {
  if (p.E > 128) return prefill_wide_eligible(p, dtype, alignment_only_failure);
  if (alignment_only_failure) *alignment_only_failure = false;
  if (p.E != p.Dv || (p.E != 64 && p.E != 128)) return false;
  return operands_eligible(p, dtype, alignment_only_failure);
}

// Head dimensions between 64 and 128 (multiples of 8, so that rows stay on the 16-byte grid of a tensor copy):
// 128-wide tiles with zero-filled columns.  Below 64 the exponentials bound a tile whatever its head dimension
// and the requests are small; those keep the CUDA-core kernel.  Measured (fp16, 16 x 16 heads x 577 x 577, head
// dimension 80): CUDA-core kernel 2463 us, these tiles 79 us with a 16-bit P, 92 us with hi + lo.
bool prefill_padded_eligible(const Problem& p, int dtype) {
  const int hi = p.E > p.Dv ? p.E : p.Dv;
  if (hi < 64 || hi > 128 || p.E % 8 != 0 || p.Dv % 8 != 0) return false;
  if (p.E == p.Dv && (p.E == 128 || p.E == 64) && !p.bias_padded) return false;
  if (hi == 64 && !p.bias_padded) return false;
  if (p.block_table != nullptr || p.k_new != nullptr || p.acc_mode != 0) return false;
  return operands_eligible(p, dtype, nullptr);
}

int plan_prefill(const Problem& p, int dtype, B200SdpaPlan* plan) {
  if (p.E > 128) return plan_prefill_wide(p, dtype, plan);
  if (!prefill_eligible(p, dtype, nullptr)) return B200_SDPA_ERR_UNSUPPORTED;
  PackGeom g;
  if (pack_geometry(p, &g)) {
    plan_per_cta(p, g.grid, g.lb * p.group, plan);
    plan->kv_splits = g.n_split;
    plan->launches = 2;
    plan->workspace_bytes = g.ws_bytes;
    return B200_SDPA_OK;
  }
  if (prefill_persistent_wanted(p)) {
    plan_prefill_persistent(p, plan);
    return B200_SDPA_OK;
  }
  const int pair_heads = pair_heads_mode(p);
  const int rows = pair_heads ? kBlockM : kRowsPerCta;
  const int n_qblk = (p.L + rows - 1) / rows;
  const long long grid = static_cast<long long>(n_qblk) * (p.Hq / (pair_heads ? 2 : 1)) * p.B;
  if (grid > 0x7fffffffLL) return B200_SDPA_ERR_UNSUPPORTED;
  plan_per_cta(p, grid, rows, plan);
  return B200_SDPA_OK;
}

int plan_prefill_padded(const Problem& p, B200SdpaPlan* plan) {
  if (prefill_persistent_wanted(p)) {
    plan_prefill_persistent(p, plan);
    return B200_SDPA_OK;
  }
  const int pair_heads = pair_heads_mode(p);
  const int rows = pair_heads ? kBlockM : kRowsPerCta;
  const long long grid = static_cast<long long>((p.L + rows - 1) / rows) * (p.Hq / (pair_heads ? 2 : 1)) * p.B;
  if (grid > 0x7fffffffLL) return B200_SDPA_ERR_UNSUPPORTED;
  plan_per_cta(p, grid, rows, plan);
  return B200_SDPA_OK;
}

// The caller has checked prefill_padded_eligible().
int launch_prefill_padded(const Problem& p, int dtype, void* workspace, uint64_t workspace_bytes, cudaStream_t stream) {
  if (prefill_persistent_wanted(p)) return launch_prefill_persistent(p, dtype, workspace, workspace_bytes, stream);
  const bool bf16 = dtype == B200_SDPA_BF16;
  if (p.bias != nullptr)
    return bf16 ? launch_variant<128, true, true, false, true>(p, stream)
                : launch_variant<128, false, true, false, true>(p, stream);
  return bf16 ? launch_variant<128, true, false, false, true>(p, stream)
              : launch_variant<128, false, false, false, true>(p, stream);
}

int launch_prefill(const Problem& p, int dtype, void* workspace, uint64_t workspace_bytes, cudaStream_t stream) {
  if (p.E > 128) return launch_prefill_wide(p, dtype, stream);
  if (!prefill_eligible(p, dtype, nullptr)) return B200_SDPA_ERR_UNSUPPORTED;
  const bool bf16 = dtype == B200_SDPA_BF16;
  PackGeom g;
  if (workspace != nullptr && reinterpret_cast<uintptr_t>(workspace) % 16 == 0 && pack_geometry(p, &g) &&
      workspace_bytes >= g.ws_bytes) {
    float* ws = reinterpret_cast<float*>(workspace);
    if (p.E == 128) return bf16 ? launch_packed<128, true>(p, g, ws, stream) : launch_packed<128, false>(p, g, ws, stream);
    return bf16 ? launch_packed<64, true>(p, g, ws, stream) : launch_packed<64, false>(p, g, ws, stream);
  }
  if (prefill_persistent_wanted(p)) return launch_prefill_persistent(p, dtype, workspace, workspace_bytes, stream);
  if (p.acc_mode != 0) {
    if (!prefill_accumulate_eligible(p)) return B200_SDPA_ERR_UNSUPPORTED;
    return bf16 ? launch_variant<128, true, false, true>(p, stream) : launch_variant<128, false, false, true>(p, stream);
  }
  if (p.bias != nullptr) {
    if (p.E == 128) return bf16 ? launch_variant<128, true, true>(p, stream) : launch_variant<128, false, true>(p, stream);
    return bf16 ? launch_variant<64, true, true>(p, stream) : launch_variant<64, false, true>(p, stream);
  }
  if (p.E == 128) return bf16 ? launch_variant<128, true, false>(p, stream) : launch_variant<128, false, false>(p, stream);
  return bf16 ? launch_variant<64, true, false>(p, stream) : launch_variant<64, false, false>(p, stream);
}

}  // namespace b200

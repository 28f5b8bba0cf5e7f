// Attention forward and backward in fp32 on CUDA cores, for head dimensions 64 and 128 with rows that can be copied
// 16 bytes at a time and without a bias.  (generic_fwd.cu and bwd_generic.cu keep every other fp32 request.)
//
// All products are fp32 FMAs: 128 a cycle and SM, 74 TFLOP/s at 1.965 GHz, is the bound, and the kernels are laid out
// so that the FMA pipe is what they wait for.  A CTA of 128 threads keeps 64 or 32 rows ("fixed") of one operand pair in
// shared memory and streams tiles of NC rows of the other past them; thread (ty, tx) owns 4 fixed rows and, of a
// score tile, the NC / TX streamed rows tx, tx + TX, ...  Two kinds of product:
//   scores      S[r][c] = sum_e F[r][e] G[c][e]: both row-major, read 4 elements of e at a time, the even and odd
//               elements summed as the two halves of one packed fp32 pair (fma.rn.f32x2: one instruction, two FMAs)
//   accumulate  acc[r][d] += sum_c O[c][r] G[c][d]: the score-shaped operand is left in shared memory transposed, so
//               that pairs of fixed rows are packed pairs; 64 or 128 columns d spread over tx
// The packed instructions leave every other issue slot to the shared-memory loads.  Those are the second bound: a
// 16-byte load costs two passes when each half of the warp reads at most 128 different bytes, four otherwise, so a warp
// covers 4 x 8 patches (TX = 8) and not 2 x 16: three quarters of the passes per FMA.
// Softmax statistics stay in registers (shuffles over the threads of a row).  Copies are asynchronous and each is
// issued as soon as its buffer has been read, so it travels under the phase that does not need it.
//
//   kernel   fixed     streamed   score products   accumulated
//   forward  Q         K, V       S                O += P V
//   dQ       Q, dO     K, V       S, dP            dQ += dS K
//   dK, dV   K, V      Q, dO      S^T, dP^T        dV += P^T dO, dK += dS^T Q   (over the group's query heads)
//
// TX = 8 (64 fixed rows) with single stream buffers, two CTAs to an SM hiding each other's copies; TX = 16 (32 rows)
// with double buffers where 64-row blocks would leave SMs without a second CTA.  Measured, causal: 2 x 8 x 512, head
// dimension 64, forward + backward 425 us on the generic kernels, 150 here (40 + 50 + 66 and launches); 2 x 16 x 1024:
// 1640 -> 595 us, FMA pipe 59 % of active cycles.  (More CTAs per SM, other unrollings and 8 x 4 patches: no faster.)
// Arithmetic as in generic_fwd.cu and
// bwd_generic.cu: expf, fp32 statistics, no scratch, no atomics.
#include "common.cuh"
#include "debug.cuh"

namespace b200 {

namespace {

constexpr int kThreads = 128;
constexpr int R = 4;   // fixed rows of a thread
#define kMaskedOut (-CUDART_INF_F)

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
  const int n = valid ? 16 : 0;   // 0: the destination is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int D> constexpr int kLd = D + 4;   // row stride in floats: eight consecutive rows start in different bank groups
template <int TX> constexpr int kLdOp = kThreads / TX * R + 4;   // row stride of the transposed operand

// `rows` rows of D floats, row stride `stride`, into a tile; rows at or beyond `n_valid` become zeros.
template <int D, int ROWS>
__device__ __forceinline__ void load_tile(float* tile, const float* src, int64_t stride, int n_valid) {
  constexpr int kChunks = D / 4;
#pragma unroll
  for (int i = 0; i < ROWS * kChunks / kThreads; ++i) {
    const int c = threadIdx.x + i * kThreads;
    const int row = c / kChunks, ch = c % kChunks;
    const bool ok = row < n_valid;
    copy16(tile + row * kLd<D> + ch * 4, src + (ok ? row * stride + ch * 4 : 0), ok);
  }
}

// S[i][j] = sum_e F[f0 + i][e] G[tx + TX j][e]
template <int D, int TX, int J>
__device__ __forceinline__ void score_patch(const float* F, const float* G, int f0, int tx, float (&s)[R][J]) {
  uint64_t acc[R][J];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j) acc[i][j] = 0ull;
#pragma unroll 4
  for (int e = 0; e < D; e += 4) {
    ulonglong2 g[J];
#pragma unroll
    for (int j = 0; j < J; ++j) g[j] = *reinterpret_cast<const ulonglong2*>(G + (tx + TX * j) * kLd<D> + e);
    ulonglong2 f[R];
#pragma unroll
    for (int i = 0; i < R; ++i) f[i] = *reinterpret_cast<const ulonglong2*>(F + (f0 + i) * kLd<D> + e);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j) acc[i][j] = fma2(f[i].x, g[j].x, acc[i][j]);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j) acc[i][j] = fma2(f[i].y, g[j].y, acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const float2 v = unpack2(acc[i][j]);
      s[i][j] = v.x + v.y;
    }
}

// Leaves the patch in shared memory transposed: O[c][fixed row].
template <int TX, int J>
__device__ __forceinline__ void store_transposed(float* O, int f0, int tx, const float (&s)[R][J]) {
#pragma unroll
  for (int j = 0; j < J; ++j)
    *reinterpret_cast<float4*>(O + (tx + TX * j) * kLdOp<TX> + f0) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
}

// acc[i][c] (+)= sum over the NC streamed rows of O[row][f0 + 2 i, + 1] G[row][column c of this thread]; the thread's
// columns are 4 tx .. 4 tx + 3 of every 4 TX
template <int D, int TX, int NC>
__device__ __forceinline__ void accumulate(const float* O, const float* G, int f0, int tx, uint64_t (&acc)[R / 2][D / TX]) {
#pragma unroll 4
  for (int row = 0; row < NC; ++row) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(O + row * kLdOp<TX> + f0);
    const uint64_t a[R / 2] = {v.x, v.y};
#pragma unroll
    for (int h = 0; h < D / (4 * TX); ++h) {
      const float4 g = *reinterpret_cast<const float4*>(G + row * kLd<D> + h * 4 * TX + tx * 4);
      const uint64_t gx = pack2(g.x, g.x), gy = pack2(g.y, g.y), gz = pack2(g.z, g.z), gw = pack2(g.w, g.w);
#pragma unroll
      for (int i = 0; i < R / 2; ++i) {
        acc[i][4 * h] = fma2(a[i], gx, acc[i][4 * h]);
        acc[i][4 * h + 1] = fma2(a[i], gy, acc[i][4 * h + 1]);
        acc[i][4 * h + 2] = fma2(a[i], gz, acc[i][4 * h + 2]);
        acc[i][4 * h + 3] = fma2(a[i], gw, acc[i][4 * h + 3]);
      }
    }
  }
}

// Writes the thread's rows of an accumulator, scaled per row, where row < n_rows.
template <int D, int TX>
__device__ __forceinline__ void store_rows(float* base, int64_t stride, int row0, int f0, int tx, int n_rows,
                                           const uint64_t (&acc)[R / 2][D / TX], const float (&mul)[R]) {
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = row0 + f0 + i;
    if (row >= n_rows) continue;
#pragma unroll
    for (int h = 0; h < D / (4 * TX); ++h) {
      float4 v;
      float* o = &v.x;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 t = unpack2(acc[i / 2][4 * h + c]);
        o[c] = ((i & 1) ? t.y : t.x) * mul[i];
      }
      *reinterpret_cast<float4*>(base + row * stride + h * 4 * TX + tx * 4) = v;
    }
  }
}

template <int D, int TX, int NC> struct Cfg {
  static constexpr int kRows = kThreads / TX * R;
  static constexpr int kStages = TX == 16 ? 2 : 1;     // buffers of each streamed operand
  static constexpr int kOps = TX == 16 ? 2 : 1;        // (dK, dV) P and dS in buffers of their own
  static constexpr int kFixed = kRows * kLd<D>, kStream = NC * kLd<D>, kOp = NC * kLdOp<TX>;   // floats
  static constexpr int kFwdBytes = 4 * (kFixed + 2 * kStages * kStream + kOp);
  static constexpr int kDqBytes = 4 * (2 * kFixed + 2 * kStages * kStream + kOp);
  static constexpr int kDkvBytes = 4 * (2 * kFixed + 2 * kStages * kStream + kOps * kOp + 2 * NC);
};

// ------------------------------------------------------------------------------------------------ forward --

template <int D, int TX, int NC>
__global__ void __launch_bounds__(kThreads) fp32_fwd_kernel(const Problem p, const int n_blk) {
  using C = Cfg<D, TX, NC>;
  constexpr int J = NC / TX;
  extern __shared__ __align__(16) float smem[];
  constexpr int ST = C::kStages;
  float *Qs = smem, *K0 = Qs + C::kFixed, *V0 = K0 + ST * C::kStream, *Op = V0 + ST * C::kStream;
  pdl_wait();
  pdl_launch_dependents();
  // latest row blocks (most keys under a causal mask) first
  const int bh = blockIdx.x % (p.Hq * p.B);
  const int h = bh % p.Hq, b = bh / p.Hq, hk = h / p.group;
  const int row0 = (n_blk - 1 - static_cast<int>(blockIdx.x / (p.Hq * p.B))) * C::kRows;
  const int tx = threadIdx.x % TX, f0 = threadIdx.x / TX * R;
  const int n_keys = valid_keys(p, b);
  int64_t end = n_keys;
  if (p.causal) {
    const int64_t lim = static_cast<int64_t>((row0 + C::kRows < p.L ? row0 + C::kRows : p.L) - 1) + p.causal_shift + 1;
    end = lim < end ? lim : end;
  }
  const int k_end = end < 0 ? 0 : static_cast<int>(end);
  const float* q = reinterpret_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1] + row0 * p.qs[2];
  const float* k = reinterpret_cast<const float*>(p.k) + b * p.ks[0] + hk * p.ks[1];
  const float* v = reinterpret_cast<const float*>(p.v) + b * p.vs[0] + hk * p.vs[1];

  uint64_t acc[R / 2][D / TX];
  float m[R], l[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m[i] = kMaskedOut;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < D / TX; ++c) acc[i / 2][c] = 0ull;
  }
  if (k_end > 0) {
    load_tile<D, C::kRows>(Qs, q, p.qs[2], p.L - row0);
    load_tile<D, NC>(K0, k, p.ks[2], k_end);
    if (ST == 2) load_tile<D, NC>(V0, v, p.vs[2], k_end);
    copy_commit();
  }
  for (int j0 = 0; j0 < k_end; j0 += NC) {
    const int stage = ST == 2 ? (j0 / NC) & 1 : 0;
    float *Ks = K0 + stage * C::kStream, *Vs = V0 + stage * C::kStream;
    const int j1 = j0 + NC;
    copy_wait<0>();
    __syncthreads();   // K (two stages: and V) is here; the last tile's V and operand have been read
    if (ST == 1) {
      load_tile<D, NC>(Vs, v + j0 * p.vs[2], p.vs[2], k_end - j0);
    } else if (j1 < k_end) {
      load_tile<D, NC>(K0 + (stage ^ 1) * C::kStream, k + j1 * p.ks[2], p.ks[2], k_end - j1);
      load_tile<D, NC>(V0 + (stage ^ 1) * C::kStream, v + j1 * p.vs[2], p.vs[2], k_end - j1);
    }
    copy_commit();
    float s[R][J], al[R];
    score_patch<D, TX, J>(Qs, Ks, f0, tx, s);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int64_t lim64 = p.causal ? static_cast<int64_t>(row0 + f0 + i) + p.causal_shift + 1 : n_keys;
      const int lim = lim64 < n_keys ? static_cast<int>(lim64 < 0 ? 0 : lim64) : n_keys;
      float mx = kMaskedOut;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        s[i][j] = j0 + tx + TX * j < lim ? s[i][j] * p.scale : kMaskedOut;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int o = TX / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m[i], mx);
      const float m_safe = m_new == kMaskedOut ? 0.f : m_new;
      const float alpha = m[i] == kMaskedOut ? 0.f : expf(m[i] - m_safe);
      m[i] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        s[i][j] = expf(s[i][j] - m_safe);
        sum += s[i][j];
      }
      l[i] = fmaf(l[i], alpha, sum);   // this thread's columns; the row's other threads are added at the end
      al[i] = alpha;
    }
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
      const uint64_t a2 = pack2(al[2 * i], al[2 * i + 1]);
#pragma unroll
      for (int c = 0; c < D / TX; ++c) acc[i][c] = mul2(acc[i][c], a2);
    }
    store_transposed<TX, J>(Op, f0, tx, s);
    if (ST == 1) copy_wait<0>();
    __syncthreads();   // V and the operand are here; K has been read
    if (ST == 1) {
      if (j1 < k_end) load_tile<D, NC>(Ks, k + j1 * p.ks[2], p.ks[2], k_end - j1);
      copy_commit();
    }
    accumulate<D, TX, NC>(Op, Vs, f0, tx, acc);
  }
  float inv[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
#pragma unroll
    for (int o = TX / 2; o > 0; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
    inv[i] = l[i] > 0.f ? 1.f / l[i] : 0.f;
    const int row = row0 + f0 + i;
    if (p.lse != nullptr && tx == 0 && row < p.L &&
        dbg_bhrc(p.status, DBG_FP32 * 100 + 1, b, p.B, h, p.Hq, row, p.L, 0, 0, 1))
      p.lse[b * p.ls[0] + h * p.ls[1] + row * p.ls[2]] = m[i] == kMaskedOut ? -CUDART_INF_F : m[i] + logf(l[i]);
  }
  if (dbg_bhrc(p.status, DBG_FP32 * 100 + 2, b, p.B, h, p.Hq, row0, p.L, 0, D, p.Dv))
    store_rows<D, TX>(reinterpret_cast<float*>(p.out) + b * p.os[0] + h * p.os[1], p.os[2], row0, f0, tx, p.L, acc, inv);
}

// ----------------------------------------------------------------------------------------------- backward --

template <int D, int TX, int NC>
__global__ void __launch_bounds__(kThreads) fp32_bwd_dq_kernel(const BwdProblem bp, const int n_blk) {
  using C = Cfg<D, TX, NC>;
  constexpr int J = NC / TX;
  const Problem& p = bp.f;
  extern __shared__ __align__(16) float smem[];
  constexpr int ST = C::kStages;
  float *Qs = smem, *Gs = Qs + C::kFixed, *K0 = Gs + C::kFixed, *V0 = K0 + ST * C::kStream, *Op = V0 + ST * C::kStream;
  const int bh = blockIdx.x % (p.Hq * p.B);
  const int h = bh % p.Hq, b = bh / p.Hq, hk = h / p.group;
  const int row0 = (n_blk - 1 - static_cast<int>(blockIdx.x / (p.Hq * p.B))) * C::kRows;
  const int tx = threadIdx.x % TX, f0 = threadIdx.x / TX * R;
  const int n_keys = valid_keys(p, b);
  int64_t end = n_keys;
  if (p.causal) {
    const int64_t lim = static_cast<int64_t>((row0 + C::kRows < p.L ? row0 + C::kRows : p.L) - 1) + p.causal_shift + 1;
    end = lim < end ? lim : end;
  }
  const int k_end = end < 0 ? 0 : static_cast<int>(end);
  const float* k = reinterpret_cast<const float*>(p.k) + b * p.ks[0] + hk * p.ks[1];
  const float* v = reinterpret_cast<const float*>(p.v) + b * p.vs[0] + hk * p.vs[1];
  const float* go = reinterpret_cast<const float*>(bp.dout) + b * bp.dos[0] + h * bp.dos[1];
  const float* o = reinterpret_cast<const float*>(p.out) + b * p.os[0] + h * p.os[1];

  uint64_t acc[R / 2][D / TX];
#pragma unroll
  for (int i = 0; i < R / 2; ++i)
#pragma unroll
    for (int c = 0; c < D / TX; ++c) acc[i][c] = 0ull;
  float lse[R], delta[R];
  if (k_end > 0) {
    load_tile<D, C::kRows>(Qs, reinterpret_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1] + row0 * p.qs[2], p.qs[2], p.L - row0);
    load_tile<D, C::kRows>(Gs, go + row0 * bp.dos[2], bp.dos[2], p.L - row0);
    load_tile<D, NC>(K0, k, p.ks[2], k_end);
    load_tile<D, NC>(V0, v, p.vs[2], k_end);
    copy_commit();
    // delta = sum(dO * out) of the thread's rows, TX threads a row
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = row0 + f0 + i;
      float d = 0.f;
      lse[i] = CUDART_INF_F;
      if (row < p.L) {
        const float l = p.lse[b * p.ls[0] + h * p.ls[1] + row * p.ls[2]];
        // -inf: no key seen, or nothing but NaN.  With +inf finite scores give 0 and NaN stays NaN, as it is in delta
        lse[i] = l == -CUDART_INF_F ? CUDART_INF_F : l;
#pragma unroll
        for (int c = 0; c < D / (4 * TX); ++c) {
          const float4 x = *reinterpret_cast<const float4*>(go + row * bp.dos[2] + c * 4 * TX + tx * 4);
          const float4 y = *reinterpret_cast<const float4*>(o + row * p.os[2] + c * 4 * TX + tx * 4);
          d = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, d))));
        }
      }
#pragma unroll
      for (int s = TX / 2; s > 0; s >>= 1) d += __shfl_xor_sync(0xffffffffu, d, s);
      delta[i] = d;
    }
  }
  for (int j0 = 0; j0 < k_end; j0 += NC) {
    const int stage = ST == 2 ? (j0 / NC) & 1 : 0;
    float *Ks = K0 + stage * C::kStream, *Vs = V0 + stage * C::kStream;
    const int j1 = j0 + NC;
    const bool more = j1 < k_end;
    copy_wait<0>();
    __syncthreads();   // K and V are here; (two stages) the last tile's K and operand have been read
    if (ST == 2 && more) {
      load_tile<D, NC>(K0 + (stage ^ 1) * C::kStream, k + j1 * p.ks[2], p.ks[2], k_end - j1);
      load_tile<D, NC>(V0 + (stage ^ 1) * C::kStream, v + j1 * p.vs[2], p.vs[2], k_end - j1);
    }
    if (ST == 2) copy_commit();
    float s[R][J], dp[R][J];
    score_patch<D, TX, J>(Qs, Ks, f0, tx, s);
    score_patch<D, TX, J>(Gs, Vs, f0, tx, dp);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int64_t lim64 = p.causal ? static_cast<int64_t>(row0 + f0 + i) + p.causal_shift + 1 : n_keys;
      const int lim = lim64 < n_keys ? static_cast<int>(lim64 < 0 ? 0 : lim64) : n_keys;
#pragma unroll
      for (int j = 0; j < J; ++j)
        s[i][j] = j0 + tx + TX * j < lim ? expf(s[i][j] * p.scale - lse[i]) * (dp[i][j] - delta[i]) : 0.f;
    }
    store_transposed<TX, J>(Op, f0, tx, s);
    __syncthreads();   // the operand is here; V has been read
    if (ST == 1 && more) load_tile<D, NC>(Vs, v + j1 * p.vs[2], p.vs[2], k_end - j1);
    accumulate<D, TX, NC>(Op, Ks, f0, tx, acc);
    if (ST == 1) {
      __syncthreads();   // K and the operand have been read
      if (more) load_tile<D, NC>(Ks, k + j1 * p.ks[2], p.ks[2], k_end - j1);
      copy_commit();
    }
  }
  float mul[R];
#pragma unroll
  for (int i = 0; i < R; ++i) mul[i] = p.scale;
  if (dbg_bhrc(p.status, DBG_FP32 * 100 + 3, b, p.B, h, p.Hq, row0, p.L, 0, D, p.E))
    store_rows<D, TX>(reinterpret_cast<float*>(bp.dq) + b * bp.dqs[0] + h * bp.dqs[1], bp.dqs[2], row0, f0, tx, p.L, acc, mul);
}

template <int D, int TX, int NC>
__global__ void __launch_bounds__(kThreads) fp32_bwd_dkv_kernel(const BwdProblem bp) {
  using C = Cfg<D, TX, NC>;
  constexpr int J = NC / TX;
  constexpr int kPerRow = kThreads / NC;   // threads that share a streamed row's delta
  const Problem& p = bp.f;
  extern __shared__ __align__(16) float smem[];
  constexpr int ST = C::kStages;
  float *Ks = smem, *Vs = Ks + C::kFixed, *Q0 = Vs + C::kFixed, *G0 = Q0 + ST * C::kStream, *Op = G0 + ST * C::kStream;
  float *st_lse = Op + C::kOps * C::kOp, *st_delta = st_lse + NC;
  // earliest key blocks (seen by the most rows under a causal mask) first
  const int bh = blockIdx.x % (p.Hkv * p.B);
  const int hk = bh % p.Hkv, b = bh / p.Hkv;
  const int key0 = static_cast<int>(blockIdx.x / (p.Hkv * p.B)) * C::kRows;
  const int tx = threadIdx.x % TX, f0 = threadIdx.x / TX * R;
  const int n_keys = valid_keys(p, b);
  int first = 0;   // first streamed row that sees a key of this block
  if (p.causal) {
    const int64_t f = static_cast<int64_t>(key0) - p.causal_shift;
    first = f <= 0 ? 0 : (f >= p.L ? p.L : static_cast<int>(f) / NC * NC);
  }
  const int per_head = (key0 < n_keys && first < p.L) ? (p.L - first + NC - 1) / NC : 0;
  const int n_tiles = per_head * p.group;

  uint64_t acc_k[R / 2][D / TX], acc_v[R / 2][D / TX];
#pragma unroll
  for (int i = 0; i < R / 2; ++i)
#pragma unroll
    for (int c = 0; c < D / TX; ++c) acc_k[i][c] = acc_v[i][c] = 0ull;
  auto load_q = [&](int t) {
    float* Qs = Q0 + (ST == 2 ? t & 1 : 0) * C::kStream;
    const int h = hk * p.group + t / per_head, row = first + t % per_head * NC;
    load_tile<D, NC>(Qs, reinterpret_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1] + row * p.qs[2], p.qs[2], p.L - row);
  };
  auto load_go = [&](int t) {
    float* Gs = G0 + (ST == 2 ? t & 1 : 0) * C::kStream;
    const int h = hk * p.group + t / per_head, row = first + t % per_head * NC;
    load_tile<D, NC>(Gs, reinterpret_cast<const float*>(bp.dout) + b * bp.dos[0] + h * bp.dos[1] + row * bp.dos[2], bp.dos[2], p.L - row);
  };
  if (n_tiles > 0) {
    load_tile<D, C::kRows>(Ks, reinterpret_cast<const float*>(p.k) + b * p.ks[0] + hk * p.ks[1] + key0 * p.ks[2], p.ks[2], n_keys - key0);
    load_tile<D, C::kRows>(Vs, reinterpret_cast<const float*>(p.v) + b * p.vs[0] + hk * p.vs[1] + key0 * p.vs[2], p.vs[2], n_keys - key0);
    load_q(0);
    load_go(0);
    copy_commit();
  }
  // log-sum-exp and delta = sum(dO * out) of the streamed rows: `out` is fetched one tile ahead (kPerRow threads a row),
  // the sum is taken when dO has arrived
  constexpr int kOuts = D / 4 / kPerRow;
  const int sr = threadIdx.x / kPerRow, sub = threadIdx.x % kPerRow;
  float4 o_next[kOuts];
  float lse_next = -CUDART_INF_F;
  auto fetch_out = [&](int t) {
    const int h = hk * p.group + t / per_head, row = first + t % per_head * NC + sr;
    lse_next = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < kOuts; ++i) o_next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < p.L) {
      lse_next = p.lse[b * p.ls[0] + h * p.ls[1] + row * p.ls[2]];
      const float* o = reinterpret_cast<const float*>(p.out) + b * p.os[0] + h * p.os[1] + row * p.os[2];
#pragma unroll
      for (int i = 0; i < kOuts; ++i) o_next[i] = *reinterpret_cast<const float4*>(o + (sub + i * kPerRow) * 4);
    }
  };
  if (n_tiles > 0) fetch_out(0);
  for (int t = 0; t < n_tiles; ++t) {
    const int row0 = first + t % per_head * NC;
    float *Qs = Q0 + (ST == 2 ? t & 1 : 0) * C::kStream, *Gs = G0 + (ST == 2 ? t & 1 : 0) * C::kStream;
    const bool more = t + 1 < n_tiles;
    copy_wait<0>();
    __syncthreads();   // Q and dO are here; the last tile's operands and statistics have been read
    if (ST == 2) {
      if (more) {
        load_q(t + 1);
        load_go(t + 1);
      }
      copy_commit();
    }
    {
      float d = 0.f;
#pragma unroll
      for (int i = 0; i < kOuts; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(Gs + sr * kLd<D> + (sub + i * kPerRow) * 4);
        const float4 y = o_next[i];
        d = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, d))));
      }
#pragma unroll
      for (int s = kPerRow / 2; s > 0; s >>= 1) d += __shfl_xor_sync(0xffffffffu, d, s);
      if (sub == 0) {
        st_delta[sr] = d;
        st_lse[sr] = lse_next;
      }
    }
    if (more) fetch_out(t + 1);
    float s[R][J], dp[R][J];
    score_patch<D, TX, J>(Ks, Qs, f0, tx, s);
    score_patch<D, TX, J>(Vs, Gs, f0, tx, dp);
    __syncthreads();   // the statistics are here
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const float lse = st_lse[tx + TX * j], delta = st_delta[tx + TX * j];
      const int row = row0 + tx + TX * j;
      const int64_t lim64 = p.causal ? static_cast<int64_t>(row) + p.causal_shift + 1 : n_keys;
      const int lim = lse == -CUDART_INF_F ? 0 : (lim64 < n_keys ? static_cast<int>(lim64 < 0 ? 0 : lim64) : n_keys);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        s[i][j] = key0 + f0 + i < lim ? expf(s[i][j] * p.scale - lse) : 0.f;
        dp[i][j] = s[i][j] * (dp[i][j] - delta);
      }
    }
    store_transposed<TX, J>(Op, f0, tx, s);
    if (C::kOps == 2) store_transposed<TX, J>(Op + C::kOp, f0, tx, dp);
    __syncthreads();   // P (and dS) are here
    accumulate<D, TX, NC>(Op, Gs, f0, tx, acc_v);
    if (C::kOps == 1) {
      __syncthreads();   // P and dO have been read
      store_transposed<TX, J>(Op, f0, tx, dp);
      if (ST == 1 && more) load_go(t + 1);
      __syncthreads();   // dS is here
    }
    accumulate<D, TX, NC>(Op + (C::kOps - 1) * C::kOp, Qs, f0, tx, acc_k);
    if (ST == 1) {
      __syncthreads();   // dS and Q have been read
      if (more) load_q(t + 1);
      copy_commit();
    }
  }
  float mul[R], one[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    mul[i] = p.scale;
    one[i] = 1.f;
  }
  if (!dbg_bhrc(p.status, DBG_FP32 * 100 + 4, b, p.B, hk, p.Hkv, key0, p.S, 0, D, p.E)) return;
  store_rows<D, TX>(reinterpret_cast<float*>(bp.dk) + b * bp.dks[0] + hk * bp.dks[1], bp.dks[2], key0, f0, tx, p.S, acc_k, mul);
  store_rows<D, TX>(reinterpret_cast<float*>(bp.dv) + b * bp.dvs[0] + hk * bp.dvs[1], bp.dvs[2], key0, f0, tx, p.S, acc_v, one);
}

// ----------------------------------------------------------------------------------------------- host side --

bool rows_ok(const void* base, const int64_t* s, int rows, int heads, int batch) {
  if (reinterpret_cast<uintptr_t>(base) % 16 || s[3] != 1) return false;
  const int n[3] = {batch, heads, rows};
  for (int i = 0; i < 3; ++i)
    if (n[i] > 1 && s[i] % 4 != 0) return false;
  return true;
}

bool common_ok(const Problem& p) {
  return p.E == p.Dv && (p.E == 64 || p.E == 128) && p.bias == nullptr && p.L >= 1 && p.S >= 1 && p.block_table == nullptr &&
         p.k_new == nullptr && p.acc_mode == 0 && rows_ok(p.q, p.qs, p.L, p.Hq, p.B) && rows_ok(p.k, p.ks, p.S, p.Hkv, p.B) &&
         rows_ok(p.v, p.vs, p.S, p.Hkv, p.B) && rows_ok(p.out, p.os, p.L, p.Hq, p.B) &&
         static_cast<int64_t>((p.L > p.S ? p.L : p.S) / 32 + 1) * p.Hq * p.B < 0x7fffffffLL;
}

// 64 fixed rows a CTA, or 32 where that gives fewer than two CTAs to an SM.
int rows_per_cta(int64_t rows, int64_t heads) { return (rows + 63) / 64 * heads < 2 * 148 ? 32 : 64; }

// The forward at head dimension 128 measured faster with 32 rows and double buffers everywhere (1 x 32/8 x 1024: 294
// against 347 us).
int fwd_rows(const Problem& p) { return p.E == 128 ? 32 : rows_per_cta(p.L, static_cast<int64_t>(p.Hq) * p.B); }

template <typename K, typename... Args>
int launch(K kern, int64_t grid, int smem, cudaStream_t stream, int kernel_id, Args... args) {
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    cudaGetLastError();
    return B200_SDPA_ERR_CUDA;
  }
  if (kernel_id == KID_GENERIC) {
    if (!launch_pdl(kern, dim3(static_cast<unsigned>(grid)), kThreads, smem, stream, args...)) return B200_SDPA_ERR_CUDA;
  } else {
    kern<<<static_cast<unsigned>(grid), kThreads, smem, stream>>>(args...);
    if (cudaGetLastError() != cudaSuccess) return B200_SDPA_ERR_CUDA;
  }
  count_launch(kernel_id);
  return B200_SDPA_OK;
}

template <int D, int TX, int NC> int launch_fwd(const Problem& p, cudaStream_t stream) {
  const int n = (p.L + Cfg<D, TX, NC>::kRows - 1) / Cfg<D, TX, NC>::kRows;
  return launch(fp32_fwd_kernel<D, TX, NC>, static_cast<int64_t>(n) * p.Hq * p.B, Cfg<D, TX, NC>::kFwdBytes, stream, KID_GENERIC, p, n);
}
template <int D, int TX, int NC> int launch_dq(const BwdProblem& bp, cudaStream_t stream) {
  const Problem& p = bp.f;
  const int n = (p.L + Cfg<D, TX, NC>::kRows - 1) / Cfg<D, TX, NC>::kRows;
  return launch(fp32_bwd_dq_kernel<D, TX, NC>, static_cast<int64_t>(n) * p.Hq * p.B, Cfg<D, TX, NC>::kDqBytes, stream, KID_BWD_DQ, bp, n);
}
template <int D, int TX, int NC> int launch_dkv(const BwdProblem& bp, cudaStream_t stream) {
  const Problem& p = bp.f;
  const int n = (p.S + Cfg<D, TX, NC>::kRows - 1) / Cfg<D, TX, NC>::kRows;
  return launch(fp32_bwd_dkv_kernel<D, TX, NC>, static_cast<int64_t>(n) * p.Hkv * p.B, Cfg<D, TX, NC>::kDkvBytes, stream, KID_BWD_DKV, bp);
}

}  // namespace

bool fp32_fwd_eligible(const Problem& p, int dtype) { return dtype == B200_SDPA_F32 && common_ok(p); }

bool fp32_bwd_eligible(const BwdProblem& bp, int dtype) {
  const Problem& p = bp.f;
  return dtype == B200_SDPA_F32 && bp.dbias == nullptr && common_ok(p) && rows_ok(bp.dout, bp.dos, p.L, p.Hq, p.B) &&
         rows_ok(bp.dq, bp.dqs, p.L, p.Hq, p.B) && rows_ok(bp.dk, bp.dks, p.S, p.Hkv, p.B) && rows_ok(bp.dv, bp.dvs, p.S, p.Hkv, p.B);
}

void plan_fp32_fwd(const Problem& p, B200SdpaPlan* plan) {
  const int rows = fwd_rows(p);
  plan->path = B200_SDPA_PATH_GENERIC;
  plan->block_m = rows;
  plan->block_n = p.E == 64 ? 64 : 32;
  plan->grid_x = static_cast<int32_t>(static_cast<int64_t>((p.L + rows - 1) / rows) * p.Hq * p.B);
  plan->grid_y = plan->grid_z = 1;
  plan->threads = kThreads;
  plan->smem_bytes = p.E == 64 ? (rows == 32 ? Cfg<64, 16, 64>::kFwdBytes : Cfg<64, 8, 64>::kFwdBytes) : Cfg<128, 16, 32>::kFwdBytes;
  plan->kv_splits = 1;
  plan->launches = 1;
  plan->workspace_bytes = 0;
}

void plan_fp32_bwd(const BwdProblem& bp, B200SdpaPlan* plan) {
  const Problem& p = bp.f;
  const int rq = rows_per_cta(p.L, static_cast<int64_t>(p.Hq) * p.B), rk = rows_per_cta(p.S, static_cast<int64_t>(p.Hkv) * p.B);
  plan->path = B200_SDPA_PATH_GENERIC;
  plan->block_m = rq;
  plan->block_n = p.E == 64 ? 64 : 32;
  plan->grid_x = static_cast<int32_t>(static_cast<int64_t>((p.L + rq - 1) / rq) * p.Hq * p.B);
  plan->grid_y = static_cast<int32_t>(static_cast<int64_t>((p.S + rk - 1) / rk) * p.Hkv * p.B);
  plan->grid_z = 1;
  plan->threads = kThreads;
  plan->smem_bytes = p.E == 64 ? (rk == 32 ? Cfg<64, 16, 64>::kDkvBytes : Cfg<64, 8, 64>::kDkvBytes)
                               : (rk == 32 ? Cfg<128, 16, 32>::kDkvBytes : Cfg<128, 8, 32>::kDkvBytes);
  plan->kv_splits = 1;
  plan->launches = 2;
  plan->workspace_bytes = 0;
}

int launch_fp32_fwd(const Problem& p, cudaStream_t stream) {
  const bool small = fwd_rows(p) == 32;
  if (p.E == 64) return small ? launch_fwd<64, 16, 64>(p, stream) : launch_fwd<64, 8, 64>(p, stream);
  return launch_fwd<128, 16, 32>(p, stream);
}

int launch_fp32_bwd(const BwdProblem& bp, cudaStream_t stream) {
  const Problem& p = bp.f;
  const bool small_q = rows_per_cta(p.L, static_cast<int64_t>(p.Hq) * p.B) == 32;
  const bool small_k = rows_per_cta(p.S, static_cast<int64_t>(p.Hkv) * p.B) == 32;
  int rc;
  if (p.E == 64) rc = small_q ? launch_dq<64, 16, 64>(bp, stream) : launch_dq<64, 8, 64>(bp, stream);
  else rc = small_q ? launch_dq<128, 16, 32>(bp, stream) : launch_dq<128, 8, 32>(bp, stream);
  if (rc != B200_SDPA_OK) return rc;
  if (p.E == 64) return small_k ? launch_dkv<64, 16, 64>(bp, stream) : launch_dkv<64, 8, 64>(bp, stream);
  return small_k ? launch_dkv<128, 16, 32>(bp, stream) : launch_dkv<128, 8, 32>(bp, stream);
}

}  // namespace b200

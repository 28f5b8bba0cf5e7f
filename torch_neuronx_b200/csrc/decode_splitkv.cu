// Split-KV flash decoding (one query row per sequence) for sm_100a.
//
// The key/value cache is the only large operand, so the kernel is organised
// around reading it exactly once at full HBM rate:
//   * grid = (key split, kv head, batch): every CTA streams one contiguous
//     chunk of one kv head's cache and serves ALL query heads of that group,
//     so grouped-query heads never re-read K/V;
//   * every lane issues 128-bit loads; a warp-wide load covers whole cache rows
//     back to back (fully coalesced), several rows in flight per lane;
//   * per-lane online softmax state in the exp2 domain; lanes, warps and finally
//     splits are merged with the usual (max, sum, weighted accumulator) rule --
//     across splits by a second small kernel that reads the fp32 partials.
// Sequences are ragged: split s of batch b covers keys [s*chunk, min((s+1)*chunk,
// kv_lens[b])) and CTAs past the end exit at once.
//
// Arithmetic restates torch_neuronx/_sdpa_math.py:79-95 for a single query row
// with a key-length mask; dead rows (no visible key) give out = 0, lse = -inf.
#include "common.cuh"
#include "debug.cuh"

#include <cstdlib>
#include <mutex>

namespace b200 {

namespace {

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kUnroll = 4;  // cache rows in flight per lane (x2 for K and V)
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

template <typename T> struct Vec;
template <> struct Vec<float> { static constexpr int N = 4; };
template <> struct Vec<__half> { static constexpr int N = 8; };
template <> struct Vec<__nv_bfloat16> { static constexpr int N = 8; };

template <typename T>
__device__ __forceinline__ void unpack(const uint4& raw, float (&f)[Vec<T>::N]);
template <>
__device__ __forceinline__ void unpack<float>(const uint4& raw, float (&f)[4]) {
  f[0] = __uint_as_float(raw.x);
  f[1] = __uint_as_float(raw.y);
  f[2] = __uint_as_float(raw.z);
  f[3] = __uint_as_float(raw.w);
}
template <>
__device__ __forceinline__ void unpack<__nv_bfloat16>(const uint4& raw, float (&f)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
template <>
__device__ __forceinline__ void unpack<__half>(const uint4& raw, float (&f)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ uint4 ld_stream_16B(const void* ptr) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(ptr));
  return r;
}

// Workspace layout (fp32): part_o[B][Hq][nsplit][D] then part_ml[B][Hq][nsplit][2]
// with ml = (running max in the exp2 domain, running sum).
template <typename T, int D, int G>
__global__ void __launch_bounds__(kThreads) decode_partial_kernel(const Problem p, const int chunk, const int nsplit,
                                                                   float* __restrict__ part_o,
                                                                   float* __restrict__ part_ml) {
  constexpr int V = Vec<T>::N;
  constexpr int LPR = D / V;       // lanes that share one cache row
  constexpr int RPW = 32 / LPR;    // rows covered by one warp-wide load
  constexpr int NSTATE = kWarps * RPW;
  static_assert(LPR <= 32 && LPR >= 1, "head dim not supported by this mapping");
  __shared__ float sm_acc[NSTATE][G][D];
  __shared__ float sm_ml[NSTATE][G][2];

  const int split = blockIdx.z;          // slowest: the launch ends on the last (short or empty) chunks
  const int hk = blockIdx.x % p.Hkv;
  const int gsub = blockIdx.x / p.Hkv;   // sub-block of the query-head group when group > G
  const int b = blockIdx.y;
  const int n_keys = valid_keys(p, b);
  const int s0 = split * chunk;
  if (s0 >= n_keys && !(split == 0)) return;  // split 0 still writes an empty partial
  const int s1 = (s0 + chunk < n_keys) ? s0 + chunk : n_keys;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPR, col = (lane % LPR) * V;
  const int h0 = hk * p.group + gsub * G;                      // first query head served here
  const int n_heads = (p.group - gsub * G) < G ? (p.group - gsub * G) : G;

  const T* __restrict__ q = reinterpret_cast<const T*>(p.q);
  const char* __restrict__ kbase = reinterpret_cast<const char*>(p.k) +
                                   (b * p.ks[0] + hk * p.ks[1] + col) * static_cast<int64_t>(sizeof(T));
  const char* __restrict__ vbase = reinterpret_cast<const char*>(p.v) +
                                   (b * p.vs[0] + hk * p.vs[1] + col) * static_cast<int64_t>(sizeof(T));
  const int64_t k_row_bytes = p.ks[2] * static_cast<int64_t>(sizeof(T));
  const int64_t v_row_bytes = p.vs[2] * static_cast<int64_t>(sizeof(T));

  const float qscale = p.scale * kLog2e;
  float qr[G][V];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int e = 0; e < V; ++e)
      qr[g][e] = g < n_heads ? to_f32<T>(q[b * p.qs[0] + (h0 + g) * p.qs[1] + (col + e) * p.qs[3]]) * qscale : 0.f;

  float m[G], l[G], acc[G][V];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -CUDART_INF_F;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < V; ++e) acc[g][e] = 0.f;
  }

  constexpr int kStep = RPW * kUnroll;  // rows per warp iteration
  for (int base = s0 + warp * kStep; base < s1; base += kWarps * kStep) {
    uint4 kraw[kUnroll], vraw[kUnroll];
    bool ok[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int row = base + u * RPW + sub;
      ok[u] = row < s1;
      const int srow = ok[u] ? row : s0;  // always a readable row of this sequence
      kraw[u] = ld_stream_16B(kbase + srow * k_row_bytes);
      vraw[u] = ld_stream_16B(vbase + srow * v_row_bytes);
    }
    float s[kUnroll][G];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      float kf[V];
      unpack<T>(kraw[u], kf);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float d = 0.f;
#pragma unroll
        for (int e = 0; e < V; ++e) d = fmaf(qr[g][e], kf[e], d);
#pragma unroll
        for (int off = LPR / 2; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
        s[u][g] = ok[u] ? d : -CUDART_INF_F;
      }
    }
    float pw[kUnroll][G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float mx = m[g];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) mx = fmaxf(mx, s[u][g]);
      const float ms = (mx == -CUDART_INF_F) ? 0.f : mx;
      const float alpha = exp2f(m[g] - ms);  // m = -inf -> 0
      m[g] = mx;
      float sum = 0.f;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        pw[u][g] = exp2f(s[u][g] - ms);
        sum += pw[u][g];
      }
      l[g] = l[g] * alpha + sum;
#pragma unroll
      for (int e = 0; e < V; ++e) acc[g][e] *= alpha;
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      float vf[V];
      unpack<T>(vraw[u], vf);
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int e = 0; e < V; ++e) acc[g][e] = fmaf(pw[u][g], vf[e], acc[g][e]);
    }
  }

  // lane states -> shared memory, then one merged partial per query head
  const int st = warp * RPW + sub;
#pragma unroll
  for (int g = 0; g < G; ++g) {
#pragma unroll
    for (int e = 0; e < V; ++e) sm_acc[st][g][col + e] = acc[g][e];
    if ((lane % LPR) == 0) {
      sm_ml[st][g][0] = m[g];
      sm_ml[st][g][1] = l[g];
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += kThreads) {
    const int g = idx / D, d = idx - g * D;
    if (g >= n_heads) continue;
    float mx = -CUDART_INF_F;
#pragma unroll
    for (int s_ = 0; s_ < NSTATE; ++s_) mx = fmaxf(mx, sm_ml[s_][g][0]);
    const float ms = (mx == -CUDART_INF_F) ? 0.f : mx;
    float o = 0.f, lsum = 0.f;
#pragma unroll
    for (int s_ = 0; s_ < NSTATE; ++s_) {
      const float w = exp2f(sm_ml[s_][g][0] - ms);
      o = fmaf(sm_acc[s_][g][d], w, o);
      lsum = fmaf(sm_ml[s_][g][1], w, lsum);
    }
    const int64_t slot = (static_cast<int64_t>(b) * p.Hq + (h0 + g)) * nsplit + split;
    if (!dbg_range(p.status, DBG_DECODE_SIMT * 100 + 1, slot, 1, static_cast<int64_t>(p.B) * p.Hq * nsplit) ||
        !dbg_range(p.status, DBG_DECODE_SIMT * 100 + 2, h0 + g, 1, p.Hq))
      continue;
    part_o[slot * D + d] = o;
    if (d == 0) {
      part_ml[slot * 2] = mx;
      part_ml[slot * 2 + 1] = lsum;
    }
  }
}

// Merge of the partials: one CTA of four warps per (batch, query head).  Every warp takes every fourth split (the
// (max, sum) pairs of all splits are read once, 32 at a time), then the four states meet in shared memory.  Bound by
// latency: two dependent rounds of loads, whatever the number of splits up to 128.  WIDE: the scratch starts on 16 bytes
// and is read in vectors; a caller's scratch need not (the partial kernels store single floats).
constexpr int kCombineWarps = 4;

template <typename T, int D, bool WIDE>
__global__ void __launch_bounds__(kCombineWarps * 32) decode_combine_kernel(const Problem p, const int chunk, const int nsplit,
                                                                            const float* __restrict__ part_o,
                                                                            const float* __restrict__ part_ml) {
  constexpr int C = D / 32;   // columns per lane
  __shared__ float sm_o[kCombineWarps][D];
  __shared__ float sm_l[kCombineWarps];
  const int h = blockIdx.x % p.Hq;
  const int b = blockIdx.x / p.Hq;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // launched as a programmatic dependent of the partial kernel: nothing may be read before it has completed
  pdl_wait();
  pdl_launch_dependents();
  const int n_keys = valid_keys(p, b);
  if (p.lens_out != nullptr && h == 0 && threadIdx.x == 0) p.lens_out[b] = n_keys;   // lengths after the append
  int used = (n_keys + chunk - 1) / chunk;
  used = used < 1 ? 1 : (used > nsplit ? nsplit : used);
  const int64_t slot0 = (static_cast<int64_t>(b) * p.Hq + h) * nsplit;
  if (!dbg_range(p.status, DBG_DECODE_SIMT * 100 + 3, slot0, used, static_cast<int64_t>(p.B) * p.Hq * nsplit) ||
      !dbg_bhrc(p.status, DBG_DECODE_SIMT * 100 + 4, b, p.B, h, p.Hq, 0, 1, lane * C, C, p.Dv))
    return;
  float mx = -CUDART_INF_F;
  for (int s = lane; s < used; s += 32) mx = fmaxf(mx, part_ml[(slot0 + s) * 2]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float ms = (mx == -CUDART_INF_F) ? 0.f : mx;
  float acc[C], lsum = 0.f;
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = 0.f;
#pragma unroll 4
  for (int s = warp; s < used; s += kCombineWarps) {
    const float* pair = part_ml + (slot0 + s) * 2;
    const float* src = part_o + (slot0 + s) * D + lane * C;
    float2 ml;
    float v[C];
    if constexpr (WIDE) {
      ml = *reinterpret_cast<const float2*>(pair);
      if constexpr (C == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src);
      else *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(src);
    } else {
      ml = make_float2(pair[0], pair[1]);
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = src[c];
    }
    const float w = exp2f(ml.x - ms);
    lsum = fmaf(ml.y, w, lsum);
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = fmaf(v[c], w, acc[c]);
  }
#pragma unroll
  for (int c = 0; c < C; ++c) sm_o[warp][lane * C + c] = acc[c];
  if (lane == 0) sm_l[warp] = lsum;
  __syncthreads();
  float l = 0.f;
#pragma unroll
  for (int w = 0; w < kCombineWarps; ++w) l += sm_l[w];
  const float inv = l > 0.f ? 1.f / l : 0.f;
  for (int d = threadIdx.x; d < D; d += kCombineWarps * 32) {
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < kCombineWarps; ++w) o += sm_o[w][d];
    reinterpret_cast<T*>(p.out)[b * p.os[0] + h * p.os[1] + d * p.os[3]] = from_f32<T>(o * inv);
  }
  if (p.lse != nullptr && threadIdx.x == 0)
    p.lse[b * p.ls[0] + h * p.ls[1]] = (mx == -CUDART_INF_F) ? -CUDART_INF_F : fmaf(mx, kLn2, logf(l));
}

int pick_group(int group) { return group >= 8 ? 8 : group > 2 ? 4 : group; }

constexpr int kMaxChunk = 2048;

// Keys per CTA.  A model of the launch, fitted to measurements (bf16, head dimension 128, 1 to 128 sequences of 512 to
// 32768 keys, within a tenth of the best chunk everywhere): up to `slots` CTAs run at a time; a CTA needs kFixed for its
// start and end and, per block of 64 keys, kBlock alone (the latency of its two-stage ring) and kShared more when all
// slots are taken (its share of the HBM rate).  Short chunks pay kFixed too often, long ones leave SMs without work.
// More CTAs than slots cost, on average, a third of a round for the last, partly filled one -- less when their lengths
// differ.  Lengths are not known here: with key lengths the cost for full caches and twice that for lengths spread
// evenly up to S are added, else full caches are assumed.  A paged cache's block costs more alone (table and address
// arithmetic).  16 sequences of 128..4000 keys, 4096 cached, 32/8 heads: 34.9 us at the 256 keys taken before, 32.3 at
// the 1024 taken now (paged, with append: 41.1 -> 33.5 at 768); one sequence of 30000 keys 41.2 -> 31.8.
// At head dimension 64 four CTAs fit on an SM (128 registers), a block's share of the HBM rate halves, and every
// partial of a (batch, head) adds `merge` to the second kernel, which is then no longer small.  242 dense and 242 paged problems
// (1 to 100 sequences of 512 to 32768 keys, 1 to 12 kv heads; device time): 3 % faster on the geometric mean than with
// the constants of 128, 5 % than with 256..2048 keys by S and the number of units alone; more than 5 % slower than
// that older rule in 42 of them (90 with the constants of 128), at worst 8 x 4096 keys ragged, 11.8 us against 14.0.
int default_chunk(const Problem& p) {
  constexpr double kFixed = 3.5;        // us
  const double slots = p.E == 64 ? 592 : 444, merge = p.E == 64 ? 0.1 : 0.0;
  const double block = p.block_table != nullptr ? 1.12 : 0.71;
  const int sub = (p.group + 15) / 16;
  const double shared = 1.6 * (p.E + p.Dv) / 256.0;
  const double units = static_cast<double>(p.B) * p.Hkv * sub;
  auto launch_us = [&](double ctas, int chunk, bool ragged) {
    const double blocks = chunk / 64.0, fill = ctas / slots;
    if (fill <= 1.0) return kFixed + blocks * (block + shared * fill);
    const double over = ragged && fill < 4.0 / 3.0 ? 3.0 * (fill - 1.0) : 1.0;
    return (fill + 0.35 * over) * (kFixed + blocks * (block + shared));
  };
  int best = 256;
  double best_us = 1e30;
  for (int chunk = 64; chunk <= kMaxChunk; chunk += chunk < 512 ? 64 : 256) {
    const int n = (p.S + chunk - 1) / chunk;
    double t = launch_us(units * n, chunk, false);
    t += merge * n;
    if (p.kv_lens != nullptr) t += 2 * launch_us(units * (n + 1) / 2, chunk, true) + merge * (n + 1);
    t *= 1.0 + 0.002 * n;   // equal: fewer partials
    if (t < best_us) {
      best_us = t;
      best = chunk;
    }
    if (chunk >= p.S) break;
  }
  return best;
}

struct DecodeGeom {
  int chunk, nsplit, g, nsub;
  uint64_t ws_bytes;
};

DecodeGeom geometry(const Problem& p, int kv_chunk) {
  DecodeGeom gm;
  gm.chunk = kv_chunk > 0 ? (kv_chunk + 31) / 32 * 32 : default_chunk(p);
  gm.nsplit = (p.S + gm.chunk - 1) / gm.chunk;
  if (gm.nsplit < 1) gm.nsplit = 1;
  gm.g = pick_group(p.group);
  gm.nsub = (p.group + gm.g - 1) / gm.g;
  gm.ws_bytes = static_cast<uint64_t>(p.B) * p.Hq * gm.nsplit * (p.Dv + 2) * sizeof(float);
  return gm;
}

template <typename T, int D>
int launch_combine(const Problem& p, const DecodeGeom& gm, float* po, float* pml, cudaStream_t stream) {
  auto kern = reinterpret_cast<uintptr_t>(po) % 16 == 0 ? decode_combine_kernel<T, D, true> : decode_combine_kernel<T, D, false>;
  if (!launch_pdl(kern, dim3(p.B * p.Hq), kCombineWarps * 32, 0, stream, p, gm.chunk, gm.nsplit, po, pml)) return B200_SDPA_ERR_CUDA;
  count_launch(KID_COMBINE);
  return B200_SDPA_OK;
}

template <typename T, int D, int G>
int launch_pg(const Problem& p, const DecodeGeom& gm, float* po, float* pml, cudaStream_t stream) {
  dim3 grid(p.Hkv * gm.nsub, p.B, gm.nsplit);
  decode_partial_kernel<T, D, G><<<grid, kThreads, 0, stream>>>(p, gm.chunk, gm.nsplit, po, pml);
  if (cudaGetLastError() != cudaSuccess) return B200_SDPA_ERR_CUDA;
  count_launch(KID_DECODE);
  return launch_combine<T, D>(p, gm, po, pml, stream);
}

// 16-bit caches go to the tensor-core partial kernel (decode_mma.cu); the CUDA-core
// kernel above keeps fp32 caches and can be forced with B200_SDPA_DECODE_SIMT=1.
bool use_mma_partial(const Problem& p, int dtype) {
  static const bool forced_simt = [] {
    const char* e = getenv("B200_SDPA_DECODE_SIMT");
    return e != nullptr && e[0] == '1';
  }();
  if (p.block_table != nullptr || p.k_new != nullptr) return true;   // only the tensor-core kernel serves these
  return !forced_simt && decode_mma_eligible(p, dtype);
}

template <typename T, int D>
int launch_g(const Problem& p, const DecodeGeom& gm, float* po, float* pml, cudaStream_t stream) {
  switch (gm.g) {
    case 1: return launch_pg<T, D, 1>(p, gm, po, pml, stream);
    case 2: return launch_pg<T, D, 2>(p, gm, po, pml, stream);
    case 4: return launch_pg<T, D, 4>(p, gm, po, pml, stream);
    default: return launch_pg<T, D, 8>(p, gm, po, pml, stream);
  }
}

}  // namespace

bool decode_eligible(const Problem& p, int dtype) {
  if (p.L != 1 || p.bias != nullptr || p.E != p.Dv) return false;
  // a paged cache or an appended row: 16-bit caches only (the tensor-core partial kernel)
  if ((p.block_table != nullptr || p.k_new != nullptr) && !decode_mma_eligible(p, dtype)) return false;
  if (p.k_new != nullptr) {
    if (p.kns[0] % 8 || p.kns[1] % 8 || p.vns[0] % 8 || p.vns[1] % 8) return false;
    if (reinterpret_cast<uintptr_t>(p.k_new) % 16 || reinterpret_cast<uintptr_t>(p.v_new) % 16) return false;
  }
  if (p.E != 64 && p.E != 128) return false;
  if (p.B > 65535 || static_cast<int64_t>(p.Hkv) * ((p.group + 7) / 8) > 65535) return false;
  // is_causal with one query row only limits keys to j <= causal_shift; the host
  // layer folds that into kv_lens, so here causal rows are left to other paths.
  if (p.causal) return false;
  const int64_t es = dtype == B200_SDPA_F32 ? 4 : 2;
  // 128-bit loads: unit inner stride, 16-byte aligned rows and bases
  if (p.ks[3] != 1 || p.vs[3] != 1) return false;
  if ((p.ks[0] * es) % 16 || (p.ks[1] * es) % 16 || (p.ks[2] * es) % 16) return false;
  if ((p.vs[0] * es) % 16 || (p.vs[1] * es) % 16 || (p.vs[2] * es) % 16) return false;
  if (reinterpret_cast<uintptr_t>(p.k) % 16 || reinterpret_cast<uintptr_t>(p.v) % 16) return false;
  return true;
}

int plan_decode(const Problem& p, int dtype, int kv_chunk, B200SdpaPlan* plan) {
  if (!decode_eligible(p, dtype)) return B200_SDPA_ERR_UNSUPPORTED;
  const DecodeGeom gm = geometry(p, kv_chunk);
  if (gm.nsplit > 65535) return B200_SDPA_ERR_UNSUPPORTED;   // grid.z
  plan->path = B200_SDPA_PATH_DECODE;
  plan->block_m = 1;
  plan->block_n = gm.chunk;
  plan->grid_x = p.Hkv * gm.nsub;
  plan->grid_y = p.B;
  plan->grid_z = gm.nsplit;
  plan->threads = kThreads;
  plan->smem_bytes = 0;
  plan->kv_splits = gm.nsplit;
  plan->launches = 2;
  plan->workspace_bytes = gm.ws_bytes;
  return B200_SDPA_OK;
}

int launch_decode(const Problem& p, int dtype, int kv_chunk, void* workspace, uint64_t workspace_bytes,
                  cudaStream_t stream) {
  if (!decode_eligible(p, dtype)) return B200_SDPA_ERR_UNSUPPORTED;
  const DecodeGeom gm = geometry(p, kv_chunk);
  if (gm.nsplit > 65535) return B200_SDPA_ERR_UNSUPPORTED;   // grid.z
  if (workspace == nullptr || workspace_bytes < gm.ws_bytes) return B200_SDPA_ERR_WORKSPACE;
  float* po = reinterpret_cast<float*>(workspace);
  float* pml = po + static_cast<uint64_t>(p.B) * p.Hq * gm.nsplit * p.Dv;
  const bool d128 = p.E == 128;
  if (use_mma_partial(p, dtype)) {
    const int rc = launch_decode_partial_mma(p, dtype, gm.chunk, gm.nsplit, po, pml, stream);
    if (rc != B200_SDPA_OK) return rc;
    if (dtype == B200_SDPA_BF16)
      return d128 ? launch_combine<__nv_bfloat16, 128>(p, gm, po, pml, stream)
                  : launch_combine<__nv_bfloat16, 64>(p, gm, po, pml, stream);
    return d128 ? launch_combine<__half, 128>(p, gm, po, pml, stream) : launch_combine<__half, 64>(p, gm, po, pml, stream);
  }
  switch (dtype) {
    case B200_SDPA_F32:
      return d128 ? launch_g<float, 128>(p, gm, po, pml, stream) : launch_g<float, 64>(p, gm, po, pml, stream);
    case B200_SDPA_F16:
      return d128 ? launch_g<__half, 128>(p, gm, po, pml, stream) : launch_g<__half, 64>(p, gm, po, pml, stream);
    case B200_SDPA_BF16:
      return d128 ? launch_g<__nv_bfloat16, 128>(p, gm, po, pml, stream)
                  : launch_g<__nv_bfloat16, 64>(p, gm, po, pml, stream);
    default: return B200_SDPA_ERR_DTYPE;
  }
}

// ---------------------------------------------------------------------------
// Decode with built-in scratch.
//
// Some hosts cannot give this library a workspace at call time: a serving
// process that handed all device memory to its own pool when it started (so a
// later cudaMalloc fails or is forbidden), or code on a path where allocator
// calls are not permitted at all.  For them the partials of the split-KV
// kernel live in the fixed array below instead of caller-provided memory.
// Every GPU that loads the library carries the array until the process exits,
// which is why it is kept modest; requests whose partials do not fit are
// rejected, never truncated.
//
// The array's name is only a host-side handle.  Its device address is looked
// up once per device with cudaGetSymbolAddress(), with that device current, the
// first time the entry point is used on the device -- so the first call per
// device should be made outside any stream capture.  All calls share the array
// and it keeps whatever the previous call left: the kernels write every slot
// they later read, so nothing has to be cleared, but two calls that overlap on
// the GPU (different streams) would race on it.
// ---------------------------------------------------------------------------
constexpr unsigned long long kStaticScratchBytes = B200_SDPA_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_decode_scratch[kStaticScratchBytes];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
void* g_scratch_ptr[kMaxDevices] = {};
}  // namespace

int launch_decode_static(const Problem& p, int dtype, int kv_chunk, cudaStream_t stream) {
  if (!decode_eligible(p, dtype)) return B200_SDPA_ERR_UNSUPPORTED;
  DecodeGeom gm = geometry(p, kv_chunk);
  // the library's own choice of chunk, which is made for speed with scratch of any size, gives way to longer ones
  for (int chunk = gm.chunk; kv_chunk <= 0 && gm.ws_bytes > kStaticScratchBytes && chunk < kMaxChunk;) {
    chunk = chunk + 256 < kMaxChunk ? chunk + 256 : kMaxChunk;
    gm = geometry(p, chunk);
  }
  if (gm.ws_bytes > kStaticScratchBytes) return B200_SDPA_ERR_TOO_LARGE;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return B200_SDPA_ERR_CUDA;
  }
  void* ptr = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_ptr[dev] == nullptr) {
      void* found = nullptr;
      if (cudaGetSymbolAddress(&found, g_decode_scratch) != cudaSuccess || found == nullptr) {
        cudaGetLastError();
        return B200_SDPA_ERR_CUDA;
      }
      g_scratch_ptr[dev] = found;
    }
    ptr = g_scratch_ptr[dev];
  }
  return launch_decode(p, dtype, gm.chunk, ptr, kStaticScratchBytes, stream);
}


}  // namespace b200

// The expanded form of latent attention for portions of prompts: keys W_uk c and values W_uv c are formed for all
// heads by library products, and this kernel attends them with 5th-generation tensor cores.  A head's key is
// [its own dim elements | the rotated part that all heads share], so the two come through tensor maps of
// their own - the shared part is read from the cached rows and never copied per head - and meet in shared
// memory as neighbouring 64-wide blocks of the K dimension; likewise the two parts of a query.  Blocks that are
// not full (dim 32, rot 16, ...) are zero-filled by TMA, so any sizes that are multiples of 8 up to
// dim 128, rot 64, vdim 128 run.  Without a rotated part the key is its own elements alone; kv_heads below heads shares
// a key and value head among a group of query heads, which makes this the prompt form of grouped attention too.
//
// A row may see only the last `window` keys (a CTA starts at the tile that holds its first row's first key), and a
// per-head sink may join the denominator.
//
// Structure as prefill_attn.cu: one CTA per (128 query rows, head), two per SM, against key tiles of 64; two buffers of S and O in
// tensor memory, P over S; warps 0-3 own one query row per thread and do the online softmax, warp 4 issues the MMAs - the
// scores two tiles ahead -, warp 5 the TMA loads.  What differs: K is 64 x up to 192 elements per tile, so that with a rotated
// part K and V have a buffer less; rows stand at positions start .. start + n - 1 of a longer key sequence.  Every wait is bounded.
// Bound by the tensor core as there.  2048 rows over 8192 keys, 16 heads of 128: 133 us, now 115; with a window of 4096: 76 and 70;
// 2000 rows, 16 heads of 128 + 64 rotated: 43 and 36 (before: one CTA per SM with two blocks of rows and tiles of 128 keys, whose
// scores had to wait for the tile before, and products issued one by one).  That form, issued as here, is still the faster one for
// much work with a rotated part: the second kernel (8192 rows of these: 272, 288 in the first).
#include <math.h>

#include <mutex>
#include <type_traits>

#include "tcgen05.cuh"

namespace axb {
namespace {

constexpr int kRows = 128, kKeys = 64, kBox = kRows * 64 * 2;  // one [128 rows][64 elements] block: 16 KB
constexpr int kKeyBox = kKeys * 64 * 2;                        // of [64 keys][64 elements]
constexpr int kThreads = 192, kMmaWarp = 4, kLoadWarp = 5;
constexpr float kLog2e = 1.4426950408889634f, kLazy = 8.0f;

struct Params {
  __nv_bfloat16 *out;
  int n, start, skv, heads, group, vdim;  // group: query heads per key and value head
  int window;                             // 0: all
  const float *sink;                      // (heads), or null
  float scale_log2;
  unsigned long long wait_ns;
};

// A thread's row of scores of a tile from key n0 on: those outside [begin, end) are masked, the running maximum m_run (of the
// scaled scores: scale may be negative or zero in principle) moves where some row of the warp found a score more than kLazy above
// it, and the weights go to tensor memory in bf16.  The sums of weights so far and the row's accumulator then owe the factor corr;
// true where it may not be one.
template <int kChunks>
__device__ __forceinline__ bool softmax_tile(uint32_t (&sr)[kChunks][32], int n0, int begin, int end, float scale_log2, uint32_t weights,
                                             float &m_run, float &corr, float (&sum4)[4]) {
  if (n0 < begin) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (n0 + c * 32 + i < begin) sr[c][i] = 0xff800000u;  // -inf
  }
  if (n0 + kChunks * 32 > end) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (n0 + c * 32 + i >= end) sr[c][i] = 0xff800000u;  // -inf
  }
  const float m_tile = row_max(sr) * scale_log2;
  corr = 1.f;
  const bool moved = __any_sync(0xffffffffu, m_tile > m_run + kLazy);
  if (moved) {
    const float m_new = fmaxf(m_run, m_tile);
    corr = fast_exp2(m_run - ((m_new == -INFINITY) ? 0.f : m_new));
    m_run = m_new;
  }
  const float m_safe = (m_run == -INFINITY) ? 0.f : m_run;
  const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2), shift2 = pack_f32x2(-m_safe, -m_safe);
#pragma unroll
  for (int i = 0; i < 4; ++i) sum4[i] *= corr;
  // neighbours first, and 128 keys together: the order of these additions shows in the last bit of the results
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    uint32_t packed[16];
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      float w[4];
#pragma unroll
      for (int u = 0; u < 4; u += 2) {
        const float2 x =
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sr[c][i + u]), __uint_as_float(sr[c][i + u + 1])), scale2, shift2));
        w[u] = fast_exp2(x.x), w[u + 1] = fast_exp2(x.y);
        packed[(i + u) >> 1] = pack_bf16x2(w[u], w[u + 1]);
      }
      sum4[(i >> 1) & 3] += w[0] + w[1];
      sum4[((i >> 1) & 3) + 1] += w[2] + w[3];
    }
    tmem_st16(weights + c * 16, packed);
  }
  return moved;
}

// A row of the accumulator times corr.
template <int kVB>
__device__ __forceinline__ void rescale_row(uint32_t acc, float corr) {
#pragma unroll
  for (int c = 0; c < kVB * 2; ++c) {
    uint32_t r[32];
    tmem_ld32(acc + c * 32, r);
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * corr);
    tmem_st32(acc + c * 32, r);
  }
}

// A row's result from its accumulator, maximum and denominator.
template <int kVB>
__device__ __forceinline__ void store_row(const Params &p, int t_row, int h, uint32_t acc, float m_run, float l_run) {
  float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
  if (p.sink) {
    const float s = p.sink[h] * kLog2e, top = fmaxf(m_run, s), w = fast_exp2(m_run - top);
    inv = w / fmaf(l_run, w, fast_exp2(s - top));
  }
  __nv_bfloat16 *dst = p.out + ((size_t)t_row * p.heads + h) * p.vdim;
#pragma unroll
  for (int c = 0; c < kVB * 2; ++c) {
    uint32_t r[32];
    tmem_ld32(acc + c * 32, r);
    if (t_row < p.n) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (c * 32 + u * 8 >= p.vdim) break;
        uint4 w;
        w.x = pack_bf16x2(__uint_as_float(r[u * 8 + 0]) * inv, __uint_as_float(r[u * 8 + 1]) * inv);
        w.y = pack_bf16x2(__uint_as_float(r[u * 8 + 2]) * inv, __uint_as_float(r[u * 8 + 3]) * inv);
        w.z = pack_bf16x2(__uint_as_float(r[u * 8 + 4]) * inv, __uint_as_float(r[u * 8 + 5]) * inv);
        w.w = pack_bf16x2(__uint_as_float(r[u * 8 + 6]) * inv, __uint_as_float(r[u * 8 + 7]) * inv);
        *reinterpret_cast<uint4 *>(dst + c * 32 + u * 8) = w;
      }
    }
  }
}

// kQB / kVB: 64-wide blocks of the heads' own key part and of the values; kRot: one more block for the rotated part
template <int kQB, int kVB, int kRot>
struct Layout {
  static constexpr int kBlocks = kQB + kRot;
  static constexpr int kQ = kBlocks * kBox, kK = kBlocks * kKeyBox, kV = kVB * kKeyBox;  // a query tile, tiles of keys and values
  static constexpr bool kDeep = kQ + 3 * kK + 2 * kV <= 112 * 1024;  // two CTAs share an SM
  static constexpr int kKStages = kDeep ? 3 : 2, kVStages = kDeep ? 2 : 1;
  static constexpr int kOffK = kQ, kOffV = kOffK + kKStages * kK, kOffBar = kOffV + kVStages * kV;
  static constexpr int kSmem = kOffBar + 256;
  static_assert(kOffBar <= 112 * 1024, "two CTAs per SM");
};

template <int kQB, int kVB, int kRot>
__global__ void __launch_bounds__(kThreads, 2)
latent_prefill_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmQr,
                      const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmKr,
                      const __grid_constant__ CUtensorMap tmV, const Params p) {
  using L = Layout<kQB, kVB, kRot>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kOffBar);
  uint64_t *bar_q = bars, *full_k = bars + 1, *empty_k = bars + 4, *full_v = bars + 7, *empty_v = bars + 9;
  uint64_t *bar_s = bars + 11, *bar_o = bars + 13;  // S_j ready (per buffer); P_j.V_j done
  uint64_t *bar_fin = bars + 14;  // the last P.V: the softmax warps skip phases of bar_o, a parity wait there would alias
  uint64_t *bar_p = bars + 15;    // P_j written (per S buffer), one arrival per softmax warp
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 17);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 18);
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicOr(&g_error_word, AXB200_ERR_WAIT_TIMEOUT);
    return;
  }
  // heaviest blocks of all heads first: the last query block has the most key tiles
  const int h = blockIdx.x % p.heads, q0 = (int)((gridDim.x - 1 - blockIdx.x) / p.heads) * kRows;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int hk = h / p.group;
  const int tile0 = p.window > 0 ? max(0, p.start + q0 + 1 - p.window) / kKeys : 0;  // the first key tile
  const int nkv = (min(p.start + min(q0 + kRows, p.n), p.skv) + kKeys - 1) / kKeys - tile0;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 15; ++i) mbar_init(&bars[i], 1);
    mbar_init(&bar_p[0], 4);
    mbar_init(&bar_p[1], 4);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_dependency_wait();
  grid_dependency_launch();
  const uint32_t tmem = *tmem_slot, tmem_o = tmem + 128;  // S buffers at columns 0 and 64; P_j over the front of its S

  if (warp == kLoadWarp) {
    if (lane == 0) {
      tma_prefetch_descriptor(&tmK);
      if (kRot) tma_prefetch_descriptor(&tmKr);
      tma_prefetch_descriptor(&tmV);
      mbar_arrive_expect_tx(bar_q, L::kQ);
      for (int b = 0; b < kQB; ++b) tma_load_3d(smem + b * kBox, &tmQ, bar_q, b * 64, h, q0);  // rows past n are zero-filled
      if (kRot) tma_load_3d(smem + kQB * kBox, &tmQr, bar_q, 0, h, q0);
      bool ok = true;
      int nk = 0, nv = 0;  // tiles asked for
      auto load_k = [&] {
        const int s = nk % L::kKStages;
        if (nk >= L::kKStages) ok = ok && mbar_wait_bounded(&empty_k[s], (nk / L::kKStages - 1) & 1, abort_flag, p.wait_ns);
        if (!ok) return;
        uint8_t *dst = smem + L::kOffK + s * L::kK;
        mbar_arrive_expect_tx(&full_k[s], L::kK);
        for (int b = 0; b < kQB; ++b) tma_load_3d(dst + b * kKeyBox, &tmK, &full_k[s], b * 64, hk, (tile0 + nk) * kKeys);
        if (kRot) tma_load_3d(dst + kQB * kKeyBox, &tmKr, &full_k[s], 0, 0, (tile0 + nk) * kKeys);
        ++nk;
      };
      // consumption order is S_0 S_1 (PV_0 S_2) (PV_1 S_3) ...: K_0 K_1 V_0 K_2 V_1 K_3 ..., K ahead where it has the buffer
      while (nk < min(nkv, L::kKStages)) load_k();
      for (; nv < nkv; ++nv) {
        const int s = nv % L::kVStages;
        if (nv >= L::kVStages) ok = ok && mbar_wait_bounded(&empty_v[s], (nv / L::kVStages - 1) & 1, abort_flag, p.wait_ns);
        if (!ok) break;
        uint8_t *dst = smem + L::kOffV + s * L::kV;
        mbar_arrive_expect_tx(&full_v[s], L::kV);
        for (int b = 0; b < kVB; ++b) tma_load_3d(dst + b * kKeyBox, &tmV, &full_v[s], b * 64, hk, (tile0 + nv) * kKeys);
        if (nk < nkv) load_k();
      }
      if (*abort_flag) {  // no copy may still be on its way when the CTA leaves
        const unsigned long long t0 = global_timer_ns();
        auto drain = [&](uint64_t *bar, uint32_t parity) {
          while (!mbar_try_wait(bar, parity) && global_timer_ns() - t0 < 100000000ull) {
          }
        };
        drain(bar_q, 0);
        for (int t = max(0, nk - L::kKStages); t < nk; ++t) drain(&full_k[t % L::kKStages], (t / L::kKStages) & 1);
        for (int t = max(0, nv - L::kVStages); t < nv; ++t) drain(&full_v[t % L::kVStages], (t / L::kVStages) & 1);
      }
    }
  } else if (warp == kMmaWarp) {
    // the warp walks, one lane issues.  fp32 accumulate, bf16 operands, M = 128.  Q.K^T: N = 64, B K-major; P.V: N = kVB * 64, B
    // MN-major
    constexpr uint32_t kBf16 = (1u << 4) | (1u << 7) | (1u << 10) | ((kRows >> 4) << 24);
    constexpr uint32_t idesc_qk = kBf16 | ((kKeys >> 3) << 17), idesc_pv = kBf16 | (1u << 16) | ((kVB * 64 >> 3) << 17);
    const uint64_t dq = smem_desc(smem_u32(smem), 16, 1024);
    const uint64_t dk = smem_desc(smem_u32(smem + L::kOffK), 16, 1024);
    const uint64_t dv = smem_desc(smem_u32(smem + L::kOffV), kKeyBox, 1024);
    RingPos k, v;
    auto issue_s = [&](int j) -> bool {
      if (!mbar_wait_warp(&full_k[k.slot], k.parity, abort_flag, p.wait_ns)) return false;
      tc_fence_after();
      const uint64_t dks = dk + (uint64_t)(k.slot * (L::kK >> 4));
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < L::kBlocks * 4; ++ks)
          umma_f16(tmem + (j & 1) * kKeys, dq + (uint64_t)(((ks >> 2) * kBox + (ks & 3) * 32) >> 4),
                   dks + (uint64_t)(((ks >> 2) * kKeyBox + (ks & 3) * 32) >> 4), idesc_qk, ks > 0);
        umma_commit(&bar_s[j & 1]);
        umma_commit(&empty_k[k.slot]);
      }
      k.next(L::kKStages);
      return true;
    };
    bool ok = mbar_wait_warp(bar_q, 0, abort_flag, p.wait_ns) && issue_s(0);
    if (ok && nkv > 1) ok = issue_s(1);
    for (int j = 0; j < nkv && ok; ++j) {
      ok = mbar_wait_warp(&bar_p[j & 1], (j >> 1) & 1, abort_flag, p.wait_ns) &&
           mbar_wait_warp(&full_v[v.slot], v.parity, abort_flag, p.wait_ns);
      if (!ok) break;
      tc_fence_after();
      const uint64_t dvs = dv + (uint64_t)(v.slot * (L::kV >> 4));
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < kKeys / 16; ++ks)  // 16 keys: 8 columns of P, 2 KB of V
          umma_f16_ts(tmem_o, tmem + (j & 1) * kKeys + ks * 8, dvs + (uint64_t)(ks * (2048 >> 4)), idesc_pv, j > 0 || ks > 0);
        umma_commit(bar_o);
        umma_commit(&empty_v[v.slot]);
        if (j == nkv - 1) umma_commit(bar_fin);
      }
      v.next(L::kVStages);
      // S_{j+2} takes the place of P_j: products of unlike shapes have no order of their own, so P_j.V_j is waited for
      if (j + 2 < nkv) ok = mbar_wait_warp(bar_o, j & 1, abort_flag, p.wait_ns) && issue_s(j + 2);
    }
  } else {
    // ---- softmax warps: thread = row ----
    const int row = threadIdx.x, t_row = q0 + row;
    const int kv_end = min(p.start + t_row + 1, p.skv), kv_begin = p.window > 0 ? max(0, p.start + t_row + 1 - p.window) : 0;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16, to = tmem_o + lane_base;
    float m_run = -INFINITY, l_run = 0.f, sum4[4] = {0.f, 0.f, 0.f, 0.f};
    bool ok = true;
    for (int j = 0; j < nkv && ok; ++j) {
      ok = mbar_wait_warp(&bar_s[j & 1], (j >> 1) & 1, abort_flag, p.wait_ns);
      if (!ok) break;
      tc_fence_after();
      const uint32_t ts = tmem + (j & 1) * kKeys + lane_base;
      uint32_t sr[2][32];
#pragma unroll
      for (int c = 0; c < 2; ++c) tmem_ld32_async(ts + c * 32, sr[c]);
      tmem_wait_ld();
      float corr;
      const bool moved =
          softmax_tile(sr, (tile0 + j) * kKeys, kv_begin, kv_end, p.scale_log2, ts, m_run, corr, sum4);
      l_run *= corr;
      if (((tile0 + j) & 1) || j == nkv - 1) {
        l_run += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) sum4[i] = 0.f;
      }
      // O is in use by P_{j-1}.V_{j-1} until that completes (P_j.V_j is not issued before this warp arrives below, so the barrier
      // cannot be more than one phase ahead of the parity asked for)
      if (j > 0 && moved) {
        ok = mbar_wait_warp(bar_o, (j - 1) & 1, abort_flag, p.wait_ns);
        if (!ok) break;
        tc_fence_after();
        rescale_row<kVB>(to, corr);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p[j & 1]);
    }
    if (ok && nkv > 0) ok = mbar_wait_warp(bar_fin, 0, abort_flag, p.wait_ns);
    tc_fence_after();
    if (ok && nkv > 0) store_row<kVB>(p, t_row, h, to, m_run, l_run);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

// The form for much work with a rotated part, 65 to 128 own elements and as many value columns: one CTA per SM has two blocks of
// rows against tiles of 128 keys.  A key's 192 elements make 64-wide scores dear (12 products of 50 cycles, 12 of 66 for twice the
// keys), and four boxes of 16 KB more are under way per CTA; but scores wait for the tile before, and the blocks are coarser.  S_g
// at g * 128, P_g over its front, O_g at 256 + g * 128; K is double-buffered, V has one buffer whose halves of 64 keys are freed
// and refilled separately.  Scores take P's place in the order of issue, which products of one shape keep.
struct Wide {
  static constexpr int kKeys = 128, kThreads = 320, kMmaWarp = 8, kLoadWarp = 9;
  static constexpr int kTile = 3 * kBox, kVHalf = 2 * kKeyBox;  // a query tile or a key tile; 64 keys' values
  static constexpr int kOffK = 2 * kTile, kOffV = kOffK + 2 * kTile, kOffBar = kOffV + 2 * kVHalf, kSmem = kOffBar + 256;
};

__global__ void __launch_bounds__(Wide::kThreads, 1)
latent_prefill_wide_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmQr,
                           const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmKr,
                           const __grid_constant__ CUtensorMap tmV, const Params p) {
  using L = Wide;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kOffBar);
  uint64_t *bar_q = bars, *full_k = bars + 1, *empty_k = bars + 3, *full_v = bars + 5, *empty_v = bars + 7;
  uint64_t *bar_s = bars + 9, *bar_fin = bars + 11, *bar_p = bars + 13;  // per block of rows
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 15);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 16);
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicOr(&g_error_word, AXB200_ERR_WAIT_TIMEOUT);
    return;
  }
  const int h = blockIdx.x % p.heads, q0 = (int)((gridDim.x - 1 - blockIdx.x) / p.heads) * 2 * kRows;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int hk = h / p.group;
  const int tile0 = p.window > 0 ? max(0, p.start + q0 + 1 - p.window) / L::kKeys : 0;
  int nkv_g[2];  // key tiles; none for a block past the last row
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int first = q0 + g * kRows;
    nkv_g[g] = first < p.n ? (min(p.start + min(first + kRows, p.n), p.skv) + L::kKeys - 1) / L::kKeys - tile0 : 0;
  }
  const int nkv = max(nkv_g[0], nkv_g[1]);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 13; ++i) mbar_init(&bars[i], 1);
    mbar_init(&bar_p[0], 4);
    mbar_init(&bar_p[1], 4);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == L::kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_dependency_wait();
  grid_dependency_launch();
  const uint32_t tmem = *tmem_slot;

  if (warp == L::kLoadWarp) {
    if (lane == 0) {
      tma_prefetch_descriptor(&tmK);
      tma_prefetch_descriptor(&tmKr);
      tma_prefetch_descriptor(&tmV);
      mbar_arrive_expect_tx(bar_q, 2 * L::kTile);
      for (int g = 0; g < 2; ++g) {  // rows past n are zero-filled
        uint8_t *dst = smem + g * L::kTile;
        for (int b = 0; b < 2; ++b) tma_load_3d(dst + b * kBox, &tmQ, bar_q, b * 64, h, q0 + g * kRows);
        tma_load_3d(dst + 2 * kBox, &tmQr, bar_q, 0, h, q0 + g * kRows);
      }
      bool ok = true;
      int nk = 0, nv[2] = {0, 0};  // tiles, and halves of them, asked for
      auto load_k = [&] {
        const int s = nk & 1;
        if (nk >= 2) ok = ok && mbar_wait_bounded(&empty_k[s], ((nk >> 1) - 1) & 1, abort_flag, p.wait_ns);
        if (!ok) return;
        uint8_t *dst = smem + L::kOffK + s * L::kTile;
        mbar_arrive_expect_tx(&full_k[s], L::kTile);
        for (int b = 0; b < 2; ++b) tma_load_3d(dst + b * kBox, &tmK, &full_k[s], b * 64, hk, (tile0 + nk) * L::kKeys);
        tma_load_3d(dst + 2 * kBox, &tmKr, &full_k[s], 0, 0, (tile0 + nk) * L::kKeys);
        ++nk;
      };
      load_k();
      for (int j = 0; j < nkv && ok; ++j) {
        if (nk < nkv) load_k();
        for (int half = 0; half < 2 && ok; ++half) {
          if (j >= 1) ok = mbar_wait_bounded(&empty_v[half], (j - 1) & 1, abort_flag, p.wait_ns);
          if (!ok) break;
          uint8_t *dst = smem + L::kOffV + half * L::kVHalf;
          mbar_arrive_expect_tx(&full_v[half], L::kVHalf);
          for (int b = 0; b < 2; ++b) tma_load_3d(dst + b * kKeyBox, &tmV, &full_v[half], b * 64, hk, (tile0 + j) * L::kKeys + half * 64);
          ++nv[half];
        }
      }
      if (*abort_flag) {  // no copy may still be on its way when the CTA leaves
        const unsigned long long t0 = global_timer_ns();
        auto drain = [&](uint64_t *bar, uint32_t parity) {
          while (!mbar_try_wait(bar, parity) && global_timer_ns() - t0 < 100000000ull) {
          }
        };
        drain(bar_q, 0);
        for (int t = max(0, nk - 2); t < nk; ++t) drain(&full_k[t & 1], (t >> 1) & 1);
        for (int half = 0; half < 2; ++half)
          if (nv[half] > 0) drain(&full_v[half], (nv[half] - 1) & 1);
      }
    }
  } else if (warp == L::kMmaWarp) {
    constexpr uint32_t idesc_qk = (1u << 4) | (1u << 7) | (1u << 10) | ((L::kKeys >> 3) << 17) | ((kRows >> 4) << 24);
    constexpr uint32_t idesc_pv = idesc_qk | (1u << 16);  // as wide; B MN-major
    const uint64_t dq = smem_desc(smem_u32(smem), 16, 1024);
    const uint64_t dk = smem_desc(smem_u32(smem + L::kOffK), 16, 1024);
    const uint64_t dv = smem_desc(smem_u32(smem + L::kOffV), kKeyBox, 1024);
    auto issue_s = [&](int g, int t) {
      const uint64_t dqg = dq + (uint64_t)(g * (L::kTile >> 4)), dks = dk + (uint64_t)((t & 1) * (L::kTile >> 4));
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 12; ++ks) {
          const uint32_t off = ((ks >> 2) * kBox + (ks & 3) * 32) >> 4;
          umma_f16(tmem + g * 128, dqg + off, dks + off, idesc_qk, ks > 0);
        }
        umma_commit(&bar_s[g]);
      }
    };
    bool ok = mbar_wait_warp(bar_q, 0, abort_flag, p.wait_ns) && mbar_wait_warp(&full_k[0], 0, abort_flag, p.wait_ns);
    if (ok) {
      tc_fence_after();
      if (nkv_g[0] > 0) issue_s(0, 0);
      if (nkv_g[1] > 0) issue_s(1, 0);
      if (elect_one()) umma_commit(&empty_k[0]);
    }
    for (int j = 0; j < nkv && ok; ++j) {
      const int last_g = nkv_g[1] > j ? 1 : 0;
      bool have_k = false;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (j >= nkv_g[g]) continue;
        ok = mbar_wait_warp(&bar_p[g], j & 1, abort_flag, p.wait_ns);
        if (!ok) break;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          ok = ok && mbar_wait_warp(&full_v[half], j & 1, abort_flag, p.wait_ns);
          if (!ok) break;
          tc_fence_after();
          const uint64_t dvh = dv + (uint64_t)(half * (L::kVHalf >> 4));
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)  // 16 keys: 8 columns of P, 2 KB of V
              umma_f16_ts(tmem + 256 + g * 128, tmem + g * 128 + half * 32 + ks * 8, dvh + (uint64_t)(ks * (2048 >> 4)), idesc_pv,
                          j > 0 || half > 0 || ks > 0);
            if (g == last_g) umma_commit(&empty_v[half]);
          }
        }
        if (!ok) break;
        if (j == nkv_g[g] - 1 && elect_one()) umma_commit(&bar_fin[g]);
        if (j + 1 < nkv_g[g]) {
          if (!have_k) ok = mbar_wait_warp(&full_k[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag, p.wait_ns);
          if (!ok) break;
          have_k = true;
          tc_fence_after();
          issue_s(g, j + 1);
        }
      }
      if (ok && j + 1 < nkv && elect_one()) umma_commit(&empty_k[(j + 1) & 1]);
    }
  } else {
    // ---- softmax warps: block of rows g, thread = row ----
    const int g = warp >> 2, my_nkv = g ? nkv_g[1] : nkv_g[0];
    const int t_row = q0 + g * kRows + (threadIdx.x & (kRows - 1));
    const int kv_end = min(p.start + t_row + 1, p.skv), kv_begin = p.window > 0 ? max(0, p.start + t_row + 1 - p.window) : 0;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16, ts = tmem + g * 128 + lane_base, to = ts + 256;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < my_nkv && ok; ++j) {
      ok = mbar_wait_warp(&bar_s[g], j & 1, abort_flag, p.wait_ns);
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32_async(ts + c * 32, sr[c]);
      tmem_wait_ld();
      float corr, sum4[4] = {0.f, 0.f, 0.f, 0.f};
      const bool moved = softmax_tile(sr, (tile0 + j) * L::kKeys, kv_begin, kv_end, p.scale_log2, ts, m_run, corr, sum4);
      l_run = l_run * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
      // S_g(j) stands where P_g(j-1) was read, so P_g(j-1).V_{j-1} is complete and O_g may be rescaled
      if (j > 0 && moved) rescale_row<2>(to, corr);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p[g]);
    }
    if (ok && my_nkv > 0) ok = mbar_wait_warp(&bar_fin[g], 0, abort_flag, p.wait_ns);
    tc_fence_after();
    if (ok && my_nkv > 0) store_row<2>(p, t_row, h, to, m_run, l_run);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == L::kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// (rows, heads, elems) with row and head strides in elements -> boxes of [box_rows rows][64 elements]
bool map_of(CUtensorMap *map, const void *base, int elems, int heads, int64_t rows, int64_t head_stride, int64_t row_stride,
            int box_rows) {
  EncodeTiledFn fn = tensor_map_encoder();
  const cuuint64_t dims[3] = {(cuuint64_t)elems, (cuuint64_t)heads, (cuuint64_t)rows};
  const cuuint64_t strides[2] = {(cuuint64_t)head_stride * 2, (cuuint64_t)row_stride * 2};
  const cuuint32_t box[3] = {64, 1, (cuuint32_t)box_rows}, es[3] = {1, 1, 1};
  return fn && fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <auto kKernel>
int launch_form(int rows, int threads, int smem, const CUtensorMap (&m)[5], const Params &p, cudaStream_t st) {
  static std::mutex mu;
  static bool opted[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return AXB200_DEVICE_ERROR;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!opted[dev]) {
      if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return AXB200_DEVICE_ERROR;
      opted[dev] = true;
    }
  }
  const dim3 grid((unsigned)p.heads * ((p.n + rows - 1) / rows));
  return launch_dependent(kKernel, grid, dim3(threads), smem, st, m[0], m[1], m[2], m[3], m[4], p);
}

template <int kQB, int kVB, int kRot>
int launch(const CUtensorMap (&m)[5], const Params &p, cudaStream_t st) {
  return launch_form<&latent_prefill_kernel<kQB, kVB, kRot>>(kRows, kThreads, Layout<kQB, kVB, kRot>::kSmem, m, p, st);
}

// Whether the wide form is the faster one.  The tensor core sets the pace from about 64 tiles of 64 keys for each of the 296 CTAs
// that run at once (wide and narrow tiles, with 16 heads: 4096 rows, 57 tiles, 76 us and 76; 8192, 223, 272 and 288; 32 heads: 3000
// rows, 63, 95 and 94; 2048 rows over 8192 keys, 194, 251 and 269); and where a CTA per SM reads keys and values that do not fit
// into L2, copies under way do (100 rows over 8100 keys: 16 heads, 66 MB, 125 and 117; 32 heads, 133 MB, 125 and 142; 128 heads 138
// and 171).
bool wide_gains(const Params &p, int kv_heads, int dim, int rot_dim) {
  if (rot_dim == 0 || dim <= 64 || p.vdim <= 64) return false;
  const int64_t blocks = ((int64_t)p.n + kRows - 1) / kRows;
  int64_t tiles = 0;
  for (int64_t b = 0; b < blocks; ++b) {
    const int64_t first = p.start + b * kRows, last = first + kRows < p.skv ? first + kRows : p.skv;
    tiles += (last + kKeys - 1) / kKeys - (p.window > 0 && first + 1 > p.window ? (first + 1 - p.window) / kKeys : 0);
  }
  const int64_t first_key = p.window > 0 && p.start + 1 > p.window ? p.start + 1 - p.window : 0;
  const int64_t bytes = (p.skv - first_key) * kv_heads * (dim + p.vdim) * 2;
  return tiles * p.heads >= 64 * 296 || (blocks * p.heads <= 148 && bytes > (int64_t)100 << 20);
}

bool al16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace axb

extern "C" {

int axb200_latent_prefill_supported(int heads, int dim, int rot_dim, int vdim, int dtype) {
  return dtype == AXB200_BFLOAT16 && heads > 0 && heads <= 65535 && dim >= 8 && dim <= 128 && dim % 8 == 0 && rot_dim >= 0 &&
         rot_dim <= 64 && rot_dim % 8 == 0 && vdim >= 8 && vdim <= 128 && vdim % 8 == 0;
}

int axb200_latent_prefill(const void *q, int64_t q_ld, const void *k, const void *v, const void *rot, int64_t rot_ld,
                          const float *sink, void *out, int n, int64_t start, int heads, int kv_heads, int dim, int rot_dim,
                          int vdim, int window, float scale, int dtype, void *stream) {
  if (!axb200_latent_prefill_supported(heads, dim, rot_dim, vdim, dtype)) return AXB200_UNSUPPORTED_TYPE;
  if (!q || !k || !v || (rot_dim > 0 && !rot) || !out) return AXB200_INVALID_PTR;
  if (n < 0 || start < 0 || start + n > 0x7fffffff - 4096 || !(scale > 0.f) || kv_heads <= 0 || heads % kv_heads != 0 || window < 0)
    return AXB200_INVALID_ARGUMENT;
  if (q_ld < (int64_t)heads * (dim + rot_dim) || rot_ld < rot_dim) return AXB200_SHAPE_MISMATCH;
  if (q_ld % 8 || rot_ld % 8 || !axb::al16(q) || !axb::al16(k) || !axb::al16(v) || !axb::al16(rot) || !axb::al16(out))
    return AXB200_UNSUPPORTED_TYPE;
  if (n == 0) return AXB200_OK;
  const int per = dim + rot_dim;
  const int64_t skv = start + n;
  axb::Params p{static_cast<__nv_bfloat16 *>(out), n, (int)start, (int)skv, heads, heads / kv_heads, vdim, window, sink,
                scale * axb::kLog2e, axb::wait_limit_ns()};
  const bool wide = axb::wide_gains(p, kv_heads, dim, rot_dim);
  const int key_rows = wide ? axb::Wide::kKeys : axb::kKeys;
  CUtensorMap m[5] = {};
  const __nv_bfloat16 *qb = static_cast<const __nv_bfloat16 *>(q);
  if (!axb::map_of(&m[0], qb, dim, heads, n, per, q_ld, axb::kRows) ||
      !axb::map_of(&m[2], k, dim, kv_heads, skv, dim, (int64_t)kv_heads * dim, key_rows) ||
      !axb::map_of(&m[4], v, vdim, kv_heads, skv, vdim, (int64_t)kv_heads * vdim, 64))
    return AXB200_INTERNAL_ERROR;
  if (rot_dim > 0 && (!axb::map_of(&m[1], qb + dim, rot_dim, heads, n, per, q_ld, axb::kRows) ||
                      !axb::map_of(&m[3], rot, rot_dim, 1, skv, rot_ld, rot_ld, key_rows)))
    return AXB200_INTERNAL_ERROR;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (wide) return axb::launch_form<&axb::latent_prefill_wide_kernel>(2 * axb::kRows, axb::Wide::kThreads, axb::Wide::kSmem, m, p, st);
  auto go = [&](auto rot_tag) {
    constexpr int kRot = decltype(rot_tag)::value;
    if (dim > 64) return vdim > 64 ? axb::launch<2, 2, kRot>(m, p, st) : axb::launch<2, 1, kRot>(m, p, st);
    return vdim > 64 ? axb::launch<1, 2, kRot>(m, p, st) : axb::launch<1, 1, kRot>(m, p, st);
  };
  return rot_dim > 0 ? go(std::integral_constant<int, 1>{}) : go(std::integral_constant<int, 0>{});
}

}  // extern "C"

// Prefill attention in FLOAT32 on the 5th-generation tensor cores: the type that the reference's own
// ScaledDotProductAttention takes (src/ops/cuda/sequence.cu:451-472), head sizes up to 128.
//
// A float is the exact sum of three bf16 parts (8 bits each, round to nearest), so a product of two floats is nine products
// of parts, of which the three smallest (2^-26 of the whole) are left out: six tcgen05.mma products per Q.K^T and per P.V,
// smallest first, stand in for fp32 multiply-adds.  What remains is the tensor core's own accumulation, which truncates: a
// running sum over all keys would lose a bit per product step, so every tile of 64 keys starts O anew in tensor memory and
// the tiles are added up in fp32 registers, rescaled as the row's maximum moves.
//
// split_kernel lays K and V out as the tiles the second kernel reads: [64 keys][64 elements] boxes with 128-byte swizzle,
// three parts in a row, so that a tile is one bulk copy.  split_attn_kernel: one CTA per (128 query rows, head), longest
// blocks first:
//   warps 0-3   thread = row: scores from tensor memory, online softmax, the three parts of P over the scores
//   warps 4-7   thread = row: adds the finished tiles of O up in registers; writes the result
//   warp 8      issues the products: Q's parts and P's stay in tensor memory (as the A operand), so that shared memory feeds
//               B alone - at N = 64 a Q in shared memory would be re-read more often than the products can hide
//   warp 9      bulk copies of K and V tiles, two stages each
// Tensor memory at head size 128: Q 192 columns, two buffers of S / P 96 each, O 128 - all 512.
//
// Non-finite inputs (inf - inf among the parts) and magnitudes that have no three normal parts are noticed while splitting:
// the flags of their tiles make the FMA kernel of prefill_tiled.cu, launched behind, redo that KV head; else it returns at once.
//
// Bound by the tensor core: 12 products per tile.  Those of P.V take 66 cycles of the possible 64, those of Q.K^T, only 64 wide,
// 50 instead of 32.  1536 tokens, 16 / 8 heads of 128, causal: 744 us on the FMA pipe, 72 here (100 while a product's issue took
// 62 to 71 cycles, see elect_one), the error against 64 bits 4.2e-7 there and 1.9e-7 here.
#include <math.h>

#include <mutex>

#include "key_split.cuh"
#include "tcgen05.cuh"

namespace axb {

int sdpa_tiled_flagged(const void *q, const void *k, const void *v, void *out, int sq, int hq, int hkv, int d, int64_t skv,
                       int is_causal, const uint32_t *kv_flags, int kv_tiles, const uint32_t *q_flags, int q_blocks,
                       cudaStream_t st);

namespace {

constexpr int kRows = 128, kKeys = 64, kBox = kKeys * 64 * 2;
constexpr int kThreads = 320, kMmaWarp = 8, kLoadWarp = 9, kSplitThreads = 256;
constexpr float kLog2e = 1.4426950408889634f;

// kB: 64-wide blocks of the head size
template <int kB>
struct Layout {
  static constexpr int kPart = kB * kBox, kTile = 3 * kPart;
  static constexpr int kOffV = 2 * kTile, kOffCorr = 4 * kTile, kOffL = kOffCorr + 2 * kRows * 4, kOffBar = kOffL + 2 * kRows * 4;
  static constexpr int kSmem = kOffBar + 256;
  static constexpr int kQCols = 96 * kB, kSpCols = 96, kColO = kQCols + 2 * kSpCols;
};

struct Params {
  const float *q, *k, *v;
  float *out;
  uint8_t *tiles;                // K tiles by head, then V tiles
  uint32_t *kv_flags, *q_flags;  // one per tile (K's, then V's); one per block of query rows, by head
  int sq, hq, hkv, skv, causal, d, n_tiles, q_blocks;
  float scale_log2;
  unsigned long long wait_ns;
};

// Three bf16 parts of each of two floats; their sum is exact.
__device__ __forceinline__ void split3(float a, float b, uint32_t &h, uint32_t &m, uint32_t &l) {
  h = pack_bf16x2(a, b);
  const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xffff0000u);
  m = pack_bf16x2(ra, rb);
  l = pack_bf16x2(ra - __uint_as_float(m << 16), rb - __uint_as_float(m & 0xffff0000u));
}

// inf, NaN, what rounds to inf in bf16, and what is so small that its lower parts are subnormal (below 2^-100)
__device__ __forceinline__ bool unsplittable(float x) {
  const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
  return u >= 0x7f7f8000u || u - 1u < (27u << 23) - 1u;
}

template <int kB>
__global__ void __launch_bounds__(kSplitThreads)
split_kernel(const Params p) {
  grid_dependency_launch();
  const int t = blockIdx.x, hk = blockIdx.y, values = blockIdx.z;
  const float *src = values ? p.v : p.k;
  const size_t tile = ((size_t)values * p.hkv + hk) * p.n_tiles + t;
  uint8_t *dst = p.tiles + tile * Layout<kB>::kTile;
  bool bad = false;
#pragma unroll
  for (int i = 0; i < 2 * kB; ++i) {
    const int id = threadIdx.x + i * kSplitThreads, row = id / (8 * kB), c = id % (8 * kB), key = t * kKeys + row;
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (key < p.skv) {
      const float *at = src + ((size_t)key * p.hkv + hk) * p.d + c * 8;
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (c * 8 + u * 4 < p.d) *reinterpret_cast<float4 *>(x + u * 4) = *reinterpret_cast<const float4 *>(at + u * 4);
    }
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int u = 0; u < 8; ++u) bad |= unsplittable(x[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u) split3(x[2 * u], x[2 * u + 1], h[u], m[u], l[u]);
    uint8_t *box = dst + (c >> 3) * kBox + row * 128 + (((c & 7) ^ (row & 7)) << 4);
    *reinterpret_cast<uint4 *>(box) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(box + Layout<kB>::kPart) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4 *>(box + 2 * Layout<kB>::kPart) = make_uint4(l[0], l[1], l[2], l[3]);
  }
  const int any = __syncthreads_or(bad);
  if (threadIdx.x == 0) p.kv_flags[tile] = any;
}

template <int kB>
__global__ void __launch_bounds__(kThreads, 1)
split_attn_kernel(const Params p, const __grid_constant__ KeySplit split, const Partials partials) {
  using L = Layout<kB>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kOffBar);
  uint64_t *full_k = bars, *empty_k = bars + 2, *full_v = bars + 4, *empty_v = bars + 6;
  uint64_t *bar_s = bars + 8;                // S_j ready, per buffer
  uint64_t *bar_o = bars + 10;               // P_j . V_j done
  uint64_t *bar_p = bars + 11;               // P_j and its rescale factor written, per buffer; one arrival per warp
  uint64_t *bar_c = bars + 13;               // O_j added up, per parity of j; one arrival per warp
  uint64_t *bar_q = bars + 15, *bar_l = bars + 16;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 17);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 18);
  int *q_bad = reinterpret_cast<int *>(bars + 19);
  float *corr_s = reinterpret_cast<float *>(smem + L::kOffCorr), *l_s = reinterpret_cast<float *>(smem + L::kOffL);
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicOr(&g_error_word, AXB200_ERR_WAIT_TIMEOUT);
    return;
  }
  const int h = blockIdx.x % p.hq, unit = blockIdx.x / p.hq;
  const int qb = split.units ? split.block[unit] : (int)((gridDim.x - 1 - blockIdx.x) / p.hq);
  const int parts = split.units ? split.parts[unit] : 1;
  const int hk = h / (p.hq / p.hkv), q0 = qb * kRows;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int kv_end_max = p.causal ? min(min(q0 + kRows, p.sq), p.skv) : p.skv;
  int nkv = (kv_end_max + kKeys - 1) / kKeys, tile0 = 0;
  if (parts > 1) {
    tile0 = split_begin(nkv, split.part[unit], parts);
    nkv = split_begin(nkv, split.part[unit] + 1, parts) - tile0;
  }

  if (threadIdx.x == 0) {
    for (int i = 0; i < 11; ++i) mbar_init(&bars[i], 1);
    for (int i = 0; i < 4; ++i) mbar_init(&bar_p[i], 4);  // and bar_c
    mbar_init(bar_q, 4 * kB);
    mbar_init(bar_l, 4);
    *abort_flag = 0;
    *q_bad = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t tmem_sp = tmem + L::kQCols, tmem_o = tmem + L::kColO;
  const int row = threadIdx.x & (kRows - 1), t_row = q0 + row;

  // One 64-wide block of the thread's query row as three parts (q is no output of the splitting kernel, and everything
  // before that one has completed).
  auto load_q = [&](int block) {
    const float *src = p.q + ((size_t)t_row * p.hq + h) * p.d + block * 64;
    bool bad = false;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t part[3][16];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int c = half * 32 + u * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t_row < p.sq && block * 64 + c < p.d) x = *reinterpret_cast<const float4 *>(src + c);
        bad |= unsplittable(x.x) || unsplittable(x.y) || unsplittable(x.z) || unsplittable(x.w);
        split3(x.x, x.y, part[0][2 * u], part[1][2 * u], part[2][2 * u]);
        split3(x.z, x.w, part[0][2 * u + 1], part[1][2 * u + 1], part[2][2 * u + 1]);
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) tmem_st16(tmem + lane_base + i * 32 * kB + block * 32 + half * 16, part[i]);
    }
    if (bad) *q_bad = 1;
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_q);
  };

  if (warp == kLoadWarp) {
    if (lane == 0) {
      grid_dependency_wait();  // the tiles
      const uint8_t *k_tiles = p.tiles + ((size_t)hk * p.n_tiles + tile0) * L::kTile;
      const uint8_t *v_tiles = k_tiles + (size_t)p.hkv * p.n_tiles * L::kTile;
      bool ok = true;
      int nk = 0, nv = 0;  // copies begun
      auto load = [&](int j, int &n, const uint8_t *src, int off, uint64_t *full, uint64_t *empty) {
        const int s = j & 1;
        if (j >= 2) ok = mbar_wait_bounded(&empty[s], ((j >> 1) - 1) & 1, abort_flag, p.wait_ns);
        if (!ok) return;
        mbar_arrive_expect_tx(&full[s], L::kTile);
        bulk_load(smem + off + s * L::kTile, src + (size_t)j * L::kTile, L::kTile, &full[s]);
        n = j + 1;
      };
      load(0, nk, k_tiles, 0, full_k, empty_k);
      if (nkv > 1) load(1, nk, k_tiles, 0, full_k, empty_k);
      for (int j = 0; j < nkv && ok; ++j) {
        load(j, nv, v_tiles, L::kOffV, full_v, empty_v);
        if (ok && j + 2 < nkv) load(j + 2, nk, k_tiles, 0, full_k, empty_k);
      }
      if (*abort_flag) {  // no copy may still be on its way when the CTA leaves
        const unsigned long long t0 = global_timer_ns();
        auto drain = [&](uint64_t *bar, uint32_t parity) {
          while (!mbar_try_wait(bar, parity) && global_timer_ns() - t0 < 100000000ull) {
          }
        };
        for (int j = max(0, nk - 2); j < nk; ++j) drain(&full_k[j & 1], (j >> 1) & 1);
        for (int j = max(0, nv - 2); j < nv; ++j) drain(&full_v[j & 1], (j >> 1) & 1);
      }
    }
  } else if (warp == kMmaWarp) {
    // fp32 accumulate, bf16 operands, M = 128, A from tensor memory.  Q.K^T: N = 64 keys, B K-major; P.V: N = the head size
    // to a multiple of 16, B MN-major
    const uint32_t bf16 = (1u << 4) | (1u << 7) | (1u << 10) | ((kRows >> 4) << 24);
    const int d_steps = (p.d + 15) / 16;
    const uint32_t idesc_qk = bf16 | ((kKeys >> 3) << 17), idesc_pv = bf16 | (1u << 16) | ((uint32_t)(d_steps * 2) << 17);
    const uint64_t dk = smem_desc(smem_u32(smem), 16, 1024), dv = smem_desc(smem_u32(smem + L::kOffV), kBox, 1024);
    constexpr int kA[6] = {0, 2, 1, 0, 1, 0}, kC[6] = {2, 0, 1, 1, 0, 0};  // parts of A and B, smallest products first
    auto issue_s = [&](int j) -> bool {
      const int s = j & 1;
      if (!mbar_wait_warp(&full_k[s], (j >> 1) & 1, abort_flag, p.wait_ns)) return false;
      tc_fence_after();
      const uint64_t dks = dk + (uint64_t)(s * (L::kTile >> 4));
      if (elect_one()) {
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int ks = 0; ks < 4 * kB; ++ks) {
            if (ks >= d_steps) break;
            umma_f16_ts(tmem_sp + s * L::kSpCols, tmem + kA[i] * 32 * kB + ks * 8,
                        dks + (uint64_t)((kC[i] * L::kPart + (ks >> 2) * kBox + (ks & 3) * 32) >> 4), idesc_qk, i > 0 || ks > 0);
          }
        umma_commit(&bar_s[s]);
        umma_commit(&empty_k[s]);
      }
      return true;
    };
    bool ok = mbar_wait_warp(bar_q, 0, abort_flag, p.wait_ns) && issue_s(0);
    if (ok && nkv > 1) ok = issue_s(1);
    for (int j = 0; j < nkv && ok; ++j) {
      const int s = j & 1;
      ok = mbar_wait_warp(&bar_p[s], (j >> 1) & 1, abort_flag, p.wait_ns) &&
           mbar_wait_warp(&full_v[s], (j >> 1) & 1, abort_flag, p.wait_ns) &&
           (j == 0 || mbar_wait_warp(&bar_c[s ^ 1], ((j - 1) >> 1) & 1, abort_flag, p.wait_ns));
      if (!ok) break;
      tc_fence_after();
      const uint64_t dvs = dv + (uint64_t)(s * (L::kTile >> 4));
      if (elect_one()) {
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int ks = 0; ks < kKeys / 16; ++ks)
            umma_f16_ts(tmem_o, tmem_sp + s * L::kSpCols + kA[i] * 32 + ks * 8,
                        dvs + (uint64_t)((kC[i] * L::kPart + ks * 2048) >> 4), idesc_pv, i > 0 || ks > 0);
        umma_commit(bar_o);
        umma_commit(&empty_v[s]);
      }
      // S_{j+2} takes the place of P_j: products of unlike shapes have no order of their own, so P_j.V_j is waited for
      if (j + 2 < nkv) ok = mbar_wait_warp(bar_o, j & 1, abort_flag, p.wait_ns) && issue_s(j + 2);
    }
  } else if (warp < 4) {
    // ---- softmax: thread = row ----
    if (kB == 2) load_q(1);
    const int kv_end = p.causal ? min(t_row + 1, p.skv) : p.skv;
    const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < nkv && ok; ++j) {
      const int s = j & 1;
      ok = mbar_wait_warp(&bar_s[s], (j >> 1) & 1, abort_flag, p.wait_ns);
      if (!ok) break;
      tc_fence_after();
      const uint32_t sp = tmem_sp + s * L::kSpCols + lane_base;
      uint32_t sr[2][32];
      tmem_ld32_async(sp, sr[0]);
      tmem_ld32_async(sp + 32, sr[1]);
      tmem_wait_ld();
      const int n0 = (tile0 + j) * kKeys;
      if (n0 + kKeys > kv_end) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (n0 + c * 32 + i >= kv_end) sr[c][i] = 0xff800000u;  // -inf
      }
      const float m_new = fmaxf(m_run, row_max(sr)), m_safe = m_new == -INFINITY ? 0.f : m_new;
      const float corr = fast_exp2((m_run - m_safe) * p.scale_log2);  // 0 at the first tile
      m_run = m_new;
      const uint64_t shift2 = pack_f32x2(-m_safe, -m_safe);
      uint64_t sum2[4] = {0, 0, 0, 0};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t part[3][16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const uint64_t x2 = add_f32x2(pack_f32x2(__uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1])), shift2);
          const float2 x = unpack_f32x2(mul_f32x2(x2, scale2));
          const float a = fast_exp2(x.x), b = fast_exp2(x.y);
          sum2[(i >> 1) & 3] = add_f32x2(sum2[(i >> 1) & 3], pack_f32x2(a, b));
          split3(a, b, part[0][i >> 1], part[1][i >> 1], part[2][i >> 1]);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) tmem_st16(sp + i * 32 + c * 16, part[i]);
      }
      const float2 sum = unpack_f32x2(add_f32x2(add_f32x2(sum2[0], sum2[1]), add_f32x2(sum2[2], sum2[3])));
      l_run = l_run * corr + (sum.x + sum.y);
      if (j >= 2) {  // the factor of tile j - 2 has been read
        ok = mbar_wait_warp(&bar_c[s], ((j >> 1) - 1) & 1, abort_flag, p.wait_ns);
        if (!ok) break;
      }
      corr_s[s * kRows + row] = corr;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p[s]);
    }
    l_s[row] = l_run;
    l_s[kRows + row] = m_run * p.scale_log2;
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_l);
  } else {
    // ---- the sum over tiles: thread = row ----
    load_q(0);
    uint64_t acc[32 * kB];
#pragma unroll
    for (int i = 0; i < 32 * kB; ++i) acc[i] = 0;
    bool ok = true;
    for (int j = 0; j < nkv && ok; ++j) {
      const int s = j & 1;
      ok = mbar_wait_warp(&bar_p[s], (j >> 1) & 1, abort_flag, p.wait_ns);
      if (!ok) break;
      const float corr = corr_s[s * kRows + row];
      const uint64_t corr2 = pack_f32x2(corr, corr);
      ok = mbar_wait_warp(bar_o, j & 1, abort_flag, p.wait_ns);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2 * kB; ++c) {
        if (c * 32 >= p.d) break;
        uint32_t r[32];
        tmem_ld32(tmem_o + lane_base + c * 32, r);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          acc[c * 16 + i] = fma_f32x2(acc[c * 16 + i], corr2, pack_f32x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_c[s]);
    }
    if (ok) ok = mbar_wait_warp(bar_l, 0, abort_flag, p.wait_ns);
    if (ok && t_row < p.sq) {
      const float l = l_s[row];
      float inv = l > 0.f ? 1.0f / l : 0.f;
      float *dst = p.out + ((size_t)t_row * p.hq + h) * p.d;
      if (parts > 1) {  // un-normalised
        const size_t at = ((size_t)(unit - split.first) * p.hq + h) * kRows + row;
        partials.ml[at] = make_float2(l_s[kRows + row], l);
        dst = partials.sums + at * p.d;
        inv = 1.f;
      }
#pragma unroll
      for (int i = 0; i < 16 * kB; ++i) {
        if (i * 4 >= p.d) break;
        const float2 a = unpack_f32x2(acc[2 * i]), b = unpack_f32x2(acc[2 * i + 1]);
        *reinterpret_cast<float4 *>(dst + i * 4) = make_float4(a.x * inv, a.y * inv, b.x * inv, b.y * inv);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) p.q_flags[h * p.q_blocks + qb] = *q_bad;  // the same from every part
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }
int blocks_of(int d) { return d > 64 ? 2 : 1; }
size_t tile_bytes(int hkv, int64_t n_tiles, int d) { return (size_t)2 * hkv * n_tiles * 3 * blocks_of(d) * kBox; }
size_t kv_flag_bytes(int hkv, int64_t n_tiles) { return up256((size_t)2 * hkv * n_tiles * 4); }

// A tile of 64 keys takes 2 to 3 us of a block, a block three tiles more (Q's parts, the first copies, the result).  1536 rows of 16
// heads of 128, not causal: 176 us whole, 140 in parts; 4096 rows of 2 heads, causal: 208 and 91.  Where the SMs are nearly full
// a division gains nothing (1536 rows of 16 heads, causal: the attention kernel alone 92 us both, before the joining), hence the five tiles.
KeySplit split_plan(int sq, int hq, int64_t skv, int is_causal) {
  const auto tiles = [&](int b) {
    const int64_t last = ((int64_t)b + 1) * kRows, end = last < sq ? last : sq;
    return (int)(((is_causal && end < skv ? end : skv) + kKeys - 1) / kKeys);
  };
  return plan_key_split(((int64_t)sq + kRows - 1) / kRows, hq, is_causal != 0, 3.f, 5.f, tiles, kSms,
                        KeySplit::kMostEntries);
}

// Keys that some row sees: the others are not split into parts (16 rows over 8192 keys, 16 / 8 heads of 128, causal: 41 us with all).
int64_t visible_keys(int sq, int64_t skv, int is_causal) { return is_causal && skv > sq ? sq : skv; }

template <int kB>
int launch(const Params &p, void *parts_at, cudaStream_t st) {
  static std::mutex mu;
  static bool opted[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return AXB200_DEVICE_ERROR;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!opted[dev]) {
      if (cudaFuncSetAttribute(split_attn_kernel<kB>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<kB>::kSmem) != cudaSuccess)
        return AXB200_DEVICE_ERROR;
      opted[dev] = true;
    }
  }
  split_kernel<kB><<<dim3(p.n_tiles, p.hkv, 2), kSplitThreads, 0, st>>>(p);
  if (cudaGetLastError() != cudaSuccess) return AXB200_DEVICE_ERROR;
  const KeySplit split = split_plan(p.sq, p.hq, p.skv, p.causal);
  const Partials partials = partials_at(parts_at, split, p.hq, kRows);
  const int rc = launch_dependent(split_attn_kernel<kB>, dim3((unsigned)p.hq * (split.units ? split.units : p.q_blocks)), dim3(kThreads),
                                  Layout<kB>::kSmem, st, p, split, partials);
  if (rc != AXB200_OK || split.units == 0) return rc;
  return launch_dependent(join_parts_kernel<float, kRows>, dim3((unsigned)p.hq * (kRows / 8), split.divided_blocks), dim3(256), 0, st,
                          split, partials, p.out, p.sq, p.hq, p.d);
}

}  // namespace

// Scratch that the split form wants for this problem; 0 where the FMA kernel serves it: problems that are one launch of few key
// tiles in a row there, waves of blocks times tiles of keys.  48 rows and keys, 16 / 8 heads of 128: 23 us in one launch, 32 in
// three.  100 rows and keys: 55 and 29; 2000 rows, 64 keys: 70 and 39; 16 rows, 128 keys, 2 heads of 64: 25 and 28.
size_t sdpa_split_scratch_bytes(int sq, int hq, int hkv, int d, int64_t skv, int is_causal) {
  skv = visible_keys(sq, skv, is_causal);
  const int64_t in_a_row = (((int64_t)sq * hq + 128 * 148 - 1) / (128 * 148)) * ((skv + kKeys - 1) / kKeys);
  const int64_t rows = (int64_t)sq * (hq / hkv);
  if (d % 4 || d > 128 || sq < 16 || hkv > 65535 || in_a_row < (rows >= kRows ? 2 : 3)) return 0;
  const int64_t n_tiles = (skv + kKeys - 1) / kKeys, q_blocks = ((int64_t)sq + kRows - 1) / kRows;
  const size_t parts = key_split_bytes(split_plan(sq, hq, skv, is_causal), hq, kRows, d);
  const size_t total = up256((size_t)hq * q_blocks * 4) + kv_flag_bytes(hkv, n_tiles) +
                       tile_bytes(hkv, n_tiles, d) + parts;
  return total <= kMostScratch ? total : 0;  // 170 K tokens of 8 heads of 128
}

// q, k, v, out and scratch on 16-byte boundaries; scratch of the size above.
int sdpa_split(const void *q, const void *k, const void *v, void *out, int sq, int hq, int hkv, int d, int64_t skv, int is_causal,
               void *scratch, cudaStream_t st) {
  skv = visible_keys(sq, skv, is_causal);
  Params p{};
  p.q = static_cast<const float *>(q);
  p.k = static_cast<const float *>(k);
  p.v = static_cast<const float *>(v);
  p.out = static_cast<float *>(out);
  p.sq = sq;
  p.hq = hq;
  p.hkv = hkv;
  p.skv = (int)skv;
  p.causal = is_causal != 0;
  p.d = d;
  p.n_tiles = (int)((skv + kKeys - 1) / kKeys);
  p.q_blocks = (sq + kRows - 1) / kRows;
  p.scale_log2 = (1.0f / sqrtf((float)d)) * kLog2e;
  p.wait_ns = wait_limit_ns();
  uint8_t *at = static_cast<uint8_t *>(scratch);
  p.q_flags = reinterpret_cast<uint32_t *>(at);
  at += up256((size_t)hq * p.q_blocks * 4);
  p.kv_flags = reinterpret_cast<uint32_t *>(at);
  p.tiles = at + kv_flag_bytes(hkv, p.n_tiles);
  void *parts_at = p.tiles + tile_bytes(hkv, p.n_tiles, d);
  const int status = blocks_of(d) == 2 ? launch<2>(p, parts_at, st) : launch<1>(p, parts_at, st);
  if (status != AXB200_OK) return status;
  return sdpa_tiled_flagged(q, k, v, out, sq, hq, hkv, d, skv, is_causal, p.kv_flags, p.n_tiles, p.q_flags, p.q_blocks, st);
}

}  // namespace axb

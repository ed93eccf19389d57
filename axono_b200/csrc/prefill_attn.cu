// Prefill attention (many queries, optional causal mask) for sm_100a on the 5th-generation tensor
// cores.  Replaces the reference's ScaledDotProductAttention / SdpaKernel
// (src/ops/cuda/sequence.cu:105-163,451-472), whose scores live in shared memory (skv*4 bytes, so it
// cannot pass ~12 K keys) and whose P.V loop is thread-serial.
//
// fp16: one CTA (four softmax warps + an MMA warp + a TMA warp, two CTAs per SM) per
// (block of 128 query rows, query head).  Q, K and V tiles are staged by TMA with 128-byte swizzle;
// S = Q.K^T (128 x 64 per tile of 64 keys) and O += P.V are tcgen05.mma (cta_group::1, kind::f16) with
// the accumulators in tensor memory (two S buffers and O: 256 columns per CTA); thread t owns query
// row t: it reads its scores with tcgen05.ld, does the online softmax in registers, writes P (fp16
// pairs) back over its S row with tcgen05.st - P.V takes its A operand from tensor
// memory, so P never crosses shared memory - and rescales its O row in tensor memory when the running
// maximum moves by more than a threshold.  One lane each of two more warps launches the MMAs and the
// TMA loads; the sides meet only on mbarriers (tcgen05.commit for MMA completion).  K/V tiles are
// multi-buffered and S is computed two tiles ahead, so tensor core and softmax overlap.  Every wait
// is bounded.  FLOAT32 goes to prefill_f32.cu, head sizes that are not a multiple of 8 up to 128 to prefill_tiled.cu, and what
// that does not take to the decode kernels, row by row.
//
// Semantics as the reference's CPU op (src/ops/cpu/sequence.cpp:236-301): q (sq,hq,d), k/v
// (skv,hkv,d) token-major, head h reads KV head h / (hq/hkv), scale 1/sqrt(d); with is_causal row t
// sees keys [0, t] when skv >= t+1 and all keys otherwise.
#include <math.h>

#include <mutex>
#include <type_traits>

#include "key_split.cuh"
#include "tcgen05.cuh"

namespace axb {

// Row-by-row evaluation on the decode kernels (defined beside them).
int sdpa_rows_fallback(const void *q, const void *k, const void *v, void *out, int sq, int hq, int hkv,
                       int d, int64_t skv, int is_causal, int dtype, void *workspace,
                       size_t workspace_bytes, cudaStream_t st);
size_t sdpa_rows_workspace_bytes(int sq, int hq, int hkv, int d, int64_t skv);
// Tiled evaluation on the FMA pipe (prefill_tiled.cu): what the tensor-core kernels do not take.
bool sdpa_tiled_supported(int sq, int hq, int hkv, int d, int64_t skv);
int sdpa_tiled(const void *q, const void *k, const void *v, void *out, int sq, int hq, int hkv, int d, int64_t skv,
               int is_causal, int dtype, cudaStream_t st);
// FLOAT32 on the tensor cores (prefill_f32.cu); the scratch it wants is 0 where it does not apply.
size_t sdpa_split_scratch_bytes(int sq, int hq, int hkv, int d, int64_t skv, int is_causal);
int sdpa_split(const void *q, const void *k, const void *v, void *out, int sq, int hq, int hkv, int d, int64_t skv, int is_causal,
               void *scratch, cudaStream_t st);

namespace {

constexpr int kBlockM = 128, kBlockN = 64, kD = 128;
constexpr int kSoftmaxWarps = 4;
constexpr int kMmaWarp = kSoftmaxWarps, kLoadWarp = kSoftmaxWarps + 1;
constexpr int kThreads = (kSoftmaxWarps + 2) * 32;  // + the MMA warp and the TMA warp
constexpr int kQTileBytes = kBlockM * kD * 2;   // 32 KB: two swizzled boxes of [128 rows][64 halves]
constexpr int kKvTileBytes = kBlockN * kD * 2;  // 16 KB: two swizzled boxes of [64 rows][64 halves]
constexpr int kKStages = 3, kVStages = 2;  // K runs ahead of V: S is computed two tiles before P.V
constexpr int kOffQ = 0, kOffK = kQTileBytes, kOffV = kOffK + kKStages * kKvTileBytes;
constexpr int kOffBar = kOffV + kVStages * kKvTileBytes;
constexpr int kSmemBytes = kOffBar + 256;  // 112 KB + barriers: two CTAs per SM
constexpr float kLog2e = 1.4426950408889634f;

struct PrefillParams {
  void *out;
  int sq, hq, hkv, skv, causal, d;
  float scale_log2;
  const __half *q, *k, *v;  // for rows that the tensor core cannot finish
};

constexpr float kLazyLog2 = 8.0f;

// What a kernel of whole blocks takes in the place of a plan: 2 KB of arguments cost a launch of 16 to 64 rows 0.3 of 4.8 us.
struct WholeBlocks {};

// Two fp16 parts of a pair of weights: hi + lo holds 22 bits of each (2^-24 absolute where a part is subnormal).
__device__ __forceinline__ uint32_t split_half2(float a, float b, uint32_t &lo) {
  const __half2 hi = __floats2half2_rn(a, b);
  const float2 f = __half22float2(hi);
  lo = pack_half2(a - f.x, b - f.y);
  return *reinterpret_cast<const uint32_t *>(&hi);
}

// The tensor core adds up by truncation: a running sum over all keys loses about a quarter of a unit of its last bit, towards zero,
// with each of the 8 products of a tile of 64 keys, two parts of the weights times 64 / 16 (1.8e-5 of the values by 8192 keys, 6e-5
// where these have a common offset).  So every kFlushTiles tiles, 1024 keys, O starts anew, and what it held joins a thread's sums
// in local memory, kept in fp32 with the rescaling they still owe.  (Out of line, so that the sums stay out of the registers of the
// loop that calls it.)  8192 keys, heads of 64: error 2.084e-4 without, 2.075e-4 so, as on the FMA pipe; with a common offset
// 2.316e-4, 2.239e-4 and 2.238e-4.  It costs 4 % of the time, twice as often 8 %.
constexpr int kFlushTiles = 16;
__device__ __noinline__ void flush_sums(float4 *sums, uint32_t tmem_o, int d, bool first, float owed) {
#pragma unroll 1
  for (int c = 0; c * 32 < d; ++c) {
    uint32_t r[32];
    tmem_ld32(tmem_o + c * 32, r);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 old = first ? make_float4(0.f, 0.f, 0.f, 0.f) : sums[c * 8 + i];
      sums[c * 8 + i] = make_float4(fmaf(old.x, owed, __uint_as_float(r[4 * i])), fmaf(old.y, owed, __uint_as_float(r[4 * i + 1])),
                                    fmaf(old.z, owed, __uint_as_float(r[4 * i + 2])), fmaf(old.w, owed, __uint_as_float(r[4 * i + 3])));
    }
  }
}

// One row over the keys [key0, key1) with a weight of one part, as the definition has it.  A weight in two parts meets V twice, and
// where V is infinite hi * V + lo * V is NaN (lo may be 0 or negative) though the row's value is +-inf; and every row of a block
// multiplies the V of all its tiles, also those that its mask hides.  So a thread whose row is not finite does it over - only
// inputs that are not finite lead here.  ml: where un-normalised sums go instead of the result.
__device__ __noinline__ void redo_narrow_row(const PrefillParams &p, int t_row, int h, int key0, int key1, float *sums, float2 *ml) {
  constexpr int kMost = kD / 8 - 1;  // 16-byte pieces of a row
  const int hk = h / (p.hq / p.hkv), pieces = p.d / 8;
  const size_t step = (size_t)p.hkv * p.d;
  const __half *k = p.k + (size_t)hk * p.d, *v = p.v + (size_t)hk * p.d;
  const uint4 *from = reinterpret_cast<const uint4 *>(p.q + ((size_t)t_row * p.hq + h) * p.d);
  uint4 q[kMost];
#pragma unroll
  for (int c = 0; c < kMost; ++c)
    if (c < pieces) q[c] = from[c];
  const auto dot2 = [](uint32_t a, uint32_t b, float s) {
    const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(&a)), y = __half22float2(*reinterpret_cast<const __half2 *>(&b));
    return fmaf(x.y, y.y, fmaf(x.x, y.x, s));
  };
  const auto score = [&](int key) {
    const uint4 *row = reinterpret_cast<const uint4 *>(k + key * step);
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < kMost; ++c)
      if (c < pieces) {
        const uint4 x = row[c];
        s = dot2(q[c].w, x.w, dot2(q[c].z, x.z, dot2(q[c].y, x.y, dot2(q[c].x, x.x, s))));
      }
    return s;
  };
  float m = -INFINITY;
  for (int key = key0; key < key1; ++key) m = fmaxf(m, score(key));
  for (int c0 = 0; c0 < p.d; c0 += 32) {
    float acc[32], l = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    for (int key = key0; key < key1; ++key) {
      const float s = score(key), w = s == -INFINITY ? 0.f : exp2f((s - m) * p.scale_log2);
      l += w;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + u * 8 < p.d) {
          const uint4 x = *reinterpret_cast<const uint4 *>(v + key * step + c0 + u * 8);
          const uint32_t part[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&part[i]));
            acc[u * 8 + 2 * i] = fmaf(w, f.x, acc[u * 8 + 2 * i]);
            acc[u * 8 + 2 * i + 1] = fmaf(w, f.y, acc[u * 8 + 2 * i + 1]);
          }
        }
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    __half *out = reinterpret_cast<__half *>(p.out) + ((size_t)t_row * p.hq + h) * p.d + c0;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (c0 + i < p.d) {
        if (ml)
          sums[c0 + i] = acc[i];
        else
          out[i] = __float2half_rn(acc[i] * inv);
      }
    if (ml) *ml = make_float2(m * p.scale_log2, l);
  }
}

// 192 threads.  Warps 0-3 (softmax): thread t owns query row t of the block (tensor-memory lane t)
// and all 64 key columns of a tile, so the row maximum and sum need no exchange.  Warp 4 issues every MMA from descriptors built
// once; warp 5 (one lane) issues every TMA load, K and V tiles
// in rings of 3 and 2 stages freed by tcgen05.commit - a single thread doing both spent two thirds of
// a tile's time on instruction issue.  The sides meet only on mbarriers (full/empty per stage; bar_s:
// S_j ready; bar_p: P_j written; bar_o: P_j.V_j done; bar_fin: the last P.V done).  Software pipeline:
// S_{j+2} = Q.K_{j+2}^T is issued once P_j.V_j has completed, while the softmax warps are already in
// tile j+1 (two S buffers).  Two CTAs share an SM (112 KB of shared memory and 256 tensor-memory
// columns each).
// Blocks start in the order of their key tiles over all heads, so that under a causal mask the last ones to start are the short
// ones (or in the order of a plan that divides the keys of some, key_split.cuh).
// Bound by the tensor core: a tile's 8 products of Q.K^T take 50 cycles each (Q is read from shared memory for 64 columns at a time) and
// its 4 of P.V 66, 1330 cycles for the tiles of the two CTAs of an SM; a tile takes 1410.  One CTA per SM with two blocks of 128
// rows and tiles of 128 keys needed a fifth less of the tensor core, but had no room for scores ahead of the softmax: a tile's
// chain of 3600 cycles was its time.  16 / 8 heads of 128, many calls in a row (under the power cap; ten calls after a pause take 235
// us at 8192): 8192 tokens, causal, 283 us in that form, 266 here - that form issued behind elect_one, as here, took 263 to 267, so 8192
// tokens owe their gain to the issue; 2048: 42 and 30; 4096, not causal: 131 and 119 (1150 TFLOP/s).
// kNarrow: head sizes below 128 (multiples of 8).  They ran on the FMA pipe at first, whose weights were fp32, so P enters
// P.V as two fp16 parts here: P's two parts take the two halves of an S buffer, and a tile costs 8 products for P.V instead of 4, as
// wide as the head.  Elements past the head size are zeros that TMA fills in; head sizes up to 64 leave the second 64-wide block
// of every tile out.  2700 x 2700 keys, 16 heads of 64, not causal: 1921 us on the FMA pipe, 88 with two blocks per CTA (whose P.V
// had to be 128 wide), 66 here, the joining included; the same error against 64 bits (2.1e-4, the rounding of the result).
template <bool kNarrow, typename Split>
__global__ void __launch_bounds__(kThreads, 2)
prefill_attn_f16_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ PrefillParams p,
                        const __grid_constant__ Split split, const Partials partials) {
  constexpr bool kDivided = std::is_same<Split, KeySplit>::value;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kOffBar);
  uint64_t *bar_q = bars;                                    // Q landed
  uint64_t *full_k = bars + 1, *empty_k = bars + 4;          // per K stage: tile landed / S that read it done
  uint64_t *full_v = bars + 7, *empty_v = bars + 9;          // per V stage: tile landed / P.V that read it done
  uint64_t *bar_s = bars + 11, *bar_o = bars + 13;           // S_j ready (per S buffer); P_j.V_j done
  uint64_t *bar_fin = bars + 14;  // the last P.V: the softmax warps skip phases of bar_o, a parity wait there would alias
  uint64_t *bar_p = bars + 15;    // P_j written (per S buffer), one arrival per softmax warp
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 17);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 18);

  // the swizzled tiles need a 1024-byte aligned base; refuse to run otherwise (nothing is written)
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicOr(&g_error_word, AXB200_ERR_WAIT_TIMEOUT);
    return;
  }
  // heaviest blocks of all heads first: under a causal mask the last query block has the most key tiles
  // (or in the plan's order, where keys are divided)
  const int h = blockIdx.x % p.hq, unit = blockIdx.x / p.hq;
  int qb, part = 0, parts = 1;
  if constexpr (kDivided) {
    const KeyUnit u = key_unit(split, unit);
    qb = u.block, part = u.part, parts = u.parts;
  } else {
    qb = (int)((gridDim.x - 1 - blockIdx.x) / p.hq);
  }
  const int hk = h / (p.hq / p.hkv);
  const int q0 = qb * kBlockM;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int t_last = min(q0 + kBlockM, p.sq) - 1;
  const int kv_end_max = p.causal ? min(t_last + 1, p.skv) : p.skv;  // reference rule: min(t+1, skv)
  int nkv = (kv_end_max + kBlockN - 1) / kBlockN, tile0 = 0;
  size_t at = 0;  // of the rows of a divided block, their places among the partial results
  if constexpr (kDivided) {
    if (parts > 1) {
      tile0 = split_begin(nkv, part, parts);
      nkv = split_begin(nkv, part + 1, parts) - tile0;
    }
    at = ((size_t)(unit - split.first) * p.hq + h) * kBlockM;
  }
  const bool two_blocks = !kNarrow || p.d > 64;
  const uint32_t kv_bytes = two_blocks ? kKvTileBytes : kKvTileBytes / 2;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 15; ++i) mbar_init(&bars[i], 1);
    // one per S buffer: a softmax warp may run a tile ahead of the others, and with a single barrier
    // its second arrival would complete the phase the slower warps have not reached
    mbar_init(&bar_p[0], kSoftmaxWarps);
    mbar_init(&bar_p[1], kSoftmaxWarps);
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
  const uint32_t tmem_base = *tmem_slot, tmem_o = tmem_base + 128;  // S buffers at columns 0 and 64

  if (warp == kLoadWarp) {
    // ================= TMA warp (one lane): Q, then K and V tiles in the order they are consumed =====
    if (lane == 0) {
      tma_prefetch_descriptor(&tmQ);
      tma_prefetch_descriptor(&tmK);
      tma_prefetch_descriptor(&tmV);
      mbar_arrive_expect_tx(bar_q, two_blocks ? kQTileBytes : kQTileBytes / 2);
      tma_load_3d(smem + kOffQ, &tmQ, bar_q, 0, h, q0);  // rows past sq are zero-filled
      if (two_blocks) tma_load_3d(smem + kOffQ + kQTileBytes / 2, &tmQ, bar_q, 64, h, q0);
      bool ok = true;
      int nk = 0, nv = 0;  // tiles asked for
      auto load = [&](int &n, int stages, int off, const CUtensorMap &map, uint64_t *full, uint64_t *empty) {
        const int j = n, s = j % stages;
        if (j >= stages) ok = ok && mbar_wait_bounded(&empty[s], (j / stages - 1) & 1, abort_flag);
        if (!ok) return;
        uint8_t *dst = smem + off + s * kKvTileBytes;
        mbar_arrive_expect_tx(&full[s], kv_bytes);
        tma_load_3d(dst, &map, &full[s], 0, hk, (tile0 + j) * kBlockN);
        if (two_blocks) tma_load_3d(dst + kKvTileBytes / 2, &map, &full[s], 64, hk, (tile0 + j) * kBlockN);
        ++n;
      };
      // consumption order is S_0 S_1 (PV_0 S_2) (PV_1 S_3) ...: K_0 K_1 K_2 V_0 K_3 V_1 ...
      while (nk < 2 && nk < nkv) load(nk, kKStages, kOffK, tmK, full_k, empty_k);
      while (nv < nkv && ok) {
        if (nk < nkv) load(nk, kKStages, kOffK, tmK, full_k, empty_k);
        load(nv, kVStages, kOffV, tmV, full_v, empty_v);
      }
      if (*abort_flag) {  // no copy may still be on its way when the CTA leaves
        const unsigned long long t0 = global_timer_ns();
        auto drain = [&](uint64_t *bar, uint32_t parity) {
          while (!mbar_try_wait(bar, parity) && global_timer_ns() - t0 < 100000000ull) {
          }
        };
        drain(bar_q, 0);
        for (int t = max(0, nk - kKStages); t < nk; ++t) drain(&full_k[t % kKStages], (t / kKStages) & 1);
        for (int t = max(0, nv - kVStages); t < nv; ++t) drain(&full_v[t % kVStages], (t / kVStages) & 1);
      }
    }
  } else if (warp == kMmaWarp) {
    // ================= MMA warp: all lanes walk, one issues =================
    {
      // instruction descriptors: fp32 accumulate, fp16 operands, M = 128.  Q.K^T: N = 64 keys, B
      // K-major; P.V: N = the head size to a multiple of 16, B MN-major (a V tile is [keys][d], d contiguous)
      const int d_steps = kNarrow ? (p.d + 15) / 16 : kD / 16;
      const uint32_t idesc_qk = (1u << 4) | ((kBlockN >> 3) << 17) | ((kBlockM >> 4) << 24);
      const uint32_t idesc_pv = (1u << 4) | (1u << 16) | ((uint32_t)(d_steps * 2) << 17) | ((kBlockM >> 4) << 24);
      // Shared-memory descriptors are built once: stepping a tile, a stage or 16 elements along K only
      // adds to the 14-bit address field (bytes >> 4), which cannot carry out of it (addresses < 256 KB).
      const uint64_t dq = smem_desc(smem_u32(smem + kOffQ), 16, 1024);
      const uint64_t dk = smem_desc(smem_u32(smem + kOffK), 16, 1024);
      const uint64_t dv = smem_desc(smem_u32(smem + kOffV), kKvTileBytes / 2, 1024);
      // S_j = Q . K_j^T into S buffer j&1; arrives on bar_s[j&1], and frees the K stage when done
      auto issue_s = [&](int j) -> bool {
        const int s = j & 1, sk = j % kKStages;
        if (!mbar_wait_warp(&full_k[sk], (j / kKStages) & 1, abort_flag, kWaitNanos)) return false;
        tc_fence_after();
        const uint64_t dks = dk + (uint64_t)(sk * (kKvTileBytes >> 4));
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {  // head_dim 128 = 8 steps of 16; each 64-wide half of d is one box
            if (kNarrow && ks >= d_steps) break;
            const uint32_t q_off = (ks >> 2) * (kQTileBytes / 2) + (ks & 3) * 32;
            const uint32_t k_off = (ks >> 2) * (kKvTileBytes / 2) + (ks & 3) * 32;
            umma_f16(tmem_base + s * kBlockN, dq + (q_off >> 4), dks + (k_off >> 4), idesc_qk, ks > 0);
          }
          umma_commit(&bar_s[s]);
          umma_commit(&empty_k[sk]);
        }
        return true;
      };
      bool ok = mbar_wait_warp(bar_q, 0, abort_flag, kWaitNanos) && issue_s(0);
      if (ok && nkv > 1) ok = issue_s(1);
      for (int j = 0; j < nkv && ok; ++j) {
        // P_j stands in S buffer j&1 (in the first 32 columns, its second part in the others): O += P_j . V_j
        const int sv = j % kVStages;
        ok = mbar_wait_warp(&bar_p[j & 1], (j >> 1) & 1, abort_flag, kWaitNanos) &&
             mbar_wait_warp(&full_v[sv], (j / kVStages) & 1, abort_flag, kWaitNanos);
        if (!ok) break;
        tc_fence_after();
        const uint64_t dvs = dv + (uint64_t)(sv * (kKvTileBytes >> 4));
        const uint32_t p_tmem = tmem_base + (j & 1) * kBlockN;
        if (elect_one()) {
#pragma unroll
          for (int part = 0; part < (kNarrow ? 2 : 1); ++part)
#pragma unroll
            for (int ks = 0; ks < kBlockN / 16; ++ks)
              // V as the MN-major B operand: the two 64-wide d atoms are one box (8 KB) apart, 8-key
              // groups 1 KB apart, 16 keys per instruction = 2 KB
              umma_f16_ts(tmem_o, p_tmem + part * 32 + ks * 8, dvs + (uint64_t)(ks * (2048 >> 4)), idesc_pv,
                          (kNarrow ? j % kFlushTiles != 0 : j > 0) || part > 0 || ks > 0);
          umma_commit(bar_o);
          umma_commit(&empty_v[sv]);
          if (j == nkv - 1) umma_commit(bar_fin);
        }
        if (j + 2 < nkv) {
          // P_j.V_j complete: P_j is consumed, so S_{j+2} may overwrite S buffer j&1 (queueing it behind
          // P_j.V_j instead would lean on issue-order execution, which is documented only for MMAs of
          // one shape; measured no faster)
          ok = mbar_wait_warp(bar_o, j & 1, abort_flag, kWaitNanos);
          if (!ok) break;
          ok = issue_s(j + 2);
        }
      }
    }
  } else {
    // ================= softmax warps =================
    const int row = threadIdx.x;
    const int t_row = q0 + row;
    const int kv_end = p.causal ? min(t_row + 1, p.skv) : p.skv;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    float m_run = -INFINITY, l_run = 0.f;
    float4 sums[kNarrow ? kD / 4 : 1];  // what flush_sums has taken, and the factor it has to be multiplied with
    float owed = 1.f;
    bool ok = true;
    for (int j = 0; j < nkv && ok; ++j) {
      const int sb = j & 1;
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bar_s[sb], (j >> 1) & 1, abort_flag));
      if (!ok) break;
      tc_fence_after();
      // ---- this thread's row of scores: 64 keys ----
      const int n0 = (tile0 + j) * kBlockN;
      uint32_t sr[2][32];
      tmem_ld32_async(tmem_base + sb * kBlockN + lane_base, sr[0]);
      tmem_ld32_async(tmem_base + sb * kBlockN + lane_base + 32, sr[1]);
      tmem_wait_ld();
      if (n0 + kBlockN > kv_end) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (n0 + c * 32 + i >= kv_end) sr[c][i] = 0xff800000u;  // -inf
      }
      // Lazy maximum: the running maximum (and with it the rescale of O in tensor memory) moves only
      // when some row of the warp found a score more than kLazyLog2 above it; until then p = 2^(s - m)
      // may reach 2^kLazyLog2, which fp16 P and the fp32 sums hold without loss.
      const float m_tile = row_max(sr) * p.scale_log2;
      float corr = 1.f;
      const bool corr_any = __any_sync(0xffffffffu, m_tile > m_run + kLazyLog2);
      if (corr_any) {
        const float m_new = fmaxf(m_run, m_tile);
        corr = fast_exp2(m_run - ((m_new == -INFINITY) ? 0.f : m_new));
        m_run = m_new;
      }
      const float m_safe = (m_run == -INFINITY) ? 0.f : m_run;
      const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), shift2 = pack_f32x2(-m_safe, -m_safe);
      uint64_t sum2[4] = {0, 0, 0, 0};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t packed[16], low[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 x = unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1])), scale2, shift2));
          const float a = fast_exp2(x.x), b = fast_exp2(x.y);
          sum2[(i >> 1) & 3] = add_f32x2(sum2[(i >> 1) & 3], pack_f32x2(a, b));
          if (kNarrow)
            packed[i >> 1] = split_half2(a, b, low[i >> 1]);
          else
            packed[i >> 1] = pack_half2(a, b);
        }
        // P_j (fp16 pairs) over this thread's own S row (all scores are in registers)
        tmem_st16(tmem_base + sb * kBlockN + lane_base + c * 16, packed);
        if (kNarrow) tmem_st16(tmem_base + sb * kBlockN + lane_base + 32 + c * 16, low);
      }
      const float2 sum = unpack_f32x2(add_f32x2(add_f32x2(sum2[0], sum2[1]), add_f32x2(sum2[2], sum2[3])));
      l_run = l_run * corr + (sum.x + sum.y);
      // rescale this row of O in tensor memory when the warp moved a maximum; O is in use by
      // P_{j-1}.V_{j-1} until that completes (P_j.V_j is not issued before this warp arrives below,
      // so the barrier cannot be more than one phase ahead of the parity asked for)
      const bool flush = kNarrow && j > 0 && j % kFlushTiles == 0;  // P_j.V_j starts O anew
      if (j > 0 && (corr_any || flush)) {
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar_o, (j - 1) & 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
        if (flush) {
          flush_sums(sums, tmem_o + lane_base, p.d, j == kFlushTiles, owed);
          owed = corr;
        } else {
          if (kNarrow) owed *= corr;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (kNarrow && c * 32 >= p.d) break;
            uint32_t r[32];
            tmem_ld32(tmem_o + lane_base + c * 32, r);
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * corr);
            tmem_st32(tmem_o + lane_base + c * 32, r);
          }
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p[sb]);
    }
    // ---- epilogue: O / l -> out ----
    if (ok && nkv > 0) ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar_fin, 0, abort_flag));
    tc_fence_after();
    at += row;
    float bad = 0.f;  // NaN once a stored sum is not finite
    const auto load_o = [&](int c, uint32_t (&r)[32]) {
      tmem_ld32(tmem_o + lane_base + c * 32, r);
      if (kNarrow && nkv > kFlushTiles) {
        const float *old = reinterpret_cast<const float *>(sums) + c * 32;
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(fmaf(old[i], owed, __uint_as_float(r[i])));
      }
    };
    if (parts > 1) {
      const bool any = ok && nkv > 0;
      if (t_row < p.sq) partials.ml[at] = any ? make_float2(m_run, l_run) : make_float2(-INFINITY, 0.f);
      if (any) {
        float *dst = partials.sums + at * p.d;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (kNarrow && c * 32 >= p.d) break;
          uint32_t r[32];
          load_o(c, r);
          if (t_row < p.sq) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              if (kNarrow && c * 32 + u * 4 >= p.d) break;
              if (kNarrow)
#pragma unroll
                for (int i = 0; i < 4; ++i) bad = fmaf(__uint_as_float(r[u * 4 + i]), 0.f, bad);
              *reinterpret_cast<uint4 *>(dst + c * 32 + u * 4) = make_uint4(r[u * 4], r[u * 4 + 1], r[u * 4 + 2], r[u * 4 + 3]);
            }
          }
        }
      }
    } else if (ok && nkv > 0) {
      const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
      __half *dst = reinterpret_cast<__half *>(p.out) + ((size_t)t_row * p.hq + h) * (kNarrow ? p.d : kD);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (kNarrow && c * 32 >= p.d) break;
        uint32_t r[32];
        load_o(c, r);
        if (t_row < p.sq) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (kNarrow && c * 32 + u * 8 >= p.d) break;
            if (kNarrow)
#pragma unroll
              for (int i = 0; i < 8; ++i) bad = fmaf(__uint_as_float(r[u * 8 + i]), 0.f, bad);
            uint4 w;
            w.x = pack_half2(__uint_as_float(r[u * 8 + 0]) * inv, __uint_as_float(r[u * 8 + 1]) * inv);
            w.y = pack_half2(__uint_as_float(r[u * 8 + 2]) * inv, __uint_as_float(r[u * 8 + 3]) * inv);
            w.z = pack_half2(__uint_as_float(r[u * 8 + 4]) * inv, __uint_as_float(r[u * 8 + 5]) * inv);
            w.w = pack_half2(__uint_as_float(r[u * 8 + 6]) * inv, __uint_as_float(r[u * 8 + 7]) * inv);
            *reinterpret_cast<uint4 *>(dst + c * 32 + u * 8) = w;
          }
        }
      }
    }
    if (kNarrow && bad != 0.f)
      redo_narrow_row(p, t_row, h, tile0 * kBlockN, min((tile0 + nkv) * kBlockN, kv_end), partials.sums + at * p.d,
                      parts > 1 ? partials.ml + at : nullptr);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem_base) : "memory");
}

// (rows, heads, d) fp16 token-major -> tensor map with boxes of [box_rows rows][64 halves], 128-byte swizzle
bool rows_map(CUtensorMap *map, const void *base, int64_t rows, int heads, int d, int box_rows) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)rows};
  cuuint64_t strides[2] = {(cuuint64_t)d * 2, (cuuint64_t)heads * d * 2};
  cuuint32_t box[3] = {64, 1, (cuuint32_t)box_rows}, es[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A tile takes about 0.7 us of a block; a block costs six tiles more.  Joining with its launch counts as 18 (it took 7 to 9 us, with
// what the parts of full SMs take from each other, and somewhat less since), as 14 where heads are few and narrow, and as 10 for one
// head and a fifth for each further part of a row.  Whole and divided, the joining included: 4096 rows of 2 heads of 128, causal: 46
// and 23 us; 2700 of 16 heads of 64, not causal: 76 and 66; 2000 of 8 heads of 128, causal: 25 both; 2048 of 16, causal: 28 and 38,
// left whole.  1100 rows, causal, at 18 tiles (whole) and here: 2 heads of 64 17.1 and 10.3, 8 heads 17.4 and 14.7, 2 heads of 128
// 16.4 and 11.3; not causal, 4 heads of 64 17.4 and 13.0.  2700 rows of one head of 128, causal: 20.8 in 22 parts, 15.7 in fewer.  One
// head of 128, not causal, whole (a plan of 448 entries did not hold the parts) and divided: 40000 rows 959 and 608; 77000, 3126 and
// 2570.
KeySplit prompt_plan(int sq, int hq, int64_t skv, int d, int is_causal) {
  const auto tiles = [&](int b) {
    const int64_t last = ((int64_t)b + 1) * kBlockM, end = last < sq ? last : sq;
    return (int)(((is_causal && end < skv ? end : skv) + kBlockN - 1) / kBlockN);
  };
  const float least_gain = hq == 1 ? 10.f : hq * d <= (is_causal ? 640 : 256) ? 14.f : 18.f;
  KeySplit plan = plan_key_split(((int64_t)sq + kBlockM - 1) / kBlockM, hq, is_causal != 0, 6.f, least_gain, tiles, 2 * kSms, 1216,
                                 hq == 1 ? 0.2f : 0.f);
  if (key_split_bytes(plan, hq, kBlockM, d) > kMostScratch) plan.units = plan.divided = 0;
  return plan;
}

// Heads below 128 in prompts: a TMA row is a multiple of 16 bytes, and below 16 rows (of 128 that a tile holds) the
// row-by-row form is the cheaper one.
bool narrow_heads(int sq, int d) { return d < kD && d % 8 == 0 && sq >= 16; }

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace axb

extern "C" {

size_t axb200_sdpa_workspace_bytes(int sq, int hq, int hkv, int d, int64_t skv, int dtype) {
  // the tensor-core kernels and the tiled FMA kernel can keep everything on chip; only the row-by-row evaluation on the decode
  // kernels needs room for partials (whatever the tensor-core path does not take - unaligned pointers, say - the tiled kernel does)
  if (hkv > 0 && hq % hkv == 0 && axb::sdpa_tiled_supported(sq, hq, hkv, d, skv)) return 0;
  return axb::sdpa_rows_workspace_bytes(sq, hq, hkv, d, skv);
}

size_t axb200_sdpa_scratch_bytes(int sq, int hq, int hkv, int d, int64_t skv, int is_causal, int dtype) {
  // what makes prompts faster: the fp32 form's tiles of parts, and what blocks with divided keys leave
  if (sq <= 0 || hq <= 0 || hkv <= 0 || d <= 0 || skv <= 0 || skv > 0x7fffffff - 4096 || hq % hkv != 0) return 0;
  if (dtype == AXB200_FLOAT32 && axb::sdpa_tiled_supported(sq, hq, hkv, d, skv))
    return axb::sdpa_split_scratch_bytes(sq, hq, hkv, d, skv, is_causal);
  if (dtype == AXB200_FLOAT16 && (d == axb::kD || axb::narrow_heads(sq, d)))
    return axb::key_split_bytes(axb::prompt_plan(sq, hq, skv, d, is_causal), hq, axb::kBlockM, d);
  return 0;
}

int axb200_sdpa(const void *q, const void *k, const void *v, void *out, int sq, int hq, int hkv, int d,
                int64_t skv, int is_causal, int dtype, void *workspace, size_t workspace_bytes, void *stream) {
  return axb200_sdpa_scratch(q, k, v, out, sq, hq, hkv, d, skv, is_causal, dtype, workspace, workspace_bytes, nullptr, 0, stream);
}

int axb200_sdpa_scratch(const void *q, const void *k, const void *v, void *out, int sq, int hq, int hkv, int d, int64_t skv,
                        int is_causal, int dtype, void *workspace, size_t workspace_bytes, void *scratch, size_t scratch_bytes,
                        void *stream) {
  if (dtype != AXB200_FLOAT16 && dtype != AXB200_FLOAT32) return AXB200_UNSUPPORTED_TYPE;
  if (!q || !k || !v || !out) return AXB200_INVALID_PTR;
  if (sq <= 0 || hq <= 0 || hkv <= 0 || d <= 0 || skv <= 0 || skv > 0x7fffffff - 4096) return AXB200_INVALID_ARGUMENT;
  if (hq % hkv != 0) return AXB200_SHAPE_MISMATCH;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool narrow = axb::narrow_heads(sq, d);
  const bool tensor_path = dtype == AXB200_FLOAT16 && (d == axb::kD || narrow) && hq <= 65535 && axb::aligned16(q) &&
                           axb::aligned16(k) && axb::aligned16(v) && axb::aligned16(out) && axb::tensor_map_encoder();
  if (!tensor_path) {
    const bool tiled = axb::sdpa_tiled_supported(sq, hq, hkv, d, skv);
    const bool split = tiled && dtype == AXB200_FLOAT32 && scratch && axb::aligned16(scratch) && axb::aligned16(q) &&
                       axb::aligned16(k) && axb::aligned16(v) && axb::aligned16(out);
    const size_t need = split ? axb::sdpa_split_scratch_bytes(sq, hq, hkv, d, skv, is_causal) : 0;
    if (need && scratch_bytes >= need) return axb::sdpa_split(q, k, v, out, sq, hq, hkv, d, skv, is_causal, scratch, st);
    if (tiled)
      return axb::sdpa_tiled(q, k, v, out, sq, hq, hkv, d, skv, is_causal, dtype, st);
    return axb::sdpa_rows_fallback(q, k, v, out, sq, hq, hkv, d, skv, is_causal, dtype, workspace, workspace_bytes, st);
  }
  CUtensorMap mq, mk, mv;
  if (!axb::rows_map(&mq, q, sq, hq, d, axb::kBlockM) || !axb::rows_map(&mk, k, skv, hkv, d, axb::kBlockN) ||
      !axb::rows_map(&mv, v, skv, hkv, d, axb::kBlockN))
    return AXB200_INTERNAL_ERROR;
  static std::mutex mu;
  static bool opted[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return AXB200_DEVICE_ERROR;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!opted[dev]) {
      const auto opt = [](auto kernel) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, axb::kSmemBytes) == cudaSuccess;
      };
      if (!opt(&axb::prefill_attn_f16_kernel<false, axb::WholeBlocks>) || !opt(&axb::prefill_attn_f16_kernel<true, axb::WholeBlocks>) ||
          !opt(&axb::prefill_attn_f16_kernel<false, axb::KeySplit>) || !opt(&axb::prefill_attn_f16_kernel<true, axb::KeySplit>))
        return AXB200_DEVICE_ERROR;
      opted[dev] = true;
    }
  }
  axb::PrefillParams p{};
  p.out = out;
  p.sq = sq;
  p.hq = hq;
  p.hkv = hkv;
  p.skv = (int)skv;
  p.causal = is_causal != 0;
  p.d = d;
  p.scale_log2 = (1.0f / sqrtf((float)d)) * axb::kLog2e;
  p.q = static_cast<const __half *>(q);
  p.k = static_cast<const __half *>(k);
  p.v = static_cast<const __half *>(v);
  axb::KeySplit split{};
  if (scratch && axb::aligned16(scratch)) {
    split = axb::prompt_plan(sq, hq, skv, d, is_causal);
    if (scratch_bytes < axb::key_split_bytes(split, hq, axb::kBlockM, d)) split.units = 0;
  }
  if (split.units == 0) {
    const dim3 grid((unsigned)hq * ((sq + axb::kBlockM - 1) / axb::kBlockM));
    auto *kernel = narrow ? axb::prefill_attn_f16_kernel<true, axb::WholeBlocks> : axb::prefill_attn_f16_kernel<false, axb::WholeBlocks>;
    kernel<<<grid, axb::kThreads, axb::kSmemBytes, st>>>(mq, mk, mv, p, axb::WholeBlocks{}, axb::Partials{nullptr, nullptr});
    return axb::launch_status();
  }
  const axb::Partials partials = axb::partials_at(scratch, split, hq, axb::kBlockM);
  auto *kernel = narrow ? axb::prefill_attn_f16_kernel<true, axb::KeySplit> : axb::prefill_attn_f16_kernel<false, axb::KeySplit>;
  kernel<<<dim3((unsigned)hq * split.units), axb::kThreads, axb::kSmemBytes, st>>>(mq, mk, mv, p, split, partials);
  if (cudaPeekAtLastError() == cudaSuccess)
    return axb::launch_dependent(axb::join_parts_kernel<__half, axb::kBlockM>, dim3((unsigned)hq * (axb::kBlockM / 8), split.divided_blocks),
                                 dim3(256), 0, st, split, partials, static_cast<__half *>(out), sq, hq, d);
  return axb::launch_status();
}

}  // extern "C"

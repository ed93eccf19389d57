// The products between two attention calls of a decode step as one launch, for up to 8 rows (a batch of decoded tokens):
//
//   stage 0   y  = attn . W_o^T + residual
//   stage 1   act = silu(gate) * up of z . [W_gate | W_up]^T, z the norm of y
//   stage 2   y' = act . W_down^T + y
//   stage 3   next = z' . W_next^T (the next layer's input product, or the logits), z' the norm of y'
//
// What bounds it: reading the weights.  As launches of their own (product, norm, product, activation, product, norm, product)
// the seven start and drain one after the other, each product being 1 to 8 us of reading.  Here one CTA per SM stays
// through all stages and asks for the next stages' first weights (192 KB per SM) before it waits for the other CTAs.  8 rows,
// width 2048, ff 6144, 4096 columns next (100 MB of weights, 15.6 us at 6.46 TB/s), in a graph: 41.3 us before, 29.6 to 32.1 now (five
// boxes).  What is left: three meetings of all CTAs and the reading of the inputs after each (about 3 us together each time), and 1.1 us per unit
// of a CTA, of which its copies into shared memory take 0.45 and its reads and products 0.4; the reading of a unit from HBM takes 1.5.
//
// Split: a unit is 32 rows of a weight matrix (16 gate and 16 up rows in stage 1, so that the activation joins values of one
// thread) over all of K; units go to pairs of CTAs (clusters) in turn.  K is cut into blocks of 64: block j belongs to warp
// j % 32 of the pair's 32.  A warp copies its tile of 32 x 64 into a ring of its own (no barrier between warps: it asks for the
// next tile where it consumed one) and multiplies it with the inputs of its block, which it holds in registers through the stage;
// the sixteen partial tiles of a CTA meet in shared memory, those of the pair through distributed shared memory, each CTA
// finishing half of the rows.  A pair and not one CTA per unit, because every CTA reads the inputs of its part of K from L2: all
// of K in each of 148 CTAs took 18 us of a stage with 32 rows.  mma.sync, weights as operand A: with 8 columns a tcgen05 product
// of 128 rows would need several CTAs' parts of K added up for every unit to fill the chip; here a tile needs no trip through
// tensor memory.  K is permuted alike in both operands so that a thread's operands are 16 bytes in a row.  Copies by TMA
// took as long (31.1 us), and prefetches of further tiles into L2 were slower (34.5).
//
// Between stages all CTAs meet at a counter, so the launch is cooperative with one CTA per SM: two launches of this
// kernel cannot be resident together (each takes most of every SM's shared memory), which is also why the counter can be the
// device's.  Every wait is bounded; after one that ran out the CTA goes through the remaining stages without meeting the others,
// sends all that its pair may wait for, arms no more barriers where it was the pair that it waited for, and leaves when what the
// other CTA sends has landed.
#include <mutex>

#include "tcgen05.cuh"
#include "vec.cuh"

namespace axb {
namespace {

constexpr int kWarps = 16, kThreads = kWarps * 32, kPair = 2;
constexpr int kBlock = 64;              // K per tile
constexpr int kUnit = 32;               // weight rows per tile
constexpr int kTile = kUnit * kBlock * 2;
constexpr int kStages = 4;
// Buffers of the exchange in a pair.  A CTA's senders send its sums of unit n behind a barrier that its owners reached after they had
// read the other CTA's sums of unit n - 2 (they read those of n - 1 beside this send).  The other CTA sent n - 2 behind a barrier that
// its owners reached after they had read what they got for unit n - 4: four can be written without asking, three cannot.
constexpr int kRecvs = 4;

constexpr int kHeld = 4;    // blocks whose inputs a warp holds
constexpr int kSlots = 3;   // tiles in flight per warp
constexpr int kRows = 8;    // input rows: the columns of a product
constexpr int kRecv = 128 * 4;  // the other CTA's sums of one unit
constexpr int kOffRed = kWarps * kSlots * kTile, kRed = kWarps * 256 * 4;  // partial tiles
constexpr int kOffRecv = kOffRed + kRed, kOffInv = kOffRecv + kRecvs * kRecv, kOffBar = kOffInv + kRows * 4;
constexpr int kSmem = kOffBar + kRecvs * 8 + 16;

struct Stage {
  const void *w;  // (n, k), in stage 1 (2 n, k)
  const void *x;  // (rows, k)
  void *out;      // (rows, n)
  int k, n;       // n: columns of out
  int blocks, units, first;  // first: the pair that has unit 0
};

struct ChainParams {
  Stage st[kStages];
  const void *res_in, *res_mid;  // (rows, width), what stages 0 and 2 are joined with; stages 1 and 3 read their sums
  const void *norm[2];           // of stages 1 and 3
  float *squares;       // (rows, grid): sums of squares of the CTAs' columns, for the norm of the stage that follows
  float eps;
  int rows;
  int weights_ready;  // weights may be read before the launch in front of this one is over
  unsigned long long wait_ns;
};

__device__ unsigned long long g_arrived = 0;  // CTAs counted at the ends of stages; a multiple of the grid between launches
__global__ void zero_arrived_kernel() { g_arrived = 0; }
struct ArrivedReset {
  ArrivedReset() { register_timeout_hook([] { zero_arrived_kernel<<<1, 1>>>(); }); }
};
ArrivedReset g_arrived_reset;

__device__ __forceinline__ uint4 lds16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// One tile: 2 x 16 weight rows x 64, times b.  Thread (g, t) = (lane / 4, lane % 4) has weight rows r and 8 + r of each
// sixteen with r = g / 2 + 4 (g % 2): the eight lanes that load together then touch all banks under the 128-byte swizzle.
// It reads the 16-byte pieces t and t + 4 of a row; words 2 i and 2 i + 1 of a piece are step i's K pairs.
__device__ __forceinline__ void tile_mma(float (&acc)[2][4], uint32_t tile, const uint4 (&b)[2], int r, int t) {
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t at = tile + m * (kTile / 2) + r * 128 + (((t + 4 * q) ^ r) << 4);
      const uint4 lo = lds16(at), hi = lds16(at + 1024);
      const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
      mma_16816(acc[m], a0, b[q].x, b[q].y);
      mma_16816(acc[m], a1, b[q].z, b[q].w);
    }
}

__device__ __forceinline__ void unpack8(const uint4 &v, float (&f)[8]) {
  const __half *e = reinterpret_cast<const __half *>(&v);
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = __half2float(e[i]);
}

// What other CTAs wrote during this launch is read through L2.
__device__ __forceinline__ uint4 load16(const void *p) { return __ldcg(reinterpret_cast<const uint4 *>(p)); }

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t v;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
  return v;
}
__device__ __forceinline__ uint32_t in_cta(const void *mine, int rank) {  // the same place in a CTA of the cluster
  uint32_t v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(v) : "r"(smem_u32(mine)), "r"(rank));
  return v;
}
// Two floats into another CTA's shared memory; its barrier counts the bytes.
__device__ __forceinline__ void send2(uint32_t to, float a, float b, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(to), "f"(a), "f"(b), "r"(bar)
               : "memory");
}

// More bytes that the barrier's phase has to wait for, without an arrival.
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// After a wait that ran out: nothing that the other CTA sends may still be on its way when this one leaves its shared memory.  The
// other sends `sent` units of kRecv bytes into the barriers in turn, whatever happened to it, and this CTA armed phases for the first
// `armed`.  What is left is added to whichever phase a barrier is in - the armed one where sums of later units landed in it, else the
// next - and one more arrival ends that; so the last phase of each completes when all bytes are there.  (A phase counts less than
// 1 MB: for more columns than any vocabulary has, the time alone has to do.)
__device__ __noinline__ void drain(uint64_t *got, int sent, int armed, unsigned long long limit_ns) {
  const unsigned long long t0 = global_timer_ns();
  for (int i = 0; i < kRecvs; ++i) {
    const int phases = (armed - i + kRecvs - 1) / kRecvs, rest = (sent - i + kRecvs - 1) / kRecvs - phases;
    auto wait = [&](int phase) {
      while (!mbar_try_wait(&got[i], phase & 1) && global_timer_ns() - t0 < limit_ns) {
      }
    };
    const bool counts = rest <= ((1 << 20) - 1) / kRecv;
    if (rest > 0 && counts) mbar_expect_tx(&got[i], (uint32_t)(rest * kRecv));
    if (phases > 0) wait(phases - 1);
    if (rest > 0) {
      if (counts) mbar_arrive(&got[i]);
      wait(phases);
    }
  }
}

// KC: blocks of the norms' width that a warp has.
template <int KC>
__global__ void __launch_bounds__(kThreads, 1) row_chain_kernel(const __grid_constant__ ChainParams p) {
  static_assert(KC <= kHeld, "inputs held in registers");
  extern __shared__ __align__(128) uint8_t smem[];
  float *const inv_of = reinterpret_cast<float *>(smem + kOffInv);
  float *const red = reinterpret_cast<float *>(smem + kOffRed);
  uint64_t *const got_all = reinterpret_cast<uint64_t *>(smem + kOffBar);  // the other CTA's sums
  volatile int *const abort_flag = reinterpret_cast<volatile int *>(got_all + kRecvs);
  const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, r = (g >> 1) | ((g & 1) << 2);
  const int half = (int)cluster_rank(), pair = blockIdx.x / kPair, pairs = gridDim.x / kPair, block0 = half * kWarps + warp;
  constexpr int kStride = kPair * kWarps;
  const uint32_t ring_at = smem_u32(smem) + warp * kSlots * kTile;
  auto first_unit = [&](int s) {
    const int d = pair - p.st[s].first;
    return d < 0 ? d + pairs : d;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kRecvs; ++i) mbar_init(&got_all[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  // the other CTA's barriers are there after the wait below; relaxed (the fence above covers the barriers), since a release waits
  // for the copies that are under way
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  grid_dependency_launch();

  // ---- the warp's tiles in the order of their use ---------------------------------------------------------------------------
  struct Cursor {
    int stage, unit, block, units, blocks;
  };
  auto enter = [&](Cursor &c, int stage) {  // the first tile of a stage, or of the next that has one for this warp
    for (c.stage = stage; c.stage < kStages; ++c.stage) {
      c.unit = first_unit(c.stage), c.units = p.st[c.stage].units, c.blocks = p.st[c.stage].blocks, c.block = block0;
      if (c.unit < c.units && c.block < c.blocks) return;
    }
  };
  auto advance = [&](Cursor &c) {
    c.block += kStride;
    if (c.block < c.blocks) return;
    c.block = block0;
    c.unit += pairs;
    if (c.unit >= c.units) enter(c, c.stage + 1);
  };
  Cursor next;  // the next tile to ask for
  enter(next, 0);
  int put = 0, get = 0;
  // Eight copies of 16 bytes per lane: copy i brings rows 4 i + lane / 8, piece lane % 8, to where the swizzle has it.
  const int c_row = lane >> 3, c_piece = lane & 7;
  auto ask = [&] {
    if (next.stage < kStages) {
      const Stage &s = p.st[next.stage];
      const bool gated = next.stage == 1;
      const int r0 = gated ? next.unit * (kUnit / 2) : next.unit * kUnit, ld = s.k * 2;
      const uint8_t *src = static_cast<const uint8_t *>(s.w) + (size_t)(r0 + c_row) * ld + next.block * (kBlock * 2) + c_piece * 16;
      const size_t far = gated ? (size_t)(s.n - kUnit / 2) * ld : 0;  // from the gate rows to the up rows
      const uint32_t dst = ring_at + put * kTile + c_row * 128;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint8_t *from = src + (size_t)(4 * i) * ld + (i >= 4 ? far : 0);
        const int bytes = r0 + 4 * i + c_row < s.n || gated ? 16 : 0;
        asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst + i * 512 + ((c_piece ^ (c_row + 4 * (i & 1))) << 4)),
                     "l"(__cvta_generic_to_global(bytes ? from : static_cast<const uint8_t *>(s.w))), "r"(bytes)
                     : "memory");
      }
      advance(next);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // an empty one at the end: every tile stays a group of its own
    put = put + 1 == kSlots ? 0 : put + 1;
  };
  if (!p.weights_ready) grid_dependency_wait();
#pragma unroll 1
  for (int i = 0; i < kSlots; ++i) ask();
  // the warp's oldest tile, and its slot given back
  auto take = [&](float(&acc)[2][4], const uint4(&b)[2]) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kSlots - 1) : "memory");
    __syncwarp();
    tile_mma(acc, ring_at + get * kTile, b, r, t);
    get = get + 1 == kSlots ? 0 : get + 1;
    __syncwarp();
    ask();
  };

  // ---- a finished unit: the first two warps have two sums of it per thread (weight rows v_f and 16 + v_f, or gate and up, for
  // input row v_n), the next two those that the other CTA of the pair finishes ------------------------------------------------
  const bool owner = threadIdx.x < 64, sender = !owner && threadIdx.x < 128;
  const int v_i = threadIdx.x & 63, v_e = v_i >> 5, v_n = 2 * t + v_e, v_f = r + 8 * half;
  float mine[2], joined[2] = {0.f, 0.f}, sq = 0.f;
  const float2 *const recv = reinterpret_cast<const float2 *>(smem + kOffRecv);
  const uint32_t peer_recv = in_cta(recv, half ^ 1), peer_got = in_cta(got_all, half ^ 1);
  RingPos sent, got;
  int units_done = 0, armed = 0;  // units whose phase thread 0 armed; ~ of it in a warp whose wait for the other CTA ran out

  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  grid_dependency_wait();

#pragma unroll 1
  for (int st = 0; st < kStages; ++st) {
    const Stage &s = p.st[st];
    const int u0 = first_unit(st);
    const bool gated = st == 1, joins = !(st & 1);
    uint4 b[kHeld][2];
    // inputs of block c as operand B: row g, pieces t and t + 4
    auto column = [&](int c, int q) { return c * kBlock + (t + 4 * q) * 8; };
    auto fetch = [&](uint4(&dst)[2], int c) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int k = column(c, q);
        dst[q] = g < p.rows && k < s.k ? load16(static_cast<const __half *>(s.x) + (size_t)g * s.k + k) : make_uint4(0, 0, 0, 0);
      }
    };
    uint4 nw[KC][2];
    if (st & 1) {  // what does not come from the stage before
#pragma unroll
      for (int c = 0; c < KC; ++c)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int k = column(block0 + kStride * c, q);
          nw[c][q] = k < s.k ? *reinterpret_cast<const uint4 *>(static_cast<const __half *>(p.norm[st >> 1]) + k) : make_uint4(0, 0, 0, 0);
        }
    }
    if (st > 0) {  // all CTAs have stored what the stage before gives
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        const unsigned long long place = atomicAdd(&g_arrived, 1ull), goal = (place / gridDim.x + 1) * gridDim.x;
        unsigned long long seen, t0 = 0;
        for (uint32_t spin = 1; !*abort_flag; ++spin) {
          asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(&g_arrived) : "memory");
          if (seen >= goal) break;
          if ((spin & 63u) == 0u) {
            const unsigned long long now = global_timer_ns();
            if (t0 == 0)
              t0 = now;
            else if (now - t0 > p.wait_ns) {
              *abort_flag = 1;
              atomicOr(&g_error_word, AXB200_ERR_WAIT_TIMEOUT);
            }
          }
        }
      }
      __syncthreads();
    }
    if (st & 1) {
#pragma unroll
      for (int c = 0; c < KC; ++c) fetch(b[c], block0 + kStride * c);
      if (warp < kRows) {
        float sum = 0.f;
        if (warp < p.rows)
          for (int i0 = lane; i0 < (int)gridDim.x; i0 += 160) {  // five loads under way together
            float v[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) v[i] = i0 + 32 * i < (int)gridDim.x ? __ldcg(p.squares + (size_t)warp * gridDim.x + i0 + 32 * i) : 0.f;
            sum += (v[0] + v[1]) + (v[2] + v[3]) + v[4];
          }
        sum = warp_sum(sum);
        if (lane == 0) inv_of[warp] = 1.0f / sqrtf(sum / (float)s.k + p.eps);
      }
      __syncthreads();
      const float inv = inv_of[g];
#pragma unroll
      for (int c = 0; c < KC; ++c)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float v[8], w[8];
          unpack8(b[c][q], v);
          unpack8(nw[c][q], w);
          uint4 z;
          z.x = pack_half2(v[0] * inv * w[0], v[1] * inv * w[1]), z.y = pack_half2(v[2] * inv * w[2], v[3] * inv * w[3]);
          z.z = pack_half2(v[4] * inv * w[4], v[5] * inv * w[5]), z.w = pack_half2(v[6] * inv * w[6], v[7] * inv * w[7]);
          b[c][q] = z;
        }
    }
    // sums of the unit, complete after the exchange
    auto finish = [&](int u) {
      if (owner) {
        if (armed >= 0 && !mbar_wait_warp(&got_all[got.slot], got.parity, abort_flag, p.wait_ns)) armed = ~armed;
        const float2 other = recv[got.slot * (kRecv / 8) + v_i];
        mine[0] += other.x, mine[1] += other.y;
      }
      got.next(kRecvs);
      if (!owner || v_n >= p.rows) return;
      if (gated) {
        const int f = u * (kUnit / 2) + v_f;
        if (f < s.n)
          static_cast<__half *>(s.out)[(size_t)v_n * s.n + f] = __float2half_rn(mine[0] / (1.0f + expf(-mine[0])) * mine[1]);
        return;
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int f = u * kUnit + 16 * m + v_f;
        if (f >= s.n) continue;
        __half *const at = static_cast<__half *>(s.out) + (size_t)v_n * s.n + f;
        if (joins) mine[m] += joined[m];
        *at = __float2half_rn(mine[m]);
        sq = fmaf(mine[m], mine[m], sq);
      }
    };
    sq = 0.f;
    int last = -1;
#pragma unroll 1
    for (int u = u0; u < s.units; u += pairs) {
      float acc[2][4] = {};
      __half joins_with[2];
      if (joins && owner) {
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int f = u * kUnit + 16 * m + v_f;
          if (v_n < p.rows && f < s.n) joins_with[m] = __ldcg(static_cast<const __half *>(st == 0 ? p.res_in : p.res_mid) + (size_t)v_n * s.n + f);
        }
      }
      if (st & 1) {
#pragma unroll
        for (int c = 0; c < KC; ++c)
          if (block0 + kStride * c < s.blocks) take(acc, b[c]);
      } else {
#pragma unroll 1
        for (int c0 = block0; c0 < s.blocks; c0 += kStride * kHeld) {
#pragma unroll
          for (int i = 0; i < kHeld; ++i)
            if (c0 + kStride * i < s.blocks) fetch(b[i], c0 + kStride * i);
#pragma unroll
          for (int i = 0; i < kHeld; ++i)
            if (c0 + kStride * i < s.blocks) take(acc, b[i]);
        }
      }
      if (last >= 0) __syncthreads();  // the last unit's partial tiles have been read
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) red[((warp * 2 + m) * 4 + i) * 32 + lane] = acc[m][i];
      __syncthreads();
      if (last >= 0) finish(last);
      if (threadIdx.x == 0 && armed >= 0) {  // this warp has waited for every phase armed so far, so none is armed twice
        mbar_arrive_expect_tx(&got_all[sent.slot], kRecv);
        ++armed;
      }
      if (owner || sender) {  // accumulators 0 and 1 are the rows of the first CTA, 2 and 3 of the second
        const int e = (owner ? half : half ^ 1) * 2 + v_e;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const float *at = red + (m * 4 + e) * 32 + lane;
          float sum = 0.f;
#pragma unroll
          for (int w = 0; w < kWarps; ++w) sum += at[w * 256];
          mine[m] = sum;
          if (joins) joined[m] = __half2float(joins_with[m]);
        }
        if (sender) send2(peer_recv + sent.slot * kRecv + v_i * 8, mine[0], mine[1], peer_got + sent.slot * 8);
      }
      sent.next(kRecvs);
      ++units_done;
      last = u;
    }
    if (last >= 0) finish(last);
    if (joins && owner) {  // over the eight rows r of a column
      sq += __shfl_xor_sync(0xffffffffu, sq, 4);
      sq += __shfl_xor_sync(0xffffffffu, sq, 8);
      sq += __shfl_xor_sync(0xffffffffu, sq, 16);
      if (g == 0 && v_n < p.rows) p.squares[(size_t)v_n * gridDim.x + blockIdx.x] = sq;
    }
  }
  // the other CTA may still be in its own waits, each as long as the limit at most: three meetings and one exchange
  if (threadIdx.x == 0 && *abort_flag) drain(got_all, units_done, armed < 0 ? ~armed : armed, kWaitNanos + 4 * min(p.wait_ns, 1ull << 60));
}

bool al16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int blocks_held(int width) { return (width / kBlock + kPair * kWarps - 1) / (kPair * kWarps); }

// Multiples of 64 for the tiles.  Up to 8 rows and 4096 wide: with more columns or more inputs per warp the products and the
// reading of the inputs by every pair cost what the launches did (chain against seven launches, both in a graph with cold weights:
// 8 rows, width 2048: 29.6 us, 41.3; 4096: 78.6, 86.5; 5120: 110.6, 100.8; forms of this kernel for 16 rows, 2048: 37.1, 40.5, and with
// the logits 161.6, 125.4; 4096: 90.3, 87.4).
bool takes(int64_t rows, int attn, int width, int ff, int next) {
  return rows >= 1 && rows <= kRows && attn > 0 && attn % 64 == 0 && width > 0 && width % 64 == 0 && ff > 0 && ff % 64 == 0 && next > 0 &&
         blocks_held(width) <= 2;
}

// A unit takes a pair about 1.45 us however little of K it has, and reads 128 KB of it up to 2048 wide; products of their own read a
// narrow K as fast as a wide one. So the chain saves about 9 us, less 1.45 (1 - width / 2048) per round of units in stages 1 and
// 3.  Launches and chain, 8 rows: width 2048, ff 6144, 4096 next, 40.7 and 32.0 us; 151936 next, 126 and 120; width 1024, ff 3072, 4096
// next, 29.2 and 23.4; 151936 next, 73 and 113; width 512, ff 1536, 1024 next, 22.2 and 16.9; 32000 next, 26.6 and 32.3.
bool gains(int width, int ff, int next) {
  const int places = 148 / kPair;
  const float rounds = (ff / (kUnit / 2) + (next + kUnit - 1) / kUnit) / (float)places;
  return 1.45f * fmaxf(0.f, 1.f - width / 2048.f) * rounds < 9.f;
}

// Pairs that the device holds at once, the same for every form of the kernel (one CTA per SM): the counter counts whole grids.
std::mutex g_pairs_mu;
int g_pairs[64] = {0};

template <int KC>
int launch(ChainParams &p, cudaStream_t st) {
  auto *kernel = row_chain_kernel<KC>;
  static bool opted[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return AXB200_DEVICE_ERROR;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[3];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kPair, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  attr[2].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[2].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  int pairs;
  {
    std::lock_guard<std::mutex> lock(g_pairs_mu);
    if (!opted[dev]) {
      int n = 0;
      cfg.numAttrs = 1;
      cfg.gridDim = dim3(kPair);
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1 || (g_pairs[dev] != 0 && n < g_pairs[dev])) {
        cudaGetLastError();
        return AXB200_DEVICE_ERROR;
      }
      if (g_pairs[dev] == 0) g_pairs[dev] = n;
      opted[dev] = true;
    }
    pairs = g_pairs[dev];
  }
  int at = 0;
  for (int i = 0; i < kStages; ++i) {
    p.st[i].first = at;
    at = (at + p.st[i].units) % pairs;
  }
  cfg.numAttrs = 3;
  cfg.gridDim = dim3(pairs * kPair);
  if (cudaLaunchKernelEx(&cfg, kernel, p) != cudaSuccess) {
    cudaGetLastError();
    return AXB200_DEVICE_ERROR;
  }
  return AXB200_OK;
}

}  // namespace
}  // namespace axb

extern "C" {

int axb200_row_chain_supported(int64_t rows, int attn, int width, int ff, int next, int dtype) {
  return dtype == AXB200_FLOAT16 && axb::takes(rows, attn, width, ff, next) ? 1 : 0;
}

int axb200_row_chain_gains(int64_t rows, int attn, int width, int ff, int next, int dtype) {
  return axb200_row_chain_supported(rows, attn, width, ff, next, dtype) && axb::gains(width, ff, next) ? 1 : 0;
}

size_t axb200_row_chain_workspace_bytes(int64_t rows, int width, int ff) {
  // activations, the sums after stage 0, sums of squares per CTA (a device has at most 1024 SMs)
  return rows <= 0 || width <= 0 || ff <= 0 ? 0 : (size_t)rows * (((size_t)width + ff) * 2 + 1024 * sizeof(float));
}

int axb200_row_chain(const void *x, const void *w_o, const void *residual, const void *norm1, const void *w_gate_up, const void *w_down,
                     const void *norm2, const void *w_next, void *residual_out, void *out, int64_t rows, int attn, int width, int ff,
                     int next, float eps, int dtype, void *workspace, size_t workspace_bytes, void *stream) {
  return axb200_row_chain_constant(x, w_o, residual, norm1, w_gate_up, w_down, norm2, w_next, residual_out, out, rows, attn, width, ff,
                                   next, eps, dtype, 0, workspace, workspace_bytes, stream);
}

int axb200_row_chain_constant(const void *x, const void *w_o, const void *residual, const void *norm1, const void *w_gate_up,
                              const void *w_down, const void *norm2, const void *w_next, void *residual_out, void *out, int64_t rows,
                              int attn, int width, int ff, int next, float eps, int dtype, int weights_ready, void *workspace,
                              size_t workspace_bytes, void *stream) {
  for (const void *q : {x, w_o, residual, norm1, w_gate_up, w_down, norm2, w_next, static_cast<const void *>(residual_out),
                        static_cast<const void *>(out), static_cast<const void *>(workspace)}) {
    if (!q) return AXB200_INVALID_PTR;
    if (!axb::al16(q)) return AXB200_INVALID_ARGUMENT;
  }
  if (dtype != AXB200_FLOAT16) return AXB200_UNSUPPORTED_TYPE;
  if (!axb::takes(rows, attn, width, ff, next) || workspace_bytes < axb200_row_chain_workspace_bytes(rows, width, ff))
    return AXB200_INVALID_ARGUMENT;
  axb::ChainParams p{};
  uint8_t *ws = static_cast<uint8_t *>(workspace);
  void *mid = ws, *act = ws + (size_t)rows * width * 2;
  p.squares = reinterpret_cast<float *>(ws + (size_t)rows * ((size_t)width + ff) * 2);
  auto blocks = [](int k) { return k / axb::kBlock; };
  auto units = [](int n, int per) { return (n + per - 1) / per; };
  p.st[0] = {w_o, x, mid, attn, width, blocks(attn), units(width, axb::kUnit), 0};
  p.st[1] = {w_gate_up, mid, act, width, ff, blocks(width), units(ff, axb::kUnit / 2), 0};
  p.st[2] = {w_down, act, residual_out, ff, width, blocks(ff), units(width, axb::kUnit), 0};
  p.st[3] = {w_next, residual_out, out, width, next, blocks(width), units(next, axb::kUnit), 0};
  p.res_in = residual, p.res_mid = mid;
  p.norm[0] = norm1, p.norm[1] = norm2;
  p.eps = eps, p.rows = (int)rows, p.weights_ready = weights_ready != 0, p.wait_ns = axb::wait_limit_ns();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return axb::blocks_held(width) <= 1 ? axb::launch<1>(p, st) : axb::launch<2>(p, st);
}

}  // extern "C"

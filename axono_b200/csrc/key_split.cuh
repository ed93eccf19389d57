// Blocks of query rows whose keys are divided among several CTAs, and the kernel that joins their partial results.
//
// The blocks of a prompt are few (a block is 128 rows of a head) and, under a causal mask, of very different length, so that
// the last of them leave most SMs without work: 2700 rows of 16 heads are 352 blocks, which two CTAs per SM take as one full wave and
// 56 more that take as long again.  A plan divides the blocks that would run alone; the parts leave un-normalised sums, their maxima and
// denominators in scratch memory.
#pragma once

#include <math.h>

#include "common.cuh"

namespace axb {

constexpr int kSms = 148;
constexpr size_t kMostScratch = (size_t)2 << 30;

// What CTAs work on, per head: unit u is part `part` of `parts` of row block `block`.  Blocks go from the last to the first; units of
// divided blocks follow one another, `divided` of them from `first` on; only they have scratch.  units == 0: blocks as they are.  Beyond
// kMostEntries units there are no entries: blocks of one length then, `even` parts for each of the divided ones at the end (else 0).
struct KeySplit {
  static constexpr int kMostEntries = 448;
  int units, first, divided, divided_blocks, blocks, even;
  uint16_t begin[kMostEntries / 2];  // of a divided block, its first part among the divided
  uint16_t block[kMostEntries];
  uint8_t part[kMostEntries], parts[kMostEntries];
};

struct KeyUnit {
  int block, part, parts;
};
__host__ __device__ inline KeyUnit key_unit(const KeySplit &plan, int unit) {
  if (plan.even == 0) return {plan.block[unit], plan.part[unit], plan.parts[unit]};
  if (unit < plan.first) return {plan.blocks - 1 - unit, 0, 1};
  const int i = unit - plan.first;
  return {plan.blocks - 1 - plan.first - i / plan.even, i % plan.even, plan.even};
}

// The first tile of part i of n.
__host__ __device__ inline int split_begin(int tiles, int part, int parts) { return (int)((int64_t)tiles * part / parts); }

// blocks row blocks of `heads` heads; tiles(b) key tiles in block b, not decreasing in b; part_cost: what a block or part costs
// beside its tiles, in tiles; least_gain: tiles in a row that a division has to save, as many as joining takes with its launch (the
// callers say what they measured); places: blocks that run at once; most_units: a plan with more is none (blocks below 65536);
// join_cost: what joining costs for each further part of a block, in tiles.
template <typename Tiles>
KeySplit plan_key_split(int64_t blocks, int heads, bool causal, float part_cost, float least_gain, Tiles tiles, int places, int most_units,
                        float join_cost = 0.f) {
  KeySplit plan{};
  if (blocks > most_units || heads > 2 * kSms) return plan;
  const int most = tiles((int)blocks - 1);
  int unsplit = 0, parts = 1, limit = 0;
  if (causal) {
    int64_t total = 0;
    for (int b = 0; b < blocks; ++b) total += tiles(b);
    // The time of parts of at most `at_most` tiles: the longest where all run at once, else an even share and half of the last.
    // Divisions only where the number of parts changes from block to block: a call makes its plan twice, and at 1433 rows the host
    // sets the pace (4 heads: 20.9 us with three divisions per block and candidate, 20.4 so).
    const auto estimate = [&](int at_most) {
      int64_t count = 0;
      int longest = 0, shortest = most, n = 1, last = 0;
      for (int b = 0; b < blocks; ++b) {
        const int t = tiles(b);
        if (t > n * at_most) {
          if (last) longest = (last + n - 1) / n > longest ? (last + n - 1) / n : longest;
          n = (t + at_most - 1) / at_most;
          shortest = t / n < shortest ? t / n : shortest;
        } else if (b == 0) {
          shortest = t < shortest ? t : shortest;
        }
        count += n;
        last = t;
      }
      longest = (last + n - 1) / n > longest ? (last + n - 1) / n : longest;
      const float alone = longest + part_cost + join_cost * ((most - 1) / at_most);
      if (count * heads <= places) return alone;
      const float even = (total + part_cost * count) * heads / places + (shortest + part_cost) / 2;
      return even > alone ? even : alone;
    };
    float best = estimate(most) - least_gain;
    const int first = (int)((total * heads + places - 1) / places);
    for (int at_most = first < 2 ? 2 : first; at_most < most && at_most < first + 8; ++at_most) {
      const float time = estimate(at_most);
      if (time < best) best = time, limit = at_most;
    }
    if (limit == 0) return plan;
  } else {
    // blocks of one length: whole waves of them as they are, the rest in parts that fill one, two or three rounds of the SMs
    const int64_t all = blocks * heads, waves = all / places;
    unsplit = (int)(waves * places / heads);
    const int64_t rest = all - (int64_t)unsplit * heads;
    float best = ((all + places - 1) / places - waves) * (most + part_cost) - least_gain;
    for (int rounds = 1; rounds <= 3; ++rounds) {
      int64_t n = rest ? rounds * places / rest : 0;
      n = n > 16 ? 16 : n;
      n = n > most / 2 ? most / 2 : n;
      const float time = n > 1 ? rounds * ((float)most / n + part_cost) + join_cost * (n - 1) : INFINITY;
      if (time < best) best = time, parts = (int)n;
    }
    if (parts == 1) return plan;
  }
  const bool entries = causal || unsplit + (blocks - unsplit) * parts <= KeySplit::kMostEntries;
  int units = 0, divided = 0;
  for (int i = 0; i < blocks; ++i) {
    const int b = (int)blocks - 1 - i;  // under a causal mask the longest first
    // causal: the longest first, so the divided ones first; else the divided ones last
    const int n = causal ? (tiles(b) + limit - 1) / limit : i < unsplit ? 1 : parts;
    if (units + n > (entries ? KeySplit::kMostEntries : most_units) || n > 255) return plan;
    if (n > 1) {
      if (divided == 0) plan.first = units;
      if (entries) plan.begin[plan.divided_blocks] = (uint16_t)divided;
      ++plan.divided_blocks;
      divided += n;
    }
    for (int part = 0; entries && part < n; ++part) {
      plan.block[units + part] = (uint16_t)b;
      plan.part[units + part] = (uint8_t)part;
      plan.parts[units + part] = (uint8_t)n;
    }
    units += n;
  }
  plan.units = units;
  plan.divided = divided;
  plan.blocks = (int)blocks;
  plan.even = entries ? 0 : parts;
  return plan;
}

// Scratch of a plan: per divided unit and head `rows` rows of d floats, and (maximum, denominator) of each row.
inline size_t key_split_bytes(const KeySplit &plan, int heads, int rows, int d) {
  return (size_t)plan.divided * heads * rows * (d + 2) * sizeof(float);
}

struct Partials {
  float *sums;  // (divided unit, head, row, d)
  float2 *ml;   // (divided unit, head, row): maximum in powers of two (-inf: no key), denominator
};
inline Partials partials_at(void *scratch, const KeySplit &plan, int heads, int rows) {
  Partials p{nullptr, nullptr};
  if (plan.units == 0) return p;
  p.ml = static_cast<float2 *>(scratch);
  p.sums = reinterpret_cast<float *>(p.ml + (size_t)plan.divided * heads * rows);
  return p;
}

// A warp per row of a divided block: out = sum_i 2^(m_i - m) sums_i / sum_i 2^(m_i - m) l_i.  blockIdx.y: divided block; blockIdx.x: head
// and 8 rows.  d: a multiple of 4 up to 128.  Bound by its launch and the way to L2: a lane has a part's maximum and denominator, and
// four parts' sums are under way at once.  One part after the other, and a block of threads launched for every part, before: fp16, 2
// heads of 64, 1100 rows, causal 11.6 us for the call, 10.3 now; 2 heads of 128, 1433 rows, not causal, 20.2 and 16.2; 16 heads of
// 64, 2700 rows, not causal, 67.7 and 65.8; fp32, 2 heads of 64, 900 rows, causal 17.4 and 15.4.  The same bits.
template <typename O, int kRowsPerBlock>
__global__ void __launch_bounds__(256)
join_parts_kernel(const __grid_constant__ KeySplit plan, const Partials p, O *out, int sq, int hq, int d) {
  const int first_unit = plan.even ? blockIdx.y * plan.even : plan.begin[blockIdx.y];  // among the divided
  const KeyUnit u = key_unit(plan, plan.first + first_unit);
  const int n = u.parts;
  grid_dependency_wait();
  const int h = blockIdx.x / (kRowsPerBlock / 8), row = blockIdx.x % (kRowsPerBlock / 8) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int64_t t = (int64_t)u.block * kRowsPerBlock + row;
  if (t >= sq) return;
  const size_t step = (size_t)hq * kRowsPerBlock, first = ((size_t)first_unit * hq + h) * kRowsPerBlock + row;
  const float2 none = make_float2(-INFINITY, 0.f);  // no key, and perhaps no sums stored
  float m = -INFINITY;
  for (int i = lane; i < n; i += 32) m = fmaxf(m, p.ml[first + i * step].x);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  float l = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int base = 0; base < n; base += 32) {
    const float2 mine = base + lane < n ? p.ml[first + (base + lane) * step] : none;
    const bool there = !(mine.x == -INFINITY && mine.y == 0.f);
    const uint32_t parts = __ballot_sync(0xffffffffu, there);
    const float weight = there ? exp2f(mine.x - m) : 0.f;
    for (int i0 = 0; i0 < 32 && base + i0 < n; i0 += 4) {
      float4 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if ((parts >> (i0 + i)) & 1 && lane * 4 < d)
          v[i] = *reinterpret_cast<const float4 *>(p.sums + (first + (base + i0 + i) * step) * d + lane * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float w = __shfl_sync(0xffffffffu, weight, i0 + i), li = __shfl_sync(0xffffffffu, mine.y, i0 + i);
        if (!((parts >> (i0 + i)) & 1)) continue;
        l = fmaf(w, li, l);
        if (lane * 4 < d) {
          acc.x = fmaf(w, v[i].x, acc.x), acc.y = fmaf(w, v[i].y, acc.y);
          acc.z = fmaf(w, v[i].z, acc.z), acc.w = fmaf(w, v[i].w, acc.w);
        }
      }
    }
  }
  if (lane * 4 >= d) return;
  const float inv = l > 0.f ? 1.0f / l : 0.f;
  O *dst = out + ((size_t)t * hq + h) * d + lane * 4;
  stf(dst, acc.x * inv);
  stf(dst + 1, acc.y * inv);
  stf(dst + 2, acc.z * inv);
  stf(dst + 3, acc.w * inv);
}

}  // namespace axb

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

// What CTAs work on, per head: unit u is part `part` of `parts` of row block `block`.  units == 0: blocks as they are.  Units of
// divided blocks follow one another: `divided` of them from `first` on; only they have scratch.  kMost: units that a plan can have (it
// travels as a kernel's argument, so a kernel for whole blocks does without).
template <int kMost>
struct KeySplit {
  static constexpr int kMostUnits = kMost;
  int units, first, divided;
  uint16_t block[kMost];
  uint8_t part[kMost], parts[kMost];
};

// The first tile of part i of n.
__host__ __device__ inline int split_begin(int tiles, int part, int parts) { return (int)((int64_t)tiles * part / parts); }

// blocks row blocks of `heads` heads; tiles(b) key tiles in block b, not decreasing in b; part_cost: what a block or part costs beside
// its tiles, in tiles; least_gain: tiles in a row that a division has to save, as many as joining takes with its launch (the callers say what they measured);
// join_cost: what joining costs for each further part of a block, in tiles; places: blocks that run at once.
template <typename Plan, typename Tiles>
Plan plan_key_split(int64_t blocks, int heads, bool causal, float part_cost, float least_gain, Tiles tiles, int places = kSms,
                    float join_cost = 0.f) {
  Plan plan{};
  if (blocks > Plan::kMostUnits || heads > 2 * kSms) return plan;
  const int most = tiles((int)blocks - 1);
  int unsplit = 0, parts = 1, limit = 0;
  if (causal) {
    // The time of parts of at most `at_most` tiles: the longest where all run at once, else an even share and half of the last.
    const auto estimate = [&](int at_most) {
      int64_t count = 0, total = 0;
      int longest = 0, shortest = most;
      for (int b = 0; b < blocks; ++b) {
        const int t = tiles(b), n = (t + at_most - 1) / at_most;
        count += n;
        total += t;
        longest = (t + n - 1) / n > longest ? (t + n - 1) / n : longest;
        shortest = t / n < shortest ? t / n : shortest;
      }
      const float alone = longest + part_cost + join_cost * ((most - 1) / at_most);
      if (count * heads <= places) return alone;
      const float even = (total + part_cost * count) * heads / places + (shortest + part_cost) / 2;
      return even > alone ? even : alone;
    };
    float best = estimate(most) - least_gain;
    int64_t total = 0;
    for (int b = 0; b < blocks; ++b) total += tiles(b);
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
  int units = 0, divided = 0;
  for (int i = 0; i < blocks; ++i) {
    const int b = (int)blocks - 1 - i;  // under a causal mask the longest first
    // causal: the longest first, so the divided ones first; else the divided ones last
    const int n = causal ? (tiles(b) + limit - 1) / limit : i < unsplit ? 1 : parts;
    if (units + n > Plan::kMostUnits || n > 255) return plan;
    if (n > 1) {
      if (divided == 0) plan.first = units;
      divided += n;
    }
    for (int part = 0; part < n; ++part, ++units) {
      plan.block[units] = (uint16_t)b;
      plan.part[units] = (uint8_t)part;
      plan.parts[units] = (uint8_t)n;
    }
  }
  plan.units = units;
  plan.divided = divided;
  return plan;
}

// Scratch of a plan: per divided unit and head `rows` rows of d floats, and (maximum, denominator) of each row.
template <typename Plan>
size_t key_split_bytes(const Plan &plan, int heads, int rows, int d) {
  return (size_t)plan.divided * heads * rows * (d + 2) * sizeof(float);
}

struct Partials {
  float *sums;  // (divided unit, head, row, d)
  float2 *ml;   // (divided unit, head, row): maximum in powers of two (-inf: no key), denominator
};
template <typename Plan>
Partials partials_at(void *scratch, const Plan &plan, int heads, int rows) {
  Partials p{nullptr, nullptr};
  if (plan.units == 0) return p;
  p.ml = static_cast<float2 *>(scratch);
  p.sums = reinterpret_cast<float *>(p.ml + (size_t)plan.divided * heads * rows);
  return p;
}

// A warp per row of a divided block: out = sum_i 2^(m_i - m) sums_i / sum_i 2^(m_i - m) l_i.  blockIdx.y: divided unit (those that are
// no first part leave at once); blockIdx.x: head and 8 rows.  d: a multiple of 4 up to 128.
template <typename O, int kRowsPerBlock, typename Plan>
__global__ void __launch_bounds__(256) join_parts_kernel(const __grid_constant__ Plan plan, const Partials p, O *out, int sq, int hq, int d) {
  const int u = plan.first + blockIdx.y, n = plan.parts[u];
  if (plan.part[u] != 0) return;
  grid_dependency_wait();
  const int h = blockIdx.x / (kRowsPerBlock / 8), row = blockIdx.x % (kRowsPerBlock / 8) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int64_t t = (int64_t)plan.block[u] * kRowsPerBlock + row;
  if (t >= sq) return;
  const size_t step = (size_t)hq * kRowsPerBlock, first = ((size_t)blockIdx.y * hq + h) * kRowsPerBlock + row;
  float m = -INFINITY;
  for (int i = 0; i < n; ++i) m = fmaxf(m, p.ml[first + i * step].x);
  float l = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = 0; i < n; ++i) {
    const float2 ml = p.ml[first + i * step];
    if (ml.x == -INFINITY && ml.y == 0.f) continue;  // no key, and perhaps nothing stored
    const float w = exp2f(ml.x - m);
    l = fmaf(w, ml.y, l);
    if (lane * 4 < d) {
      const float4 v = *reinterpret_cast<const float4 *>(p.sums + (first + i * step) * d + lane * 4);
      acc.x = fmaf(w, v.x, acc.x), acc.y = fmaf(w, v.y, acc.y), acc.z = fmaf(w, v.z, acc.z), acc.w = fmaf(w, v.w, acc.w);
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

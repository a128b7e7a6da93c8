// Work distribution of the decode GEMVs: which CTA takes which weight rows of which experts.
#pragma once

#include "dst_common.cuh"

namespace dst {
namespace {

// A work unit is (expert, pass, block of RI weight rows): pass i covers the expert's token rows
// ra + i MT .. (MT at most). Only experts with rows have units; they are numbered expert by expert, pass by pass, row
// block by row block, and every CTA takes an equal, contiguous run of them, so a pass's token rows are staged once per CTA.
// Experts without rows get no share of the grid: a decode step that reaches 6 of 384 experts ran on ten of the 592 CTAs
// when the runs were cut over all experts' row blocks (one token, two stacked terms: 563 us for both GEMVs, 31 now).
// P: a parameter block with offsets, E, T and NT (the 128-row tiles of an expert).
template <int RI>
__host__ __device__ __forceinline__ int blocks_per_expert(int NT) { return (NT * 128 + RI - 1) / RI; }

// Passes at most of T rows on E experts: the sum of ceil(rows / MT) over the experts that have some.
template <int MT>
inline long long max_passes(long long E, long long T) { return (T + (MT - 1) * (E < T ? E : T)) / MT; }

// a / b for 0 <= a, 0 < b < 2^31, in 32 bits where a allows it (a 64-bit division is some hundred instructions)
__device__ __forceinline__ long long div_small(long long a, int b) {
  return a <= 0xffffffffLL ? (long long)((uint32_t)a / (uint32_t)b) : a / b;
}

struct Unit {
  int e, n0;           // expert and first weight row
  int64_t ra, rb, m0;  // the expert's token rows [ra, rb) and the pass's first one
};

// A warp's position in the unit sequence (the same in all its lanes; every call is made by the whole warp).
template <int MT, int RI>
struct UnitWalk {
  int block, blocks;  // row block inside the pass
  Unit u;
  // local = the unit's index among the units of expert e (which has rows)
  template <typename P>
  __device__ __forceinline__ void start(const P& p, int e, long long local) {
    blocks = blocks_per_expert<RI>(p.NT);
    u.e = e;
    row_range(p.offsets, e, p.T, u.ra, u.rb);
    const long long pass = div_small(local, blocks);
    block = (int)(local - pass * blocks);
    u.m0 = u.ra + pass * MT;
    u.n0 = block * RI;
  }
  template <typename P>
  __device__ __forceinline__ void next(const P& p) {
    if (++block == blocks) {
      block = 0;
      u.m0 += MT;
      if (u.m0 >= u.rb) {
        // the next expert with rows, 32 at a time (an empty or inverted range has none)
        const int lane = threadIdx.x & 31;
        for (int e0 = u.e + 1; e0 < p.E; e0 += 32) {
          int64_t a = 0, b = 0;
          if (e0 + lane < p.E) row_range(p.offsets, e0 + lane, p.T, a, b);
          const uint32_t some = __ballot_sync(0xffffffffu, b > a);
          if (some) {
            const int src = __ffs(some) - 1;
            u.e = e0 + src;
            u.ra = __shfl_sync(0xffffffffu, a, src);
            u.rb = __shfl_sync(0xffffffffu, b, src);
            break;
          }
        }
        u.m0 = u.ra;
      }
    }
    u.n0 = block * RI;
  }
};

// The CTA's run of units, found by all its threads together: every thread counts the units of a contiguous run of experts,
// a block-wide scan gives their number and the expert that holds the CTA's first unit. scratch: one long long per warp.
struct UnitRun {
  long long count;    // units of this CTA
  long long local;    // the first one's index among the units of expert e
  int e;
};
template <int MT, int RI, int THREADS, typename P>
__device__ __forceinline__ void find_run(const P& p, long long* scratch, UnitRun* run) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (p.E + THREADS - 1) / THREADS;
  const int e0 = threadIdx.x * per, e1 = e0 + per < p.E ? e0 + per : p.E;
  const int blocks = blocks_per_expert<RI>(p.NT);
  auto units_of = [&](int e) -> long long {
    int64_t a, b;
    row_range(p.offsets, e, p.T, a, b);
    return (b - a + MT - 1) / MT * blocks;
  };
  // this CTA's share of `total` units: equal runs. Fewer units than CTAs: one each for the first CTAs, which start on different
  // SMs (spread over all CTAs instead, every second one of a grid twice the units left half of the SMs idle)
  auto share = [&](long long total, long long& u0, long long& u1) {
    const int b = (int)blockIdx.x;
    const long long base = div_small(total, (int)gridDim.x), more = total - base * (long long)gridDim.x;
    u0 = base * b + (b < more ? b : more);
    u1 = u0 + base + (b < more ? 1 : 0);
  };
  if (p.E == 1) {  // one matrix: nothing to look for
    if (threadIdx.x == 0) {
      long long u0, u1;
      share(units_of(0), u0, u1);
      run->e = 0;
      run->local = u0;
      run->count = u1 - u0;
    }
    __syncthreads();
    return;
  }
  long long sum = 0;
  for (int e = e0; e < e1; ++e) sum += units_of(e);
  long long incl = sum;
  for (int d = 1; d < 32; d <<= 1) {
    const long long up = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += up;
  }
  if (lane == 31) scratch[warp] = incl;
  if (threadIdx.x == 0) run->count = 0;
  __syncthreads();
  long long before = incl - sum, total = 0;
  for (int w = 0; w < THREADS / 32; ++w) {
    if (w < warp) before += scratch[w];
    total += scratch[w];
  }
  long long u0, u1;
  share(total, u0, u1);
  if (u0 < u1 && u0 >= before && u0 < before + sum) {
    long long left = u0 - before;
    for (int e = e0; e < e1; ++e) {
      const long long n = units_of(e);
      if (left < n) {
        run->e = e;
        run->local = left;
        run->count = u1 - u0;
        break;
      }
      left -= n;
    }
  }
  __syncthreads();
}

}  // namespace
}  // namespace dst

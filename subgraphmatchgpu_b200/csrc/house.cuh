// Houses of a root task by two-path counters (device code).
//
// The house (Q4) is an edge a - b (a < b) with a common neighbour c (the roof)
// and a three-path a - x - y - b beside it.  The LIGHT program, rooted at a,
// holds every (a, b, x) as a path and intersects N(b) with N(x) for each,
// ranking every y in the roofs.  Per root a, with c(y) = the number of
// two-paths a - x - y:
//
//   t_b = |N(a) ∩ N(b)| = c(b)                        roofs of a - b
//   Q_b = sum over y in N(b), y != a, of c(y) - 1     three-paths (x = b left out)
//   houses of a - b = t_b Q_b - sum over c in N(a) ∩ N(b) of
//                     [(c(c) - 1) + (|N(b) ∩ N(c)| - 1)]
//
// The bracket takes away the three-paths that pass through the roof, as y or
// as x.  Everything but |N(b) ∩ N(c)| comes from the counters: one shared-
// memory increment per two-path and one read per element of N(b).  The last
// term is a level program of its own (one intersection per triangle instead of
// one per (a, b, x); the caller subtracts it).  Needs a symmetric graph with
// strictly increasing lists and no self loop.
//
// 1024 roots of degree <= 1024 of R-MAT s18 ef16, whole calls: 8.8-11.9 ms by
// the level program, 1.30 ms by this (k_house 0.4, the triangles' intersections
// 0.3; with a root's ranges one after another and the triangles on the warp
// kernel 2.3 ms).
#pragma once

#include "cycle.cuh"
#include "kernels.cuh"

namespace sme {
namespace dev {

// A root takes the counters when it has at most kHouseCand neighbours (one
// per thread) and its neighbours above it times the elements of all its
// neighbours' lists (a measure of what the level program intersects) reach
// kHouseWork per counter range; the others stay with the level program.  A
// range costs a CTA about 12 us (81 ns of the device), a path of the level
// program 1-3 ns of the device on short lists and up to 300 us of one warp
// between two hubs: a flat graph of degree 8 (a product of 256) is better off
// with the level program, one of degree 32 (16 000) with the counters, and so
// is a root of few neighbours that are hubs.
constexpr uint32_t kHouseCand = CYC_THREADS;
constexpr uint32_t kHouseWork = 4096;
constexpr uint32_t kHouseTile = kCycleTable / 2;  // 16-bit counters per range
constexpr size_t kHouseSmem = kCycleCtaSmem + (size_t)kHouseCand * 8;
constexpr uint32_t kHouseMark = 0x8000u;  // y is in N(a); c(y) <= 1024 stays below

// Sorts the roots, one warp each.
__global__ void __launch_bounds__(WARP_BLOCK) k_house_split(DGraph G, const uint32_t* __restrict__ roots, uint32_t P,
                                                            uint64_t least, uint32_t* kept, uint32_t* left,
                                                            uint32_t* n) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t p = gw; p < P; p += nw) {
    const uint32_t a = __ldg(roots + p);
    const uint32_t* L;
    uint32_t d;
    AdjList(G, a, L, d);
    uint32_t above = 0;
    unsigned long long work = 0;
    if (d <= kHouseCand)
      for (uint32_t i = lane; i < d; i += 32) {
        const uint32_t x = __ldg(L + i);
        above += x > a;
        work += __ldg(G.rp + x + 1) - __ldg(G.rp + x);
      }
    above = __reduce_add_sync(FULL, above);
    work = WarpSum(work);
    if (lane == 0) {
      if (above * work >= least) kept[atomicAdd(n, 1u)] = a;
      else left[atomicAdd(n + 1, 1u)] = a;
    }
  }
}

// One CTA per root and range of y (the ranges of a large root run on different
// SMs); Q_b and t_b add up in `Qs` and `roofs`, kHouseCand of them per root
// (cleared by the caller), and k_house_sum multiplies them.  Thread i has
// neighbour i; the neighbours' lists, cut to the range, are concatenated and
// walked in segments (k_cycle4_cta's way), first to count, then, from the
// first neighbour above a on, to read.
__global__ void __launch_bounds__(CYC_THREADS, 1) k_house(DGraph G, uint32_t n, const uint32_t* __restrict__ roots,
                                                          uint32_t items, uint32_t ranges, uint32_t* next,
                                                          unsigned long long* Qs, uint32_t* roofs,
                                                          unsigned long long* acc) {
  extern __shared__ uint64_t hs_sh[];
  uint64_t* off = hs_sh;
  uint64_t* ptr = off + CYC_THREADS + 2;
  unsigned long long* Q = reinterpret_cast<unsigned long long*>(ptr + CYC_THREADS);
  uint32_t* table = reinterpret_cast<uint32_t*>(Q + kHouseCand);
  __shared__ uint64_t wtot[32];
  __shared__ uint32_t s_item;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  unsigned long long local = 0, bytes = 0;
  while (true) {
    if (tid == 0) s_item = atomicAdd(next, 1u);
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= items) break;
    const uint32_t slot = it / ranges;
    const uint32_t a = __ldg(roots + slot);
    const uint32_t* L;
    uint32_t d;
    AdjList(G, a, L, d);
    const uint32_t r0 = WarpLowerBound(L, d, a + 1);  // first neighbour above a
    const uint32_t v = tid < d ? __ldg(L + tid) : 0xFFFFFFFFu;
    const uint32_t* vl = nullptr;
    uint32_t vn = 0;
    if (tid < d) AdjList(G, v, vl, vn);
    Q[tid] = 0;
    {
      const uint64_t t0 = (uint64_t)(it % ranges) * kHouseTile;
      const uint64_t t1 = t0 + kHouseTile < n ? t0 + kHouseTile : n;
      uint4* q = reinterpret_cast<uint4*>(table);
      for (uint32_t i = tid; i < (uint32_t)((t1 - t0 + 7) / 8); i += CYC_THREADS) q[i] = make_uint4(0, 0, 0, 0);
      const uint32_t done = t0 ? LowerBound(vl, vn, (uint32_t)t0) : 0;
      const uint32_t len = (t1 >= n ? vn : LowerBound(vl, vn, (uint32_t)t1)) - done;
      const uint64_t incl = CtaInclusive(len, wtot);
      off[tid] = incl - len;
      ptr[tid] = (uint64_t)(uintptr_t)(vl + done);
      const uint64_t sum = wtot[31];
      if (tid == 0) off[CYC_THREADS] = sum;
      __syncthreads();  // offsets, pointers and the cleared counters are visible
      const uint64_t from = off[r0 < CYC_THREADS ? r0 : CYC_THREADS];
      if (tid == 0) bytes += 4ULL * sum + 4ULL * (sum - from);
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
        // pass 0 counts every element; pass 1 reads those of the lists above a
        for (uint64_t f0 = (pass ? from : 0) + (uint64_t)wid * kCycleSeg; f0 < sum;
             f0 += (uint64_t)(CYC_THREADS / 32) * kCycleSeg) {
          int j = 0;  // last list whose offset is <= f0 (uniform in the warp)
#pragma unroll
          for (int o = CYC_THREADS / 2; o > 0; o >>= 1)
            if (off[j + o] <= f0) j += o;
          const uint64_t f1 = f0 + kCycleSeg < sum ? f0 + kCycleSeg : sum;
          int jq = j;  // list of the running sum
          unsigned long long run = 0;
          for (uint64_t f = f0 + lane; f < f1; f += 128) {
            uint32_t y[4];
            int js[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const uint64_t g = f + 32 * t;
              if (g < f1) {
                while (off[j + 1] <= g) ++j;  // ends: off[CYC_THREADS] = sum > g
                y[t] = __ldg(reinterpret_cast<const uint32_t*>(ptr[j]) + (g - off[j]));
              }
              js[t] = j;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              if (f + 32 * t >= f1) break;
              const uint32_t k = (uint32_t)(y[t] - t0), sh = (k & 1) * 16;
              if (pass == 0) {
                atomicAdd(table + (k >> 1), 1u << sh);
              } else if (y[t] != a) {
                const uint32_t c = (table[k >> 1] >> sh) & 0xFFFFu;
                const uint32_t w = (c & (kHouseMark - 1)) - 1;  // b itself is among the x
                if (js[t] != jq) {
                  if (run) atomicAdd(Q + jq, run);
                  jq = js[t];
                  run = 0;
                }
                run += w;
                if (c & kHouseMark) local -= w;  // y is a roof: three-paths through it
              }
            }
          }
          if (pass) {
            // mostly every lane ends in the segment's only list
            __syncwarp();
            const int j0 = __shfl_sync(FULL, jq, 0);
            if (__all_sync(FULL, jq == j0)) {
              run = WarpSum(run);
              if (lane == 0 && run) atomicAdd(Q + j0, run);
            } else if (run) {
              atomicAdd(Q + jq, run);
            }
          }
        }
        __syncthreads();
        if (pass == 0) {
          if (v >= t0 && v < t1) {  // (an unused thread's v is above every range)
            const uint32_t k = (uint32_t)(v - t0), sh = (k & 1) * 16;
            roofs[(size_t)slot * kHouseCand + tid] = (table[k >> 1] >> sh) & (kHouseMark - 1);
            atomicOr(table + (k >> 1), kHouseMark << sh);
          }
          __syncthreads();
        }
      }
    }
    if (Q[tid]) atomicAdd(Qs + (size_t)slot * kHouseCand + tid, Q[tid]);
    if (tid == 0) bytes += 12ULL * d;
    __syncthreads();  // Q and s_item are rewritten
  }
  local = WarpSum(local);
  if (lane == 0 && local) atomicAdd(acc, local);
  if (tid == 0 && bytes) atomicAdd(acc + 1, bytes);
}

// Sum of t_b Q_b over the roots' neighbours above them (Q_b is 0 for the rest).
__global__ void __launch_bounds__(WARP_BLOCK) k_house_sum(const unsigned long long* __restrict__ Qs,
                                                          const uint32_t* __restrict__ roofs, uint64_t entries,
                                                          unsigned long long* acc) {
  unsigned long long local = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < entries; i += (uint64_t)gridDim.x * blockDim.x)
    local += Qs[i] * roofs[i];
  local = WarpSum(local);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(acc, local);
}

}  // namespace dev
}  // namespace sme

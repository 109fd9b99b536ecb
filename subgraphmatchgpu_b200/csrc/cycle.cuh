// 4-cycles of a root task by counting two-paths (device code).
//
// The level programs of Q1 intersect N(u0) with N(u2) once per two-path
// u0 - u1 - u2.  The same number follows from the two-paths alone: with
// u0 < u1, u2, u3 and u1 < u3, the cycles through a root u0 and an opposite
// vertex w are the pairs of distinct u1 in N(u0) ∩ N(w), all above u0, so a
// root contributes sum over w of c(w)(c(w)-1)/2, c(w) = the number of
// two-paths u0 - u1 - w with u1, w > u0.  Each two-path is one increment of
// a counter whose previous value is added to the count (0 + 1 + ... + c-1).
// That needs u1 in N(w) whenever w is in N(u1): the graph must be symmetric
// with strictly increasing lists and no self loop (k_check_simple).
//
// What bounds it: one list element read (L2) and one shared-memory atomic per
// two-path, against a search or a walk of dozens of elements per two-path in
// the level program.  Whole calls, level program against this: R-MAT s20
// ef16, 512 roots of degree <= 1024 (9 300 two-paths a root) 3.79 -> 0.27 ms
// (0.47 with a root's counter ranges one after another in one CTA);
// a Barabasi-Albert graph of 30 011 vertices and 9 edges a vertex, every root
// (113 two-paths a root) 3.83 -> 0.23 ms.
#pragma once

#include "kernels.cuh"

namespace sme {
namespace dev {

// ---- input contract of the counting kernels ---------------------------------
// flag bit 0: a list is not strictly increasing or holds its own vertex;
// bit 1 (sym): some v in N(u) has no u in N(v).  Warps take chunks of
// consecutive edges, so a hub's list is spread over many warps.
constexpr uint32_t kNotSimple = 1u, kNotSymmetric = 2u;

// Last u in [0, n) with rp[u] <= e (the owner of edge e), by the whole warp.
__device__ __forceinline__ uint32_t WarpOwner(const uint64_t* __restrict__ rp, uint32_t n, uint64_t e) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = 0, len = n;  // first index with rp > e lies in [lo, lo + len]
  while (len > 32) {
    const uint32_t step = (len + 31) / 32;
    const uint32_t idx = lo + lane * step;
    const bool le = idx < lo + len && __ldg(rp + idx) <= e;
    const uint32_t k = __popc(__ballot_sync(FULL, le));
    if (k == 0) return lo ? lo - 1 : 0;
    const uint32_t nlo = lo + (k - 1) * step + 1;
    const uint32_t nhi = min(lo + k * step, lo + len);
    lo = nlo;
    len = nhi - nlo;
  }
  const bool le = lane < len && __ldg(rp + lo + lane) <= e;
  lo += __popc(__ballot_sync(FULL, le));
  return lo ? lo - 1 : 0;
}

template <bool SYM>
__global__ void __launch_bounds__(WARP_BLOCK) k_check_simple(DGraph G, uint32_t n, uint64_t m, uint32_t chunk,
                                                             uint32_t* flag) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t bad = 0;
  for (uint64_t c0 = gw * chunk; c0 < m; c0 += nw * chunk) {
    const uint64_t c1 = c0 + chunk < m ? c0 + chunk : m;
    uint32_t u = WarpOwner(G.rp, n, c0);
    for (uint64_t e = c0 + lane; e < c1; e += 32) {
      while (__ldg(G.rp + u + 1) <= e) ++u;  // ends: rp[n] = m > e
      const uint32_t x = __ldg(G.cols + e);
      if (x == u || (e > __ldg(G.rp + u) && __ldg(G.cols + e - 1) >= x)) bad |= kNotSimple;
      if (SYM && x != u) {
        const uint32_t* bm = HubBitmap(G, x);
        bool in;
        if (bm) {
          in = BitTest(bm, u);
        } else {
          const uint32_t* a;
          uint32_t len;
          AdjList(G, x, a, len);
          const uint32_t pos = LowerBound(a, len, u);
          in = pos < len && __ldg(a + pos) == u;
        }
        if (!in) bad |= kNotSymmetric;
      }
    }
  }
  bad = __reduce_or_sync(FULL, bad);
  if (lane == 0 && bad) atomicOr(flag, bad);
}

// ---- shared-memory counters ---------------------------------------------------
constexpr uint32_t kNoKey = 0xFFFFFFFFu;

// One more two-path to w in an open-addressed table of 2^lg slots (16-bit
// counters, two to a word); returns how many there were before.  The callers
// keep the number of insertions below the number of slots, so a free slot or
// w's own is always found.
__device__ __forceinline__ uint32_t HashBump(uint32_t* keys, uint32_t* cnt, uint32_t lg, uint32_t w) {
  const uint32_t mask = (1u << lg) - 1;
  uint32_t h = (w * 2654435761u) >> (32 - lg);
  while (true) {
    uint32_t k = keys[h];
    if (k == kNoKey) k = atomicCAS(keys + h, kNoKey, w);
    if (k == kNoKey || k == w) break;
    h = (h + 1) & mask;
  }
  const uint32_t sh = (h & 1) * 16;
  return (atomicAdd(cnt + (h >> 1), 1u << sh) >> sh) & 0xFFFFu;
}

// Roots of at most kCycleWarpMax two-paths: one warp and a table of its own
// each (sixteen warps of 6 KB, two CTAs per SM).  The others go to `queue`.
// The lanes hold 32 of the root's neighbours at a time and walk the
// concatenation of their clipped lists, so short lists keep every lane busy.
constexpr int CYW_THREADS = 512;
constexpr int CYW_WARPS = CYW_THREADS / 32;
constexpr uint32_t kCycleWarpLg = 10;
constexpr uint32_t kCycleWarpMax = 640;
constexpr uint32_t kCycleWarpCand = 64;  // a warp searches 32 lists at a time, a CTA 1024
constexpr size_t kCycleWarpSmem = (size_t)CYW_WARPS * ((4u << kCycleWarpLg) + (2u << kCycleWarpLg));

// The part of u1's list above u0 (u1 = the i-th candidate), per lane.
__device__ __forceinline__ void TwoPathRange(const DGraph& G, uint32_t u1, uint32_t u0, const uint32_t*& a,
                                             uint32_t& len) {
  AdjList(G, u1, a, len);
  const uint32_t lo = LowerBound(a, len, u0 + 1);
  a += lo;
  len -= lo;
}

__global__ void __launch_bounds__(CYW_THREADS, 2) k_cycle4_warp(DGraph G, const uint32_t* __restrict__ roots,
                                                                uint32_t P, uint32_t* next, uint32_t* queue,
                                                                uint32_t* nqueue, unsigned long long* acc) {
  extern __shared__ uint32_t cy_sh[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t* keys = cy_sh + wid * (3u << (kCycleWarpLg - 1));
  uint32_t* cnt = keys + (1u << kCycleWarpLg);
  unsigned long long local = 0, bytes = 0;
  while (true) {
    uint32_t p = 0;
    if (lane == 0) p = atomicAdd(next, 1u);
    p = __shfl_sync(FULL, p, 0);
    if (p >= P) break;
    const uint32_t u0 = __ldg(roots + p);
    const uint32_t* L;
    uint32_t d;
    AdjList(G, u0, L, d);
    const uint32_t r0 = WarpLowerBound(L, d, u0 + 1);
    L += r0;
    d -= r0;
    const uint32_t* a = nullptr;
    uint32_t len = 0, total = d > kCycleWarpCand ? kCycleWarpMax + 1 : 0;
    for (uint32_t i0 = 0; i0 < d && total <= kCycleWarpMax; i0 += 32) {
      len = 0;
      if (i0 + lane < d) TwoPathRange(G, __ldg(L + i0 + lane), u0, a, len);
      const uint32_t capped = min(len, kCycleWarpMax + 1);  // 32 of them stay far below 2^32
      total += __reduce_add_sync(FULL, capped);
    }
    if (total > kCycleWarpMax) {
      if (lane == 0) queue[atomicAdd(nqueue, 1u)] = p;
      continue;
    }
    if (total < 2) continue;
    if (lane == 0) bytes += 12ULL * d + 4ULL * total;
    // a table of at least 1.6 slots per two-path
    uint32_t lg = 33 - __clz(total);
    if (lg < 5) lg = 5;
    if (lg > kCycleWarpLg) lg = kCycleWarpLg;
    for (uint32_t i = lane; i < (1u << lg); i += 32) keys[i] = kNoKey;
    for (uint32_t i = lane; i < (1u << (lg - 1)); i += 32) cnt[i] = 0;
    __syncwarp();
    for (uint32_t i0 = 0; i0 < d; i0 += 32) {
      if (d > 32) {  // else the lanes still hold the only chunk
        len = 0;
        if (i0 + lane < d) TwoPathRange(G, __ldg(L + i0 + lane), u0, a, len);
      }
      uint32_t incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
      }
      const uint32_t sum = __shfl_sync(FULL, incl, 31);
      for (uint32_t f0 = 0; f0 < sum; f0 += 32) {
        const uint32_t f = f0 + lane;
        // owner: the number of lanes whose inclusive length is <= f
        int j = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const uint32_t y = __shfl_sync(FULL, incl, j + o - 1);
          if (y <= f) j += o;
        }
        const uint32_t before = __shfl_sync(FULL, incl - len, j & 31);
        const uint64_t base = __shfl_sync(FULL, (unsigned long long)(uintptr_t)a, j & 31);
        if (f < sum) {
          const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(base) + (f - before));
          local += HashBump(keys, cnt, lg, w);
        }
      }
    }
    __syncwarp();  // the table is cleared for the next root
  }
  local = WarpSum(local);
  if (lane == 0 && local) atomicAdd(acc, local);
  if (lane == 0 && bytes) atomicAdd(acc + 1, bytes);
}

// Roots with more two-paths.  Up to kCycleHashMax of them go through one
// table in a CTA's shared memory (TILED 0).  More are counted in direct 16-bit
// counters (32-bit ones when the root has 65536 or more candidates), one
// range of w at a time; the ranges are independent, so they are queued and
// different CTAs take them (TILED 1).  Neighbours are taken 1024 at a time,
// one per thread; their clipped lists are concatenated and cut into segments
// of kCycleSeg elements, a warp finding a segment's first list by one search
// and keeping four loads in flight per lane.
constexpr int CYC_THREADS = 1024;
constexpr uint32_t kCycleHashLg = 15;
constexpr uint32_t kCycleHashMax = 24576;  // 3/4 of the slots
constexpr uint32_t kCycleSeg = 256;
constexpr uint32_t kCycleTable = (4u << kCycleHashLg) + (2u << kCycleHashLg);  // bytes
constexpr size_t kCycleCtaSmem = kCycleTable + (size_t)(CYC_THREADS + 2) * 8 + CYC_THREADS * 8;

// Inclusive sum over the CTA's threads (CYC_THREADS of them).
__device__ __forceinline__ uint64_t CtaInclusive(uint64_t v, uint64_t* wtot) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(FULL, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) wtot[wid] = v;
  __syncthreads();
  if (wid == 0) {
    uint64_t t = wtot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(FULL, t, o);
      if (lane >= o) t += y;
    }
    wtot[lane] = t;
  }
  __syncthreads();
  return v + (wid ? wtot[wid - 1] : 0);
}

// A range costs a CTA its clearing and two searches in every neighbour's list,
// 50 ns of the device and 0.31 a neighbour, a two-path of the level program
// 0.42 ns and more (trees under 64 and 512 roots with 10, 100 and 300
// neighbours in graphs of 2^18 to 2^25 vertices).  A root whose two-paths are
// fewer than its ranges ask for goes to `left`, which the level program takes:
// 512 roots of 30 000 two-paths and 300 neighbours each, 2^25 vertices, 24.1
// ms by counters, 5.1 by the level program; 2^22 vertices 2.1 and 5.
__device__ __forceinline__ bool RangesPay(uint64_t two_paths, uint32_t ranges, uint32_t d) {
  return ranges == 1 || two_paths >= (uint64_t)ranges * (128 + 3ull * d / 4);
}

// Entries of `tiles`: queued root index << 32 | range.
template <bool TILED>
__global__ void __launch_bounds__(CYC_THREADS, 1) k_cycle4_cta(DGraph G, uint32_t n,
                                                               const uint32_t* __restrict__ roots,
                                                               const uint32_t* __restrict__ queue,
                                                               const uint32_t* __restrict__ nqueue, uint32_t* next,
                                                               uint64_t* tiles, uint32_t* ntiles, uint32_t tiles_cap,
                                                               uint32_t* left, uint32_t* nleft, uint32_t* err,
                                                               unsigned long long* acc) {
  extern __shared__ uint64_t cyc_sh[];
  uint64_t* off = cyc_sh;                 // exclusive offsets of the chunk's lists, then their sum
  uint64_t* ptr = off + CYC_THREADS + 2;  // first element of each (16-byte aligned, as is the table)
  uint32_t* table = reinterpret_cast<uint32_t*>(ptr + CYC_THREADS);
  __shared__ uint64_t wtot[32];
  __shared__ uint32_t s_item;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t nq = TILED ? min(*ntiles, tiles_cap) : *nqueue;
  unsigned long long local = 0, bytes = 0;
  while (true) {
    if (tid == 0) s_item = atomicAdd(next, 1u);
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= nq) break;
    const uint32_t slot = TILED ? (uint32_t)(tiles[it] >> 32) : it;
    const uint32_t u0 = __ldg(roots + queue[slot]);
    const uint32_t* L;
    uint32_t d;
    AdjList(G, u0, L, d);
    const uint32_t r0 = WarpLowerBound(L, d, u0 + 1);
    L += r0;
    d -= r0;
    const bool wide = d > 0xFFFFu;
    const uint64_t tile = kCycleTable / (wide ? 4 : 2);  // counters per range
    const uint32_t* a = nullptr;
    uint32_t len = 0, lg = 10, clear, nkeys = 0;
    uint64_t t0 = 0, t1 = 0;
    if (TILED) {
      t0 = (uint64_t)u0 + 1 + (uint32_t)tiles[it] * tile;
      t1 = t0 + tile < n ? t0 + tile : n;
      clear = (uint32_t)(((t1 - t0) * (wide ? 4 : 2) + 15) / 16);
    } else {
      // two-paths of the root (ranges of up to 1024 candidates stay in registers)
      uint64_t mine = 0;
      for (uint32_t i = tid; i < d; i += CYC_THREADS) {
        TwoPathRange(G, __ldg(L + i), u0, a, len);
        mine += len;
      }
      CtaInclusive(mine, wtot);
      const uint64_t total = wtot[31];
      __syncthreads();  // wtot and s_item are rewritten
      if (tid == 0) bytes += 12ULL * d + 4ULL * total;
      if (total > kCycleHashMax) {
        const uint32_t ranges = (uint32_t)((n - 1 - (uint64_t)u0 + tile - 1) / tile);
        if (tid == 0) {
          const bool pay = RangesPay(total, ranges, d);
          if (!pay) left[atomicAdd(nleft, 1u)] = u0;  // a queued root once at most
          const uint32_t count = pay ? ranges : 0;
          const uint32_t at = atomicAdd(ntiles, count);
          for (uint32_t k = 0; k < count; ++k)
            if (at + k < tiles_cap) tiles[at + k] = (uint64_t)slot << 32 | k;
            else atomicOr(err, ENGINE_ERR_BOUNDS);
        }
        continue;
      }
      while ((3u << lg) / 4 < total) ++lg;  // <= kCycleHashLg
      clear = (6u << lg) / 16;
      nkeys = (4u << lg) / 16;
    }
    uint32_t* cnt = table + (1u << lg);  // hash: counters after the keys
    uint4* q = reinterpret_cast<uint4*>(table);
    for (uint32_t i = tid; i < clear; i += CYC_THREADS)
      q[i] = i < nkeys ? make_uint4(kNoKey, kNoKey, kNoKey, kNoKey) : make_uint4(0, 0, 0, 0);
    for (uint32_t i0 = 0; i0 < d; i0 += CYC_THREADS) {
      if (TILED) {
        len = 0;
        if (i0 + tid < d) {
          AdjList(G, __ldg(L + i0 + tid), a, len);
          const uint32_t s0 = LowerBound(a, len, (uint32_t)t0);
          const uint32_t s1 = t1 >= n ? len : LowerBound(a, len, (uint32_t)t1);
          a += s0;
          len = s1 - s0;
        }
      } else if (d > CYC_THREADS) {
        len = 0;
        if (i0 + tid < d) TwoPathRange(G, __ldg(L + i0 + tid), u0, a, len);
      }
      const uint64_t incl = CtaInclusive(len, wtot);
      off[tid] = incl - len;
      ptr[tid] = (uint64_t)(uintptr_t)a;
      const uint64_t sum = wtot[31];
      if (tid == 0) off[CYC_THREADS] = sum;
      __syncthreads();  // offsets, pointers and the cleared table are visible
      for (uint64_t f0 = (uint64_t)wid * kCycleSeg; f0 < sum; f0 += (uint64_t)(CYC_THREADS / 32) * kCycleSeg) {
        // last list whose offset is <= f0 (uniform in the warp)
        int j = 0;
#pragma unroll
        for (int o = CYC_THREADS / 2; o > 0; o >>= 1)
          if (off[j + o] <= f0) j += o;
        const uint64_t f1 = f0 + kCycleSeg < sum ? f0 + kCycleSeg : sum;
        for (uint64_t f = f0 + lane; f < f1; f += 128) {
          uint32_t w[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const uint64_t g = f + 32 * t;
            if (g < f1) {
              while (off[j + 1] <= g) ++j;  // ends: off[CYC_THREADS] = sum > g
              w[t] = __ldg(reinterpret_cast<const uint32_t*>(ptr[j]) + (g - off[j]));
            }
          }
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            if (f + 32 * t >= f1) break;
            if (!TILED) {
              local += HashBump(table, cnt, lg, w[t]);
            } else {
              const uint32_t k = (uint32_t)(w[t] - t0);
              if (wide) {
                local += atomicAdd(table + k, 1u);
              } else {
                const uint32_t sh = (k & 1) * 16;
                local += (atomicAdd(table + (k >> 1), 1u << sh) >> sh) & 0xFFFFu;
              }
            }
          }
        }
      }
      __syncthreads();  // the next chunk rewrites the offsets, the next root the table
    }
    __syncthreads();  // s_item is rewritten (a root without candidates passes no barrier above)
  }
  local = WarpSum(local);
  if (lane == 0 && local) atomicAdd(acc, local);
  if (tid == 0 && bytes) atomicAdd(acc + 1, bytes);
}

}  // namespace dev
}  // namespace sme

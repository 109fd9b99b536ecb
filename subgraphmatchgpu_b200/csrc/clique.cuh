// k-cliques (k = 3 to 6) of a root task on bit matrices (device code).
//
// The level programs of Q0, Q3, Q7 and Q11 hold every edge, triangle (and, for the
// larger cliques, every 4- and 5-clique) as a path and intersect lists once
// per path.  Here a root's candidates R = N(u0) above u0 (d of them) get a
// d x d bit matrix of the edges among them, built by one intersection per
// candidate; the (k-1)-cliques of R are then counted on its rows: k - 3 levels
// of one AND of two rows each and a last one of AND + popcount.  Rows are
// triangular (bit j of row i only for i < j), so a clique is counted once.
// Triangles need no matrix, the build's hits are the count; they come here
// only as a task of every root (see ORIENT).  Nothing is
// materialised and nothing leaves the SM but the count.  Whole
// calls, level program against this: 4-cliques of R-MAT s18 ef16, every root
// 73.0 -> 2.1 ms; 5-cliques of the oriented R-MAT s17 ef16 187 -> 5.0 ms;
// 4-cliques of 16 384 roots of R-MAT s20 ef16 0.91 -> 0.31 ms.
//
// Few roots are bound by the latency of the build's loads (hub bitmap words
// from HBM): hence four of them in flight per lane, 32 lists fetched at once
// and many warps per root (4-cliques, s20 roots: 0.80 -> 0.40 ms; 0.31 with the
// small class beside class M).  Many roots
// are bound by instruction issue: hence the candidates' hash table (1-2
// shared-memory reads per looked-up element, a binary search takes 8), the
// member lists compacted from their parent's by ballot (5-cliques, s17: 18 ->
// 8.5 ms together; expanding the bits of every AND took the other half) and,
// on short rows, pairs of members instead of a warp per member (-> 5.6 ms).
//
// A root's cost grows with d, so roots are sorted into classes by d: up to 32
// a warp and one word per row (k_clique_small); up to 256, 512 and 1024 (896
// for k = 6) a CTA with the matrix in shared memory; up to 4096 a CTA with
// the matrix in global scratch.  CTAs that find no root left help with the rows
// of large ones, each with a matrix of its own (CliqueParts); where large roots
// are few the level program takes them (CliqueLeast).
//
// ORIENT: the task is every root of a symmetric graph, whose count does not
// depend on the order of the vertices; the lists are then cut to the
// neighbours of higher (degree, id) first (k_orient), which bounds d by the
// square root of the stored edges (on R-MAT s18 the largest list falls from 15
// thousand to a few hundred).  The lists stay sorted by id, the matrix by
// index.
#pragma once

#include "cycle.cuh"
#include "kernels.cuh"

namespace sme {
namespace dev {

struct CView {
  DGraph G;
  const uint2* rng;       // ORIENT: list of v is ocols[rng[v].x .. rng[v].y)
  const uint32_t* ocols;
};

template <bool ORIENT>
__device__ __forceinline__ void CList(const CView& V, uint32_t v, const uint32_t*& a, uint32_t& len) {
  if (ORIENT) {
    const uint2 r = __ldg(V.rng + v);
    a = V.ocols + r.x;
    len = r.y - r.x;
  } else {
    AdjList(V.G, v, a, len);
  }
}

// ---- orientation by (degree, id) ------------------------------------------------
constexpr int ORI_THREADS = 256;
// Edges a warp takes: a chain of loads per 32 of them, so few while the graph
// is small (R-MAT s14, 230 000 edges: 27 + 42 us with 512, 8 + 11 with 64).
__host__ __device__ constexpr uint32_t OriWarp(uint64_t m) { return m < (4u << 20) ? 64 : 512; }
constexpr uint32_t OriTile(uint64_t m) { return OriWarp(m) * (ORI_THREADS / 32); }  // edges a CTA takes

__device__ __forceinline__ bool KeepsEdge(const uint64_t* rp, uint32_t u, uint64_t du, uint32_t x) {
  const uint64_t dx = __ldg(rp + x + 1) - __ldg(rp + x);
  return dx > du || (dx == du && x > u);
}

// FILL 0: one bit per edge into `keep` and the kept edges per tile into bs;
// FILL 1: bs holds their exclusive sums, the kept edges are written to ocols
// and every list's range to rng (cleared by the caller, so an empty list's
// range is empty).  Only the first pass gathers degrees.
template <bool FILL>
__global__ void __launch_bounds__(ORI_THREADS) k_orient(const uint64_t* __restrict__ rp,
                                                        const uint32_t* __restrict__ cols, uint32_t n, uint64_t m,
                                                        uint32_t* keep, uint64_t* bs, uint32_t* ocols, uint2* rng) {
  __shared__ uint32_t wkept[ORI_THREADS / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t per = OriWarp(m);
  const uint64_t c0 = ((uint64_t)blockIdx.x * (ORI_THREADS / 32) + wid) * per;
  const uint64_t c1 = c0 + per < m ? c0 + per : m;
  uint32_t kept = 0, mine = 0;  // mine: the warp's bits, lane k those of its k-th 32 edges
  if (FILL && c0 + 32ull * lane < c1 && lane < per / 32) mine = __ldg(keep + (c0 >> 5) + lane);
  uint32_t u = c0 < m ? WarpOwner(rp, n, c0) : 0;
  if (!FILL) {
    if (c0 < m) {
#pragma unroll 4
      for (uint32_t k = 0; k < per / 32; ++k) {
        const uint64_t e = c0 + k * 32 + lane;
        bool yes = false;
        if (e < c1) {
          const uint32_t x = __ldg(cols + e);
          while (__ldg(rp + u + 1) <= e) ++u;  // ends: rp[n] = m > e
          yes = KeepsEdge(rp, u, __ldg(rp + u + 1) - __ldg(rp + u), x);
        }
        const uint32_t bits = __ballot_sync(FULL, yes);
        if (lane == k) mine = bits;
      }
      if (lane < per / 32 && c0 + 32ull * lane < c1) keep[(c0 >> 5) + lane] = mine;
    }
  }
  kept = __reduce_add_sync(FULL, (unsigned)__popc(mine));
  if (lane == 0) wkept[wid] = kept;
  __syncthreads();
  if (!FILL) {
    if (threadIdx.x == 0) {
      uint32_t t = 0;
      for (int w = 0; w < ORI_THREADS / 32; ++w) t += wkept[w];
      bs[blockIdx.x] = t;
    }
    return;
  }
  uint64_t at = bs[blockIdx.x];
  for (int w = 0; w < wid; ++w) at += wkept[w];
  if (c0 >= m) return;
  for (uint32_t k = 0; k < per / 32; ++k) {
    const uint64_t e = c0 + k * 32 + lane;
    const uint32_t bits = __shfl_sync(FULL, mine, k);
    const bool yes = (bits >> lane) & 1;
    const uint32_t pos = (uint32_t)at + __popc(bits & ((1u << lane) - 1));
    if (e < c1) {
      while (__ldg(rp + u + 1) <= e) ++u;
      if (yes) ocols[pos] = __ldg(cols + e);
      if (e == __ldg(rp + u)) rng[u].x = pos;
      if (e + 1 == __ldg(rp + u + 1)) rng[u].y = pos + (yes ? 1 : 0);
    }
    at += __popc(bits);
  }
}

// ---- classes --------------------------------------------------------------------
constexpr uint32_t kCliqueS = 32, kCliqueM = 256, kCliqueL = 512, kCliqueG = 4096;
constexpr int kCliqueMThreads = 256;
constexpr uint32_t CliqueX(int k) { return k == 6 ? 896 : 1024; }
constexpr int kCliqueParts = 8;  // most CTAs of a root

// CTAs a root of d candidates may occupy: its counting work grows faster than
// the matrix that each of them builds.  Every root is first taken by one CTA;
// the others come after all roots have been, claim rows that are not counted
// yet and find nothing to build where the first one is through (5-cliques, 1500
// roots of 600 candidates without an edge among them: 1.88 ms with five fixed
// parts a root, 1.12 by the level program, 0.75 so; every root of R-MAT s18
// 17.5 ms and 16.8).  Triangles are counted while the rows are found, so there
// the rows are cut beforehand.
__device__ __forceinline__ uint32_t CliqueParts(int k, uint32_t d) {
  if (d <= kCliqueM) return 1;
  if (k == 3) return min((uint32_t)kCliqueParts, (d + 127) / 128);
  if (k == 4) return d <= 1024 ? 1 : min(8u, (d + 511) / 512);
  return min((uint32_t)kCliqueParts, (d + 127) / 128);
}

// Roots from which on classes L (cls 2), X and G are worth their kernels.  One root's
// matrix keeps a few CTAs busy for milliseconds while the level program spreads
// it over the device (blocks of R-MAT s18 and s20, matrices and level program):
// 5-cliques, 1 root of 513-1024 candidates 0.89 and 0.40 ms, 16 roots 1.04 and
// 1.05; 1 of 2501-4096 100 and 12 ms, 16 100 and 74, 64 153 and 278; 4-cliques,
// 1 of 1025-1500 0.69 and 0.23, 256 of them 3.0 and 5.8, of 1501-2500 5.7-7.2
// and 6.0, of 2501-4096 20-25 and 51; 6-cliques, 1 of 257-512 5.1 and 1.3, 16
// 5.1 and 2.8, 16 of 513-1024 11.4 and 9.0.  Classes L and X stay where classes M and L keep
// the device busy for as long anyway (5-cliques of the oriented R-MAT
// s17 5.0 ms, 5.4 with its few X roots in the level program).
constexpr uint32_t CliqueLeast(int k, int cls) {
  return k == 4 ? (cls == 4 ? 128 : 1) : cls == 4 ? 32 : k == 5 ? (cls == 3 ? 12 : 1) : (cls == 3 ? 32 : 48);
}

// Whether class G pays by how many of kCliqueSamples sampled pairs a root are
// joined: the matrix costs a look-up per list element whatever it holds, the
// level program ends where nothing is joined.  1000 roots with the same 1400 or
// 3000 candidates, matrices and level program, 4-cliques: no pair joined 3.1
// and 0.8, 11.9 and 1.6 ms, 1% 4.4 and 4.3, 19.1 and 17.5, 5% 5.6 and 18.6,
// 31.2 and 91.3; 5-cliques, 128 roots: 1% 1.1 and 0.8, 5.6 and 3.2, 5% 4.2 and
// 5.8, 43.5 and 38.8, 10% 11.9 and 24.2, 143 and 208; where the joined pairs are
// clustered the matrices win from fewer on (R-MAT s18, 256 roots of 1025-1500,
// between 3 and 6%: 17.7 and 90.8).
constexpr uint32_t kCliqueSamples = 4;
constexpr bool CliqueDense(int k, uint64_t joined, uint64_t roots) {
  return joined * 100 >= (k == 4 ? 2 : 3) * kCliqueSamples * roots;
}

struct CliqueQueues {
  uint32_t* q[5];   // S, M, L, X, G
  uint32_t* taken;  // rows claimed of each entry of L, then X and G (cleared)
  uint32_t cap[5];
  uint32_t* n;      // entries of each, left roots, joined pairs of G's samples, then the taken entries
  uint32_t* left;   // roots (vertex ids) above every class
  uint32_t left_cap;
  uint32_t* nleft;
  uint32_t top;     // largest d of class G (of class X when there is no room for scratch)
  uint32_t* err;
};

// Sorts the roots (by index) into the queues, whose capacities hold every
// possible entry (one that did not fit would raise the error flag).
template <int K, bool ORIENT>
__global__ void __launch_bounds__(256) k_clique_classify(CView V, const uint32_t* __restrict__ roots, uint32_t P,
                                                         CliqueQueues Q) {
  const int lane = threadIdx.x & 31;
  const uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
  for (uint32_t base = w0; base < P; base += gridDim.x * blockDim.x) {
    const uint32_t p = base + lane;
    uint32_t d = 0, u0 = 0;
    const uint32_t* a = nullptr;
    if (p < P) {
      u0 = __ldg(roots + p);
      CList<ORIENT>(V, u0, a, d);
      if (!ORIENT) {
        const uint32_t r0 = LowerBound(a, d, u0 + 1);
        a += r0;
        d -= r0;
      }
    }
    int cls = -1;
    if (d >= K - 1)
      cls = d <= kCliqueS ? 0 : d <= kCliqueM ? 1 : d <= kCliqueL ? 2 : d <= CliqueX(K) ? 3 : d <= Q.top ? 4 : 5;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const unsigned mask = __ballot_sync(FULL, cls == c);
      if (!mask) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(Q.n + c, (uint32_t)__popc(mask));
      at = __shfl_sync(FULL, at, 0) + __popc(mask & ((1u << lane) - 1));
      if (cls == c) {
        if (at < Q.cap[c]) Q.q[c][at] = p;
        else atomicOr(Q.err, ENGINE_ERR_BOUNDS);
      }
    }
    if (cls >= 2 && cls <= 4) {
      const uint32_t at = atomicAdd(Q.n + cls, 1u);
      if (at < Q.cap[cls]) Q.q[cls][at] = p;
      else atomicOr(Q.err, ENGINE_ERR_BOUNDS);
    }
    if (!ORIENT && cls == 4) {  // d is above a thousand
      uint32_t joined = 0;
      for (uint32_t t = 1; t <= kCliqueSamples; ++t) {
        const uint32_t h = (p * kCliqueSamples + t) * 2654435761u;
        const uint32_t i = (h >> 16) % d, k = (i + 1 + (h & 0xFFFFu) % (d - 1)) % d;  // k != i
        const uint32_t x = __ldg(a + min(i, k)), y = __ldg(a + max(i, k));
        const uint32_t* bm = HubBitmap(V.G, x);
        if (bm) {
          joined += BitTest(bm, y);
        } else {
          const uint32_t* b;
          uint32_t len;
          AdjList(V.G, x, b, len);
          const uint32_t pos = LowerBound(b, len, y);
          joined += pos < len && __ldg(b + pos) == y;
        }
      }
      if (joined) atomicAdd(Q.n + 6, joined);
    }
    if (cls == 5) {
      const uint32_t at = atomicAdd(Q.nleft, 1u);
      if (at < Q.left_cap) Q.left[at] = u0;
      else atomicOr(Q.err, ENGINE_ERR_BOUNDS);
    }
  }
}

// Roots (vertex ids) of a queue's entries.
__global__ void k_clique_roots(const uint32_t* __restrict__ roots, const uint32_t* __restrict__ q, uint32_t count,
                               uint32_t* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    out[i] = __ldg(roots + q[i]);
}

// Two lower bounds at once (LowerBound's steps, the loads of both in flight).
__device__ __forceinline__ void LowerBound2(const uint32_t* a, uint32_t na, uint32_t x, const uint32_t* b, uint32_t nb,
                                            uint32_t y, uint32_t& ra, uint32_t& rb) {
  const uint32_t *pa = a, *pb = b;
  uint32_t ca = na, cb = nb;
  while (ca > 1 || cb > 1) {
    const uint32_t ha = ca >> 1, hb = cb >> 1;  // 0 once one is down to an element
    const uint32_t va = ha ? __ldg(pa + ha) : 0xFFFFFFFFu, vb = hb ? __ldg(pb + hb) : 0xFFFFFFFFu;
    pa = va < x ? pa + ha : pa;
    pb = vb < y ? pb + hb : pb;
    ca -= ha;
    cb -= hb;
  }
  ra = na ? (uint32_t)(pa - a) + (__ldg(pa) < x ? 1u : 0u) : 0;
  rb = nb ? (uint32_t)(pb - b) + (__ldg(pb) < y ? 1u : 0u) : 0;
}

// ---- up to 32 candidates: a warp each ----------------------------------------------
template <int K>
__device__ __forceinline__ unsigned long long SmallCliques(const uint32_t* rows, uint32_t s) {
  // (K)-cliques inside the candidate bits s
  if constexpr (K == 1) {
    return __popc(s);
  } else {
    unsigned long long c = 0;
    for (uint32_t b = s; b; b &= b - 1) c += SmallCliques<K - 1>(rows, s & rows[__ffs(b) - 1]);
    return c;
  }
}

// The d(d-1)/2 pairs of candidates are spread over the lanes; a lane finds its
// pair's edge in the list of the lower one (ORIENT: of the one of lower
// (degree, id), whose list holds it), by a hub bitmap or a search.
template <int K, bool ORIENT>
__global__ void __launch_bounds__(WARP_BLOCK, 6) k_clique_small(CView V, const uint32_t* __restrict__ roots,
                                                                const uint32_t* __restrict__ q,
                                                                const uint32_t* __restrict__ nq, uint32_t cap,
                                                                unsigned long long* acc) {
  __shared__ uint32_t srows[WARP_BLOCK / 32][32];
  const int lane = threadIdx.x & 31;
  uint32_t* rows = srows[threadIdx.x >> 5];
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t count = min(*nq, cap);
  unsigned long long local = 0, bytes = 0;
  for (uint32_t i = gw; i < count; i += nw) {
    const uint32_t u0 = __ldg(roots + q[i]);
    const uint32_t* L;
    uint32_t d;
    CList<ORIENT>(V, u0, L, d);
    if (!ORIENT) {
      const uint32_t r0 = WarpLowerBound(L, d, u0 + 1);
      L += r0;
      d -= r0;
    }
    uint32_t x = 0, ln = 0, deg = 0;
    const uint32_t* lp = nullptr;
    const uint32_t* bm = nullptr;
    if (lane < d) {
      x = __ldg(L + lane);
      CList<ORIENT>(V, x, lp, ln);
      if (ORIENT) deg = (uint32_t)(__ldg(V.G.rp + x + 1) - __ldg(V.G.rp + x));
      else bm = HubBitmap(V.G, x);
    }
    rows[lane] = 0;
    __syncwarp();
    const uint32_t np = d * (d - 1) / 2;
    for (uint32_t f0 = 0; f0 < np; f0 += 64) {
      // two pairs per lane, their searches side by side
      uint32_t lo[2], hi[2], want[2], sn[2];
      const uint32_t* sp[2];
      bool in[2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const uint32_t f = f0 + t * 32 + lane;
        uint32_t b = (uint32_t)((1.0f + sqrtf(1.0f + 8.0f * (float)f)) * 0.5f);
        while (b * (b - 1) / 2 > f) --b;
        while ((b + 1) * b / 2 <= f) ++b;
        const uint32_t a = f - b * (b - 1) / 2;  // pair a < b
        const uint32_t xa = __shfl_sync(FULL, x, a & 31), xb = __shfl_sync(FULL, x, b & 31);
        uint32_t src = a & 31;
        want[t] = xb;
        if (ORIENT) {
          const uint32_t da = __shfl_sync(FULL, deg, a & 31), db = __shfl_sync(FULL, deg, b & 31);
          if (db < da || (db == da && xb < xa)) {
            src = b & 31;
            want[t] = xa;
          }
        }
        sp[t] = reinterpret_cast<const uint32_t*>(__shfl_sync(FULL, (unsigned long long)(uintptr_t)lp, src));
        sn[t] = __shfl_sync(FULL, ln, src);
        const uint32_t* sb =
            ORIENT ? nullptr
                   : reinterpret_cast<const uint32_t*>(__shfl_sync(FULL, (unsigned long long)(uintptr_t)bm, src));
        lo[t] = a;
        hi[t] = b;
        in[t] = false;
        if (f >= np) sn[t] = 0;
        if (sb && f < np) {  // a hub: its bitmap answers, nothing to search
          in[t] = BitTest(sb, want[t]);
          sn[t] = 0;
        }
      }
      uint32_t pos[2];
      LowerBound2(sp[0], sn[0], want[0], sp[1], sn[1], want[1], pos[0], pos[1]);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (pos[t] < sn[t] && __ldg(sp[t] + pos[t]) == want[t]) in[t] = true;
        if (in[t]) atomicOr(rows + lo[t], 1u << hi[t]);
      }
    }
    __syncwarp();
    if (lane < d) local += SmallCliques<K - 2>(rows, rows[lane]);
    __syncwarp();  // the rows are cleared for the next root
    if (lane == 0) bytes += 12ULL * d + 8ULL * np;
  }
  local = WarpSum(local);
  if (lane == 0 && local) atomicAdd(acc, local);
  if (lane == 0 && bytes) atomicAdd(acc + 1, bytes);
}

// ---- a CTA per root (part) ------------------------------------------------------
__device__ __forceinline__ uint32_t LowerBoundSmem(const uint32_t* a, uint32_t n, uint32_t x) {
  const uint32_t* base = a;
  while (n > 1) {
    const uint32_t half = n >> 1;
    base = base[half] < x ? base + half : base;
    n -= half;
  }
  return (uint32_t)(base - a) + (base[0] < x ? 1u : 0u);
}

// The candidates' positions by value: an open-addressed table of 2^lg slots,
// at most half full.  Most looked-up values are no candidate and stop at the
// first free slot, where a binary search takes log2(d) dependent steps.
__device__ __forceinline__ uint32_t TableSlot(uint32_t x, uint32_t lg) { return (x * 2654435761u) >> (32 - lg); }
__device__ __forceinline__ void TablePut(uint32_t* keys, uint16_t* at, uint32_t lg, uint32_t x, uint32_t i) {
  uint32_t h = TableSlot(x, lg);
  while (atomicCAS(keys + h, kNoKey, x) != kNoKey) h = (h + 1) & ((1u << lg) - 1);
  at[h] = (uint16_t)i;
}
// Position of x, or kNoKey.
__device__ __forceinline__ uint32_t TableGet(const uint32_t* keys, const uint16_t* at, uint32_t lg, uint32_t x) {
  uint32_t h = TableSlot(x, lg);
  while (true) {
    const uint32_t k = keys[h];
    if (k == x) return at[h];
    if (k == kNoKey) return kNoKey;
    h = (h + 1) & ((1u << lg) - 1);
  }
}
constexpr uint32_t TableLg(uint32_t dmax) { return dmax <= 256 ? 10 : 11; }

// The indexes of the bits of words [w0, W) of `row` into `list`; the number
// of them.
__device__ __forceinline__ uint32_t Expand(const uint32_t* row, uint32_t w0, uint32_t W, uint16_t* list) {
  const int lane = threadIdx.x & 31;
  uint32_t total = 0;
  for (uint32_t wb = w0 & ~31u; wb < W; wb += 32) {
    const uint32_t w = wb + lane;
    uint32_t s = w >= w0 && w < W ? row[w] : 0;
    const uint32_t c = __popc(s);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    uint32_t at = total + incl - c;
    for (; s; s &= s - 1) list[at++] = (uint16_t)(w * 32 + (__ffs(s) - 1));
    total += __shfl_sync(FULL, incl, 31);
  }
  return total;
}

// A row of the matrix is an odd number of units, so that rows spread over the
// banks.  The unit is a word, except in class M for k >= 5, whose inner loop
// is the pairs below: there it is a 16-byte quad, four words per load and loop
// step (5-cliques of the oriented R-MAT s17: class M 4.0-4.3 ms with quads and
// pairs, 6.0 without; 4-cliques and class L, whose rows are read from the
// middle on, are faster on words: 1.5 against 1.7 and 1.2 against 1.5 ms).
constexpr bool CliqueQuads(int k, int threads, bool global) {
  return k >= 5 && threads == kCliqueMThreads && !global;
}
// Classes whose roots several CTAs may take.
constexpr bool CliqueCut(int k, int threads, bool global) {
  return global || (k != 4 && threads != kCliqueMThreads);
}
template <bool QUADS>
struct RowUnit {
  typedef uint32_t T;
  static constexpr int kShift = 5;  // log2 of a unit's bits
  static __device__ __forceinline__ uint32_t And(uint32_t x, uint32_t y) { return x & y; }
  static __device__ __forceinline__ uint32_t Pop(uint32_t x) { return __popc(x); }
  static __device__ __forceinline__ uint32_t Zero() { return 0; }
};
template <>
struct RowUnit<true> {
  typedef uint4 T;
  static constexpr int kShift = 7;
  static __device__ __forceinline__ uint4 And(const uint4& x, const uint4& y) {
    return make_uint4(x.x & y.x, x.y & y.y, x.z & y.z, x.w & y.w);
  }
  static __device__ __forceinline__ uint32_t Pop(const uint4& x) {
    return __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
  }
  static __device__ __forceinline__ uint4 Zero() { return make_uint4(0, 0, 0, 0); }
};
constexpr uint32_t RowUnits(uint32_t d, bool quads) { return quads ? (d + 127) / 128 : (d + 31) / 32; }

// D-cliques inside the set S, whose nl members `list` holds, on the rows of
// `mat` (ws units apart, W units each); lane-local partial counts.
template <int D, bool QUADS, typename T = typename RowUnit<QUADS>::T>
__device__ __forceinline__ unsigned long long RowCliques(const T* S, const uint16_t* list, uint32_t nl,
                                                         const T* mat, uint32_t ws, uint32_t W, uint16_t* lists,
                                                         uint32_t lcap, T* sets, uint32_t wcap) {
  typedef RowUnit<QUADS> U;
  const int lane = threadIdx.x & 31;
  unsigned long long c = 0;
  if constexpr (D == 2) {
    for (uint32_t t = lane; t < nl; t += 32) {
      const uint32_t l = list[t];
      const T* row = mat + (size_t)l * ws;
      uint32_t s = 0;
#pragma unroll 4
      for (uint32_t w = l >> U::kShift; w < W; ++w) s += U::Pop(U::And(S[w], row[w]));
      c += s;
    }
  } else {
    if (QUADS && D == 3) {
      // short rows: the pairs of members over the lanes, each joined pair
      // counting the third members in S and both rows.  A warp per member
      // leaves most lanes idle here (a member is joined to a dozen others).
      const uint32_t pairs = nl * (nl - 1) / 2;
      uint32_t t = 0, o = lane;  // pair (t, t + 1 + o)
      for (uint32_t f = lane; f < pairs; f += 32, o += 32) {
        while (o >= nl - 1 - t) {  // f < pairs: a row with pairs is left
          o -= nl - 1 - t;
          ++t;
        }
        const uint32_t l = list[t], x = list[t + 1 + o];
        const T* row = mat + (size_t)l * ws;
        if ((reinterpret_cast<const uint32_t*>(row)[x >> 5] >> (x & 31)) & 1u) {
          const T* other = mat + (size_t)x * ws;
          uint32_t s = 0;
          for (uint32_t w = x >> U::kShift; w < W; ++w) s += U::Pop(U::And(U::And(S[w], row[w]), other[w]));
          c += s;
        }
      }
      return c;
    }
    for (uint32_t t = 0; t + D - 1 < nl; ++t) {
      const uint32_t l = list[t];
      const T* row = mat + (size_t)l * ws;
      __syncwarp();  // the previous round's set and list are read out
      for (uint32_t w = (l >> U::kShift) + lane; w < W; w += 32) sets[w] = U::And(S[w], row[w]);
      // the members after l that l is joined to
      uint32_t n2 = 0;
      for (uint32_t k0 = t + 1; k0 < nl; k0 += 32) {
        const uint32_t k = k0 + lane;
        const uint32_t x = k < nl ? list[k] : 0;
        const bool in = k < nl && ((reinterpret_cast<const uint32_t*>(row)[x >> 5] >> (x & 31)) & 1u);
        const unsigned mask = __ballot_sync(FULL, in);
        if (in) lists[n2 + __popc(mask & ((1u << lane) - 1))] = (uint16_t)x;
        n2 += __popc(mask);
      }
      __syncwarp();
      if (n2 >= D - 1)
        c += RowCliques<D - 1, QUADS>(sets, lists, n2, mat, ws, W, lists + lcap, lcap, sets + wcap, wcap);
    }
  }
  return c;
}

// Shared memory of a CTA: the matrix (unless it is in global scratch), per warp
// K - 4 sets, the candidates and their table (not with the matrix in scratch),
// and per warp K - 3 member lists.
constexpr size_t CliqueSmem(int k, uint32_t dmax, int threads, bool global) {
  const bool quads = CliqueQuads(k, threads, global);
  const size_t W = RowUnits(dmax, quads), unit = quads ? 16 : 4, warps = threads / 32;
  return (global || k == 3 ? 0 : (size_t)dmax * (W | 1) * unit) + warps * (k > 4 ? k - 4 : 0) * W * unit +
         (size_t)dmax * 4 +
         (global ? 0 : (size_t)6 << TableLg(dmax)) + warps * (k - 3) * (size_t)dmax * 2;
}
constexpr size_t CliqueScratchWords(uint32_t dmax) { return (size_t)dmax * (RowUnits(dmax, false) | 1); }

template <int K, bool ORIENT, int THREADS, bool GLOBAL>
__global__ void __launch_bounds__(THREADS) k_clique_cta(CView V, const uint32_t* __restrict__ roots,
                                                        const uint32_t* __restrict__ q,
                                                        const uint32_t* __restrict__ nq, uint32_t cap,
                                                        uint32_t* next, uint32_t* taken, uint32_t dmax,
                                                        uint32_t* scratch, unsigned long long* acc) {
  extern __shared__ uint4 cq_sh[];
  constexpr int WARPS = THREADS / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr bool QUADS = CliqueQuads(K, THREADS, GLOBAL);
  typedef typename RowUnit<QUADS>::T Unit;
  constexpr uint32_t kWords = sizeof(Unit) / 4;
  const uint32_t wcap = RowUnits(dmax, QUADS);
  Unit* sh = reinterpret_cast<Unit*>(cq_sh);
  Unit* mat = GLOBAL ? reinterpret_cast<Unit*>(scratch + (size_t)blockIdx.x * CliqueScratchWords(dmax)) : sh;
  constexpr int kSets = K > 4 ? K - 4 : 0;
  Unit* sets0 = GLOBAL || K == 3 ? sh : sh + (size_t)dmax * (wcap | 1);
  Unit* sets = sets0 + (size_t)wid * kSets * wcap;
  uint32_t* R = reinterpret_cast<uint32_t*>(sets0 + (size_t)WARPS * kSets * wcap);
  const uint32_t tlg = TableLg(dmax);
  uint32_t* keys = R + dmax;
  uint16_t* at = reinterpret_cast<uint16_t*>(keys + (1u << tlg));
  uint16_t* lists = (GLOBAL ? reinterpret_cast<uint16_t*>(keys) : at + (1u << tlg)) + (size_t)wid * (K - 3) * dmax;  // K = 3: none
  __shared__ uint32_t s_more, s_entry, s_part, s_taken, s_row;
  constexpr bool kParts = CliqueCut(K, THREADS, GLOBAL);
  const uint32_t count = min(*nq, cap);
  const uint32_t items = count * (kParts ? CliqueParts(K, dmax) : 1);
  unsigned long long local = 0, bytes = 0;
  while (true) {
    if (tid == 0) {
      const uint32_t it = atomicAdd(next, 1u);
      s_more = it < items;
      if (it < items) {
        s_entry = kParts ? it % count : it;
        s_part = kParts ? it / count : 0;
        s_taken = kParts && K > 3 && it >= count ? __ldcg(taken + it % count) : 0;
      }
      s_row = 0;
    }
    __syncthreads();
    if (!s_more) break;
    const uint32_t u0 = __ldg(roots + q[s_entry]);
    const uint32_t* L;
    uint32_t d;
    CList<ORIENT>(V, u0, L, d);
    if (!ORIENT) {
      const uint32_t r0 = WarpLowerBound(L, d, u0 + 1);
      L += r0;
      d -= r0;
    }
    if (kParts && (s_part >= CliqueParts(K, d) || s_taken >= d)) {
      __syncthreads();  // the item is rewritten
      continue;
    }
    const uint32_t W = RowUnits(d, QUADS), ws = W | 1;
    uint32_t* bits_of = reinterpret_cast<uint32_t*>(mat);  // row i's words start at i * ws * kWords
    for (uint32_t i = tid; i < d; i += THREADS) R[i] = __ldg(L + i);
    if (K > 3)
      for (uint32_t i = tid; i < d * ws; i += THREADS) mat[i] = RowUnit<QUADS>::Zero();
    if (!GLOBAL) {
      for (uint32_t i = tid; i < (1u << tlg); i += THREADS) keys[i] = kNoKey;
      __syncthreads();
      for (uint32_t i = tid; i < d; i += THREADS) TablePut(keys, at, tlg, R[i], i);
    }
    __syncthreads();
    // rows wid, wid + WARPS, ... (triangles: of the part's rows, every parts-th
    // one): the lanes fetch the lists of 32 rows at a time, then the warp
    // builds them one by one, four loads in flight per lane (the loads are
    // what a row waits for)
    const uint32_t row0 = K == 3 && kParts ? s_part : 0, rstep = K == 3 && kParts ? CliqueParts(K, d) : 1;
    const uint32_t nrows = d > row0 ? (d - row0 + rstep - 1) / rstep : 0;
    for (uint32_t i0 = wid; i0 < nrows; i0 += WARPS * 32) {
      const uint32_t mine = i0 + lane * WARPS;
      const uint32_t* ma = nullptr;
      const uint32_t* mb = nullptr;
      uint32_t mlen = 0;
      if (mine < nrows) {
        CList<ORIENT>(V, R[row0 + mine * rstep], ma, mlen);
        if (!ORIENT) mb = HubBitmap(V.G, R[row0 + mine * rstep]);
      }
      const uint32_t rows = min(32u, (nrows - i0 + WARPS - 1) / WARPS);
      for (uint32_t k = 0; k < rows; ++k) {
        const uint32_t i = row0 + (i0 + k * WARPS) * rstep;
        const uint32_t* a = reinterpret_cast<const uint32_t*>(__shfl_sync(FULL, (unsigned long long)(uintptr_t)ma, k));
        const uint32_t len = __shfl_sync(FULL, mlen, k);
        const uint32_t* bm =
            ORIENT ? nullptr
                   : reinterpret_cast<const uint32_t*>(__shfl_sync(FULL, (unsigned long long)(uintptr_t)mb, k));
        // index order: either test every later candidate in v's list (one
        // bitmap word each for a hub, a search else) or look every element of
        // the list up among the candidates, whichever takes fewer steps
        const uint32_t steps = (d - i + 30) / 32, lg = 32 - __clz(len | 1u);
        if (!ORIENT && bm) {
          for (uint32_t jb = (i + 1) & ~31u; jb < d; jb += 128) {
            uint32_t x[4], word[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const uint32_t j = jb + t * 32 + lane;
              x[t] = j < d ? R[j] : 0;
              word[t] = j > i && j < d ? __ldg(bm + (x[t] >> 5)) : 0;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const unsigned bits = __ballot_sync(FULL, (word[t] >> (x[t] & 31)) & 1u);
              if (K == 3) local += lane == 0 ? __popc(bits) : 0;
              else if (lane == 0 && bits) bits_of[(size_t)i * ws * kWords + (jb >> 5) + t] = bits;  // this warp's row
            }
          }
          if (lane == 0) bytes += 12ULL + 8ULL * (d - i);
        } else if (!ORIENT && steps * lg * 2 < (len + 31) / 32) {
          for (uint32_t jb = (i + 1) & ~31u; jb < d; jb += 32) {
            const uint32_t j = jb + lane;
            bool in = j > i && j < d;
            if (in) {
              const uint32_t x = R[j], pos = LowerBound(a, len, x);
              in = pos < len && __ldg(a + pos) == x;
            }
            const unsigned bits = __ballot_sync(FULL, in);
            if (K == 3) local += lane == 0 ? __popc(bits) : 0;
            else if (lane == 0 && bits) bits_of[(size_t)i * ws * kWords + (jb >> 5)] = bits;
          }
          if (lane == 0) bytes += 12ULL + 8ULL * (d - i);
        } else {
          for (uint32_t e0 = lane; e0 < len; e0 += 128) {
            uint32_t x[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) x[t] = e0 + t * 32 < len ? __ldg(a + e0 + t * 32) : 0xFFFFFFFFu;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              if (e0 + t * 32 >= len) break;
              uint32_t c;
              if (GLOBAL) {
                c = LowerBoundSmem(R, d, x[t]);
                if (c < d && R[c] != x[t]) c = d;
              } else {
                c = TableGet(keys, at, tlg, x[t]);
              }
              if (c < d && (ORIENT || c > i)) {
                const uint32_t lo = min(i, c), hi = max(i, c);
                if (K == 3) ++local;
                else atomicOr(bits_of + (size_t)lo * ws * kWords + (hi >> 5), 1u << (hi & 31));
              }
            }
          }
          if (lane == 0) bytes += 12ULL + 8ULL * len;
        }
      }
    }
    __syncthreads();
    while (K > 3) {
      uint32_t i = 0;
      if (lane == 0) i = atomicAdd(kParts ? taken + s_entry : &s_row, 1u);
      i = __shfl_sync(FULL, i, 0);
      if (i >= d) break;
      const Unit* row = mat + (size_t)i * ws;
      __syncwarp();
      const uint32_t nl = Expand(reinterpret_cast<const uint32_t*>(row), i >> 5, W * kWords, lists);
      __syncwarp();
      if constexpr (K > 3)
        if (nl >= K - 2)
          local += RowCliques<K - 2, QUADS>(row, lists, nl, mat, ws, W, lists + dmax,
                                              dmax, sets, wcap);
    }
    __syncthreads();  // the matrix is rebuilt for the next root
  }
  local = WarpSum(local);
  if (lane == 0 && local) atomicAdd(acc, local);
  if (lane == 0 && bytes) atomicAdd(acc + 1, bytes);
}

}  // namespace dev
}  // namespace sme

// Device engine: level-by-level extension of partial instances with
// memory-bounded batches, depth first over batches.
//
// Host control mirrors HybridGPUProcessor::ProcessLevel
// (src/gpu/impl/common/HybridGPUProcessor.cuh:14-50): per level, estimate each
// path's output (children estimate), split the frontier into batches that fit
// the level's memory budget (BatchManager::OrganizeBatch,
// src/gpu/utils/batch/BatchManager.cuh:42-110), execute the batch, recurse.
// Differences by design:
//   * one device allocation per context, used as a LIFO stack (no allocator
//     calls in the loop; the reference uses cnmem + per-op DeviceArray);
//   * intersections write in a single pass into a gapped buffer sized by the
//     children estimate, instead of count pass + scan + DToH + write pass
//     (GpsmBinSearch, src/gpu/utils/ops/intersect/GPSMBinSearch.cuh:144-197);
//   * candidate sets are (pointer, count) views: a set that is a sub-range of
//     an adjacency list or of an earlier set is not copied;
//   * counts accumulate on the device; the host reads one uint64 at the end.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>

#include "clique.cuh"
#include "cycle.cuh"
#include "engine.h"
#include "house.cuh"
#include "kernels.cuh"

namespace sme {

using namespace dev;

#define CK(x)                                                                            \
  do {                                                                                   \
    cudaError_t e_ = (x);                                                                \
    if (e_ != cudaSuccess) Fail(SME_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// sme_stats.phase_ms indices
constexpr int kPhaseCompute = 0, kPhaseMaterialize = 1, kPhaseFilter = 2, kPhaseComputeCount = 3,
              kPhasePathCount = 4, kPhaseCount = 5, kPhaseOrganize = 6, kPhaseExternal = 7;

// A timed region on the execution stream (two CUDA events) and its phase.
struct Timed {
  cudaEvent_t a, b;
  int phase;
};

// ---------------------------------------------------------------- kernels --
namespace {

__global__ void k_iota(uint32_t* out, uint32_t n, uint32_t start, uint32_t stride) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = start + i * stride;
}

// ---- inclusive scan of uint64 (tile 4096 = 512 threads x 8) -------------
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;
constexpr uint32_t SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ uint64_t BlockExclusiveScan(uint64_t v, uint64_t* total) {
  __shared__ uint64_t warp_tot[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    uint64_t t = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t y = __shfl_up_sync(FULL, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nw) warp_tot[lane] = t;
  }
  __syncthreads();
  uint64_t warp_prefix = wid > 0 ? warp_tot[wid - 1] : 0;
  uint64_t excl = warp_prefix + x - v;
  if (total) *total = warp_tot[(blockDim.x >> 5) - 1];
  __syncthreads();
  return excl;
}

// What a scan sums per path:
//   E_LIST  an intersection step's smallest list (the pivot size), an upper
//           bound of the candidate count (ThreadEstimatePathCount<MIN>,
//           CheckConstraintsCommon.cuh:161-189); with a second output, also
//           the elements of the adjacency lists the path reads (external mode:
//           what a batch must load, EXTEstimateIntersectCost,
//           src/gpu/impl/light/ext/EXTLIGHTOrganizeBatch.cuh:11-53)
//   E_SET   the size of u's candidate set
//   E_CHILD the children of the path when u is materialised: the set's range
//           clipped by < and >, minus the excluded values in it (`first`, when
//           given, receives where the range starts)
enum EstKind { E_LIST, E_SET, E_CHILD };

template <EstKind KIND>
__device__ __forceinline__ uint64_t EstOf(const DFront& F, const DStep& s, const DCond& c,
                                          const uintE* __restrict__ rp, uint32_t p, uint64_t* lists,
                                          uint32_t* first) {
  if (KIND == E_LIST) {
    uint64_t m = ~0ULL, sd = 0;
    for (int i = 0; i < s.nconn; ++i) {
      const uint32_t v = F.inst[s.conn[i]][p];
      const uint64_t d = __ldg(rp + v + 1) - __ldg(rp + v);
      m = min(m, d);
      sd += d;
    }
    *lists = sd;
    if (s.reuse >= 0) {
      const uint32_t* ptr;
      uint32_t len;
      GetSet(F, s.reuse, p, ptr, len);
      m = min(m, (uint64_t)len);
    }
    return m == ~0ULL ? 0 : m;
  }
  const uint32_t* a;
  uint32_t n;
  GetSet(F, s.u, p, a, n);
  if (KIND == E_SET) return n;
  Bounds bd = MakeBounds(c, F, p);
  uint32_t r0, r1, ex[MAXV];
  Range(a, n, bd, r0, r1);
  if (first) first[p] = r0;
  return (uint64_t)(r1 - r0 - Exclusions(a, r0, r1, bd, ex));
}

// Inclusive sums of the tile's estimates into `out` (and `out2`), the tile
// sums into bs (bs2 = bs + nb + 1); the last block to finish turns the tile
// sums into exclusive ones with the total after them.  One tile needs nothing
// more; k_scan_add adds the tile sums otherwise.  The estimate, its scan and
// the total were four launches and the host's split query before.  ITEMS 1
// for frontiers of up to kScanSmall paths an SM (an estimate is a chain of loads:
// one per thread, over as many SMs as there are tiles), else SCAN_ITEMS.
constexpr uint32_t kScanSmall = 4 * SCAN_THREADS;
template <EstKind KIND, bool TWO, int ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_est_scan(DFront F, DStep s, DCond c,
                                                           const uintE* __restrict__ rp, uint64_t* out,
                                                           uint64_t* out2, uint32_t* first, uint64_t* bs,
                                                           uint32_t* ticket) {
  const uint64_t base = (uint64_t)blockIdx.x * (SCAN_THREADS * ITEMS);
  const uint32_t nb = gridDim.x;
  uint64_t v[ITEMS], v2[TWO ? ITEMS : 1];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint64_t i = base + (uint64_t)k * SCAN_THREADS + threadIdx.x;
    uint64_t lists = 0;
    v[k] = i < F.P ? EstOf<KIND>(F, s, c, rp, (uint32_t)i, &lists, first) : 0;
    if (TWO) v2[k] = lists;
  }
  uint64_t run = 0, run2 = 0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint64_t i0 = base + (uint64_t)k * SCAN_THREADS;
    if (i0 >= F.P) break;  // uniform in the block
    const uint64_t i = i0 + threadIdx.x;
    uint64_t total;
    const uint64_t e = BlockExclusiveScan(v[k], &total);
    if (i < F.P) out[i] = run + e + v[k];
    run += total;
    if (TWO) {
      const uint64_t e2 = BlockExclusiveScan(v2[k], &total);
      if (i < F.P) out2[i] = run2 + e2 + v2[k];
      run2 += total;
    }
  }
  uint64_t* bs2 = bs + nb + 1;
  __shared__ uint32_t s_last;
  if (threadIdx.x == 0) {
    bs[blockIdx.x] = run;
    if (TWO) bs2[blockIdx.x] = run2;
    __threadfence();
    s_last = atomicAdd(ticket, 1u) == nb - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();  // the other blocks' sums, read past L1
  const uint32_t per = (nb + SCAN_THREADS - 1) / SCAN_THREADS;
  for (int w = 0; w < (TWO ? 2 : 1); ++w) {
    uint64_t* t = w ? bs2 : bs;
    const uint32_t b = min(nb, threadIdx.x * per), e = min(nb, b + per);
    uint64_t sum = 0, total;
    for (uint32_t i = b; i < e; ++i) sum += __ldcg(t + i);
    uint64_t at = BlockExclusiveScan(sum, &total);
    for (uint32_t i = b; i < e; ++i) {
      const uint64_t x = __ldcg(t + i);
      t[i] = at;
      at += x;
    }
    if (threadIdx.x == 0) t[nb] = total;
  }
  if (threadIdx.x == 0) *ticket = 0;  // for the next launch on the stream
}

template <bool TWO, int ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_add(uint64_t* out, uint64_t* out2, uint32_t n,
                                                           const uint64_t* __restrict__ bs) {
  const uint64_t base = (uint64_t)(blockIdx.x + 1) * (SCAN_THREADS * ITEMS);  // tile 0 stays as it is
  const uint32_t nb = gridDim.x + 1;
  const uint64_t add = bs[blockIdx.x + 1], add2 = TWO ? bs[nb + 1 + blockIdx.x + 1] : 0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const uint64_t i = base + (uint64_t)k * SCAN_THREADS + threadIdx.x;
    if (i < n) {
      out[i] += add;
      if (TWO) out2[i] += add2;
    }
  }
}

// ---- COMPUTE over one list: a view per path --------------------------------
// The candidate set of a step that reads one list (or one earlier set) and has
// no `!=` condition is a sub-range of it: one thread per path clips it; no
// estimate, no scan and no data buffer.
__global__ void __launch_bounds__(WARP_BLOCK) k_view(DFront F, DStep s, DGraph G, uint64_t* out_ptr,
                                                     uint32_t* out_cnt, unsigned long long* acc) {
  unsigned long long bytes = 0;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < F.P; p += gridDim.x * blockDim.x) {
    const uint32_t* a;
    uint32_t n;
    if (s.nconn) AdjList(G, F.inst[s.conn[0]][p], a, n);
    else GetSet(F, s.reuse, p, a, n);
    const BoundsT<0> bd = MakeBounds<0>(s.cond, F, p);
    uint32_t r0, r1;
    Range(a, n, bd, r0, r1);
    out_ptr[p] = (uint64_t)(a + r0);
    out_cnt[p] = r1 - r0;
    bytes += 12ULL * s.nconn;
  }
  bytes = WarpSum(bytes);
  if ((threadIdx.x & 31) == 0 && bytes) atomicAdd(acc + 1, bytes);
}

__global__ void k_scan_reduce(const uint64_t* __restrict__ in, uint32_t n, uint64_t* bs) {
  uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
  uint64_t s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    uint64_t i = base + (uint64_t)k * SCAN_THREADS + threadIdx.x;
    if (i < n) s += in[i];
  }
  __shared__ uint64_t red[SCAN_THREADS / 32];
  s = WarpSum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    uint64_t t = threadIdx.x < SCAN_THREADS / 32 ? red[threadIdx.x] : 0;
    t = WarpSum(t);
    if (threadIdx.x == 0) bs[blockIdx.x] = t;
  }
}

// Exclusive scan of the block sums in place (one block).
__global__ void k_scan_partials(uint64_t* bs, uint32_t nb) {
  uint32_t per = (nb + blockDim.x - 1) / blockDim.x;
  uint32_t b = threadIdx.x * per, e = min(nb, b + per);
  uint64_t s = 0;
  for (uint32_t i = b; i < e; ++i) s += bs[i];
  uint64_t run = BlockExclusiveScan(s, nullptr);
  for (uint32_t i = b; i < e; ++i) {
    uint64_t v = bs[i];
    bs[i] = run;
    run += v;
  }
}

__global__ void k_scan_apply(uint64_t* data, uint32_t n, const uint64_t* __restrict__ bs) {
  uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
  uint64_t v[SCAN_ITEMS];
  uint64_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    uint64_t i = base + k;
    v[k] = i < n ? data[i] : 0;
    s += v[k];
  }
  uint64_t run = BlockExclusiveScan(s, nullptr) + bs[blockIdx.x];
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    uint64_t i = base + k;
    run += v[k];
    if (i < n) data[i] = run;
  }
}

// Batch boundaries: for threshold k, the first path whose inclusive cost
// exceeds cost(start-1) + (k+1)*budget (SplitBatchKernel,
// src/gpu/utils/batch/SplitBatch.cuh:38-87).  cost(p) = pf*(p+1) + cf*est_incl[p].
__global__ void k_split(const uint64_t* __restrict__ incl, const uint64_t* __restrict__ incl2, uint32_t P,
                        uint32_t start, double pf, double cf, double cg, double budget, uint32_t K,
                        uint64_t* out) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  auto cost = [&](uint32_t p) {  // inclusive cost of paths [0, p]
    double c = pf * (double)(p + 1) + cf * (double)incl[p];
    if (incl2) c += cg * (double)incl2[p];
    return c;
  };
  double c0 = start == 0 ? 0.0 : cost(start - 1);
  double t = c0 + (double)(k + 1) * budget;
  uint32_t lo = start, hi = P;  // first p in [start,P) with cost(p) > t
  while (lo < hi) {
    uint32_t mid = lo + (hi - lo) / 2;
    double c = cost(mid);
    if (c > t) hi = mid;
    else lo = mid + 1;
  }
  if (lo == start) ++lo;  // a single path above the budget: its own batch
  out[3 * k] = lo;
  out[3 * k + 1] = incl[lo - 1];  // lo > start >= 0
  out[3 * k + 2] = incl2 ? incl2[lo - 1] : 0;
}

// ---- paths grouped by the hub they probe ------------------------------------
// A count step's membership tests land on the dense bitmap of the hub whose
// list is searched.  Taken in frontier order, consecutive paths probe
// different hubs and every 4-byte test pulls a 32-byte sector from DRAM (the
// bitmaps do not fit L2); taken hub by hub, a hub's bitmap stays in L2 while
// its paths run.  A counting sort by hub slot (non-hubs in one last bucket)
// gives the order: warp-aggregated counts, a scan, a warp-aggregated scatter.
__global__ void k_hub_hist(DFront F, uint8_t kv, const int32_t* __restrict__ hub, uint32_t nb,
                           unsigned long long* cnt) {
  const int lane = threadIdx.x & 31;
  const uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = w0; base < F.P; base += stride) {
    const uint32_t p = base + lane;
    uint32_t key = 0xffffffffu;
    if (p < F.P) {
      const int32_t h = __ldg(hub + F.inst[kv][p]);
      key = h < 0 ? nb - 1 : (uint32_t)h;
    }
    const unsigned same = __match_any_sync(FULL, key);
    if (key != 0xffffffffu && lane == __ffs(same) - 1) atomicAdd(cnt + key, (unsigned long long)__popc(same));
  }
}

__global__ void k_hub_cursor(const unsigned long long* __restrict__ incl, const unsigned long long* cnt,
                             uint32_t nb, unsigned long long* cur) {
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x)
    cur[b] = incl[b] - cnt[b];
}

__global__ void k_hub_scatter(DFront F, uint8_t kv, const int32_t* __restrict__ hub, uint32_t nb,
                              unsigned long long* cur, uint32_t* perm) {
  const int lane = threadIdx.x & 31;
  const uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = w0; base < F.P; base += stride) {
    const uint32_t p = base + lane;
    uint32_t key = 0xffffffffu;
    if (p < F.P) {
      const int32_t h = __ldg(hub + F.inst[kv][p]);
      key = h < 0 ? nb - 1 : (uint32_t)h;
    }
    const unsigned same = __match_any_sync(FULL, key);
    const int leader = __ffs(same) - 1;
    unsigned long long at = 0;
    if (key != 0xffffffffu && lane == leader) at = atomicAdd(cur + key, (unsigned long long)__popc(same));
    at = __shfl_sync(FULL, at, leader);
    if (key != 0xffffffffu) perm[at + __popc(same & ((1u << lane) - 1))] = p;
  }
}

// ---- mapped reuse: the sibling path's cached intersection ----------------
// In the reuse plan the level-1 paths of a root M[0] are its neighbours N(M[0])
// in order (one contiguous run per root; the compiler checks level 1 has no
// condition), and the level-2 store holds, per level-1 path (M[0], y) of the
// current batch, the intersection N(M[0]) ∩ N(y).  A path whose ancestor is
// (M[0], M[1]) at store index s finds the sibling (M[0], M[x]) at index
// s + rank(M[x]) - rank(M[1]), ranks taken in N(M[0]) (FastLocateCache over
// the prefix tree, src/gpu/impl/common/CheckConstraintsReuseCommon.cuh:114-289,
// reduced to two binary searches by that layout).  `sib` stays null when the
// sibling is not in the store (another batch), and the step intersects the
// lists instead.
__device__ __forceinline__ void SiblingSet(const DFront& F, const DStep& s, const DGraph& G, uint32_t p,
                                           const uint32_t*& sib, uint32_t& sibn) {
  sib = nullptr;
  sibn = 0;
  if (s.msrc < 0) return;
  const uint32_t m0 = F.inst[0][p], m1 = F.inst[1][p], mx = F.inst[s.mx][p];
  if ((s.mop == 0 && !(mx < m0)) || (s.mop == 1 && !(mx > m0))) return;  // not a level-1 candidate
  const uint32_t* n0;
  uint32_t d0;
  AdjList(G, m0, n0, d0);
  const uint32_t ia = LowerBound(n0, d0, m1), ib = LowerBound(n0, d0, mx);
  if (ib >= d0 || __ldg(n0 + ib) != mx) return;
  const int64_t s2 = (int64_t)SetIndex(F, s.msrc, p) + (int64_t)ib - (int64_t)ia;
  if (s2 < 0 || s2 >= (int64_t)F.nset[s.msrc]) return;
  sib = reinterpret_cast<const uint32_t*>(F.set[s.msrc].ptr[s2]);
  sibn = F.set[s.msrc].cnt[s2];
}

// ---- intersection (COMPUTE / COMPUTE_COUNT / COMPUTE_PATH_COUNT) ---------
// One warp per path.  The pivot is the smallest list (ThreadChoosePivotLevel,
// CheckConstraintsCommon.cuh:10-29); < and > conditions clip the pivot to a
// sub-range by binary search before the scan; every pivot element is checked
// in the other lists by a per-lane binary search whose lower end advances with
// the lane's previous hit (each lane sees increasing candidates).
// MODE 0 writes the sorted candidate set, MODE 1 counts (optionally ranked
// into a partner set), MODE 2 stores only the per-path count.  MINB is the
// minimum resident blocks per SM asked of the register allocator (the
// kernels are latency bound: more resident warps, more searches in flight).
// NLM bounds the lists a step intersects (backward lists + cached set), so a
// step with two or three lists keeps fewer values live; NEX = 0 is for steps
// without `!=` conditions (no exclusion array).  The launcher guarantees
// both bounds.
// DEFER (two lists, no `!=`): a path whose clipped pivot holds at least
// hv.min_len elements is queued for k_compute_cta instead.  MAPPED (reuse
// plan, s.msrc >= 0): the set cached by the sibling path replaces the lists
// of s.mmask when the sibling is in the current batch (see SiblingSet).
template <int MODE, int MINB = 1, int NLM = MAXV, int NEX = MAXV, bool DEFER = false, bool MAPPED = false,
          bool PERM = false>
__global__ void __launch_bounds__(WARP_BLOCK, MINB) k_compute(
    DFront F, DStep s, DGraph G, const uint64_t* __restrict__ est_incl, uint32_t b0, uint64_t* out_ptr,
    uint32_t* out_cnt, uint32_t* out_data, uint64_t out_cap, unsigned long long* acc, uint32_t* err,
    DHeavy hv) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const unsigned lt = (1u << lane) - 1;
  unsigned long long local = 0, bytes = 0, hits = 0;
  const uint64_t base = b0 == 0 ? 0 : est_incl[b0 - 1];

  for (uint32_t pi = gw; pi < F.P; pi += nw) {
    const uint32_t p = PERM ? __ldg(hv.perm + pi) : pi;
    const uint32_t* L[NLM];
    const uint32_t* B[NLM];  // hub bitmap of the list (null: binary search)
    uint32_t N[NLM];
    int nl = 0;
    const uint32_t* sib = nullptr;
    uint32_t sibn = 0;
    if constexpr (MAPPED) SiblingSet(F, s, G, p, sib, sibn);
    if (MAPPED && sib) {
      // the lists outside the mask, then the sibling's cached set
#pragma unroll
      for (int i = 0; i < NLM; ++i) {
        if (i < s.nconn && !((s.mmask >> i) & 1)) {
          const uint32_t v = F.inst[s.conn[i]][p];
          const uint32_t* lp;
          uint32_t ln;
          AdjList(G, v, lp, ln);
#pragma unroll
          for (int t = 0; t < NLM; ++t)
            if (t == nl) {
              L[t] = lp;
              N[t] = ln;
              B[t] = HubBitmap(G, v);
            }
          ++nl;
        }
      }
#pragma unroll
      for (int t = 0; t < NLM; ++t)
        if (t == nl) {
          L[t] = sib;
          N[t] = sibn;
          B[t] = nullptr;
        }
      ++nl;
      if (lane == 0) ++hits;
    } else {
#pragma unroll
      for (int i = 0; i < NLM; ++i) {
        B[i] = nullptr;
        if (i < s.nconn) {
          uint32_t v = F.inst[s.conn[i]][p];
          AdjList(G, v, L[i], N[i]);
          B[i] = HubBitmap(G, v);
          nl = i + 1;
        }
      }
    }
    if (s.reuse >= 0) {
#pragma unroll
      for (int i = 0; i < NLM; ++i)
        if (i == nl) GetSet(F, s.reuse, p, L[i], N[i]);
      ++nl;
    }
    if (lane == 0) bytes += 12ULL * s.nconn;  // row pointers + gathered instance vertices
    // pivot to slot 0
#pragma unroll
    for (int i = 1; i < NLM; ++i) {
      if (i < nl && N[i] < N[0]) {
        const uint32_t* tp = L[0];
        L[0] = L[i];
        L[i] = tp;
        tp = B[0];
        B[0] = B[i];
        B[i] = tp;
        uint32_t tn = N[0];
        N[0] = N[i];
        N[i] = tn;
      }
    }
    BoundsT<NEX> bd = MakeBounds<NEX>(s.cond, F, p);
    uint32_t r0 = 0, r1 = 0;
    if (nl > 0) WarpRange(L[0], N[0], bd, r0, r1);
    if (DEFER && nl == 2 && r1 - r0 >= hv.min_len) {
      uint32_t slot = 0;
      if (lane == 0) slot = atomicAdd(hv.q, 1u);
      slot = __shfl_sync(FULL, slot, 0);
      if (slot < hv.cap) {
        if (lane == 0) hv.q[1 + slot] = p;
        continue;
      }
    }

    uint64_t out_off = 0;
    if (MODE == 0) {
      out_off = (p + b0 == 0 ? 0 : est_incl[p + b0 - 1]) - base;
      if (nl == 1 && !s.noview) {
        // single list: the candidate set is a sub-range unless an excluded
        // value falls inside it
        uint32_t ex[MAXV];
        int ne = Exclusions(L[0], r0, r1, bd, ex);
        if (ne == 0) {
          if (lane == 0) {
            out_ptr[p] = (uint64_t)(L[0] + r0);
            out_cnt[p] = r1 - r0;
          }
          continue;
        }
      }
    }
    // partner set for ranked counting
    const uint32_t* W = nullptr;
    uint32_t WN = 0;
    if (MODE == 1 && s.with_u >= 0) GetSet(F, s.with_u, p, W, WN);

    // every element of the clipped pivot is read once and tested against
    // each other list (one bitmap word or one list element answers a test)
    if (lane == 0) bytes += 4ULL * (r1 - r0) * (uint64_t)nl;
    uint32_t cur[NLM];
#pragma unroll
    for (int i = 0; i < NLM; ++i) cur[i] = 0;
    uint32_t written = 0;
    for (uint32_t bi = r0; bi < r1; bi += 32) {
      uint32_t i = bi + lane;
      bool ok = i < r1;
      uint32_t x = ok ? __ldg(L[0] + i) : 0;
#pragma unroll
      for (int k = 0; k < NEX; ++k)
        if (k < bd.nne && x == bd.ne[k]) ok = false;
#pragma unroll
      for (int j = 1; j < NLM; ++j) {
        if (j < nl && ok) {
          if (B[j]) {
            ok = BitTest(B[j], x);
          } else {
            uint32_t pos = cur[j] + LowerBound(L[j] + cur[j], N[j] - cur[j], x);
            cur[j] = pos;
            ok = pos < N[j] && __ldg(L[j] + pos) == x;
          }
        }
      }
      unsigned mask = __ballot_sync(FULL, ok);
      if (MODE == 0) {
        uint64_t o = out_off + written + __popc(mask & lt);
        if (ok) {
          if (o < out_cap) out_data[o] = x;
          else atomicOr(err, ENGINE_ERR_BOUNDS);
        }
      } else if (MODE == 1) {
        if (W != nullptr) {
          if (ok) local += RankCount(W, WN, x, s.with_op);
        } else if (lane == 0) {
          local += __popc(mask);
        }
      }
      written += __popc(mask);
    }
    if (lane == 0) {
      if (MODE == 0) {
        out_ptr[p] = (uint64_t)(out_data + out_off);
        out_cnt[p] = written;
        bytes += 4ULL * written;
      } else if (MODE == 2) {
        out_ptr[p] = 0;
        out_cnt[p] = written;
      }
    }
  }
  if (MODE == 1) {
    local = WarpSum(local);
    if (lane == 0 && local) atomicAdd(acc, local);
  }
  if (lane == 0 && bytes) atomicAdd(acc + 1, bytes);
  if (MAPPED && lane == 0 && hits) atomicAdd(acc + 5, hits);
}

// ---- common neighbours of two vertices ----------------------------------------
// Counting steps over two adjacency lists without any condition (the diamond's
// path count, the house's triangles).  One warp per path: two hubs whose
// shorter list is long are counted on their bitmaps, AND and popcount in
// 16-byte loads; else the shorter list is walked, 128 elements at a time so
// that four loads and then four tests per lane are in flight (a walk 32 at a
// time waits for two dependent loads per step).  The bitmaps win from about a
// list element per kAndWords words: a walked element costs a 32-byte sector of
// the bitmap it hits, a word of both bitmaps 8 bytes.  `simple`: no list holds
// an element twice (a bitmap would count it once).  House on 1024 roots of
// R-MAT s18 (270 000 triangles): 969 us by k_compute, 315 us here.
constexpr uint32_t kAndWords = 6;

template <int MODE>
__global__ void __launch_bounds__(WARP_BLOCK, 5) k_pair_count(DFront F, int c0, int c1, DGraph G, bool simple,
                                                              uint64_t* out_ptr, uint32_t* out_cnt,
                                                              unsigned long long* acc) {
  static_assert(MODE == 1 || MODE == 2, "counts only");
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  unsigned long long local = 0, bytes = 0;
  for (uint32_t p = gw; p < F.P; p += nw) {
    uint32_t v = F.inst[c0][p], w = F.inst[c1][p];
    const uint32_t *a, *b;
    uint32_t na, nb;
    AdjList(G, v, a, na);
    AdjList(G, w, b, nb);
    const uint32_t* ma = HubBitmap(G, v);
    const uint32_t* mb = HubBitmap(G, w);
    if (nb < na) {  // walk the shorter list, test in the longer one
      const uint32_t* t = a;
      a = b;
      b = t;
      t = ma;
      ma = mb;
      mb = t;
      const uint32_t tn = na;
      na = nb;
      nb = tn;
    }
    uint32_t c = 0;
    if (simple && ma && mb && na > G.words / kAndWords) {
      const uint4* qa = reinterpret_cast<const uint4*>(ma);
      const uint4* qb = reinterpret_cast<const uint4*>(mb);
#pragma unroll 4
      for (uint32_t i = lane; i < G.words / 4; i += 32) {
        const uint4 x = __ldg(qa + i), y = __ldg(qb + i);
        c += __popc(x.x & y.x) + __popc(x.y & y.y) + __popc(x.z & y.z) + __popc(x.w & y.w);
      }
    } else if (mb) {
      for (uint32_t i = lane; i < na; i += 128) {
        uint32_t x[4], t[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = i + 32 * k < na ? __ldg(a + i + 32 * k) : 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) t[k] = i + 32 * k < na ? __ldg(mb + (x[k] >> 5)) : 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) c += (t[k] >> (x[k] & 31)) & 1u;
      }
    } else {
      uint32_t cur = 0;
      for (uint32_t i = lane; i < na; i += 32) {
        const uint32_t x = __ldg(a + i);
        cur += LowerBound(b + cur, nb - cur, x);
        c += cur < nb && __ldg(b + cur) == x;
      }
    }
    if (MODE == 1) {
      local += c;
    } else {
      c = __reduce_add_sync(FULL, c);
      if (lane == 0) {
        out_ptr[p] = 0;
        out_cnt[p] = c;
      }
    }
    if (lane == 0) bytes += 24ULL + 8ULL * na;  // as the warp kernel counts them
  }
  if (MODE == 1) {
    local = WarpSum(local);
    if (lane == 0 && local) atomicAdd(acc, local);
  }
  if (lane == 0 && bytes) atomicAdd(acc + 1, bytes);
}

// ---- intersection of the root's list with one other list -------------------
// Steps that intersect exactly two adjacency lists, one of them the list of
// the plan's first vertex (the root of the task: the 4-cycle's and the
// triangle's count steps, the diamond's path count, the 4-clique's second
// level).  The frontier keeps the paths of a root together (materialisation
// preserves the parents' order), so a CTA holds the root's list as an n-bit
// bitmap in shared memory and rebuilds it only when the root changes between
// runs of paths.  Per path a warp then takes the cheapest of: walking the
// other list's clipped range and testing each element in the shared bitmap
// (no search at all), walking the root's clipped range and testing the other
// vertex's hub bitmap (one load each), or walking the root's clipped range
// with a binary search in the other list (the warp kernel's way).  Costs are
// compared in warp iterations, a binary search counting log2 of the list.
// Results equal k_compute's: MODE 0 writes the sorted set (both walks visit
// ascending values), MODE 1 counts, MODE 2 stores the count.  CTAs take
// chunks of RM_CHUNK paths from a counter.
constexpr int RM_THREADS = 1024;
constexpr int RM_WARPS = RM_THREADS / 32;
constexpr uint32_t RM_CHUNK = 2048;
constexpr uint32_t kRootMapMaxBytes = 200u << 10;  // bitmaps up to n = 1 638 400
constexpr uint32_t kNoRoot = 0xFFFFFFFFu;

template <int MODE, int NEX>
__global__ void __launch_bounds__(RM_THREADS, 2) k_compute_rootmap(
    DFront F, DStep s, DGraph G, int ru, int other, const uint64_t* __restrict__ est_incl, uint32_t b0,
    uint64_t* out_ptr, uint32_t* out_cnt, uint32_t* out_data, uint64_t out_cap, unsigned long long* acc,
    uint32_t* err, uint32_t* next_chunk, uint32_t words) {
  extern __shared__ uint32_t rmap[];
  __shared__ uint32_t s_chunk, s_end;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1;
  for (uint32_t i = threadIdx.x; i < words; i += RM_THREADS) rmap[i] = 0;
  unsigned long long local = 0, bytes = 0;
  const uint64_t base = (MODE == 0 && b0 > 0) ? est_incl[b0 - 1] : 0;
  const uint32_t* rootcol = F.inst[ru];
  const uint32_t* othercol = F.inst[other];
  uint32_t cur_root = kNoRoot;
  __syncthreads();
  while (true) {
    if (threadIdx.x == 0) s_chunk = atomicAdd(next_chunk, 1u);
    __syncthreads();
    const uint64_t c0 = (uint64_t)s_chunk * RM_CHUNK;
    __syncthreads();  // s_chunk is rewritten only after the next barrier pair
    if (c0 >= F.P) break;
    const uint32_t c1 = (uint32_t)(c0 + RM_CHUNK < F.P ? c0 + RM_CHUNK : F.P);
    uint32_t p = (uint32_t)c0;
    while (p < c1) {
      const uint32_t r = __ldg(rootcol + p);
      if (threadIdx.x == 0) s_end = c1;
      __syncthreads();
      for (uint32_t q = p + threadIdx.x; q < c1; q += RM_THREADS)
        if (__ldg(rootcol + q) != r) {
          atomicMin(&s_end, q);
          break;
        }
      __syncthreads();
      const uint32_t e = s_end;
      if (r != cur_root) {
        const uint32_t* L;
        uint32_t N;
        if (cur_root != kNoRoot) {
          AdjList(G, cur_root, L, N);
          for (uint32_t i = threadIdx.x; i < N; i += RM_THREADS) rmap[__ldg(L + i) >> 5] = 0;
          __syncthreads();
        }
        AdjList(G, r, L, N);
        for (uint32_t i = threadIdx.x; i < N; i += RM_THREADS) {
          const uint32_t x = __ldg(L + i);
          atomicOr(rmap + (x >> 5), 1u << (x & 31));
        }
        __syncthreads();
        cur_root = r;
      }
      const uint32_t* Lr;
      uint32_t Nr;
      AdjList(G, r, Lr, Nr);
      for (uint32_t pp = p + wid; pp < e; pp += RM_WARPS) {
        const uint32_t v = __ldg(othercol + pp);
        const uint32_t* Lv;
        uint32_t Nv;
        AdjList(G, v, Lv, Nv);
        const uint32_t* Bv = HubBitmap(G, v);
        const uint32_t* Cv = HubCoarse(G, v);
        BoundsT<NEX> bd = MakeBounds<NEX>(s.cond, F, pp);
        uint32_t a0, a1, v0, v1;
        WarpRange(Lr, Nr, bd, a0, a1);
        WarpRange(Lv, Nv, bd, v0, v1);
        // algorithmic bytes as the warp kernel counts them: the smaller
        // list is the pivot, its clipped range read and tested once
        if (lane == 0) bytes += 24ULL + 8ULL * (Nv < Nr ? v1 - v0 : a1 - a0);
        const uint32_t wv = (v1 - v0 + 31) >> 5, wr = (a1 - a0 + 31) >> 5;
        int how = 0;  // 0: walk v's range, test the shared bitmap
        if (Bv) {
          if (wr < wv) how = 1;  // walk the root's range, test v's hub bitmap
        } else {
          const uint32_t lg = 32 - __clz(Nv | 1u);
          if (wr * lg < wv) how = 2;  // walk the root's range, search v's list
        }
        const uint32_t* W = how == 0 ? Lv : Lr;
        const uint32_t w0 = how == 0 ? v0 : a0, w1 = how == 0 ? v1 : a1;
        uint64_t out_off = 0;
        if (MODE == 0) out_off = (pp + b0 == 0 ? 0 : est_incl[pp + b0 - 1]) - base;
        uint32_t cur = 0, written = 0;
        for (uint32_t bi = w0; bi < w1; bi += 32) {
          const uint32_t i = bi + lane;
          bool ok = i < w1;
          const uint32_t x = ok ? __ldg(W + i) : 0;
#pragma unroll
          for (int k = 0; k < NEX; ++k)
            if (k < bd.nne && x == bd.ne[k]) ok = false;
          if (ok) {
            if (how == 0) {
              ok = (rmap[x >> 5] >> (x & 31)) & 1u;
            } else if (how == 1) {
              ok = BitTest2(Bv, Cv, x);
            } else {
              const uint32_t pos = cur + LowerBound(Lv + cur, Nv - cur, x);
              cur = pos;
              ok = pos < Nv && __ldg(Lv + pos) == x;
            }
          }
          const unsigned mask = __ballot_sync(FULL, ok);
          if (MODE == 0) {
            const uint64_t o = out_off + written + __popc(mask & lt);
            if (ok) {
              if (o < out_cap) out_data[o] = x;
              else atomicOr(err, ENGINE_ERR_BOUNDS);
            }
          } else if (MODE == 1 && lane == 0) {
            local += __popc(mask);
          }
          written += __popc(mask);
        }
        if (lane == 0) {
          if (MODE == 0) {
            out_ptr[pp] = (uint64_t)(out_data + out_off);
            out_cnt[pp] = written;
            bytes += 4ULL * written;
          } else if (MODE == 2) {
            out_ptr[pp] = 0;
            out_cnt[pp] = written;
          }
        }
      }
      __syncthreads();  // the bitmap may change for the next run
      p = e;
    }
  }
  if (MODE == 1) {
    local = WarpSum(local);
    if (lane == 0 && local) atomicAdd(acc, local);
  }
  if (lane == 0 && bytes) atomicAdd(acc + 1, bytes);
}

// ---- intersection, one CTA per long-pivot path ----------------------------
// The paths k_compute<..., DEFER> queued: two lists, no `!=` conditions, a
// clipped pivot of at least DHeavy::min_len elements.  All CTA_THREADS
// threads walk one path's pivot.  When the other list is not a hub (no
// bitmap), its window between the pivot's first and last value is staged in
// shared memory first: the 16-byte-aligned interior by one bulk copy
// (cp.async.bulk global -> shared, completion on an mbarrier, the source this
// GPU's own memory), the at most three elements on either ragged end by plain
// loads; every binary search then probes shared memory instead of L2.  The
// window is staged only when it fits `win_cap` elements and holds at most
// kStageRatio elements per pivot element (else the copy would read more than
// the searches).  Results equal k_compute's: MODE 0 writes the sorted set at
// the path's offset (block-ordered compaction), MODE 1 counts (ranked into a
// partner set when the step has one), MODE 2 stores the count.
constexpr int CTA_THREADS = 512;
constexpr int CTA_WARPS = CTA_THREADS / 32;
constexpr uint32_t kStageRatio = 16;
constexpr uint32_t kMbarSpins = 1u << 22;

__device__ __forceinline__ uint32_t LowerBoundShared(const uint32_t* a, uint32_t n, uint32_t x) {
  if (n == 0) return 0;
  const uint32_t* base = a;
  while (n > 1) {
    const uint32_t half = n >> 1;
    base = base[half] < x ? base + half : base;
    n -= half;
  }
  return (uint32_t)(base - a) + (base[0] < x ? 1u : 0u);
}

__device__ __forceinline__ bool MbarTryWait(uint32_t bar, uint32_t phase) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(phase)
      : "memory");
  return done != 0;
}

// Waits (bounded) for the phase of `bar` to complete; false if it gave up.
__device__ __forceinline__ bool MbarWait(uint32_t bar, uint32_t phase) {
  for (uint32_t i = 0; i < kMbarSpins; ++i)
    if (MbarTryWait(bar, phase)) return true;
  return false;
}

template <int MODE>
__global__ void __launch_bounds__(CTA_THREADS, 2) k_compute_cta(
    DFront F, DStep s, DGraph G, const uint64_t* __restrict__ est_incl, uint32_t b0, uint64_t* out_ptr,
    uint32_t* out_cnt, uint32_t* out_data, uint64_t out_cap, unsigned long long* acc, uint32_t* err,
    const uint32_t* __restrict__ hq, uint32_t hq_cap, uint32_t win_cap) {
  extern __shared__ __align__(128) uint32_t win[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t wtot[CTA_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&mbar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  uint32_t phase = 0;
  unsigned long long local = 0, bytes = 0;
  const uint64_t base = (MODE == 0 && b0 > 0) ? est_incl[b0 - 1] : 0;
  const uint32_t nheavy = min(hq[0], hq_cap);
  for (uint32_t i = blockIdx.x; i < nheavy; i += gridDim.x) {
    const uint32_t p = hq[1 + i];
    // the two lists (backward lists, then the reused set), pivot first
    const uint32_t* L[2];
    const uint32_t* Bm[2] = {nullptr, nullptr};
    uint32_t N[2];
    int nl = 0;
    for (int k = 0; k < 2 && k < s.nconn; ++k) {
      const uint32_t v = F.inst[s.conn[k]][p];
      AdjList(G, v, L[k], N[k]);
      Bm[k] = HubBitmap(G, v);
      nl = k + 1;
    }
    if (s.reuse >= 0 && nl < 2) {
      GetSet(F, s.reuse, p, L[nl], N[nl]);
      Bm[nl] = nullptr;
      ++nl;
    }
    if (N[1] < N[0]) {
      const uint32_t* t = L[0];
      L[0] = L[1];
      L[1] = t;
      t = Bm[0];
      Bm[0] = Bm[1];
      Bm[1] = t;
      const uint32_t tn = N[0];
      N[0] = N[1];
      N[1] = tn;
    }
    BoundsT<0> bd = MakeBounds<0>(s.cond, F, p);
    uint32_t r0 = 0, r1 = 0;
    Range(L[0], N[0], bd, r0, r1);
    if (tid == 0) bytes += 4ULL * (r1 - r0) * 2ULL;
    // the other list's window [a, e) over the pivot's value range
    const uint32_t* W = L[1];
    uint32_t WN = N[1];
    bool staged = false;
    uint32_t pad = 0;
    if (!Bm[1] && r1 > r0) {
      const uint32_t a = LowerBound(L[1], N[1], __ldg(L[0] + r0));
      const uint32_t e = a + LowerBound(L[1] + a, N[1] - a, __ldg(L[0] + r1 - 1) + 1);
      W = L[1] + a;
      WN = e - a;
      const uintptr_t lo = (uintptr_t)W, hi = (uintptr_t)(W + WN);
      const uintptr_t alo = (lo + 15) & ~(uintptr_t)15, ahi = hi & ~(uintptr_t)15;
      const uint32_t head = (uint32_t)((alo - lo) >> 2);  // elements before the aligned interior
      pad = (4 - (head & 3)) & 3;
      staged = WN >= 64 && pad + WN <= win_cap && WN <= kStageRatio * (r1 - r0) && ahi > alo;
      if (staged) {
        const uint32_t bytes_in = (uint32_t)(ahi - alo);
        if (tid == 0) {
          // shared memory the previous path read is overwritten by the async proxy
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes_in)
                       : "memory");
          const uint32_t dst = (uint32_t)__cvta_generic_to_shared(win + pad + head);
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
              "l"(alo), "r"(bytes_in), "r"(bar)
              : "memory");
        }
        // ragged ends by plain loads
        const uint32_t tail0 = (uint32_t)((ahi - lo) >> 2);
        if (tid < (int)head) win[pad + tid] = __ldg(W + tid);
        if (tid >= 4 && tid < 4 + (int)(WN - tail0)) win[pad + tail0 + (tid - 4)] = __ldg(W + tail0 + (tid - 4));
        const bool done = MbarWait(bar, phase);
        // one decision for the whole CTA (and the ragged ends made visible)
        if (__syncthreads_or(!done)) {
          // the copy did not complete: flag it, give it one more bounded
          // wait (it writes this CTA's shared memory) and stop this CTA
          if (tid == 0) atomicOr(err, ENGINE_ERR_TIMEOUT);
          MbarWait(bar, phase);
          return;
        }
        phase ^= 1;
      }
    }
    const uint32_t* Ws = staged ? win + pad : W;
    const uint32_t* Bo = Bm[1];
    const uint32_t* P2 = nullptr;  // ranked-count partner set
    uint32_t P2N = 0;
    if (MODE == 1 && s.with_u >= 0) GetSet(F, s.with_u, p, P2, P2N);
    const uint64_t out_off = MODE == 0 ? (p + b0 == 0 ? 0 : est_incl[p + b0 - 1]) - base : 0;
    uint32_t cur = 0, written = 0;
    for (uint32_t bi = r0; bi < r1; bi += CTA_THREADS) {
      const uint32_t k = bi + tid;
      bool ok = k < r1;
      const uint32_t x = ok ? __ldg(L[0] + k) : 0;
      if (ok && nl == 2) {
        if (Bo) {
          ok = BitTest(Bo, x);
        } else if (staged) {
          const uint32_t pos = cur + LowerBoundShared(Ws + cur, WN - cur, x);
          cur = pos;
          ok = pos < WN && Ws[pos] == x;
        } else {
          const uint32_t pos = cur + LowerBound(Ws + cur, WN - cur, x);
          cur = pos;
          ok = pos < WN && __ldg(Ws + pos) == x;
        }
      }
      const unsigned mask = __ballot_sync(FULL, ok);
      if (MODE == 1) {
        if (ok) local += P2 ? RankCount(P2, P2N, x, s.with_op) : 1ULL;
      } else {
        if (lane == 0) wtot[wid] = __popc(mask);
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < CTA_WARPS; ++w) {
          const uint32_t c = wtot[w];
          before += w < wid ? c : 0;
          total += c;
        }
        if (MODE == 0 && ok) {
          const uint64_t o = out_off + written + before + __popc(mask & ((1u << lane) - 1));
          if (o < out_cap) out_data[o] = x;
          else atomicOr(err, ENGINE_ERR_BOUNDS);
        }
        written += total;
        __syncthreads();  // wtot is rewritten by the next chunk
      }
    }
    if (tid == 0 && MODE != 1) {
      out_ptr[p] = MODE == 0 ? (uint64_t)(out_data + out_off) : 0;
      out_cnt[p] = written;
      if (MODE == 0) bytes += 4ULL * written;
    }
    __syncthreads();  // the window is free for the next path
  }
  if (MODE == 1) {
    local = WarpSum(local);
    if (lane == 0 && local) atomicAdd(acc, local);
  }
  if (tid == 0 && bytes) atomicAdd(acc + 1, bytes);
}

// ---- intersection, flattened over 32 paths per warp ------------------------
// Same result as k_compute.  Each lane first prepares one path (lists, pivot,
// clipped pivot range, excluded values) into shared memory; the warp then
// walks the concatenation of the 32 pivot ranges 32 elements at a time, so
// short pivots (the common case on skewed graphs) keep every lane busy.  A
// lane finds its element's path by binary search over the 32 range offsets.
// Sets stay sorted and compact per path: the rank of an element is its path's
// running count plus the valid lanes before it in the same path segment.
template <int NLM, int NEX>
struct FlatPath {
  const uint32_t* L[NLM];  // L[0] = pivot (already offset by r0); others cut to the pivot's value range
  const uint32_t* B[NLM];  // hub bitmaps (null: binary search)
  uint32_t N[NLM];
  uint32_t ne[NEX > 0 ? NEX : 1];
  const uint32_t* W;       // ranked-count partner set
  uint32_t WN;
  uint64_t out_off;
  uint32_t written;
  uint8_t nl, nne;
};
constexpr int FLAT_WARPS = WARP_BLOCK / 32;

// Specialised like k_compute: NLM bounds the intersected lists, NEX = 0 for
// steps without `!=` conditions (the launcher guarantees both).
template <int MODE, int MINB = 1, int NLM = MAXV, int NEX = MAXV>
__global__ void __launch_bounds__(WARP_BLOCK, MINB) k_compute_flat(
    DFront F, DStep s, DGraph G, const uint64_t* __restrict__ est_incl, uint32_t b0, uint64_t* out_ptr,
    uint32_t* out_cnt, uint32_t* out_data, uint64_t out_cap, unsigned long long* acc, uint32_t* err) {
  __shared__ FlatPath<NLM, NEX> sp[FLAT_WARPS][32];
  __shared__ uint32_t soff[FLAT_WARPS][33];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  unsigned long long local = 0, bytes = 0;
  const uint64_t base = (MODE == 0 && b0 > 0) ? est_incl[b0 - 1] : 0;
  for (uint32_t p0 = gw * 32; p0 < F.P; p0 += nw * 32) {
    const uint32_t p = p0 + lane;
    uint32_t len = 0;
    bool view = false;
    if (p < F.P) {
      FlatPath<NLM, NEX>& fp = sp[wl][lane];
      const uint32_t* L[NLM];
      const uint32_t* B[NLM];
      uint32_t N[NLM];
      int nl = 0;
#pragma unroll
      for (int i = 0; i < NLM; ++i) {
        B[i] = nullptr;
        if (i < s.nconn) {
          uint32_t v = F.inst[s.conn[i]][p];
          AdjList(G, v, L[i], N[i]);
          B[i] = HubBitmap(G, v);
          nl = i + 1;
        }
      }
      if (s.reuse >= 0) {
#pragma unroll
        for (int i = 0; i < NLM; ++i)
          if (i == nl) GetSet(F, s.reuse, p, L[i], N[i]);
        ++nl;
      }
      uint64_t b = 12ULL * s.nconn;  // row pointers + gathered instance vertices
#pragma unroll
      for (int i = 1; i < NLM; ++i) {
        if (i < nl && N[i] < N[0]) {
          const uint32_t* tp = L[0];
          L[0] = L[i];
          L[i] = tp;
          tp = B[0];
          B[0] = B[i];
          B[i] = tp;
          uint32_t tn = N[0];
          N[0] = N[i];
          N[i] = tn;
        }
      }
      BoundsT<NEX> bd = MakeBounds<NEX>(s.cond, F, p);
      uint32_t r0 = 0, r1 = 0;
      if (nl > 0) Range(L[0], N[0], bd, r0, r1);
      if (MODE == 0) {
        fp.out_off = (p + b0 == 0 ? 0 : est_incl[p + b0 - 1]) - base;
        if (nl == 1 && !s.noview) {
          uint32_t ex[MAXV];
          if (Exclusions(L[0], r0, r1, bd, ex) == 0) {
            out_ptr[p] = (uint64_t)(L[0] + r0);
            out_cnt[p] = r1 - r0;
            view = true;
          }
        }
      }
      if (!view) b += 4ULL * (r1 - r0) * (uint64_t)nl;  // pivot elements x lists tested
      bytes += b;
      fp.W = nullptr;
      fp.WN = 0;
      if (MODE == 1 && s.with_u >= 0) GetSet(F, s.with_u, p, fp.W, fp.WN);
      fp.L[0] = L[0] + r0;
      fp.N[0] = r1 - r0;
      // the other lists only matter between the pivot's first and last value
      const uint32_t lo_v = r1 > r0 ? __ldg(L[0] + r0) : 0, hi_v = r1 > r0 ? __ldg(L[0] + r1 - 1) : 0;
#pragma unroll
      for (int i = 1; i < NLM; ++i) {
        fp.B[i] = B[i];
        fp.L[i] = L[i];
        fp.N[i] = N[i];
        if (i < nl && !B[i] && r1 > r0) {
          const uint32_t a = LowerBound(L[i], N[i], lo_v);
          const uint32_t e = a + LowerBound(L[i] + a, N[i] - a, hi_v + 1);
          fp.L[i] = L[i] + a;
          fp.N[i] = e - a;
        }
      }
#pragma unroll
      for (int i = 0; i < NEX; ++i) fp.ne[i] = bd.ne[i];
      fp.nne = (uint8_t)bd.nne;
      fp.nl = (uint8_t)nl;
      fp.written = 0;
      len = view ? 0 : r1 - r0;
    }
    // exclusive scan of the pivot ranges of the 32 paths
    uint32_t x = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    soff[wl][lane] = x - len;
    const uint32_t total = __shfl_sync(FULL, x, 31);
    if (lane == 31) soff[wl][32] = total;
    __syncwarp();
    for (uint32_t fb = 0; fb < total; fb += 32) {
      const uint32_t f = fb + lane;
      const bool in = f < total;
      // path of element f: last j with soff[j] <= f
      int j = 0;
      if (in) {
        int lo = 0, hi = 31;
        while (lo < hi) {
          int mid = (lo + hi + 1) >> 1;
          if (soff[wl][mid] <= f) lo = mid;
          else hi = mid - 1;
        }
        j = lo;
      }
      const FlatPath<NLM, NEX>& fp = sp[wl][j];
      bool ok = in;
      uint32_t v = 0;
      if (ok) {
        v = __ldg(fp.L[0] + (f - soff[wl][j]));
#pragma unroll
        for (int k = 0; k < NEX; ++k)
          if (k < fp.nne && v == fp.ne[k]) ok = false;
#pragma unroll
        for (int q = 1; q < NLM; ++q) {
          if (q < fp.nl && ok) {
            if (fp.B[q]) {
              ok = BitTest(fp.B[q], v);
            } else {
              uint32_t pos = LowerBound(fp.L[q], fp.N[q], v);
              ok = pos < fp.N[q] && __ldg(fp.L[q] + pos) == v;
            }
          }
        }
      }
      const unsigned valid = __ballot_sync(FULL, ok);
      if (MODE == 1) {
        if (ok) local += fp.W ? RankCount(fp.W, fp.WN, v, s.with_op) : 1;
      } else {
        // segments of lanes that belong to the same path
        const int jprev = __shfl_up_sync(FULL, j, 1);
        const unsigned start = __ballot_sync(FULL, in && (lane == 0 || jprev != j));
        const unsigned le = (lane == 31) ? FULL : ((2u << lane) - 1);
        const int seg = 31 - __clz(start & le);
        const unsigned segmask = (lane == 31 ? FULL : ((2u << lane) - 1)) & ~((1u << seg) - 1);
        const uint32_t before = __popc(valid & segmask & ((1u << lane) - 1));
        const uint32_t w0 = in ? sp[wl][j].written : 0;
        if (MODE == 0 && ok) {
          uint64_t o = fp.out_off + w0 + before;
          if (o < out_cap) out_data[o] = v;
          else atomicOr(err, ENGINE_ERR_BOUNDS);
        }
        __syncwarp();
        // the last lane of each segment advances its path's running count
        const int jnext = __shfl_down_sync(FULL, j, 1);
        const bool last = in && (lane == 31 || f + 1 >= total || jnext != j);
        if (last) sp[wl][j].written = w0 + before + (ok ? 1 : 0);
        __syncwarp();
      }
      (void)valid;
    }
    if (MODE != 1 && p < F.P && !view) {  // views were published above
      const FlatPath<NLM, NEX>& fp = sp[wl][lane];
      out_ptr[p] = MODE == 0 ? (uint64_t)(out_data + fp.out_off) : 0;
      out_cnt[p] = fp.written;
      if (MODE == 0) bytes += 4ULL * fp.written;
    }
    __syncwarp();
  }
  if (MODE == 1) {
    local = WarpSum(local);
    if (lane == 0 && local) atomicAdd(acc, local);
  }
  bytes = WarpSum(bytes);
  if (lane == 0 && bytes) atomicAdd(acc + 1, bytes);
}

// ---- MATERIALIZE ---------------------------------------------------------
// Expands each path's valid candidates into child rows: materialised columns
// (broadcast from the parent) plus the new vertex, and the set index of every
// live candidate set (Materialize, src/gpu/impl/light/op/LIGHTMaterialize.cuh:23-162,
// fused: expand + filter + compact + per-column gather in one pass).  Work is
// cut by child rows, not by parents: a warp takes kMatChunk consecutive rows,
// finds the parent of the first one with a warp-cooperative search over the
// inclusive child counts, and walks forward through the parents the chunk
// covers; the k-th child of a parent is its k-th candidate in the clipped
// range that is not excluded.  A parent with tens of thousands of children
// (a hub's list) is spread over many warps instead of holding one.  Only
// parents of more than `big` children are expanded here (the rest, whose
// per-parent set-up a chunk would serialise, take k_mat_write); the parents
// a chunk covers are scanned 32 at a time, one coalesced load per lane.
constexpr uint32_t kMatChunk = 1024;
constexpr uint64_t kMatBig = 2048;

// First p in [0, n) with a[p] > c, by the whole warp (`a` non-decreasing).
__device__ __forceinline__ uint32_t WarpUpperBound64(const uint64_t* __restrict__ a, uint32_t n, uint64_t c) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = 0, len = n;
  while (len > 32) {
    const uint32_t step = (len + 31) / 32;
    const uint32_t idx = lo + lane * step;
    const bool le = idx < lo + len && __ldg(a + idx) <= c;
    const uint32_t k = __popc(__ballot_sync(0xffffffffu, le));
    if (k == 0) return lo;
    const uint32_t nlo = lo + (k - 1) * step + 1;
    const uint32_t nhi = min(lo + k * step, lo + len);
    lo = nlo;
    len = nhi - nlo;
  }
  const bool le = lane < len && __ldg(a + lo + lane) <= c;
  return lo + __popc(__ballot_sync(0xffffffffu, le));
}

__global__ void __launch_bounds__(WARP_BLOCK) k_mat_write_big(DFront F, DCond c, DMatOut o,
                                                              const uint64_t* __restrict__ incl,
                                                              uint64_t total, uint64_t big, uint32_t* err) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const int u = o.u;
  for (uint64_t c0 = (uint64_t)gw * kMatChunk; c0 < total; c0 += (uint64_t)nw * kMatChunk) {
    const uint64_t c1 = c0 + kMatChunk < total ? c0 + kMatChunk : total;
    // the parents overlapping [c0, c1) start at the parent of row c0; they
    // are scanned 32 at a time and only the large ones expanded
    uint32_t p = WarpUpperBound64(incl, F.P, c0);
    while (p < F.P) {
      const uint32_t q = p + lane;
      bool cand = false, past = false;
      if (q < F.P) {
        const uint64_t qe = __ldg(incl + q), qo = q == 0 ? 0 : __ldg(incl + q - 1);
        past = qo >= c1;
        cand = !past && qe - qo > big;  // qe > c0 holds for every q at or after the first parent
      }
      const unsigned mp = __ballot_sync(FULL, past);
      unsigned todo = __ballot_sync(FULL, cand);
      if (mp) todo &= (1u << (__ffs(mp) - 1)) - 1;
      while (todo) {
        const uint32_t pp = p + (__ffs(todo) - 1);
        todo &= todo - 1;
        const uint64_t off = pp == 0 ? 0 : __ldg(incl + pp - 1);
        const uint64_t end = __ldg(incl + pp);
        const uint32_t* a;
        uint32_t n;
        GetSet(F, u, pp, a, n);
        Bounds bd = MakeBounds(c, F, pp);
        uint32_t r0, r1, ex[MAXV];
        WarpRange(a, n, bd, r0, r1);
        int ne = Exclusions(a, r0, r1, bd, ex);
        uint32_t vals[MAXV], idx[MAXV];
#pragma unroll
        for (int i = 0; i < MAXV; ++i) {
          vals[i] = 0;
          idx[i] = 0;
          if (i < o.nmat && o.mat[i] != u) vals[i] = F.inst[o.mat[i]][pp];
          if (i < o.nsets) idx[i] = SetIndex(F, o.sets[i], pp);
        }
        const uint64_t s0 = off > c0 ? off : c0, s1 = end < c1 ? end : c1;
        for (uint64_t w = s0 + lane; w < s1; w += 32) {
          // the (w - off)-th candidate of [r0, r1) that is not excluded
          uint32_t j = r0 + (uint32_t)(w - off);
#pragma unroll
          for (int k = 0; k < MAXV; ++k)
            if (k < ne && ex[k] <= j) ++j;
          if (j >= r1) {
            atomicOr(err, ENGINE_ERR_BOUNDS);
            continue;
          }
          const uint32_t x = __ldg(a + j);
#pragma unroll
          for (int i = 0; i < MAXV; ++i) {
            if (i < o.nmat) o.inst[o.mat[i]][w] = o.mat[i] == u ? x : vals[i];
            if (i < o.nsets) o.cidx[o.sets[i]][w] = idx[i];
          }
        }
      }
      if (mp) break;
      p += 32;
    }
  }
}

// The same without `!=` conditions, where a parent's children are one range of
// its set starting at first[p] (null: at the set's start): one lane per child
// row.  A warp takes `rows` consecutive rows, finds the parents of the first
// and the last one together and each lane its row's between them, so neither
// a long parent nor many short ones hold a warp up (a warp per parent waited
// for its longest one, a warp per 1024 rows for its parents' set-up).  32 rows
// while the warps fit the device, kMatRows beyond.  Triangles of R-MAT s14,
// 114 000 rows: 73 us by the two kernels below and above, 10 us here.
constexpr uint32_t kMatRows = 128;

__global__ void __launch_bounds__(WARP_BLOCK) k_mat_rows(DFront F, DMatOut o, const uint64_t* __restrict__ incl,
                                                         const uint32_t* __restrict__ first, uint64_t total,
                                                         uint32_t rows) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int u = o.u;
  for (uint64_t c0 = gw * rows; c0 < total; c0 += nw * rows) {
    const uint64_t c1 = c0 + rows < total ? c0 + rows : total;
    const uint32_t pa = WarpUpperBound64(incl, F.P, c0);
    const uint32_t pb = pa + WarpUpperBound64(incl + pa, F.P - pa, c1 - 1);
    for (uint64_t w = c0 + lane; w < c1; w += 32) {
      uint32_t lo = pa, hi = pb;  // first p with incl[p] > w
      while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (__ldg(incl + mid) > w) hi = mid;
        else lo = mid + 1;
      }
      const uint64_t off = lo == 0 ? 0 : __ldg(incl + lo - 1);
      const uint32_t s = SetIndex(F, u, lo);
      const uint32_t* a = reinterpret_cast<const uint32_t*>(F.set[u].ptr[s]);
      const uint32_t x = __ldg(a + (first ? __ldg(first + lo) : 0) + (uint32_t)(w - off));
#pragma unroll
      for (int i = 0; i < MAXV; ++i) {
        if (i < o.nmat) o.inst[o.mat[i]][w] = o.mat[i] == u ? x : F.inst[o.mat[i]][lo];
        if (i < o.nsets) o.cidx[o.sets[i]][w] = SetIndex(F, o.sets[i], lo);
      }
    }
  }
}

// Parents of at most `big` children: one warp each (the large ones are
// k_mat_write_big's).
__global__ void __launch_bounds__(WARP_BLOCK) k_mat_write(DFront F, DCond c, DMatOut o,
                                                          const uint64_t* __restrict__ incl,
                                                          uint64_t total, uint64_t big, uint32_t* err) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const int u = o.u;
  for (uint32_t p = gw; p < F.P; p += nw) {
    if ((p == 0 ? incl[0] : incl[p] - incl[p - 1]) > big) continue;  // k_mat_write_big's
    const uint32_t* a;
    uint32_t n;
    GetSet(F, u, p, a, n);
    Bounds bd = MakeBounds(c, F, p);
    uint32_t r0, r1, ex[MAXV];
    Range(a, n, bd, r0, r1);
    int ne = Exclusions(a, r0, r1, bd, ex);
    uint64_t off = (p == 0 ? 0 : incl[p - 1]);
    uint32_t vals[MAXV], idx[MAXV];
#pragma unroll
    for (int i = 0; i < MAXV; ++i) {
      vals[i] = 0;
      idx[i] = 0;
      if (i < o.nmat && o.mat[i] != u) vals[i] = F.inst[o.mat[i]][p];
      if (i < o.nsets) idx[i] = SetIndex(F, o.sets[i], p);
    }
    for (uint32_t j = r0 + lane; j < r1; j += 32) {
      int before = 0;
      bool skip = false;
#pragma unroll
      for (int k = 0; k < MAXV; ++k) {
        if (k < ne) {
          if (ex[k] == j) skip = true;
          if (ex[k] < j) ++before;
        }
      }
      if (skip) continue;
      uint64_t w = off + (j - r0) - before;
      if (w >= total) {
        atomicOr(err, ENGINE_ERR_BOUNDS);
        continue;
      }
      uint32_t x = __ldg(a + j);
#pragma unroll
      for (int i = 0; i < MAXV; ++i) {
        if (i < o.nmat) o.inst[o.mat[i]][w] = o.mat[i] == u ? x : vals[i];
        if (i < o.nsets) o.cidx[o.sets[i]][w] = idx[i];
      }
    }
  }
}

// ---- FILTER_COMPUTE ------------------------------------------------------
// Re-applies conditions to a computed set (FilterCandidate,
// src/gpu/impl/light/op/LIGHTFilterCompute.cuh:22-155).  A filtered set with
// no excluded value inside its range is a view of the old set.
__global__ void __launch_bounds__(WARP_BLOCK) k_filter(DFront F, int u, DCond c,
                                                       const uint64_t* __restrict__ est_incl, uint32_t b0,
                                                       uint64_t* out_ptr, uint32_t* out_cnt,
                                                       uint32_t* out_data, uint64_t out_cap, uint32_t* err) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint64_t base = b0 == 0 ? 0 : est_incl[b0 - 1];
  for (uint32_t p = gw; p < F.P; p += nw) {
    const uint32_t* a;
    uint32_t n;
    GetSet(F, u, p, a, n);
    Bounds bd = MakeBounds(c, F, p);
    uint32_t r0, r1, ex[MAXV];
    Range(a, n, bd, r0, r1);
    int ne = Exclusions(a, r0, r1, bd, ex);
    if (ne == 0) {
      if (lane == 0) {
        out_ptr[p] = (uint64_t)(a + r0);
        out_cnt[p] = r1 - r0;
      }
      continue;
    }
    uint64_t off = (p + b0 == 0 ? 0 : est_incl[p + b0 - 1]) - base;
    for (uint32_t j = r0 + lane; j < r1; j += 32) {
      int before = 0;
      bool skip = false;
      for (int k = 0; k < ne; ++k) {
        if (ex[k] == j) skip = true;
        if (ex[k] < j) ++before;
      }
      if (skip) continue;
      uint64_t w = off + (j - r0) - before;
      if (w < out_cap) out_data[w] = __ldg(a + j);
      else atomicOr(err, ENGINE_ERR_BOUNDS);
    }
    if (lane == 0) {
      out_ptr[p] = (uint64_t)(out_data + off);
      out_cnt[p] = r1 - r0 - ne;
    }
  }
}

// ---- COUNT (LIGHTCount / LIGHTDirectCount) -------------------------------
// One unmaterialised vertex: sum of set sizes.
__global__ void k_count1(DFront F, int u, unsigned long long* acc) {
  unsigned long long s = 0;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < F.P; p += gridDim.x * blockDim.x)
    s += F.set[u].cnt[SetIndex(F, u, p)];
  s = WarpSum(s);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(acc, s);
}

// Two unmaterialised vertices u0,u1 with condition (x0 op x1): each element of
// the smaller set is ranked in the larger one
// (GeneralCountTwoComputedVertices, src/gpu/impl/light/op/LIGHTCount.cuh:22-116).
__global__ void __launch_bounds__(WARP_BLOCK) k_count2(DFront F, int u0, int u1, uint8_t op,
                                                       unsigned long long* acc) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  unsigned long long s = 0;
  for (uint32_t p = gw; p < F.P; p += nw) {
    const uint32_t *A, *B;
    uint32_t na, nb;
    GetSet(F, u0, p, A, na);
    GetSet(F, u1, p, B, nb);
    if (na <= nb) {
      for (uint32_t i = lane; i < na; i += 32) s += RankCount(B, nb, __ldg(A + i), op);
    } else {
      // count x in A with (x op y) for each y in B
      uint8_t rop = op == 0 ? 1 : (op == 1 ? 0 : 2);
      for (uint32_t i = lane; i < nb; i += 32) s += RankCount(A, na, __ldg(B + i), rop);
    }
  }
  s = WarpSum(s);
  if (lane == 0 && s) atomicAdd(acc, s);
}

// Closed forms over candidate-set sizes (ThreadDirectCount,
// src/gpu/impl/light/op/LIGHTDirectCount.cuh:21-79).
__device__ unsigned long long DirectCount(const unsigned long long* c, int q) {
  unsigned long long r = 0;
  switch (q) {
    case 0: r = c[2]; break;
    case 1: r = c[3]; break;
    case 2: r = c[1] > 0 ? c[1] * (c[1] - 1) / 2 : 0; break;
    case 3: r = c[3]; break;
    case 5:
      r = c[1] * c[3] * c[5];
      if (r > 0) r = r - c[3] * (c[1] - 1 + c[5] - 1) - c[3] * c[3];
      break;
    case 6:
      if (c[4] > 0 && c[2] > 0) r = c[4] * c[2] - c[2];
      break;
    case 7: r = c[4]; break;
    case 8: r = c[4]; break;
    case 10: r = c[2] > 0 ? c[2] * (c[2] - 1) / 2 : 0; break;
    case 11: r = c[5]; break;
    default: r = 0;
  }
  return r;
}

__global__ void k_count_direct(DFront F, uint8_t nu, uint8_t u0, uint8_t u1, uint8_t u2, int q,
                               unsigned long long* acc) {
  unsigned long long s = 0;
  const uint8_t us[3] = {u0, u1, u2};
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < F.P; p += gridDim.x * blockDim.x) {
    unsigned long long c[MAXV] = {0, 0, 0, 0, 0, 0};
    for (int i = 0; i < nu; ++i) c[us[i]] = F.set[us[i]].cnt[SetIndex(F, us[i], p)];
    s += DirectCount(c, q);
  }
  s = WarpSum(s);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(acc, s);
}

// ---- external mode: per-batch subgraph ------------------------------------
// Marks the adjacency lists a batch's intersections read
// (InspectRequiredAdjLists, src/gpu/impl/common/ext/EXTGraphGPUCommon.cuh:157-184).
// External mode keeps the adjacency lists a batch reads in a device list
// cache: coff[v] is the first element of v's list in the cache, kAbsent when
// it is not there.  A batch claims the lists it needs that are missing
// (IncInspectRequiredAdjLists, src/gpu/impl/common/ext/EXTIncGraphGPUCommon.cuh:20-75:
// lists already in device memory are not loaded again), places them after
// the cache's last list and gathers them from pinned, mapped host memory;
// lists stay for later batches and steps until the cache is full, when it
// starts over.  Only the lists of a batch cross the host link, and no work
// scales with the vertex count except a start-over.
constexpr uint64_t kAbsent = ~0ULL, kPending = ~0ULL - 1;

// Claims, places and gathers in one launch: a lane takes one list reference
// of the batch, the lane that wins a missing list's claim places it after the
// cache's last one, and the warp then copies the lists its lanes won from
// pinned, mapped host memory (coalesced reads over the host link; replaces the
// host-thread gather + synchronous H2D of LoadSubgraph,
// src/gpu/impl/common/ext/LoadSubgraph.h:10-42, EXTGraphGPUCommon.cuh:60-149).
// A list that does not fit raises `over` and stays pending; the host then
// starts the cache over.
__global__ void __launch_bounds__(WARP_BLOCK) k_ext_load(DFront F, DStep s, const uintE* __restrict__ rp,
                                                         const uint32_t* __restrict__ host_cols, uint64_t* coff,
                                                         uint32_t* __restrict__ cache, uint64_t cap,
                                                         unsigned long long* used, unsigned long long* over) {
  const int lane = threadIdx.x & 31;
  const uint64_t items = (uint64_t)F.P * s.nconn;
  const uint64_t w0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull;
  for (uint64_t b = w0; b < items; b += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t it = b + lane;
    uint64_t from = 0, to = 0;
    uint32_t len = 0;
    if (it < items) {
      const uint32_t v = F.inst[s.conn[it % s.nconn]][it / s.nconn];
      const uint64_t r = __ldg(rp + v);
      const uint32_t n = (uint32_t)(__ldg(rp + v + 1) - r);
      if (n && __ldcg(coff + v) == kAbsent &&
          atomicCAS(reinterpret_cast<unsigned long long*>(coff + v), kAbsent, kPending) == kAbsent) {
        const uint64_t o = atomicAdd(used, (unsigned long long)n);
        if (o + n <= cap) {
          coff[v] = o;
          from = r;
          to = o;
          len = n;
        } else {
          *over = 1;
        }
      }
    }
    for (unsigned won = __ballot_sync(FULL, len > 0); won; won &= won - 1) {
      const int k = __ffs(won) - 1;
      const uint32_t n = __shfl_sync(FULL, len, k);
      const uint32_t* src = host_cols + __shfl_sync(FULL, (unsigned long long)from, k);
      uint32_t* dst = cache + __shfl_sync(FULL, (unsigned long long)to, k);
      // a read over the host link takes microseconds: sixteen per lane at once
      for (uint32_t j0 = 0; j0 < n; j0 += 512) {
        uint32_t x[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          const uint32_t j = j0 + t * 32 + lane;
          x[t] = j < n ? src[j] : 0;
        }
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          const uint32_t j = j0 + t * 32 + lane;
          if (j < n) dst[j] = x[t];
        }
      }
    }
  }
}

// Writes complete instances (all vertices materialised) from instance `at` on,
// in output slots: one thread per output word, so the writes are whole lines
// (cols.p[s]: the column of output slot s).  The position of a frontier's
// instances is the number emitted before it, which the host knows: no counter.
struct EmitCols {
  const uint32_t* p[MAXV];
};
__global__ void k_emit(EmitCols cols, uint32_t P, uint32_t n, uint64_t at, uint32_t* out, uint64_t cap) {
  const uint64_t fit = at < cap ? (cap - at < P ? cap - at : P) : 0;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < fit * n;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t p = e / n;
    out[at * n + e] = __ldg(cols.p[e - p * n] + p);
  }
}

}  // namespace

// ---------------------------------------------------------------- runtime --
void* Arena::Alloc(size_t bytes) {
  size_t b = (bytes + 255) & ~size_t(255);
  if (b > cap - top)
    Fail(SME_ERR_OOM, "device arena exhausted: need " + std::to_string(b) + " bytes, " +
                          std::to_string(cap - top) + " free of " + std::to_string(cap));
  void* p = base + top;
  top += b;
  peak = std::max(peak, top);
  return p;
}

int DeviceCount() {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

namespace {
int SmCount(int device) {
  static int cached[64] = {0};
  if (device >= 0 && device < 64 && cached[device]) return cached[device];
  int v = 148;
  cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
  if (device >= 0 && device < 64) cached[device] = v;
  return v;
}
}  // namespace

DeviceContext::~DeviceContext() {}

DeviceContext* CreateContext(int device, uint64_t bytes) {
  if (DeviceCount() <= device || device < 0) Fail(SME_ERR_NO_DEVICE, "no CUDA device " + std::to_string(device));
  CK(cudaSetDevice(device));
  auto* c = new DeviceContext();
  c->device = device;
  try {
    CK(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
    for (auto& e : c->copy_ev) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    uint64_t want = bytes ? bytes : (uint64_t)(fr * 0.80);
    if (want > fr) want = (uint64_t)(fr * 0.95);
    CK(cudaMalloc((void**)&c->arena.base, want));
    c->arena.cap = want;
    c->pinned_words = 1 << 14;
    CK(cudaMallocHost((void**)&c->h_pinned, c->pinned_words * sizeof(uint64_t)));
  } catch (...) {
    DestroyContext(c);
    throw;
  }
  return c;
}

void DestroyContext(DeviceContext* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  if (c->copy_stream) cudaStreamSynchronize(c->copy_stream);
  if (c->arena.base) cudaFree(c->arena.base);
  if (c->h_pinned) cudaFreeHost(c->h_pinned);
  if (c->h_stage) cudaFreeHost(c->h_stage);
  if (c->stream) cudaStreamDestroy(c->stream);
  if (c->copy_stream) cudaStreamDestroy(c->copy_stream);
  for (auto e : c->copy_ev)
    if (e) cudaEventDestroy(e);
  for (auto e : c->events) cudaEventDestroy(e);
  delete c;
}

namespace {
__global__ void k_build_bitmaps(const uintE* __restrict__ rp, const uint32_t* __restrict__ cols,
                                const uint32_t* __restrict__ hubs, uint32_t words, uint32_t* bm) {
  const uint32_t v = hubs[blockIdx.x];
  uint32_t* row = bm + (size_t)blockIdx.x * words;
  for (uintE j = rp[v] + threadIdx.x; j < rp[v + 1]; j += blockDim.x) {
    uint32_t w = cols[j];
    atomicOr(row + (w >> 5), 1u << (w & 31));
  }
}

// One hub's bitmap per CTA, built in shared memory and written out whole in
// 16-byte stores (no memset of the bitmaps and no global atomics); for
// bitmaps of up to kSmemBitmapBytes.  `words` is a multiple of 4.
constexpr uint32_t kSmemBitmapBytes = 200u << 10;
__global__ void __launch_bounds__(1024) k_build_bitmaps_smem(const uintE* __restrict__ rp,
                                                             const uint32_t* __restrict__ cols,
                                                             const uint32_t* __restrict__ hubs, uint32_t words,
                                                             uint32_t* bm, uint32_t* coarse, uint32_t cwords) {
  extern __shared__ uint4 row_v[];
  uint32_t* row_s = reinterpret_cast<uint32_t*>(row_v);
  const uint32_t quads = words / 4;
  for (uint32_t i = threadIdx.x; i < quads; i += blockDim.x) row_v[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  const uint32_t v = hubs[blockIdx.x];
  for (uintE j = rp[v] + threadIdx.x; j < rp[v + 1]; j += blockDim.x) {
    const uint32_t w = cols[j];
    atomicOr(row_s + (w >> 5), 1u << (w & 31));
  }
  __syncthreads();
  uint4* row = reinterpret_cast<uint4*>(bm + (size_t)blockIdx.x * words);
  for (uint32_t i = threadIdx.x; i < quads; i += blockDim.x) row[i] = row_v[i];
  // coarse row: bit b of word cw set when bitmap word 32 cw + b is not zero
  uint32_t* crow = coarse + (size_t)blockIdx.x * cwords;
  for (uint32_t cw = threadIdx.x; cw < cwords; cw += blockDim.x) {
    uint32_t bits = 0;
    for (uint32_t b = 0; b < 32; ++b) {
      const uint32_t wi = cw * 32 + b;
      if (wi < words && row_s[wi]) bits |= 1u << b;
    }
    crow[cw] = bits;
  }
}

__global__ void k_set_slots(const uint32_t* __restrict__ hubs, uint32_t nh, int32_t* slot) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x)
    slot[hubs[i]] = (int32_t)i;
}

// Bitmaps for the vertices of highest degree (>= kHubMinDegree) within a
// byte budget (SME_HUB_BITMAP_MB, default 1 GiB, at most a quarter of the
// device memory `room` the caller can spare); a bitmap is n bits.  Measured
// on R-MAT s20 (root blocks of the bench): 256 MiB 9.5e9, 512 MiB 9.8e9,
// 1 GiB 10.5e9, 2 GiB 10.7e9 instances/s, flat beyond; whole-graph counts
// flat from 512 MiB.  The hub choice is cached on the host graph; hubs take
// slots in id order, so the hubs of a vertex range are a slot range.
struct HubPlan {
  std::shared_ptr<const std::vector<uint32_t>> sel;  // sorted ids; slot i holds (*sel)[i]
  const std::vector<uint32_t>& hubs() const { return *sel; }
  uint32_t* d_hubs = nullptr;
  uint32_t words = 0;
  bool smem = false;
};

// Chooses the hubs, allocates slot index + bitmaps + hub list with `alloc`,
// and queues on `st` the hub-list copy, the slot fill and (global build only)
// the clearing of the bitmaps.  False when no vertex gets a bitmap.
template <typename Alloc>
bool PlanHubBitmaps(DeviceGraph* d, const HostGraph& g, cudaStream_t st, Alloc alloc, uint64_t room, HubPlan* hp) {
  uint64_t kHubMinDegree = 256;
  if (const char* e = std::getenv("SME_HUB_MIN_DEGREE")) kHubMinDegree = std::strtoull(e, nullptr, 10);
  uint64_t budget = 1024ULL << 20;
  if (const char* e = std::getenv("SME_HUB_BITMAP_MB")) budget = std::strtoull(e, nullptr, 10) << 20;
  budget = std::min<uint64_t>(budget, room / 4);
  // n bits, rounded up to whole 16-byte quads (rows start 16-byte aligned)
  const uint32_t words = (uint32_t)(((g.n + 31) / 32 + 3) & ~uint64_t(3));
  if (budget == 0 || words == 0) return false;
  const uint64_t max_hubs = budget / ((uint64_t)words * 4);
  if (max_hubs == 0) return false;
  hp->sel = g.HubSelection(kHubMinDegree, max_hubs);
  if (hp->sel->empty()) return false;
  const uint32_t nh = (uint32_t)hp->sel->size();
  hp->words = words;
  hp->smem = (uint64_t)words * 4 <= kSmemBitmapBytes;
  d->hub_slot = (int32_t*)alloc(g.n * sizeof(int32_t));
  d->bitmaps = (uint32_t*)alloc((size_t)nh * words * 4);
  if (hp->smem) {  // built beside the bitmap by the shared-memory builder
    d->cwords = (words + 31) / 32;
    d->coarse = (uint32_t*)alloc((size_t)nh * d->cwords * 4);
  }
  hp->d_hubs = (uint32_t*)alloc((size_t)nh * 4);
  CK(cudaMemcpyAsync(hp->d_hubs, hp->sel->data(), (size_t)nh * 4, cudaMemcpyHostToDevice, st));
  CK(cudaMemsetAsync(d->hub_slot, 0xFF, g.n * sizeof(int32_t), st));
  k_set_slots<<<std::min<uint32_t>((nh + 255) / 256, 1184), 256, 0, st>>>(hp->d_hubs, nh, d->hub_slot);
  if (!hp->smem) CK(cudaMemsetAsync(d->bitmaps, 0, (size_t)nh * words * 4, st));
  d->words = words;
  d->nhubs = nh;
  return true;
}

// Builds the bitmaps of slots [first, first + count) from the device lists.
void BuildHubRange(const DeviceGraph* d, const HubPlan& hp, uint32_t first, uint32_t count, cudaStream_t st) {
  if (!count) return;
  if (hp.smem) {
    CK(cudaFuncSetAttribute(k_build_bitmaps_smem, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)kSmemBitmapBytes));
    k_build_bitmaps_smem<<<count, 1024, (size_t)hp.words * 4, st>>>(
        d->row_ptrs, d->cols, hp.d_hubs + first, hp.words, d->bitmaps + (size_t)first * hp.words,
        d->coarse + (size_t)first * d->cwords, d->cwords);
  } else {
    k_build_bitmaps<<<count, 256, 0, st>>>(d->row_ptrs, d->cols, hp.d_hubs + first, hp.words,
                                           d->bitmaps + (size_t)first * hp.words);
  }
}

// Plan + build of every hub, queued on `stream`: the caller keeps the plan (the
// hub list is copied from it) until it has waited for the stream.  Returns the
// host->device bytes.
template <typename Alloc>
uint64_t BuildHubBitmaps(DeviceGraph* d, const HostGraph& g, cudaStream_t stream, Alloc alloc, uint64_t room,
                         HubPlan* hp) {
  if (!PlanHubBitmaps(d, g, stream, alloc, room, hp)) return 0;
  BuildHubRange(d, *hp, 0, (uint32_t)hp->hubs().size(), stream);
  CK(cudaGetLastError());
  return (uint64_t)hp->hubs().size() * 4;
}

// ------------------------------------------------------------ packed lists --
// rp[0] = 0, rp[i + 1] = deg[i] (then an inclusive scan of rp + 1).
__global__ void k_deg_to_rp(const uint32_t* __restrict__ deg, uint64_t n, uintE* rp) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i <= n; i += (uint64_t)gridDim.x * blockDim.x)
    rp[i] = i ? deg[i - 1] : 0;
}

// Expands the packed lists (format: PackedLists, sme_internal.h) of lists
// [v0, v1) into cols; their segments after the first are segs[s0, s1).
// One warp per (list, segment): warps [0, v1 - v0) take segment 0 of list
// v0 + w, the next s1 - s0 warps the segments named in segs.  The warp reads
// the segment's block widths (one per lane), scans the blocks' byte sizes to
// place every block, then per block extracts one delta per lane and adds the
// running value through a warp scan.  Every offset read from the buffer is
// checked against the stream before use: a bad one sets *flag and skips the
// segment.
__global__ void __launch_bounds__(256) k_unpack_lists(const uint32_t* __restrict__ deg,
                                                      const uint32_t* __restrict__ woff,
                                                      const uint64_t* __restrict__ segs, uint64_t n, uint64_t v0,
                                                      uint64_t v1, uint64_t s0, uint64_t s1,
                                                      const uint32_t* __restrict__ stream, uint64_t stream_words,
                                                      const uintE* __restrict__ rp, uint64_t m, uintV* cols,
                                                      uint32_t* flag) {
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nv = v1 - v0;
  if (w >= nv + (s1 - s0)) return;  // uniform in the warp
  uint64_t v;
  uint32_t s;
  if (w < nv) {
    v = v0 + w;
    s = 0;
  } else {
    const uint64_t e = segs[s0 + (w - nv)];
    v = e >> 32;
    s = (uint32_t)e;
  }
  if (v >= n) {
    if (lane == 0) atomicOr(flag, 1u);
    return;
  }
  const uint64_t d = deg[v];
  const uint64_t nseg = (d + kPackSegment - 1) / kPackSegment;
  if (s >= nseg) {
    if (s > 0 && lane == 0) atomicOr(flag, 1u);
    return;
  }
  const uint64_t stream_bytes = stream_words * 4;
  const uint64_t list = (uint64_t)woff[v] * 4;
  uint32_t base = 0;
  uint64_t seg = list + 8 * (nseg - 1);
  if (s > 0) {
    const uint64_t ti = (list >> 2) + 2 * (uint64_t)(s - 1);
    if (ti + 1 >= stream_words) {
      if (lane == 0) atomicOr(flag, 1u);
      return;
    }
    base = stream[ti];
    seg = list + stream[ti + 1];
  }
  const uint64_t e0 = (uint64_t)s * kPackSegment;
  const uint32_t ne = (uint32_t)(d - e0 < kPackSegment ? d - e0 : kPackSegment);
  const uint32_t nb = (ne + 31) / 32;
  const uint64_t out0 = rp[v] + e0;
  if (seg + nb + 8 > stream_bytes || out0 + ne > m) {
    if (lane == 0) atomicOr(flag, 1u);
    return;
  }
  const uint8_t* bytes = reinterpret_cast<const uint8_t*>(stream);
  const uint32_t width = lane < nb ? bytes[seg + lane] : 0;
  const uint32_t cnt = lane < nb ? min(32u, ne - 32 * lane) : 0;
  const uint32_t sz = (cnt * width + 7) / 8;
  uint32_t incl = sz;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  if (__any_sync(FULL, width > 32) || seg + nb + total + 8 > stream_bytes) {
    if (lane == 0) atomicOr(flag, 1u);
    return;
  }
  const uint64_t off = seg + nb + (incl - sz);  // byte start of this lane's block
  uintV* out = cols + out0;
  uint32_t prev = base;
  for (uint32_t t = 0; t < nb; ++t) {
    const uint32_t b = __shfl_sync(FULL, width, t);
    const uint32_t c = __shfl_sync(FULL, cnt, t);
    const uint64_t o = __shfl_sync(FULL, (unsigned long long)off, t);
    uint32_t delta = 0;
    if (lane < c && b) {
      const uint64_t bit = o * 8 + (uint64_t)lane * b;
      const uint64_t wi = bit >> 5;
      delta = __funnelshift_r(stream[wi], stream[wi + 1], (uint32_t)bit & 31);
      if (b < 32) delta &= (1u << b) - 1u;
    }
#pragma unroll
    for (int o2 = 1; o2 < 32; o2 <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, delta, o2);
      if (lane >= o2) delta += y;
    }
    const uint32_t val = prev + delta;
    if (lane < c) out[32 * t + lane] = val;
    prev = __shfl_sync(FULL, val, 31);
  }
}

uint32_t ScanBlocks(uint64_t n) { return (uint32_t)((n + SCAN_TILE - 1) / SCAN_TILE); }

// row_ptrs from the packed degrees in `scratch` (copied there already).
void PackedRowPtrs(const PackedLists& pk, const uint8_t* scratch, uint64_t* bs, uintE* rp, cudaStream_t st) {
  const uint64_t n = pk.n;
  const uint32_t* deg = reinterpret_cast<const uint32_t*>(scratch + pk.deg_at);
  k_deg_to_rp<<<(unsigned)std::min<uint64_t>((n + 256) / 256, 148 * 8), 256, 0, st>>>(deg, n, rp);
  if (n) {
    const uint32_t nb = ScanBlocks(n);
    k_scan_reduce<<<nb, SCAN_THREADS, 0, st>>>(rp + 1, (uint32_t)n, bs);
    k_scan_partials<<<1, 1024, 0, st>>>(bs, nb);
    k_scan_apply<<<nb, SCAN_THREADS, 0, st>>>(rp + 1, (uint32_t)n, bs);
  }
}

// Expands lists [v0, v1) (segments segs[s0, s1)) from `scratch` into cols.
void UnpackRange(const PackedLists& pk, const uint8_t* scratch, const uintE* rp, uintV* cols, uint32_t* flag,
                 uint64_t v0, uint64_t v1, uint64_t s0, uint64_t s1, cudaStream_t st) {
  const uint64_t items = (v1 - v0) + (s1 - s0);
  if (!items) return;
  k_unpack_lists<<<(unsigned)((items * 32 + 255) / 256), 256, 0, st>>>(
      reinterpret_cast<const uint32_t*>(scratch + pk.deg_at), reinterpret_cast<const uint32_t*>(scratch + pk.woff_at),
      reinterpret_cast<const uint64_t*>(scratch + pk.segs_at), pk.n, v0, v1, s0, s1,
      reinterpret_cast<const uint32_t*>(scratch + pk.stream_at), pk.stream_bytes / 4, rp, pk.m, cols, flag);
}

// Copies the packed lists into `scratch` (device, pk.total bytes) and expands
// them into rp (n + 1) and cols (m) on `st`.  `bs` holds ScanBlocks(n) words,
// `flag` one word (set by a bad offset).
void UnpackLists(const PackedLists& pk, uint8_t* scratch, uint64_t* bs, uint32_t* flag, uintE* rp, uintV* cols,
                 cudaStream_t st) {
  CK(cudaMemcpyAsync(scratch, pk.base, pk.total, cudaMemcpyHostToDevice, st));
  CK(cudaMemsetAsync(flag, 0, sizeof(uint32_t), st));
  PackedRowPtrs(pk, scratch, bs, rp, st);
  UnpackRange(pk, scratch, rp, cols, flag, 0, pk.n, 0, pk.nsegs, st);
  CK(cudaGetLastError());
}

void CheckPacked(const HostGraph& g, const PackedLists& pk) {
  if (pk.n != g.n || pk.m != g.m) Fail(SME_ERR_INVALID_ARG, "packed lists do not match the graph");
  if (pk.n > UINT32_MAX) Fail(SME_ERR_INVALID_ARG, "packed upload needs n < 2^32");
}

void FailOnFlag(uint32_t flag) {
  if (flag) Fail(SME_ERR_CUDA, "packed lists are corrupt: an offset points outside the stream");
}

// Per-call packed upload into the arena, copy and expansion overlapped: the
// header (degrees, list offsets, segment ids) and then kUploadChunks byte
// ranges of the stream, cut at list boundaries, go over the context's copy
// stream; the execution stream scans the degrees into row_ptrs, then, as each
// range lands, expands its lists and builds the bitmaps of its hubs.  Hub
// bitmaps are allocated below the copy's scratch, which is released when the
// upload is done.  Returns the host->device bytes beyond the packed buffer.
uint64_t UploadPackedPipelined(const HostGraph& g, const PackedLists& pk, DeviceGraph* d, DeviceContext& ctx,
                               uint32_t* flag) {
  auto arena_alloc = [&ctx](size_t b) { return ctx.arena.Alloc(b); };
  const uint64_t n = pk.n;
  const uint64_t scratch_bytes = pk.total + (uint64_t)ScanBlocks(n) * 8 + 512;
  HubPlan hp;
  const uint64_t room = ctx.arena.Free() > scratch_bytes ? ctx.arena.Free() - scratch_bytes : 0;
  const bool hubs = PlanHubBitmaps(d, g, ctx.stream, arena_alloc, room, &hp);
  const size_t mark = ctx.arena.Mark();
  uint8_t* scratch = (uint8_t*)arena_alloc(pk.total);
  uint64_t* bs = (uint64_t*)arena_alloc((size_t)ScanBlocks(n) * 8);
  CK(cudaMemsetAsync(flag, 0, sizeof(uint32_t), ctx.stream));

  // chunk boundaries: list ids where the stream offset passes k/K of it
  const uint32_t* woff = reinterpret_cast<const uint32_t*>(pk.base + pk.woff_at);
  const uint64_t* segs = reinterpret_cast<const uint64_t*>(pk.base + pk.segs_at);
  const uint64_t lists_words = (pk.stream_bytes - 8) / 4;
  const int K = pk.stream_bytes >= (8ULL << 20) ? kUploadChunks : 1;
  uint64_t vb[kUploadChunks + 1];
  vb[0] = 0;
  vb[K] = n;
  for (int k = 1; k < K; ++k)
    vb[k] = std::max<uint64_t>(vb[k - 1],
                               (uint64_t)(std::lower_bound(woff, woff + n, (uint32_t)(lists_words * k / K)) - woff));
  auto byte_at = [&](uint64_t v) { return v < n ? (uint64_t)woff[v] * 4 : pk.stream_bytes; };
  auto seg_at = [&](uint64_t v) {
    return (uint64_t)(std::lower_bound(segs, segs + pk.nsegs, v << 32) - segs);
  };

  CK(cudaMemcpyAsync(scratch, pk.base, pk.stream_at, cudaMemcpyHostToDevice, ctx.copy_stream));
  CK(cudaEventRecord(ctx.copy_ev[0], ctx.copy_stream));
  for (int k = 0; k < K; ++k) {
    const uint64_t b0 = k == 0 ? 0 : byte_at(vb[k]), b1 = k + 1 == K ? pk.stream_bytes : byte_at(vb[k + 1]);
    if (b1 > b0)
      CK(cudaMemcpyAsync(scratch + pk.stream_at + b0, pk.base + pk.stream_at + b0, b1 - b0,
                         cudaMemcpyHostToDevice, ctx.copy_stream));
    CK(cudaEventRecord(ctx.copy_ev[k + 1], ctx.copy_stream));
  }
  CK(cudaStreamWaitEvent(ctx.stream, ctx.copy_ev[0], 0));
  PackedRowPtrs(pk, scratch, bs, d->row_ptrs, ctx.stream);
  for (int k = 0; k < K; ++k) {
    CK(cudaStreamWaitEvent(ctx.stream, ctx.copy_ev[k + 1], 0));
    UnpackRange(pk, scratch, d->row_ptrs, d->cols, flag, vb[k], vb[k + 1], seg_at(vb[k]), seg_at(vb[k + 1]),
                ctx.stream);
    if (hubs) {
      const std::vector<uint32_t>& H = hp.hubs();
      const uint32_t h0 = (uint32_t)(std::lower_bound(H.begin(), H.end(), (uint32_t)vb[k]) - H.begin());
      const uint32_t h1 = vb[k + 1] >= n ? (uint32_t)H.size()
                                         : (uint32_t)(std::lower_bound(H.begin(), H.end(), (uint32_t)vb[k + 1]) -
                                                      H.begin());
      BuildHubRange(d, hp, h0, h1 - h0, ctx.stream);
    }
  }
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(ctx.stream));
  ctx.arena.Release(mark);
  return hubs ? (uint64_t)hp.hubs().size() * 4 : 0;
}
}  // namespace

namespace {
DGraph ViewOf(const DeviceGraph& g) {
  if (g.hub_slot)
    return DGraph{g.row_ptrs, g.cols, g.hub_slot, g.bitmaps, g.words, nullptr, g.coarse, g.cwords};
  return DGraph{g.row_ptrs, g.cols, nullptr, nullptr, 0, nullptr, nullptr, 0};
}

// Queues k_check_simple on `st` (`flag` cleared by the caller).
void LaunchCheck(const DeviceGraph& g, bool sym, uint32_t* flag, cudaStream_t st) {
  if (!g.m) return;
  // a chunk is a serial chain for its warp: short ones while there are few
  const uint32_t chunk = g.m < (4u << 20) ? 64 : 512;
  const unsigned grid = (unsigned)std::min<uint64_t>((g.m + (uint64_t)chunk * 8 - 1) / ((uint64_t)chunk * 8),
                                                     (uint64_t)SmCount(g.device) * 8);
  if (sym)
    k_check_simple<true><<<grid, WARP_BLOCK, 0, st>>>(ViewOf(g), (uint32_t)g.n, g.m, chunk, flag);
  else
    k_check_simple<false><<<grid, WARP_BLOCK, 0, st>>>(ViewOf(g), (uint32_t)g.n, g.m, chunk, flag);
}
}  // namespace

DeviceGraph* UploadGraph(const HostGraph& g, int device, cudaStream_t stream, uint64_t* h2d) {
  CK(cudaSetDevice(device));
  auto* d = new DeviceGraph();
  d->device = device;
  d->n = g.n;
  d->m = g.m;
  uint64_t bytes = 0;
  std::shared_ptr<const PackedLists> pk = g.packed;
  uint8_t* scratch = nullptr;
  HubPlan hp;
  try {
    // one word after the row pointers for k_check_simple's flag
    CK(cudaMalloc((void**)&d->row_ptrs, (g.n + 2) * sizeof(uintE)));
    CK(cudaMalloc((void**)&d->cols, std::max<uint64_t>(g.m, 1) * sizeof(uintV)));
    if (pk) {
      CheckPacked(g, *pk);
      const uint64_t bs_at = (pk->total + 15) & ~uint64_t(15);
      CK(cudaMalloc((void**)&scratch, bs_at + (uint64_t)ScanBlocks(g.n) * 8 + 16));
      uint32_t* flag = reinterpret_cast<uint32_t*>(scratch + bs_at + (uint64_t)ScanBlocks(g.n) * 8);
      UnpackLists(*pk, scratch, reinterpret_cast<uint64_t*>(scratch + bs_at), flag, d->row_ptrs, d->cols, stream);
      uint32_t h_flag = 0;
      CK(cudaMemcpyAsync(&h_flag, flag, 4, cudaMemcpyDeviceToHost, stream));
      CK(cudaStreamSynchronize(stream));
      cudaFree(scratch);
      scratch = nullptr;
      FailOnFlag(h_flag);
      bytes = pk->total;
    } else {
      CK(cudaMemcpyAsync(d->row_ptrs, g.row_ptrs, (g.n + 1) * sizeof(uintE), cudaMemcpyHostToDevice, stream));
      if (g.m) CK(cudaMemcpyAsync(d->cols, g.cols, g.m * sizeof(uintV), cudaMemcpyHostToDevice, stream));
      bytes = (g.n + 1) * sizeof(uintE) + g.m * sizeof(uintV);
    }
    auto dev_alloc = [](size_t b) {
      void* p = nullptr;
      CK(cudaMalloc(&p, b));
      return p;
    };
    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    bytes += BuildHubBitmaps(d, g, stream, dev_alloc, fr, &hp);
    uint32_t* flag = reinterpret_cast<uint32_t*>(d->row_ptrs + g.n + 1);
    CK(cudaMemsetAsync(flag, 0, sizeof(uint32_t), stream));
    LaunchCheck(*d, true, flag, stream);
    uint32_t defects = 0;
    CK(cudaMemcpyAsync(&defects, flag, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));  // the upload's only wait (a packed one has another)
    CK(cudaGetLastError());
    d->defects = (int)defects;
    if (hp.d_hubs) cudaFree(hp.d_hubs);
  } catch (...) {
    cudaStreamSynchronize(stream);  // copies and kernels on the arrays freed below
    if (scratch) cudaFree(scratch);
    if (hp.d_hubs) cudaFree(hp.d_hubs);
    FreeDeviceGraph(d);
    throw;
  }
  if (h2d) *h2d += bytes;
  return d;
}

DeviceGraph* UploadGraphToArena(const HostGraph& g, DeviceContext& ctx, uint64_t* h2d) {
  CK(cudaSetDevice(ctx.device));
  auto* d = new DeviceGraph();
  d->device = ctx.device;
  d->n = g.n;
  d->m = g.m;
  d->in_arena = true;
  uint64_t bytes = 0;
  std::shared_ptr<const PackedLists> pk = g.packed;
  HubPlan hp;
  try {
    QuiesceOnError quiesce(ctx);
    auto arena_alloc = [&ctx](size_t b) { return ctx.arena.Alloc(b); };
    d->row_ptrs = (uintE*)arena_alloc((g.n + 1) * sizeof(uintE));
    d->cols = (uintV*)arena_alloc(std::max<uint64_t>(g.m, 1) * sizeof(uintV));
    uint32_t* flag = nullptr;
    if (pk) {
      CheckPacked(g, *pk);
      flag = (uint32_t*)arena_alloc(sizeof(uint32_t));
      bytes = pk->total + UploadPackedPipelined(g, *pk, d, ctx, flag);
    } else {
      CK(cudaMemcpyAsync(d->row_ptrs, g.row_ptrs, (g.n + 1) * sizeof(uintE), cudaMemcpyHostToDevice, ctx.stream));
      if (g.m) CK(cudaMemcpyAsync(d->cols, g.cols, g.m * sizeof(uintV), cudaMemcpyHostToDevice, ctx.stream));
      bytes = (g.n + 1) * sizeof(uintE) + g.m * sizeof(uintV);
      bytes += BuildHubBitmaps(d, g, ctx.stream, arena_alloc, ctx.arena.Free(), &hp);
    }
    if (flag) {
      CK(cudaMemcpyAsync(ctx.h_pinned, flag, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.stream));
      CK(cudaStreamSynchronize(ctx.stream));
      FailOnFlag(*reinterpret_cast<const uint32_t*>(ctx.h_pinned));
    }
    CK(cudaStreamSynchronize(ctx.stream));
    quiesce.done = true;
  } catch (...) {
    delete d;
    throw;
  }
  if (h2d) *h2d += bytes;
  return d;
}

void FreeDeviceGraph(DeviceGraph* d) {
  if (!d) return;
  if (d->in_arena) {  // released with the arena mark taken before the upload
    delete d;
    return;
  }
  cudaSetDevice(d->device);
  if (d->row_ptrs) cudaFree(d->row_ptrs);
  if (d->cols && !d->host_mapped) cudaFree(d->cols);
  if (d->hub_slot) cudaFree(d->hub_slot);
  if (d->bitmaps) cudaFree(d->bitmaps);
  if (d->coarse) cudaFree(d->coarse);
  delete d;
}

// --------------------------------------------------------------- executor --
namespace {

DCond ToDCond(const std::vector<StepCond>& c) {
  DCond d{};
  d.n = (uint8_t)c.size();
  for (size_t i = 0; i < c.size(); ++i) {
    d.op[i] = c[i].op;
    d.operand[i] = c[i].operand;
  }
  return d;
}

DStep ToDStep(const Step& s) {
  DStep d{};
  d.u = s.u;
  d.nconn = (uint8_t)s.conn.size();
  for (size_t i = 0; i < s.conn.size(); ++i) d.conn[i] = s.conn[i];
  d.reuse = s.reuse_src;
  d.cond = ToDCond(s.cond);
  d.with_u = s.with_u;
  d.with_op = s.with_op;
  d.msrc = s.map_src;
  d.mx = s.map_x;
  d.mmask = s.map_mask;
  d.mop = s.map_op;
  return d;
}

// Timing events a context keeps between runs.
constexpr size_t kKeptEvents = 256;
// Free arena below which every count runs its level program.
constexpr uint64_t kFormArena = 64ULL << 20;

class Executor {
 public:
  Executor(const Program& prog, const DeviceGraph& g, DeviceContext& ctx, uint32_t* d_out, uint64_t cap)
      : prog_(prog), g_(g), ctx_(ctx), A_(ctx.arena), st_(ctx.stream), out_(d_out), cap_(cap), steps_(&prog.steps) {
    sms_ = SmCount(ctx.device);
    mat_misses_.assign(std::max(prog.steps.size(), prog.minus.size()), 0);
    mat_skips_ = mat_misses_;
    lists_simple_ = g.defects >= 0 && !((uint32_t)g.defects & kNotSimple);
  }

  ~Executor() {
    for (auto& e : events_) {
      cudaEventDestroy(e.a);
      cudaEventDestroy(e.b);
    }
  }

  // External mode: adjacency lists are read from `host_cols` (pinned and
  // mapped host memory) into a per-batch device subgraph; g_.row_ptrs holds
  // the global row pointers on the device (GraphDevTracker,
  // src/gpu/graph/GraphDevTracker.cuh:12-79).
  void SetExternal(const uint32_t* host_cols) { ext_cols_ = host_cols; }
  uint64_t ext_h2d_bytes() const { return ext_bytes_; }

  RunResult Run(const RootTask& task) {
    QuiesceOnError quiesce(ctx_);
    const uint32_t stride = task.stride ? task.stride : 1;
    auto t0 = std::chrono::steady_clock::now();
    size_t mark = A_.Mark();
    A_.peak = mark;  // high-water mark of this run
    ctrl_ = (unsigned long long*)A_.Alloc(kCtrl * sizeof(unsigned long long));
    acc_ = ctrl_;
    if (ext_cols_) AllocExternalCache();
    const cudaEvent_t ev0 = TakeEvent(), ev1 = TakeEvent();
    CK(cudaEventRecord(ev0, st_));
    CK(cudaMemsetAsync(ctrl_, 0, kCtrl * sizeof(unsigned long long), st_));
    const Step& s0 = (*steps_)[0];
    // roots: inst column + next level estimate + scan temporaries
    const uint64_t per_root = 4 + 8 + 8;
    uint64_t chunk = std::max<uint64_t>(1, Budget(0) / per_root);
    chunk = std::min<uint64_t>(chunk, 0x7fffffffULL);
    // the task's roots in chunks of `chunk` roots
    const uint64_t nroots = task.Count();
    for (uint64_t i0 = 0; i0 < nroots; i0 += chunk) {
      uint32_t P = (uint32_t)std::min<uint64_t>(chunk, nroots - i0);
      size_t m = A_.Mark();
      uint32_t* col = (uint32_t*)A_.Alloc((size_t)P * 4);
      if (task.list) {
        CK(cudaMemcpyAsync(col, task.list + i0, (size_t)P * 4, cudaMemcpyHostToDevice, st_));
        root_h2d_ += (uint64_t)P * 4;
      } else {
        k_iota<<<Grid(P, 256), 256, 0, st_>>>(col, P, (uint32_t)(task.begin + i0 * stride), stride);
        Launched();
      }
      DFront F{};
      F.P = P;
      F.inst[s0.u] = col;
      ++batches_;
      if (!CountByForm(task, col, P)) Level(1, F);
      if (i0 + P >= nroots) break;  // what the last chunk left is told by the final read
      if (left_) RunLeft((uint32_t)ReadU64((const uint64_t*)(ctrl_ + 14)));
      A_.Release(m);
    }
    unsigned long long h[kCtrl];
    auto finish = [&] {
      CK(cudaEventRecord(ev1, st_));
      CK(cudaMemcpyAsync(h, ctrl_, sizeof(h), cudaMemcpyDeviceToHost, st_));
      CK(cudaStreamSynchronize(st_));
    };
    finish();
    if (h[14]) {
      RunLeft((uint32_t)h[14]);
      finish();
    }
    quiesce.done = true;
    float dev_ms = 0;
    cudaEventElapsedTime(&dev_ms, ev0, ev1);
    CK(cudaGetLastError());
    if (h[3])
      Fail(SME_ERR_CUDA, std::string(h[3] & ENGINE_ERR_BOUNDS ? "device bounds check failed" : "") +
                             (h[3] & ENGINE_ERR_TIMEOUT ? " bulk-copy wait gave up" : "") + " (engine error flags " +
                             std::to_string(h[3]) + ")");
    RunResult r;
    r.count = prog_.enumerate ? emitted_ : h[0] - (h[8] - minus_paths_);
    r.emitted = emitted_;
    r.stats.algorithmic_bytes = h[1] + h[9];
    r.stats.reuse_hits = h[5];
    ext_bytes_ += h[6] * 4;
    r.stats.kernel_launches = launches_;
    r.stats.batches = batches_;
    r.stats.peak_device_bytes = A_.peak;
    r.stats.paths_processed = paths_;
    HarvestTimers();
    ctx_.events.push_back(ev0);
    ctx_.events.push_back(ev1);
    while (ctx_.events.size() > kKeptEvents) {
      cudaEventDestroy(ctx_.events.back());
      ctx_.events.pop_back();
    }
    const double* phase = phase_;
    for (int i = 0; i < 8; ++i) r.stats.phase_ms[i] = phase[i];
    // the intersection kernels: COMPUTE, COMPUTE_COUNT, COMPUTE_PATH_COUNT
    r.stats.kernel_ms = phase[kPhaseCompute] + phase[kPhaseComputeCount] + phase[kPhasePathCount];
    r.stats.device_ms = dev_ms;
    r.stats.hot_launches = hot_;
    r.stats.h2d_bytes = root_h2d_;
    r.stats.elapsed_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    A_.Release(mark);
    return r;
  }

 private:
  const Program& prog_;
  const DeviceGraph& g_;
  DeviceContext& ctx_;
  Arena& A_;
  cudaStream_t st_;
  uint32_t* out_;
  uint64_t cap_;
  const std::vector<Step>* steps_;  // the level program being run
  int sms_ = 148;
  bool lists_simple_ = false;  // known to hold no element twice
  int verdict_[2] = {-1, -1};  // Defects without and with symmetry, -1 not asked
  // [0] count [1] bytes [3] error flags [4] list cache overflow
  // [5] reuse hits [6] list cache elements [7] ticket of k_est_scan; [8..13]
  // count, bytes and hits of Program::minus [14] roots in left_
  static constexpr int kCtrl = 16;
  unsigned long long* ctrl_ = nullptr;
  unsigned long long* acc_ = nullptr;  // counters of the program being run
  uint32_t* left_ = nullptr;           // roots that CountCycles leaves to the steps
  uint64_t emitted_ = 0;               // instances written (or counted past the capacity)
  uint64_t minus_paths_ = 0;           // paths of the last step of Program::minus
  uint64_t launches_ = 0, batches_ = 0, paths_ = 0, hot_ = 0, root_h2d_ = 0;
  const uint32_t* ext_cols_ = nullptr;
  uint64_t ext_bytes_ = 0;
  uint64_t* ext_off_ = nullptr;      // per vertex: list offset in the cache
  uint32_t* ext_cache_ = nullptr;    // device list cache
  uint64_t ext_cap_ = 0, ext_bound_ = 0;
  double ext_overlap_ = 32.0;
  int ext_misses_ = 0;  // counting frontiers whose lists did not fit at once
  // per step: frontiers whose children did not fit the budget at once, less
  // three times those whose children did
  std::vector<int> mat_misses_, mat_skips_;

  // The steps over the roots left_[0..n).
  void RunLeft(uint32_t n) {
    DFront F{};
    F.P = n;
    F.inst[(*steps_)[0].u] = left_;
    left_ = nullptr;
    CK(cudaMemsetAsync(ctrl_ + 14, 0, sizeof(unsigned long long), st_));
    Level(1, F);
  }

  // The resident graph with its hub bitmaps (`use_bitmaps_` false: lists only).
  DGraph Resident() const {
    if (use_bitmaps_) return ViewOf(g_);
    return DGraph{g_.row_ptrs, g_.cols, nullptr, nullptr, 0, nullptr, nullptr, 0};
  }

  // k_check_simple's verdict on the graph (found at upload for a resident
  // one, else here, once per call; one on symmetry is one on the lists too).
  uint32_t Defects(bool sym) {
    if (g_.defects >= 0) return (uint32_t)g_.defects;
    if (verdict_[1] >= 0) return (uint32_t)verdict_[1];
    if (!sym && verdict_[0] >= 0) return (uint32_t)verdict_[0];
    const size_t mark = A_.Mark();
    uint32_t* flag = (uint32_t*)A_.Alloc(sizeof(uint32_t));
    CK(cudaMemsetAsync(flag, 0, sizeof(uint32_t), st_));
    LaunchCheck(g_, sym, flag, st_);
    Launched();
    verdict_[sym] = (int)ReadU32(flag);
    A_.Release(mark);
    return (uint32_t)verdict_[sym];
  }

  // Counts the roots col[0..P) with the program's own kernel when it has one
  // and the graph and the arena allow it; false: run the steps.  Below
  // kFormArena of free arena the steps' batches stay in charge, whose budget
  // a caller has set.
  bool CountByForm(const RootTask& task, const uint32_t* col, uint32_t P) {
    if (prog_.form == C_STEPS || ext_cols_ || g_.n > 0xFFFFFFFEu || A_.Free() < kFormArena + (uint64_t)P * 8)
      return false;
    // a graph that came with the call is checked in it: 3.6 ps an edge for the
    // lists, 28 with symmetry, and a host round trip (R-MAT s20: 0.11 and 0.88
    // ms of kernel).  A root saves 20 ns of the 4-clique's level program (0.66
    // ms for 16 384 roots, 0.26 on the matrices; 85 ns for 5-cliques) and 6 us
    // of the 4-cycle's and the house's: few roots of a large graph keep it
    // (2 000 roots of R-MAT s20: 0.26 ms, 0.31 with the check; 4 000: equal)
    if (g_.defects < 0 && (uint64_t)P * (prog_.form == C_CLIQUE ? 6000 : 1 << 17) < g_.m) return false;
    if (prog_.form == C_CYCLE4) return !Defects(true) && CountCycles(col, P);
    if (prog_.form == C_HOUSE) return !Defects(true) && CountHouses(col, P);
    const bool all = !task.list && task.begin == 0 && task.end >= g_.n && task.stride <= 1 && P == g_.n;
    if (prog_.n == 3 && (!all || oriented_)) return false;  // (see below): no need to ask
    const uint32_t bad = Defects(all && !oriented_);
    if (bad & kNotSimple) return false;
    const bool orient = all && !oriented_ && !(bad & kNotSymmetric) && g_.m / 2 < 0xFFFFFFFFull;
    switch (prog_.n) {
      // triangles of a block of roots: the level program (4096 roots of R-MAT
      // s20 0.21 ms, 0.27 here); of every root: R-MAT s20 21.5 -> 7.8 ms, s18
      // 3.0 -> 1.4, a flat graph of 65 536 vertices 0.35 -> 0.15
      case 3: return orient && CountCliques<3, true>(task, col, P);
      case 4: return orient ? CountCliques<4, true>(task, col, P) : CountCliques<4, false>(task, col, P);
      case 5: return orient ? CountCliques<5, true>(task, col, P) : CountCliques<5, false>(task, col, P);
      case 6: return orient ? CountCliques<6, true>(task, col, P) : CountCliques<6, false>(task, col, P);
      default: return false;
    }
  }

  template <int K, bool ORIENT, int THREADS, bool GLOBAL>
  void LaunchCliqueClass(const CView& V, const uint32_t* col, const CliqueQueues& Q, int cls, uint32_t dmax,
                         uint32_t* scratch, cudaStream_t st) {
    const size_t smem = CliqueSmem(K, dmax, THREADS, GLOBAL);
    auto kernel = k_clique_cta<K, ORIENT, THREADS, GLOBAL>;
    // one attribute per instantiation and device (the largest class of it;
    // setting it twice from two threads is harmless)
    constexpr size_t kMost = GLOBAL       ? CliqueSmem(K, kCliqueG, THREADS, true)
                             : THREADS == kCliqueMThreads ? CliqueSmem(K, kCliqueM, THREADS, false)
                                                          : CliqueSmem(K, CliqueX(K), THREADS, false);
    static std::atomic<int> per_sm_of[64][2];  // resident CTAs: class L or the only one, class X
    const int dv = ctx_.device, slot = cls == 3 ? 1 : 0;
    int per_sm = dv >= 0 && dv < 64 ? per_sm_of[dv][slot].load(std::memory_order_acquire) : 0;
    if (!per_sm) {
      CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, THREADS, smem));
      per_sm = std::max(per_sm, 1);
      if (dv >= 0 && dv < 64) per_sm_of[dv][slot].store(per_sm, std::memory_order_release);
    }
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)sms_ * (GLOBAL ? 1 : per_sm),
                                                       (uint64_t)Q.cap[cls] * kCliqueParts);
    uint32_t* taken = Q.taken + (cls > 2 ? Q.cap[2] : 0) + (cls > 3 ? Q.cap[3] : 0);
    kernel<<<grid, THREADS, smem, st>>>(V, col, Q.q[cls], Q.n + cls, Q.cap[cls], Q.n + 8 + cls, taken, dmax, scratch,
                                         ctrl_);
    Launched();
  }

  // Houses over the roots col[0..P) (house.cuh): the counters' sum, less what
  // the program `minus` counts; roots that do not take the counters run the
  // steps.
  bool CountHouses(const uint32_t* col, uint32_t P) {
    static std::atomic<bool> set[64];  // per device, once (twice is harmless)
    const int dv = ctx_.device;
    if (dv < 0 || dv >= 64 || !set[dv].load(std::memory_order_acquire)) {
      CK(cudaFuncSetAttribute(k_house, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHouseSmem));
      if (dv >= 0 && dv < 64) set[dv].store(true, std::memory_order_release);
    }
    if ((uint64_t)P * 8 > A_.Free() / 4) return false;
    const size_t mark = A_.Mark();
    uint32_t* ctl = (uint32_t*)A_.Alloc(4 * sizeof(uint32_t));  // kept, left, next
    uint32_t* kept = (uint32_t*)A_.Alloc((size_t)P * 4);
    uint32_t* left = (uint32_t*)A_.Alloc((size_t)P * 4);
    CK(cudaMemsetAsync(ctl, 0, 4 * sizeof(uint32_t), st_));
    const uint32_t ranges = (uint32_t)((g_.n + kHouseTile - 1) / kHouseTile);
    k_house_split<<<WarpGrid(P), WARP_BLOCK, 0, st_>>>(ViewOf(g_), col, P, (uint64_t)kHouseWork * ranges, kept, left,
                                                       ctl);
    Launched();
    CK(cudaMemcpyAsync(ctx_.h_pinned, ctl, 8, cudaMemcpyDeviceToHost, st_));
    CK(cudaStreamSynchronize(st_));
    const uint32_t nk = (uint32_t)ctx_.h_pinned[0], nl = (uint32_t)(ctx_.h_pinned[0] >> 32);
    DFront F{};
    if (nk) {
      paths_ += nk;
      // sums and roofs of a slice of the roots at a time (12 KB a root, in at
      // most half of the arena; items below 2^32)
      const uint32_t slice = (uint32_t)std::min<uint64_t>(
          {nk, A_.Free() / 2 / (kHouseCand * 12), 65536, 0xFFFFFFFFull / ranges});
      const size_t qmark = A_.Mark();
      unsigned long long* Qs = (unsigned long long*)A_.Alloc((size_t)slice * kHouseCand * 12);
      Timed t = TimerStart();
      for (uint32_t k = 0; k < nk; k += slice) {
        const uint32_t m = std::min(slice, nk - k);
        CK(cudaMemsetAsync(Qs, 0, (size_t)m * kHouseCand * 12, st_));  // roofs follow
        CK(cudaMemsetAsync(ctl + 2, 0, sizeof(uint32_t), st_));
        uint32_t* roofs = (uint32_t*)(Qs + (size_t)m * kHouseCand);
        k_house<<<(unsigned)std::min<uint64_t>(sms_, (uint64_t)m * ranges), CYC_THREADS, kHouseSmem, st_>>>(
            ViewOf(g_), (uint32_t)g_.n, kept + k, m * ranges, ranges, ctl + 2, Qs, roofs, ctrl_);
        k_house_sum<<<Grid((uint64_t)m * kHouseCand, WARP_BLOCK), WARP_BLOCK, 0, st_>>>(
            Qs, roofs, (uint64_t)m * kHouseCand, ctrl_);
        launches_ += 2;
      }
      TimerStop(t, kPhaseComputeCount);
      A_.Release(qmark);
      steps_ = &prog_.minus;
      acc_ = ctrl_ + 8;
      F.P = nk;
      F.inst[(*steps_)[0].u] = kept;
      Level(1, F);
      steps_ = &prog_.steps;
      acc_ = ctrl_;
    }
    if (nl) {
      F = DFront{};
      F.P = nl;
      F.inst[(*steps_)[0].u] = left;
      Level(1, F);
    }
    A_.Release(mark);
    return true;
  }

  // k-cliques over the roots col[0..P) by bit matrices (clique.cuh).  Roots
  // above every class, and few large ones, run the level program; ORIENT has
  // none to hand back, so there a root above every class sends the whole task
  // to it (false).
  template <int K, bool ORIENT>
  bool CountCliques(const RootTask& task, const uint32_t* col, uint32_t P) {
    if (P > 0xFFFFFFFFu / kCliqueParts) return false;
    // entries a class can hold: distinct roots of more than c candidates are
    // at most m / c
    auto most = [&](uint32_t above) {
      return (uint32_t)(task.list ? P : std::min<uint64_t>(P, g_.m / (above + 1) + 1));
    };
    // largest possible list: ORIENT keeps neighbours of at least the same
    // degree, so d of them hold d * d of the m stored edges
    const uint64_t bound = ORIENT ? (uint64_t)std::sqrt((double)g_.m) + 1 : g_.n;
    CliqueQueues Q{};
    Q.cap[0] = Q.cap[1] = P;
    Q.cap[2] = most(kCliqueM);
    Q.cap[3] = most(kCliqueL);
    Q.cap[4] = Q.left_cap = most(CliqueX(K));
    const uint64_t tiles = (g_.m + OriTile(g_.m) - 1) / OriTile(g_.m);
    const uint64_t ntaken = K == 3 ? 0 : (uint64_t)Q.cap[2] + Q.cap[3] + Q.cap[4];
    uint64_t need = 4096 + Q.left_cap * 4ull + ntaken * 4;
    for (int c = 0; c < 5; ++c) need += Q.cap[c] * 4ull + 256;
    if (ORIENT) need += g_.n * sizeof(uint2) + (g_.m / 2 + 1) * 4 + tiles * 8 + g_.m / 8 + 2048;
    if (need > A_.Free() / 2) return false;
    const size_t mark = A_.Mark();
    uint32_t* ctl = (uint32_t*)A_.Alloc(16 * sizeof(uint32_t));
    for (int c = 0; c < 5; ++c) Q.q[c] = (uint32_t*)A_.Alloc(std::max<size_t>(Q.cap[c], 1) * 4);
    Q.left = (uint32_t*)A_.Alloc(std::max<size_t>(Q.left_cap, 1) * 4);
    if (ntaken && bound > kCliqueM) {
      Q.taken = (uint32_t*)A_.Alloc(ntaken * 4);
      CK(cudaMemsetAsync(Q.taken, 0, ntaken * 4, st_));
    }
    Q.n = ctl;
    Q.nleft = ctl + 5;
    Q.err = (uint32_t*)(ctrl_ + 3);
    Q.top = CliqueX(K);
    uint32_t* scratch = nullptr;
    const size_t scratch_bytes = (size_t)sms_ * CliqueScratchWords(kCliqueG) * 4;
    if (bound > Q.top && A_.Free() / 2 > scratch_bytes) Q.top = kCliqueG;
    CView V{oriented_ ? ViewOf(g_) : Resident(), nullptr, nullptr};
    CK(cudaMemsetAsync(ctl, 0, 16 * sizeof(uint32_t), st_));
    paths_ += P;
    Timed to = TimerStart();
    if (ORIENT) {
      uint2* rng = (uint2*)A_.Alloc((size_t)g_.n * sizeof(uint2));
      uint32_t* ocols = (uint32_t*)A_.Alloc((g_.m / 2 + 1) * 4);
      uint64_t* bs = (uint64_t*)A_.Alloc(std::max<size_t>(tiles, 1) * 8);
      uint32_t* keep = (uint32_t*)A_.Alloc((size_t)(g_.m / 32 + 1) * 4);
      CK(cudaMemsetAsync(rng, 0, (size_t)g_.n * sizeof(uint2), st_));
      if (tiles) {
        k_orient<false><<<(unsigned)tiles, ORI_THREADS, 0, st_>>>(g_.row_ptrs, g_.cols, (uint32_t)g_.n, g_.m, keep,
                                                                  bs, ocols, rng);
        k_scan_partials<<<1, 1024, 0, st_>>>(bs, (uint32_t)tiles);
        k_orient<true><<<(unsigned)tiles, ORI_THREADS, 0, st_>>>(g_.row_ptrs, g_.cols, (uint32_t)g_.n, g_.m, keep,
                                                                 bs, ocols, rng);
        launches_ += 3;
      }
      V.rng = rng;
      V.ocols = ocols;
    }
    if (Q.top == kCliqueG) scratch = (uint32_t*)A_.Alloc(scratch_bytes);
    k_clique_classify<K, ORIENT><<<Grid(P, 256), 256, 0, st_>>>(V, col, P, Q);
    Launched();
    TimerStop(to, kPhaseOrganize);
    // roots for the level program: those above every class, and those of L, X
    // and G where they are few (of G also where their candidates are hardly
    // joined).  Oriented lists have no such program.
    uint32_t nsteps = 0;
    uint32_t* steps_roots = nullptr;
    bool run[5] = {true, true, true, bound > kCliqueL, Q.top == kCliqueG};
    if (ORIENT ? bound > Q.top : bound > (K == 4 ? CliqueX(K) : K == 5 ? kCliqueL : kCliqueM)) {
      CK(cudaMemcpyAsync(ctx_.h_pinned, ctl, 7 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st_));
      CK(cudaStreamSynchronize(st_));
      uint32_t n[5];
      std::memcpy(n, ctx_.h_pinned, sizeof(n));
      for (int c = 0; c < 5; ++c) n[c] = std::min(n[c], Q.cap[c]);
      const uint32_t left = std::min(reinterpret_cast<const uint32_t*>(ctx_.h_pinned)[5], Q.left_cap);
      const uint32_t joined = reinterpret_cast<const uint32_t*>(ctx_.h_pinned)[6];
      if (left && ORIENT) {
        A_.Release(mark);
        paths_ -= P;
        return false;
      }
      const bool busy = (uint64_t)n[1] + 6ull * n[2] >= (K == 6 ? 8000 : 2000);
      nsteps = left;
      for (int c = 2; c < 5; ++c)
        if (!ORIENT && (c == 4 ? n[c] < CliqueLeast(K, c) || !CliqueDense(K, joined, n[c])
                               : n[c] < CliqueLeast(K, c) && !busy)) {
          run[c] = false;
          nsteps += n[c];
        }
      if (nsteps) {
        steps_roots = (uint32_t*)A_.Alloc((size_t)nsteps * 4);
        if (left) CK(cudaMemcpyAsync(steps_roots, Q.left, (size_t)left * 4, cudaMemcpyDeviceToDevice, st_));
        uint32_t at = left;
        for (int c = 2; c < 5; ++c) {
          if (run[c] || !n[c]) continue;
          k_clique_roots<<<Grid(n[c], 256), 256, 0, st_>>>(col, Q.q[c], n[c], steps_roots + at);
          Launched();
          at += n[c];
        }
      }
    }
    Timed t = TimerStart();
    // the classes are independent: the few large roots (first) and the small
    // ones run on the context's second stream beside class M, so neither waits
    // for the other's last CTAs; a class no list can reach is not launched
    constexpr int kWide = K <= 4 ? 1024 : 512;
    const bool fork = bound > kCliqueM;
    if (fork) {
      CK(cudaEventRecord(ctx_.copy_ev[0], st_));
      CK(cudaStreamWaitEvent(ctx_.copy_stream, ctx_.copy_ev[0], 0));
      if (run[4])
        LaunchCliqueClass<K, ORIENT, 256, true>(V, col, Q, 4, kCliqueG, scratch, ctx_.copy_stream);
      if (run[3])
        LaunchCliqueClass<K, ORIENT, kWide, false>(V, col, Q, 3, CliqueX(K), nullptr, ctx_.copy_stream);
      if (run[2])
        LaunchCliqueClass<K, ORIENT, kWide, false>(V, col, Q, 2, kCliqueL, nullptr, ctx_.copy_stream);
    }
    if (bound > kCliqueS)
      LaunchCliqueClass<K, ORIENT, kCliqueMThreads, false>(V, col, Q, 1, kCliqueM, nullptr, st_);
    k_clique_small<K, ORIENT><<<WarpGrid(P), WARP_BLOCK, 0, fork ? ctx_.copy_stream : st_>>>(V, col, Q.q[0], Q.n,
                                                                                             Q.cap[0], ctrl_);
    Launched();
    if (fork) CK(cudaEventRecord(ctx_.copy_ev[1], ctx_.copy_stream));
    if (fork) CK(cudaStreamWaitEvent(st_, ctx_.copy_ev[1], 0));
    TimerStop(t, kPhaseComputeCount);
    if (nsteps) {
      DFront F{};
      F.P = nsteps;
      F.inst[(*steps_)[0].u] = steps_roots;
      Level(1, F);
    }
    A_.Release(mark);
    return true;
  }

  // 4-cycles through the roots col[0..P) by two-path counters (cycle.cuh).
  bool CountCycles(const uint32_t* col, uint32_t P) {
    // ranges of a root's counters, at most (the narrowest: 32-bit counters,
    // which a graph of 65536 vertices or fewer never needs)
    const uint64_t per = kCycleTable / (g_.n > 0xFFFFu ? 4 : 2);
    const uint64_t ranges = (g_.n + per - 1) / per;
    if (P * ranges > 0xFFFFFFFFull || P * (ranges * 8 + 8) > A_.Free() / 2) return false;
    left_ = (uint32_t*)A_.Alloc((size_t)P * 4);  // released with the chunk of roots
    uint32_t* nleft = (uint32_t*)(ctrl_ + 14);
    const size_t mark = A_.Mark();
    static std::atomic<bool> set[64];  // per device, once (twice is harmless)
    const int dv = ctx_.device;
    if (dv < 0 || dv >= 64 || !set[dv].load(std::memory_order_acquire)) {
      CK(cudaFuncSetAttribute(k_cycle4_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCycleWarpSmem));
      CK(cudaFuncSetAttribute(k_cycle4_cta<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCycleCtaSmem));
      CK(cudaFuncSetAttribute(k_cycle4_cta<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCycleCtaSmem));
      if (dv >= 0 && dv < 64) set[dv].store(true, std::memory_order_release);
    }
    // next root, queued roots, next queued, queued ranges, next range
    uint32_t* ctl = (uint32_t*)A_.Alloc(8 * sizeof(uint32_t));
    uint32_t* queue = (uint32_t*)A_.Alloc((size_t)P * 4);
    uint64_t* tiles = (uint64_t*)A_.Alloc((size_t)P * ranges * 8);
    uint32_t* err = (uint32_t*)(ctrl_ + 3);
    const DGraph G = ViewOf(g_);
    paths_ += P;
    Timed t = TimerStart();
    CK(cudaMemsetAsync(ctl, 0, 8 * sizeof(uint32_t), st_));
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)sms_ * 2, (P + CYW_WARPS - 1) / CYW_WARPS);
    const unsigned ctas = (unsigned)std::min<uint64_t>(sms_, P);
    k_cycle4_warp<<<grid, CYW_THREADS, kCycleWarpSmem, st_>>>(G, col, P, ctl, queue, ctl + 1, ctrl_);
    k_cycle4_cta<false><<<ctas, CYC_THREADS, kCycleCtaSmem, st_>>>(G, (uint32_t)g_.n, col, queue, ctl + 1, ctl + 2,
                                                                    tiles, ctl + 3, (uint32_t)(P * ranges), left_,
                                                                    nleft, err, ctrl_);
    launches_ += 2;
    // more two-paths than the table takes need more than kCycleHashMax edges
    if (g_.m > kCycleHashMax) {
      const unsigned most = (unsigned)std::min<uint64_t>(sms_, (uint64_t)P * ranges);
      k_cycle4_cta<true><<<most, CYC_THREADS, kCycleCtaSmem, st_>>>(G, (uint32_t)g_.n, col, queue, ctl + 1, ctl + 4,
                                                                     tiles, ctl + 3, (uint32_t)(P * ranges), left_,
                                                                     nleft, err, ctrl_);
      ++launches_;
    }
    TimerStop(t, kPhaseComputeCount);
    A_.Release(mark);
    return true;
  }

  struct Batch {
    uint32_t b0, b1;
    uint64_t e0, e1;  // inclusive estimate before b0 / at b1-1
    uint64_t lists;   // external mode: elements of the lists its paths read
  };

  // Loads the adjacency lists that step `ds` intersects for the paths of Fb and
  // that the device list cache does not hold yet.
  // `elems`: the elements of all those lists, counted per path.  What the
  // cache holds is known here only as a bound (`ext_bound_`: the batches'
  // elements since the last look); the device's own count is read when the
  // bound no longer fits.  False: the batch's lists do not fit the empty cache.
  bool LoadLists(const DFront& Fb, const DStep& ds, uint64_t elems) {
    Timed tl = TimerStart();
    unsigned long long* seen = ctrl_ + 4;  // [4] overflow, [6] elements held
    auto load = [&] {
      k_ext_load<<<Grid((uint64_t)Fb.P * std::max<int>(ds.nconn, 1), WARP_BLOCK), WARP_BLOCK, 0, st_>>>(
          Fb, ds, g_.row_ptrs, ext_cols_, ext_off_, ext_cache_, ext_cap_, ctrl_ + 6, ctrl_ + 4);
      Launched();
    };
    auto look = [&] {  // true: no overflow
      CK(cudaMemcpyAsync(ctx_.h_pinned, seen, 24, cudaMemcpyDeviceToHost, st_));
      CK(cudaStreamSynchronize(st_));
      ext_bound_ = ctx_.h_pinned[2];
      return ctx_.h_pinned[0] == 0;
    };
    auto clear = [&] {
      ext_bytes_ += std::min<uint64_t>(ext_bound_, ext_cap_) * 4;
      CK(cudaMemsetAsync(ext_off_, 0xff, (size_t)(g_.n + 1) * 8, st_));
      CK(cudaMemsetAsync(ctrl_ + 4, 0, 8, st_));
      CK(cudaMemsetAsync(ctrl_ + 6, 0, 8, st_));
      ext_bound_ = 0;
    };
    bool fits = true;
    load();
    if (ext_bound_ + elems <= ext_cap_) {
      ext_bound_ += elems;
    } else if (!look()) {  // the cache is full: start over with this batch's lists
      clear();
      load();
      if (elems <= ext_cap_) {
        ext_bound_ = elems;
      } else if (!look()) {
        clear();
        fits = false;
      }
    }
    TimerStop(tl, kPhaseExternal);
    return fits;
  }

  DGraph View() const {
    return ext_cols_ ? DGraph{g_.row_ptrs, ext_cache_, nullptr, nullptr, 0, ext_off_, nullptr, 0} : Resident();
  }

  // A batch whose lists do not fit the cache, as two (`incl`, `incl2`: the
  // paths' inclusive estimates and list elements), the first on top.
  void Halve(const Batch& b, const uint64_t* incl, const uint64_t* incl2, std::vector<Batch>& todo) {
    if (b.b1 - b.b0 < 2)
      Fail(SME_ERR_OOM, "external mode: the lists one batch reads (" + std::to_string(b.lists * 4) +
                            " bytes) exceed the device list cache (" + std::to_string(ext_cap_ * 4) + " bytes)");
    ext_overlap_ = std::max(1.0, ext_overlap_ / 2);
    const uint32_t mid = b.b0 + (b.b1 - b.b0) / 2;
    const uint64_t em = ReadU64(incl + mid - 1);
    const uint64_t lm = ReadU64(incl2 + mid - 1) - (b.b0 ? ReadU64(incl2 + b.b0 - 1) : 0);
    todo.push_back(Batch{mid, b.b1, em, b.e1, b.lists - lm});
    todo.push_back(Batch{b.b0, mid, b.e0, em, lm});
  }

  uint64_t ReadU32(const unsigned int* d) {
    CK(cudaMemcpyAsync(ctx_.h_pinned, d, sizeof(unsigned int), cudaMemcpyDeviceToHost, st_));
    CK(cudaStreamSynchronize(st_));
    return *reinterpret_cast<const unsigned int*>(ctx_.h_pinned);
  }

  // External mode: the device list cache takes about half of the arena that
  // is free when the run starts (the frontiers keep the rest).
  void AllocExternalCache() {
    ext_off_ = (uint64_t*)A_.Alloc((size_t)(g_.n + 1) * 8);
    CK(cudaMemsetAsync(ext_off_, 0xff, (size_t)(g_.n + 1) * 8, st_));
    const uint64_t bytes = std::max<uint64_t>(A_.Free() / 2, 1 << 20) & ~uint64_t(255);
    ext_cache_ = (uint32_t*)A_.Alloc(bytes);
    ext_cap_ = bytes / 4;
    ext_bound_ = 0;
  }

  // What a batch of step k may cost at least.  In memory a budget below 1 MiB
  // is taken for 1 MiB: batches of a few thousand paths cost more launches than
  // they save memory.  In external mode only while the levels after this one
  // can take as much: batches there are not held small by the lists they load,
  // and levels that each took 1 MiB of an arena of a few left none for the
  // next.  (The last step is a count, which takes next to nothing.)
  uint64_t AtLeast(size_t k, uint64_t budget) const {
    uint64_t least = 1 << 20;
    if (ext_cols_) least = std::min(least, (uint64_t)((double)A_.Free() * 0.85 / (double)((*steps_).size() - k)));
    return std::max(budget, least);
  }

  // Batch cost of an external step in frontier-budget units: the subgraph
  // bytes count against the list cache (cg scales them so that frontier
  // bytes / budget + list bytes / (cache x ext_overlap_) <= 1).  The list bytes
  // are counted per path, and the paths of a batch share most of their lists,
  // so a batch is first given ext_overlap_ times the cache; one whose lists do
  // not fit after all is halved, and so is the factor.  R-MAT s16, 13 MiB:
  // 4-cliques 1.07 s in 11 855 batches -> 0.19 s in 2 418.
  double ExtListCost(size_t k, uint64_t budget) const {
    return ext_cols_ && ext_cap_ ? 4.0 * (double)AtLeast(k, budget) / ((double)(ext_cap_ * 4) * ext_overlap_) : 0.0;
  }
  std::vector<Timed> events_;  // recorded regions
  double phase_[8] = {0, 0, 0, 0, 0, 0, 0, 0};

  void Launched() { ++launches_; }

  unsigned Grid(uint64_t items, int per_block) const {
    uint64_t b = (items + per_block - 1) / per_block;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(b, (uint64_t)sms_ * 16));
  }
  unsigned WarpGrid(uint64_t paths) const { return Grid(paths * 32, WARP_BLOCK); }

  // The order in which a count step takes its paths: grouped by the hub
  // slot of the step's last list vertex (the most recently materialised one,
  // which changes fastest along the frontier), or nullptr to keep the
  // frontier order (no bitmaps, a small frontier, no room, or turned off).
  const uint32_t* GroupByHub(const DFront& F, const DStep& ds) {
    if (!group_by_hub_ || !use_bitmaps_ || !g_.hub_slot || g_.nhubs == 0 || ds.nconn == 0 || F.P < (1u << 16))
      return nullptr;
    const uint32_t nb = g_.nhubs + 1;
    const size_t need = (size_t)F.P * 4 + (size_t)nb * 24 + (((size_t)nb + SCAN_TILE - 1) / SCAN_TILE) * 8 + 4096;
    if (A_.Free() < need + (16u << 20)) return nullptr;
    Timed to = TimerStart();
    const uint8_t kv = ds.conn[ds.nconn - 1];
    unsigned long long* cnt = (unsigned long long*)A_.Alloc((size_t)nb * 8);
    unsigned long long* incl = (unsigned long long*)A_.Alloc((size_t)nb * 8);
    unsigned long long* cur = (unsigned long long*)A_.Alloc((size_t)nb * 8);
    uint32_t* perm = (uint32_t*)A_.Alloc((size_t)F.P * 4);
    CK(cudaMemsetAsync(cnt, 0, (size_t)nb * 8, st_));
    k_hub_hist<<<Grid(F.P, 256), 256, 0, st_>>>(F, kv, g_.hub_slot, nb, cnt);
    CK(cudaMemcpyAsync(incl, cnt, (size_t)nb * 8, cudaMemcpyDeviceToDevice, st_));
    Scan(reinterpret_cast<uint64_t*>(incl), nb);
    k_hub_cursor<<<Grid(nb, 256), 256, 0, st_>>>(incl, cnt, nb, cur);
    k_hub_scatter<<<Grid(F.P, 256), 256, 0, st_>>>(F, kv, g_.hub_slot, nb, cur, perm);
    launches_ += 3;
    TimerStop(to, kPhaseOrganize);
    return perm;
  }

  // Window of k_compute_cta in dynamic shared memory (64 KiB: two CTAs of
  // 512 threads per SM), the attribute set once per device.
  template <int MODE>
  size_t CtaWindowBytes() {
    constexpr size_t kBytes = 64 << 10;
    // per device, once (server slots on several host threads may race here;
    // setting the attribute twice is harmless)
    static std::atomic<bool> set[64];
    const int d = ctx_.device;
    if (d >= 0 && d < 64 && !set[d].load(std::memory_order_acquire)) {
      CK(cudaFuncSetAttribute(k_compute_cta<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBytes));
      set[d].store(true, std::memory_order_release);
    }
    return kBytes;
  }

  template <int MODE, int MINB, int NLM>
  void LaunchWarp(bool ne, const DFront& F, const DStep& ds, const DGraph& G, const uint64_t* est, uint32_t b0,
                  uint64_t* ptr, uint32_t* cnt, uint32_t* data, uint64_t cap, unsigned long long* acc,
                  uint32_t* err) {
    if (ne)
      k_compute<MODE, MINB, NLM, MAXV><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(F, ds, G, est, b0, ptr, cnt, data,
                                                                             cap, acc, err, DHeavy{});
    else
      k_compute<MODE, MINB, NLM, 0><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(F, ds, G, est, b0, ptr, cnt, data, cap,
                                                                          acc, err, DHeavy{});
  }

  template <int MODE, int MINB, int NLM>
  void LaunchFlat(bool ne, const DFront& F, const DStep& ds, const DGraph& G, const uint64_t* est, uint32_t b0,
                  uint64_t* ptr, uint32_t* cnt, uint32_t* data, uint64_t cap, unsigned long long* acc,
                  uint32_t* err) {
    const unsigned grid = WarpGrid((F.P + 31) / 32);
    if (ne)
      k_compute_flat<MODE, MINB, NLM, MAXV><<<grid, WARP_BLOCK, 0, st_>>>(F, ds, G, est, b0, ptr, cnt, data, cap,
                                                                         acc, err);
    else
      k_compute_flat<MODE, MINB, NLM, 0><<<grid, WARP_BLOCK, 0, st_>>>(F, ds, G, est, b0, ptr, cnt, data, cap, acc,
                                                                      err);
  }

  // The root's list as a shared-memory bitmap (k_compute_rootmap), the
  // attribute for its dynamic shared memory set once per device.
  template <int MODE, int NEX>
  void LaunchRootMapAs(int ru, int other, const DFront& F, const DStep& ds, const DGraph& G, const uint64_t* est,
                       uint32_t b0, uint64_t* ptr, uint32_t* cnt, uint32_t* data, uint64_t cap,
                       unsigned long long* acc, uint32_t* err) {
    // per device, once (server slots on several host threads may race here;
    // setting the attribute twice is harmless)
    static std::atomic<bool> set[64];
    const int d = ctx_.device;
    if (d >= 0 && d < 64 && !set[d].load(std::memory_order_acquire)) {
      CK(cudaFuncSetAttribute(k_compute_rootmap<MODE, NEX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kRootMapMaxBytes));
      set[d].store(true, std::memory_order_release);
    }
    const uint32_t words = (uint32_t)((g_.n + 31) / 32);
    const size_t bytes = (size_t)words * 4;
    const size_t mark = A_.Mark();
    uint32_t* next = (uint32_t*)A_.Alloc(4);
    CK(cudaMemsetAsync(next, 0, 4, st_));
    // two CTAs of 1024 threads per SM while two bitmaps fit shared memory
    const uint64_t per_sm = bytes <= (112u << 10) ? 2 : 1;
    const unsigned grid =
        (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(sms_ * per_sm, (F.P + RM_CHUNK - 1) / RM_CHUNK));
    k_compute_rootmap<MODE, NEX><<<grid, RM_THREADS, bytes, st_>>>(F, ds, G, ru, other, est, b0, ptr, cnt, data,
                                                                    cap, acc, err, next, words);
    A_.Release(mark);
  }

  // Intersection launch: warp per path, specialised (granularity 0 auto, 3),
  // warp per path generic (1) or flattened over 32 paths per warp (2); in the
  // auto launches, a two-list step that reads the root's list takes
  // k_compute_rootmap (SME_ROOT_MAP=0 turns it off).
  template <int MODE>
  void Compute(const DFront& F, const DStep& ds, const DGraph& G, const uint64_t* est, uint32_t b0, uint64_t* ptr,
               uint32_t* cnt, uint32_t* data, uint64_t cap, const uint32_t* perm = nullptr) {
    unsigned long long* acc = acc_;
    uint32_t* err = (uint32_t*)(ctrl_ + 3);
    Timed t = TimerStart();
    const int gran = gran_;
    const int nlists = ds.nconn + (ds.reuse >= 0 ? 1 : 0);
    bool has_ne = false;
    for (int i = 0; i < ds.cond.n; ++i) has_ne |= ds.cond.op[i] == 2;
    const int ru = (*steps_)[0].u;
    int ri = -1;
    for (int i = 0; i < ds.nconn; ++i)
      if (ds.conn[i] == ru) ri = i;
    // the bitmap pays only where a root has many paths (its rebuild and the
    // CTA's barriers are per run of paths): three or more materialised
    // vertices (the 4-cycle's count step, not the diamond's or the
    // 4-clique's second level, measured 3.4x and 2.2x slower there)
    int nmat = 0;
    for (int v = 0; v < MAXV; ++v) nmat += F.inst[v] != nullptr;
    const bool rootmap = root_map_ && nmat >= 3 && !perm && ds.msrc < 0 && ds.reuse < 0 && ds.nconn == 2 && ri >= 0 &&
                         (gran == 0 || gran == 3) && (MODE != 1 || ds.with_u < 0) && !G.coff && g_.n > 0 &&
                         (g_.n + 31) / 32 * 4 <= kRootMapMaxBytes && F.inst[ru] && F.inst[ds.conn[1 - ri]];
    // two lists and nothing else (see k_pair_count); long runs of paths per
    // root keep the shared-memory bitmap
    const bool pair = MODE != 0 && !rootmap && !perm && ds.msrc < 0 && ds.reuse < 0 && ds.nconn == 2 &&
                      ds.cond.n == 0 && ds.with_u < 0 && gran == 0 && !G.coff;
    if (pair) {
      if constexpr (MODE != 0)
        k_pair_count<MODE><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(F, ds.conn[0], ds.conn[1], G,
                                                                          lists_simple_, ptr, cnt, acc);
    } else if (rootmap) {
      const int other = ds.conn[1 - ri];
      if (has_ne)
        LaunchRootMapAs<MODE, MAXV>(ru, other, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
      else
        LaunchRootMapAs<MODE, 0>(ru, other, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
    } else if (MODE == 1 && perm && ds.msrc < 0 && (gran == 0 || gran == 3) && nlists <= 3) {
      // count step, paths taken hub by hub (see k_hub_hist)
      if constexpr (MODE == 1) {
        DHeavy hv{};
        hv.perm = perm;
        if (nlists <= 2) {
          if (has_ne)
            k_compute<1, 8, 2, MAXV, false, false, true><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(
                F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, hv);
          else
            k_compute<1, 8, 2, 0, false, false, true><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(
                F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, hv);
        } else {
          if (has_ne)
            k_compute<1, 8, 3, MAXV, false, false, true><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(
                F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, hv);
          else
            k_compute<1, 8, 3, 0, false, false, true><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(
                F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, hv);
        }
      }
    } else if (ds.msrc >= 0) {
      // mapped reuse: the warp kernel that looks up the sibling's set
      if (has_ne)
        k_compute<MODE, 4, MAXV, MAXV, false, true><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(
            F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, DHeavy{});
      else
        k_compute<MODE, 4, MAXV, 0, false, true><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(
            F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, DHeavy{});
    } else if (gran == 4 && nlists == 2 && !has_ne) {
      // warp per path; paths with a long clipped pivot go to a CTA each
      const size_t mark = A_.Mark();
      const uint32_t qcap = (uint32_t)std::min<uint64_t>(F.P, 1u << 16);
      uint32_t* q = (uint32_t*)A_.Alloc(((size_t)qcap + 1) * 4);
      CK(cudaMemsetAsync(q, 0, 4, st_));
      k_compute<MODE, 8, 2, 0, true><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(
          F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, DHeavy{q, qcap, heavy_min_});
      Launched();
      const size_t win_bytes = CtaWindowBytes<MODE>();
      k_compute_cta<MODE><<<(unsigned)sms_ * 2, CTA_THREADS, win_bytes, st_>>>(
          F, ds, G, est, b0, ptr, cnt, data, cap, acc, err, q, qcap, (uint32_t)(win_bytes / 4));
      hot_ += 1;
      A_.Release(mark);
    } else if (gran == 0 || gran == 3 || gran == 4) {
      // warp per path, specialised on the number of intersected lists and
      // on the presence of `!=` conditions; fewer live values let more warps
      // reside, which is what counts: the searches are L2-latency bound.
      // Auto: eight blocks per SM for two or three lists, six otherwise
      // (measured fastest on every plan at R-MAT s20); 3: six throughout.
      const int nl = ds.nconn + (ds.reuse >= 0 ? 1 : 0);
      bool ne = false;
      for (int i = 0; i < ds.cond.n; ++i) ne |= ds.cond.op[i] == 2;
      const bool dense = gran != 3;
      if (nl <= 2)
        dense ? LaunchWarp<MODE, 8, 2>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err)
              : LaunchWarp<MODE, 6, 2>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
      else if (nl <= 3)
        dense ? LaunchWarp<MODE, 8, 3>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err)
              : LaunchWarp<MODE, 6, 3>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
      else
        LaunchWarp<MODE, 6, MAXV>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
    } else if (gran == 1) {
      k_compute<MODE><<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(F, ds, G, est, b0, ptr, cnt, data, cap, acc, err,
                                                             DHeavy{});
    } else {
      // flattened, specialised the same way
      const int nl = ds.nconn + (ds.reuse >= 0 ? 1 : 0);
      bool ne = false;
      for (int i = 0; i < ds.cond.n; ++i) ne |= ds.cond.op[i] == 2;
      if (nl <= 2)
        LaunchFlat<MODE, 8, 2>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
      else if (nl <= 3)
        LaunchFlat<MODE, 6, 3>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
      else
        LaunchFlat<MODE, 4, MAXV>(ne, F, ds, G, est, b0, ptr, cnt, data, cap, acc, err);
    }
    TimerStop(t, MODE == 0 ? kPhaseCompute : MODE == 1 ? kPhaseComputeCount : kPhasePathCount);
    Launched();
  }

 public:
  int gran_ = 0;
  uint32_t heavy_min_ = 2048;  // granularity 4: shortest pivot that gets a CTA
  bool group_by_hub_ = false;  // count steps take their paths hub by hub
  bool use_bitmaps_ = true;
  bool oriented_ = false;  // each edge once, towards the higher id
  bool root_map_ = true;  // two-list steps on the root's list: k_compute_rootmap

 private:

  uint64_t Budget(size_t k) const {
    size_t rem = (*steps_).size() - k + 1;
    return (uint64_t)((double)A_.Free() * 0.85 / (double)rem);
  }

  // Timing events come from the context's free list and go back to it.
  cudaEvent_t TakeEvent() {
    if (!ctx_.events.empty()) {
      cudaEvent_t e = ctx_.events.back();
      ctx_.events.pop_back();
      return e;
    }
    cudaEvent_t e = nullptr;
    CK(cudaEventCreate(&e));
    return e;
  }
  // Adds the finished regions to their phases (the stream has passed them).
  void HarvestTimers() {
    for (auto& e : events_) {
      float ms = 0;
      cudaEventElapsedTime(&ms, e.a, e.b);
      phase_[e.phase] += ms;
      ctx_.events.push_back(e.a);
      ctx_.events.push_back(e.b);
    }
    events_.clear();
  }

  Timed TimerStart() {
    Timed e;
    e.a = TakeEvent();
    e.b = TakeEvent();
    cudaEventRecord(e.a, st_);
    e.phase = 0;
    return e;
  }
  // Records the end of a timed region of `phase` (sme_stats.phase_ms index).
  void TimerStop(Timed e, int phase) {
    cudaEventRecord(e.b, st_);
    e.phase = phase;
    events_.push_back(e);
    if (phase == kPhaseCompute || phase == kPhaseComputeCount || phase == kPhasePathCount) ++hot_;
  }

  void Scan(uint64_t* d, uint32_t n) {
    if (n == 0) return;
    uint32_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    size_t m = A_.Mark();
    uint64_t* bs = (uint64_t*)A_.Alloc((size_t)nb * 8);
    k_scan_reduce<<<nb, SCAN_THREADS, 0, st_>>>(d, n, bs);
    k_scan_partials<<<1, 1024, 0, st_>>>(bs, nb);
    k_scan_apply<<<nb, SCAN_THREADS, 0, st_>>>(d, n, bs);
    launches_ += 3;
    A_.Release(m);
  }

  uint64_t ReadU64(const uint64_t* d) {
    CK(cudaMemcpyAsync(ctx_.h_pinned, d, 8, cudaMemcpyDeviceToHost, st_));
    CK(cudaStreamSynchronize(st_));
    return ctx_.h_pinned[0];
  }

  // Inclusive sums of a step's estimates over the paths into `est` (external
  // mode: of its list elements into `est2`), and their totals.
  struct Totals {
    uint64_t est, lists;
  };
  template <EstKind KIND, int ITEMS>
  void LaunchEstScan(const DFront& F, const DStep& ds, const DCond& dc, uint64_t* est, uint64_t* est2,
                     uint32_t* first, uint32_t nb, uint64_t* bs) {
    uint32_t* ticket = (uint32_t*)(ctrl_ + 7);
    if (est2)
      k_est_scan<E_LIST, true, ITEMS><<<nb, SCAN_THREADS, 0, st_>>>(F, ds, dc, g_.row_ptrs, est, est2, nullptr, bs,
                                                                    ticket);
    else
      k_est_scan<KIND, false, ITEMS><<<nb, SCAN_THREADS, 0, st_>>>(F, ds, dc, g_.row_ptrs, est, nullptr, first, bs,
                                                                  ticket);
    Launched();
    if (nb == 1) return;
    if (est2) k_scan_add<true, ITEMS><<<nb - 1, SCAN_THREADS, 0, st_>>>(est, est2, F.P, bs);
    else k_scan_add<false, ITEMS><<<nb - 1, SCAN_THREADS, 0, st_>>>(est, nullptr, F.P, bs);
    Launched();
  }
  // `read`: the totals are wanted (a host round trip; else zeros).
  template <EstKind KIND>
  Totals EstScan(const DFront& F, const DStep& ds, const DCond& dc, uint64_t* est, uint64_t* est2,
                 uint32_t* first = nullptr, bool read = true) {
    const uint32_t tile = F.P <= kScanSmall * (uint32_t)sms_ ? SCAN_THREADS : SCAN_TILE;
    const uint32_t nb = (F.P + tile - 1) / tile;
    const size_t m = A_.Mark();
    uint64_t* bs = (uint64_t*)A_.Alloc(((size_t)nb + 1) * 16);
    if (tile == SCAN_THREADS) LaunchEstScan<KIND, 1>(F, ds, dc, est, est2, first, nb, bs);
    else LaunchEstScan<KIND, SCAN_ITEMS>(F, ds, dc, est, est2, first, nb, bs);
    if (!read) {
      A_.Release(m);
      return Totals{0, 0};
    }
    CK(cudaMemcpyAsync(ctx_.h_pinned, bs + nb, 8, cudaMemcpyDeviceToHost, st_));
    if (est2) CK(cudaMemcpyAsync(ctx_.h_pinned + 1, bs + 2 * nb + 1, 8, cudaMemcpyDeviceToHost, st_));
    CK(cudaStreamSynchronize(st_));
    if (events_.size() >= kKeptEvents / 2) HarvestTimers();
    A_.Release(m);
    return Totals{ctx_.h_pinned[0], est2 ? ctx_.h_pinned[1] : 0};
  }

  // The batches of P paths: one when the whole cost fits the budget, else cut
  // on the device.
  std::vector<Batch> Batches(const uint64_t* incl, uint32_t P, double pf, double cf, uint64_t budget, Totals t,
                             const uint64_t* incl2 = nullptr, double cg = 0) {
    if (pf * P + cf * (double)t.est + cg * (double)t.lists <= (double)budget)
      return {Batch{0, P, 0, t.est, t.lists}};
    return Split(incl, P, pf, cf, budget, incl2, cg);
  }

  std::vector<Batch> Split(const uint64_t* incl, uint32_t P, double pf, double cf, uint64_t budget,
                           const uint64_t* incl2 = nullptr, double cg = 0) {
    std::vector<Batch> out;
    if (P == 0) return out;
    const uint32_t K = (uint32_t)std::min<size_t>(ctx_.pinned_words / 3, (64 << 10) / 24);
    size_t m = A_.Mark();
    uint64_t* d = (uint64_t*)A_.Alloc((size_t)K * 24);
    uint32_t start = 0;
    uint64_t e_start = 0, l_start = 0;
    while (start < P) {
      k_split<<<(K + 255) / 256, 256, 0, st_>>>(incl, incl2, P, start, pf, cf, cg, (double)budget, K, d);
      Launched();
      CK(cudaMemcpyAsync(ctx_.h_pinned, d, (size_t)K * 24, cudaMemcpyDeviceToHost, st_));
      CK(cudaStreamSynchronize(st_));
      const uint64_t* h = ctx_.h_pinned;
      for (uint32_t k = 0; k < K && start < P; ++k) {
        uint32_t end = (uint32_t)std::min<uint64_t>(h[3 * k], P);
        if (end <= start) continue;
        out.push_back(Batch{start, end, e_start, h[3 * k + 1], h[3 * k + 2] - l_start});
        start = end;
        e_start = h[3 * k + 1];
        l_start = h[3 * k + 2];
      }
    }
    A_.Release(m);
    return out;
  }

  static DFront Slice(const DFront& F, uint32_t b0, uint32_t b1) {
    DFront G = F;
    G.P = b1 - b0;
    for (int v = 0; v < MAXV; ++v) {
      if (F.inst[v]) G.inst[v] = F.inst[v] + b0;
      if (F.cidx[v]) G.cidx[v] = F.cidx[v] + b0;
      else G.ident_off[v] = F.ident_off[v] + b0;
    }
    return G;
  }

  void Emit(const DFront& F) {
    EmitCols cols{};
    for (int v = 0; v < prog_.n; ++v) cols.p[prog_.out_slot[v]] = F.inst[v];
    if (emitted_ < cap_) {
      k_emit<<<Grid((uint64_t)F.P * prog_.n, 256), 256, 0, st_>>>(cols, F.P, (uint32_t)prog_.n, emitted_, out_, cap_);
      Launched();
    }
    emitted_ += F.P;
  }

  void ClipViews(const DFront& F, const DStep& ds, const DGraph& G, uint64_t* ptr, uint32_t* cnt) {
    Timed t = TimerStart();
    k_view<<<Grid(F.P, WARP_BLOCK), WARP_BLOCK, 0, st_>>>(F, ds, G, ptr, cnt, acc_);
    TimerStop(t, kPhaseCompute);
    Launched();
  }

  static bool HasNe(const DCond& c) {
    for (int i = 0; i < c.n; ++i)
      if (c.op[i] == 2) return true;
    return false;
  }
  // Where each path's children start in its set: needed when conditions clip
  // the set and none excludes single values.
  uint32_t* FirstOf(const DCond& dc, uint32_t P) {
    return dc.n && !HasNe(dc) ? (uint32_t*)A_.Alloc((size_t)P * 4) : nullptr;
  }

  // Expands the paths of F into their C children (`cnt`: inclusive child
  // counts, `first`: see FirstOf) and runs the next level on them.
  void Materialize(size_t k, const DFront& F, const DCond& dc, const uint64_t* cnt, const uint32_t* first,
                   uint64_t C) {
    if (C == 0) return;
    if (C > 0x7fffffffULL) Fail(SME_ERR_OOM, "materialised batch exceeds 2^31 partial instances");
    const Step& s = (*steps_)[k];
    uint32_t* err = (uint32_t*)(ctrl_ + 3);
    DMatOut o{};
    o.u = s.u;
    o.keep = s.keep_set;
    o.nmat = (uint8_t)s.mat_after.size();
    for (size_t i = 0; i < s.mat_after.size(); ++i) {
      o.mat[i] = s.mat_after[i];
      o.inst[s.mat_after[i]] = (uint32_t*)A_.Alloc(C * 4);
    }
    o.nsets = (uint8_t)s.sets_after.size();
    for (size_t i = 0; i < s.sets_after.size(); ++i) {
      o.sets[i] = s.sets_after[i];
      o.cidx[s.sets_after[i]] = (uint32_t*)A_.Alloc(C * 4);
    }
    Timed tm = TimerStart();
    if (!HasNe(dc)) {
      const uint32_t rows = C <= (uint64_t)sms_ * 64 * 32 ? 32 : kMatRows;
      k_mat_rows<<<WarpGrid((C + rows - 1) / rows), WARP_BLOCK, 0, st_>>>(F, o, cnt, first, C, rows);
      Launched();
    } else {
      k_mat_write<<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(F, dc, o, cnt, C, kMatBig, err);
      Launched();
      if (C > kMatBig) {  // else no parent has more
        k_mat_write_big<<<WarpGrid((C + kMatChunk - 1) / kMatChunk), WARP_BLOCK, 0, st_>>>(F, dc, o, cnt, C, kMatBig,
                                                                                           err);
        Launched();
      }
    }
    TimerStop(tm, kPhaseMaterialize);
    DFront Fn{};
    Fn.P = (uint32_t)C;
    for (int v = 0; v < MAXV; ++v) Fn.inst[v] = o.inst[v];
    for (uint8_t w : s.sets_after) {
      Fn.set[w] = F.set[w];
      Fn.nset[w] = F.nset[w];
      Fn.cidx[w] = o.cidx[w];
    }
    Level(k + 1, Fn);
  }

  void Level(size_t k, const DFront& F) {
    if (F.P == 0) return;
    if (k == (*steps_).size()) {
      if (prog_.enumerate) Emit(F);
      return;
    }
    const Step& s = (*steps_)[k];
    DStep ds = ToDStep(s);
    ds.noview = ext_cols_ != nullptr;
    unsigned long long* acc = ctrl_;
    uint32_t* err = (uint32_t*)(ctrl_ + 3);
    switch (s.kind) {
      case S_COMPUTE_COUNT: {
        paths_ += F.P;
        if (steps_ == &prog_.minus) minus_paths_ += F.P;
        if (!ext_cols_) {
          const size_t mg = A_.Mark();
          const uint32_t* perm = GroupByHub(F, ds);
          Compute<1>(F, ds, Resident(), nullptr, 0, nullptr, nullptr, nullptr, 0, perm);
          A_.Release(mg);
          return;
        }
        // external: the whole frontier when its lists fit the cache (they are
        // shared by most of its paths, so this is tried before anything is
        // estimated, while it keeps working), else batches whose lists do
        if (ext_misses_ < 4) {
          if (LoadLists(F, ds, ~0ull >> 1)) {
            ++batches_;
            Compute<1>(F, ds, View(), nullptr, 0, nullptr, nullptr, nullptr, 0);
            return;
          }
          ++ext_misses_;
        }
        const size_t m0 = A_.Mark();
        uint64_t* est = (uint64_t*)A_.Alloc((size_t)F.P * 8);
        uint64_t* sd = (uint64_t*)A_.Alloc((size_t)F.P * 8);
        const Totals tot = EstScan<E_LIST>(F, ds, DCond{}, est, sd);
        // a count takes no memory beyond these two: only its lists are bounded
        const uint64_t bk = std::max<uint64_t>(Budget(k), 1 << 20);
        const std::vector<Batch> bs =
            Batches(sd, F.P, 12.0, 0.0, bk, Totals{tot.lists, tot.lists}, sd, ExtListCost(k, bk));
        std::vector<Batch> todo(bs.rbegin(), bs.rend());
        while (!todo.empty()) {
          const Batch b = todo.back();
          todo.pop_back();
          DFront Fb = Slice(F, b.b0, b.b1);
          if (!LoadLists(Fb, ds, b.lists)) {
            Halve(b, sd, sd, todo);
            continue;
          }
          ++batches_;
          Compute<1>(Fb, ds, View(), nullptr, 0, nullptr, nullptr, nullptr, 0);
        }
        A_.Release(m0);
        return;
      }
      case S_ALIAS: {
        DFront Fn = F;
        const int a = s.alias_of;
        Fn.set[s.u] = F.set[a];
        Fn.cidx[s.u] = F.cidx[a];
        Fn.ident_off[s.u] = F.ident_off[a];
        Fn.nset[s.u] = F.nset[a];
        Level(k + 1, Fn);
        return;
      }
      case S_COUNT: {
        Timed tc = TimerStart();
        if (s.direct) {
          uint8_t us[3] = {0, 0, 0};
          for (size_t i = 0; i < s.unmat.size() && i < 3; ++i) us[i] = s.unmat[i];
          k_count_direct<<<Grid(F.P, 256), 256, 0, st_>>>(F, (uint8_t)s.unmat.size(), us[0], us[1], us[2],
                                                          prog_.query_type, acc);
        } else if (s.unmat.size() == 1) {
          k_count1<<<Grid(F.P, 256), 256, 0, st_>>>(F, s.unmat[0], acc);
        } else {
          k_count2<<<WarpGrid(F.P), WARP_BLOCK, 0, st_>>>(F, s.unmat[0], s.unmat[1], s.pair_op, acc);
        }
        TimerStop(tc, kPhaseCount);
        Launched();
        return;
      }
      default:
        break;
    }
    const size_t mark0 = A_.Mark();
    const DCond dc = ToDCond(s.cond);
    const bool has_ne = HasNe(dc);
    uint64_t* est = nullptr;
    uint64_t* sumdeg = nullptr;  // external mode: list elements per path
    std::vector<Batch> batches;
    // a step over one list without `!=` writes views, a path count nothing but
    // counts: when one batch holds them there is nothing to estimate
    const bool view = s.kind == S_COMPUTE && !ext_cols_ && ds.msrc < 0 && ds.nconn + (ds.reuse >= 0 ? 1 : 0) == 1 &&
                      !has_ne && (gran_ == 0 || gran_ == 2);
    const double fixed = 12 + 16;  // estimate, pointer and count per path
    if ((view || (s.kind == S_PATH_COUNT && !ext_cols_)) && fixed * F.P <= (double)Budget(k)) {
      batches.push_back(Batch{0, F.P, 0, 0, 0});
    } else if (s.kind == S_MATERIALIZE) {
      // one batch when all children fit, counted exactly; else batches by the
      // set sizes, an upper bound, each counted in its turn.  A step that
      // misses three times as often as it fits tries one frontier in eight:
      // under a small budget its frontiers would all be counted twice (R-MAT
      // s14, diamonds under 4 MiB by the reuse plan: 6.5 ms without tries, 7.6
      // with one per frontier, 6.7 so; 5-cliques under 8 MiB by GPSM, which fit:
      // 35, 22 and 22 ms; 4-cliques of R-MAT s16, external, 13 MiB: 189 ms with
      // one per frontier, 205 where three misses end the tries, 183 so).
      const double pf = 16, cf = 4.0 * (s.mat_after.size() + s.sets_after.size()) + 16;
      if (mat_misses_[k] < 3 || ++mat_skips_[k] % 8 == 0) {
        Timed to = TimerStart();
        uint64_t* cnt = (uint64_t*)A_.Alloc((size_t)F.P * 8);
        uint32_t* first = FirstOf(dc, F.P);
        const Totals t = EstScan<E_CHILD>(F, ds, dc, cnt, nullptr, first);
        TimerStop(to, kPhaseOrganize);
        if (pf * F.P + cf * (double)t.est <= (double)Budget(k) && t.est <= 2000000000ull) {
          ++batches_;
          mat_misses_[k] = std::max(mat_misses_[k] - 3, -8);
          Materialize(k, F, dc, cnt, first, t.est);
          A_.Release(mark0);
          return;
        }
        mat_misses_[k] = std::min(mat_misses_[k] + 1, 3);
        A_.Release(mark0);
      }
      est = (uint64_t*)A_.Alloc((size_t)F.P * 8);
      Timed to = TimerStart();
      EstScan<E_SET>(F, ds, dc, est, nullptr, nullptr, false);
      TimerStop(to, kPhaseOrganize);
      // child counts of a batch stay within 31-bit path indices
      const uint64_t bk = std::min<uint64_t>(Budget(k), (uint64_t)(cf * 2.0e9));
      batches = Split(est, F.P, pf, cf, AtLeast(k, bk));
    } else {  // COMPUTE, PATH_COUNT, FILTER
      Timed to = TimerStart();
      est = (uint64_t*)A_.Alloc((size_t)F.P * 8);
      if (ext_cols_ && s.kind != S_FILTER) sumdeg = (uint64_t*)A_.Alloc((size_t)F.P * 8);
      const Totals t = s.kind == S_FILTER ? EstScan<E_SET>(F, ds, dc, est, nullptr)
                                          : EstScan<E_LIST>(F, ds, dc, est, sumdeg);
      TimerStop(to, kPhaseOrganize);
      const double cf = s.kind == S_PATH_COUNT ? 0 : 4;
      const uint64_t bk = std::min<uint64_t>(Budget(k), (uint64_t)(std::max(cf, 1.0) * 2.0e9));
      batches = Batches(est, F.P, fixed, cf, AtLeast(k, bk), t, sumdeg, ExtListCost(k, bk));
    }
    std::reverse(batches.begin(), batches.end());
    while (!batches.empty()) {
      const Batch b = batches.back();
      batches.pop_back();
      const size_t mark = A_.Mark();
      DFront Fb = Slice(F, b.b0, b.b1);
      const uint32_t Pb = b.b1 - b.b0;
      if (sumdeg && !LoadLists(Fb, ds, b.lists)) {
        Halve(b, est, sumdeg, batches);
        continue;
      }
      ++batches_;
      switch (s.kind) {
        case S_COMPUTE:
        case S_PATH_COUNT: {
          paths_ += Pb;
          uint64_t* ptr = (uint64_t*)A_.Alloc((size_t)Pb * 8);
          uint32_t* cnt = (uint32_t*)A_.Alloc((size_t)Pb * 4);
          uint64_t cap = s.kind == S_COMPUTE && !view ? b.e1 - b.e0 : 0;
          uint32_t* data = cap ? (uint32_t*)A_.Alloc(cap * 4) : nullptr;
          const DGraph gv = View();
          if (view)
            ClipViews(Fb, ds, gv, ptr, cnt);
          else if (s.kind == S_COMPUTE)
            Compute<0>(Fb, ds, gv, est, b.b0, ptr, cnt, data, cap);
          else
            Compute<2>(Fb, ds, gv, est, b.b0, ptr, cnt, nullptr, 0);
          DFront Fn = Fb;
          Fn.set[s.u] = DSet{ptr, cnt};
          Fn.nset[s.u] = Pb;
          Fn.cidx[s.u] = nullptr;
          Fn.ident_off[s.u] = 0;
          Level(k + 1, Fn);
          break;
        }
        case S_FILTER: {
          uint64_t* ptr = (uint64_t*)A_.Alloc((size_t)Pb * 8);
          uint32_t* cnt = (uint32_t*)A_.Alloc((size_t)Pb * 4);
          uint64_t cap = b.e1 - b.e0;
          uint32_t* data = cap ? (uint32_t*)A_.Alloc(cap * 4) : nullptr;
          Timed tf = TimerStart();
          k_filter<<<WarpGrid(Pb), WARP_BLOCK, 0, st_>>>(Fb, s.u, ToDCond(s.cond), est, b.b0, ptr, cnt, data,
                                                         cap, err);
          TimerStop(tf, kPhaseFilter);
          Launched();
          DFront Fn = Fb;
          Fn.set[s.u] = DSet{ptr, cnt};
          Fn.nset[s.u] = Pb;
          Fn.cidx[s.u] = nullptr;
          Fn.ident_off[s.u] = 0;
          Level(k + 1, Fn);
          break;
        }
        case S_MATERIALIZE: {
          uint64_t* cnt = (uint64_t*)A_.Alloc((size_t)Pb * 8);
          Timed tm = TimerStart();
          uint32_t* first = FirstOf(dc, Pb);
          const uint64_t C = EstScan<E_CHILD>(Fb, ds, dc, cnt, nullptr, first).est;
          TimerStop(tm, kPhaseMaterialize);
          Materialize(k, Fb, dc, cnt, first, C);
          break;
        }
        default:
          Fail(SME_ERR_INVALID_ARG, "unexpected step kind");
      }
      A_.Release(mark);
    }
    A_.Release(mark0);
  }
};

}  // namespace

RunResult RunProgram(const Program& prog, const DeviceGraph& g, DeviceContext& ctx, const RootTask& task,
                     uint32_t* d_out, uint64_t cap, int tuning) {
  CK(cudaSetDevice(ctx.device));
  RootTask t = task;
  if (!t.list) {
    if (t.end > g.n) t.end = g.n;
    if (t.begin > t.end) t.begin = t.end;
  }
  Executor ex(prog, g, ctx, d_out, cap);
  ex.gran_ = tuning & 0xff;
  ex.use_bitmaps_ = !(tuning & 0x100);
  ex.oriented_ = (tuning & 0x200) != 0;
  if (const char* e = std::getenv("SME_HEAVY_PIVOT")) ex.heavy_min_ = (uint32_t)std::max(32L, std::atol(e));
  if (const char* e = std::getenv("SME_GROUP_BY_HUB")) ex.group_by_hub_ = std::atoi(e) != 0;
  if (const char* e = std::getenv("SME_ROOT_MAP")) ex.root_map_ = std::atoi(e) != 0;
  return ex.Run(t);
}

// EXTERNAL_GPU: the graph stays in host memory.
//   EXT_CACHE  global row pointers on the device; for every intersection
//              batch, the required adjacency lists are gathered by the GPU
//              from pinned, mapped host memory into a device subgraph
//              (EXTLIGHTGPUProcessor::PrepareBatch/LoadSubgraph,
//              src/gpu/impl/light/ext/EXTLIGHTGPUProcessor.cuh:20-90).
//   EXT_UMA    the adjacency lists live in managed memory and migrate on
//              demand (EXTUMALIGHTGPUComp, src/gpu/impl/light/ext/uma/).
RunResult RunProgramExternal(const Program& prog, const HostGraph& hg, DeviceContext& ctx, const RootTask& task,
                             int ext_variant, uint64_t graph_budget_bytes) {
  (void)graph_budget_bytes;
  CK(cudaSetDevice(ctx.device));
  RootTask t = task;
  if (!t.list) {
    if (t.end > hg.n) t.end = hg.n;
    if (t.begin > t.end) t.begin = t.end;
  }
  DeviceGraph dg;
  dg.device = ctx.device;
  dg.n = hg.n;
  dg.m = hg.m;
  uint64_t h2d = (hg.n + 1) * sizeof(uintE);
  CK(cudaMalloc((void**)&dg.row_ptrs, (hg.n + 1) * sizeof(uintE)));
  RunResult r;
  bool registered = false;
  uint32_t* managed = nullptr;
  try {
    CK(cudaMemcpyAsync(dg.row_ptrs, hg.row_ptrs, (hg.n + 1) * sizeof(uintE), cudaMemcpyHostToDevice, ctx.stream));
    if (ext_variant == SME_EXT_UMA) {
      CK(cudaMallocManaged((void**)&managed, std::max<uint64_t>(hg.m, 1) * sizeof(uintV)));
      if (hg.m) std::memcpy(managed, hg.cols, hg.m * sizeof(uintV));
      dg.cols = managed;
      Executor ex(prog, dg, ctx, nullptr, 0);
      r = ex.Run(t);
      h2d += hg.m * sizeof(uintV);
    } else {
      const uint32_t* dcols = nullptr;
      if (hg.m) {
        cudaError_t e = cudaHostRegister(hg.cols, hg.m * sizeof(uintV), cudaHostRegisterMapped | cudaHostRegisterReadOnly);
        if (e == cudaSuccess) {
          registered = true;
        } else if (e == cudaErrorHostMemoryAlreadyRegistered) {
          cudaGetLastError();
        } else {
          Fail(SME_ERR_CUDA, std::string("cudaHostRegister: ") + cudaGetErrorString(e));
        }
        CK(cudaHostGetDevicePointer((void**)&dcols, hg.cols, 0));
      }
      Executor ex(prog, dg, ctx, nullptr, 0);
      ex.SetExternal(dcols);
      r = ex.Run(t);
      h2d += ex.ext_h2d_bytes();
    }
  } catch (...) {
    cudaStreamSynchronize(ctx.stream);
    if (registered) cudaHostUnregister(hg.cols);
    if (managed) cudaFree(managed);
    cudaFree(dg.row_ptrs);
    throw;
  }
  if (registered) cudaHostUnregister(hg.cols);
  if (managed) cudaFree(managed);
  cudaFree(dg.row_ptrs);
  r.stats.h2d_bytes += h2d;
  return r;
}

}  // namespace sme

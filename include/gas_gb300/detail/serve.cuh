// Round-at-a-time kernels of the serving loop.
//
// A served batch (Q queries of one program on one resident graph) advances
// by ordinary launches, one or two per round, on the stream of its lane.
// No kernel here waits on another block, so batches on different lanes --
// different graphs, programs and sizes -- share the SMs freely and overlap;
// nothing depends on co-residency (unlike the persistent kernels, whose
// grid barriers need every block resident).
//
// BFS / SSSP reuse the batched units of batch.cuh (the (vertex, query) pair
// frontier and SSSP distance buckets included): round r is
//   batch_round_kernel(r)  bounds, resets, pair / push / pull pass, count
//   batch_tail_kernel(r)   end test (sets done, rounds) or compaction
// and both return at once when the batch is done, so the host may queue
// rounds ahead of the end test.
//
// Personalised PageRank (PPR, alpha 0.15, teleport to the source) runs
// every query of a batch in lock step, pulling over in-edges:
//   rank'[v][q] = tele(v,q) + (1-alpha) * (sum over in-edges u->v, in CSC
//                 order, of rank[u][q] / outdeg(u))      for active v
//   rank'[v][q] = rank[v][q]                              otherwise
// with the engine's active sets A0 = every vertex, A(k+1) = out-neighbours
// of A(k) (apply always returns true).  Sums use correctly rounded float
// operations without contraction; for vertices of in-degree <= kPprChunk
// each is the left fold from 0 in CSC order, so those ranks equal a
// single-source run of the reference engine's CPU loop (refgas.h:140-166
// with the program of pagerank.cu:27-73 and a teleport term) bit for bit.
// Every sum depends on the graph alone: a query's ranks are the same in
// every batch and mix.
#pragma once

#include "batch.cuh"

namespace gas {
namespace detail {

// ---------------------------------------------------------------- BFS/SSSP

template <int W, int KIND>
__global__ void __launch_bounds__(256) batch_round_kernel(const BatchArgs a, int r,
                                                          const unsigned *done) {
  if (ld_acquire(done)) return;
  __shared__ int32_t sBound[32 * W];
  __shared__ unsigned sNear[W];
  __shared__ PairSmem sPairs;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  const long long gw = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  // list entries are dealt to warps block-first (warp k of every block, then
  // warp k+1), so a short list spreads over every SM
  const long long gwl = (long long)(threadIdx.x / 32) * gridDim.x + blockIdx.x;
  const size_t maskWords = (size_t)a.nVertices * W;
  const int rc = r % 3, rn = (r + 1) % 3;
  const bool buckets = KIND == kBatchSSSP && a.delta > 0;
  const BatchBucket bk{buckets ? sBound : nullptr, buckets ? sNear : nullptr};
  if (buckets) {  // this round's bounds (as in batch_run_kernel)
    const int32_t *tPrev = (r & 1) ? a.thresh[1] : a.thresh[0];
    int32_t *tNext = (r & 1) ? a.thresh[0] : a.thresh[1];
    const unsigned *nPrev = a.nearFlag[(r + 2) % 3];
    for (int q = threadIdx.x; q < 32 * W; q += blockDim.x) {
      int32_t t = __ldcg(tPrev + q);
      if (r > 0 && !((__ldcg(nPrev + q / 32) >> (q % 32)) & 1u)) t += a.delta;
      sBound[q] = t;
      if (blockIdx.x == 0) tNext[q] = t;
    }
    if (threadIdx.x < W) sNear[threadIdx.x] = 0u;
    if (blockIdx.x == 0 && threadIdx.x < W) a.nearFlag[rn][threadIdx.x] = 0u;
    __syncthreads();
  }
  unsigned *cur = a.mask[rc];
  unsigned *nxt = a.mask[rn];
  unsigned *clr = a.mask[(r + 2) % 3];
  const unsigned long long lc = a.listCnt[rc];
  const long long nList = (long long)(lc >> 32);
  const long long eOut = (long long)(lc & 0xffffffffull);
  const bool push = a.pairMode || buckets || eOut * a.alpha <= (long long)a.nEdges;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.cnt[rn] = 0ull;
    a.listCnt[(r + 2) % 3] = 0ull;
  }
  if (!a.pairMode)  // pair rounds from the mask clear the words they read
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < maskWords;
         i += (size_t)gridDim.x * blockDim.x)
      clr[i] = 0u;
  unsigned long long changed = 0ull;
  if (a.pairMode) {
    if (KIND == kBatchSSSP || a.pairMode == kPairsMask)
      batch_pairs_round<W, KIND>(a, r, cur, nxt, sPairs, changed, bk);
    else
      batch_pair_list<W>(a, r, nList, a.listCnt + rn, changed);
  } else if (push) {
    for (long long i = gwl; i < nList; i += warps)
      batch_push_unit<W, KIND>(a, a.list[rc][i], a.listC[rc][i], r, cur, nxt, a.list[rn],
                               a.listC[rn], a.listCnt + rn, changed, bk);
  } else {
    batch_pull_round<W, KIND>(a, gw, warps, r, cur, nxt, changed);
  }
  changed = warp_sum_u64(changed);
  if ((threadIdx.x & 31) == 0 && changed) atomicAdd(a.cnt + rc, changed);
  if (buckets) {
    __syncthreads();
    if (threadIdx.x < W && sNear[threadIdx.x]) atomicOr(a.nearFlag[rc] + threadIdx.x, sNear[threadIdx.x]);
  }
}

// End of round r: no change -> done (rounds = r, as the persistent kernel
// reports); a pull round -> list its changed vertices for round r + 1.
template <int W>
__global__ void __launch_bounds__(256) batch_tail_kernel(const BatchArgs a, int r,
                                                         unsigned *done) {
  if (ld_acquire(done)) return;
  if (a.cnt[r % 3] == 0ull) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      *a.roundsOut = r;
      st_release(done, 1u);
    }
    return;
  }
  const unsigned long long lc = a.listCnt[r % 3];
  const bool push = a.pairMode || a.delta > 0 ||
                    (long long)(lc & 0xffffffffull) * a.alpha <= (long long)a.nEdges;
  if (push) return;
  const int rn = (r + 1) % 3;
  batch_compact<W>(a, a.mask[rn], a.list[rn], a.listC[rn], a.listCnt + rn);
}

// ---------------------------------------------------------------- PPR

// A vertex's in-edges form one work unit, or -- above kPprChunk edges --
// several units of kPprChunk edges whose partial sums the last unit to
// finish adds in chunk order.  Each (vertex, query) value is therefore a
// left fold in CSC order (bit for bit the reference loop's FP32 sum) for
// every vertex of in-degree <= kPprChunk, and a fixed-order sum of left-
// folded chunks above it: either way a function of the graph alone, the
// same in every batch.
constexpr int kPprChunk = 4096;

struct PprArgs {
  int32_t nVertices;
  int32_t nQueries;           // queries in the batch (<= row)
  int32_t row;                // floats of a vertex row (ppr_row_width)
  const int32_t *inSources;   // CSC
  const int32_t *outDegree;   // [V]
  int32_t nUnits;             // work units: hub chunks, then longest first
  int32_t nLong;              // of them hub chunks or longer than kPprLong
  const int4 *unit;           // {vertex, CSC begin, edges | last active round << 16,
                              //  partial-sum slot of a hub chunk or -1}
  const int32_t *slotFirst;   // [slots] first slot of the slot's vertex
  const int32_t *slotCount;   // [slots] chunks of that vertex
  const int32_t *slotHub;     // [slots] hub index (arrival counter)
  float *partial;             // [slots][row] (per batch)
  unsigned *arrive;           // [hubs][ppr_slices(row)] arrivals, never reset within a batch
  const int32_t *sources;     // [nQueries], readable to a multiple of 4
  float *rank[2];             // [V][row]
  float *contrib[2];          // [V][row] rank / outdeg (0 where outdeg is 0)
  float damp;                 // 1 - alpha, as the program computes it in float
  float teleport;             // alpha
};

// Row width of a batch of n queries: a power of two up to 32 (a lane per
// query), then whole 32-byte sectors (100 queries: 104 floats and not 128).
inline int ppr_row_width(int n) {
  if (n > 32) return (n + 7) / 8 * 8;
  int w = 1;
  while (w < n) w *= 2;
  return w;
}
// The kernels' template argument for a row: its power of two.
inline int ppr_row_class(int row) {
  int c = 1;
  while (c < row) c *= 2;
  return c;
}
// Slices of 32 queries that a row's hub chunks are summed in.
__host__ __device__ inline int ppr_slices(int row) { return (row + 31) / 32; }

// Units longer than this go through the ring, a slice of 32 queries at a time
// (ppr_long_units).  Short chains count while a round's rows are few (R-MAT-16,
// 100 queries: 4.4 ms with 256, 4.9 with 1024, 6.6 with hub chunks only);
// once they take longer than the chains, whole rows read by 16-byte words
// move more (R-MAT-19, 100 queries: 24.4, 20.5 and 22.2 ms).
constexpr int kPprLong[2] = {256, 1024};
constexpr long long kPprFewBytes = 1500000000ll;  // gathered a round

// The graph part of PprArgs, from a graph's PPR arrays (the block `mem`
// holds unit records (4 words each) | slotFirst | slotCount | slotHub,
// `units` and `slots` entries long).
inline void ppr_args_graph(PprArgs &a, const int32_t *inSources, const int32_t *outDegree,
                           const int32_t *mem, int32_t units, const int32_t (&nLong)[2], int32_t slots,
                           long long nEdges, int row) {
  const size_t nu = (size_t)(units > 0 ? units : 1), ns = (size_t)(slots > 0 ? slots : 1);
  a.inSources = inSources;
  a.outDegree = outDegree;
  a.nUnits = units;
  a.row = row;
  a.nLong = nLong[4 * nEdges * row < kPprFewBytes ? 0 : 1];
  a.unit = reinterpret_cast<const int4 *>(mem);
  a.slotFirst = mem + 4 * nu;
  a.slotCount = a.slotFirst + ns;
  a.slotHub = a.slotCount + ns;
}

// Completes the unit records: the last round in which each vertex is active.
static __global__ void ppr_unit_active_kernel(int4 *unit, int32_t nUnits, const uint8_t *lastActive) {
  for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < nUnits; u += gridDim.x * blockDim.x)
    unit[u].z |= (int)lastActive[unit[u].x] << 16;
}

__device__ __forceinline__ float ppr_contrib(float rank, int deg) {
  return deg > 0 ? __fdiv_rn(rank, (float)deg) : 0.0f;
}

// The engine's active sets do not depend on the source: A0 = every vertex,
// A(k+1) = out-neighbours of A(k).  v is in A(k) iff a walk of length k
// ends at v, so membership only shrinks with k: lastActive[v] = the largest
// such k (capped).  One pull step per launch: nxt = out-neighbours of cur.
static __global__ void ppr_active_step_kernel(int32_t nVertices, const int32_t *inOffsets,
                                              const int32_t *inSources, const uint8_t *cur,
                                              uint8_t *nxt, uint8_t *lastActive, int k) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long v = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
       v < nVertices; v += warps) {
    const int beg = inOffsets[v], end = inOffsets[v + 1];
    bool any = false;
    for (int e = beg + lane; e < end && !any; e += 32) any = cur[inSources[e]] != 0;
    any = __any_sync(kFullMask, any);
    if (lane == 0) {
      nxt[v] = any;
      if (any) lastActive[v] = (uint8_t)k;
    }
  }
}

// rank := 1 at each query's source, 0 elsewhere (pagerank-style init of a
// personalised run).
static __global__ void ppr_init_kernel(const PprArgs a) {
  const size_t n = (size_t)a.nVertices * a.row;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    a.rank[0][i] = 0.0f;
    a.contrib[0][i] = 0.0f;
  }
}

static __global__ void ppr_sources_kernel(const PprArgs a) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= a.nQueries) return;
  const int s = a.sources[q];
  a.rank[0][(size_t)s * a.row + q] = 1.0f;
  a.contrib[0][(size_t)s * a.row + q] = ppr_contrib(1.0f, a.outDegree[s]);
}

// This round's buffers (selects, not indexes, keep the parameters out of
// local memory).
struct PprRound {
  const float *rk, *ct;
  float *rk2, *ct2;
  int r;
};
__device__ __forceinline__ PprRound ppr_buffers(const PprArgs &a, int r) {
  const bool odd = (r & 1) != 0;
  return {odd ? a.rank[1] : a.rank[0], odd ? a.contrib[1] : a.contrib[0], odd ? a.rank[0] : a.rank[1],
          odd ? a.contrib[0] : a.contrib[1], r};
}

// Element idx (vertex v, query q) of the next rank and contribution.
__device__ __forceinline__ void ppr_finish(const PprArgs &a, const PprRound &b, int v, int q, size_t idx, bool act,
                                           float acc, int odeg) {
  if (act) {
    const float tele = (q < a.nQueries && a.sources[q] == v) ? a.teleport : 0.0f;
    const float nr = __fadd_rn(tele, __fmul_rn(a.damp, acc));
    b.rk2[idx] = nr;
    b.ct2[idx] = ppr_contrib(nr, odeg);
  } else {
    b.rk2[idx] = __ldcg(b.rk + idx);
    b.ct2[idx] = __ldcg(b.ct + idx);
  }
}

// The left fold, in CSC order, of up to 32 neighbouring queries over the `len`
// edges src[0..len) of a unit by one warp, lane q holding query q: the rows'
// slices (C 16-byte words from `col` on, rows `row` floats apart) come through
// a ring in shared memory, stages of 64 words with cp.async, and are added
// from there.  A long unit's time is its chain; loads into registers leave one
// batch of 16 or 32 rows in flight at a time and wait for all of it (two or
// three L2 round trips of about 0.6 us for 32 edges, so that one 4,096-edge
// chunk bounded every round of graphs up to R-MAT-18), the ring kPprStages
// batches that arrive one by one.
constexpr int kPprStages = 5;
constexpr int kPprStageWords = 64;
struct PprRing {
  float4 word[kPprStages][kPprStageWords];
};
__device__ __forceinline__ float ppr_fold_ring(const int32_t *src, const float *col, size_t row, int C, int len,
                                               PprRing &ring, int lane) {
  const int SE = C > 4 ? 8 : C > 2 ? 16 : 32;  // edges of a stage: SE * C <= 64 words
  const int e0 = lane / C, c0 = lane % C, e1 = (lane + 32) / C, c1 = (lane + 32) % C;
  int blk = lane < len ? __ldg(src + lane) : 0;  // ids of the 32 edges being asked for
  int next = 32 + lane < len ? __ldg(src + 32 + lane) : 0;
  auto ask = [&](int t) {  // stage t
    const int at = t * SE;
    if (t > 0 && (at & 31) == 0) {  // the next 32 ids (warp-uniform)
      blk = next;
      next = at + 32 + lane < len ? __ldg(src + at + 32 + lane) : 0;
    }
    float4 *to = ring.word[t % kPprStages];
    const int s0 = __shfl_sync(kFullMask, blk, (at + e0) & 31), s1 = __shfl_sync(kFullMask, blk, (at + e1) & 31);
    if (e0 < SE && at + e0 < len) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(to + lane);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(col + (size_t)s0 * row + 4 * c0)
                   : "memory");
    }
    if (e1 < SE && at + e1 < len) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(to + lane + 32);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(col + (size_t)s1 * row + 4 * c1)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int stages = (len + SE - 1) / SE;
  float acc = 0.0f;
  for (int t = 0; t < kPprStages; ++t) ask(t);
  for (int t = 0; t < stages; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPprStages - 1) : "memory");
    __syncwarp();
    if (lane < 4 * C) {
      const float *in = reinterpret_cast<const float *>(ring.word[t % kPprStages]) + lane;
      const int n = min(SE, len - t * SE);
      if (n == SE) {
        for (int e = 0; e < SE; e += 8) {
          float x[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) x[k] = in[(e + k) * 4 * C];
#pragma unroll
          for (int k = 0; k < 8; ++k) acc = __fadd_rn(acc, x[k]);
        }
      } else {
        for (int e = 0; e < n; ++e) acc = __fadd_rn(acc, in[e * 4 * C]);
      }
    }
    __syncwarp();
    ask(t + kPprStages);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  return acc;
}

// A hub chunk publishes its partial sums (this thread's: column q, counter
// `counter`, lanes `mask` of the warp together, `lead` one of them); the last
// of the vertex to arrive takes their sum in chunk order.  False: not the
// last.
__device__ __forceinline__ bool ppr_combine(const PprArgs &a, int slot, int q, bool mine, size_t counter,
                                            unsigned mask, int leadLane, bool lead, float &acc) {
  if (mine) a.partial[(size_t)slot * a.row + q] = acc;
  __threadfence();
  __syncwarp(mask);
  unsigned last = 0u;
  if (lead) {
    const unsigned old = atomicAdd(a.arrive + counter, 1u);
    last = (old + 1u) % (unsigned)a.slotCount[slot] == 0u ? 1u : 0u;
  }
  last = __shfl_sync(mask, last, leadLane);
  if (!last) return false;
  __threadfence();
  const int first = a.slotFirst[slot], cnt = a.slotCount[slot];
  float sum = 0.0f;
  if (mine)
    for (int c = 0; c < cnt; ++c) sum = __fadd_rn(sum, __ldcg(a.partial + (size_t)(first + c) * a.row + q));
  acc = sum;
  return true;
}

// The warps that take a long unit and no other: the round lasts as long as
// the longest of their chains, and short units dealt to them come on top.
// Where long units would keep more than three quarters of the warps from the
// short ones, every warp takes both.  20 rounds, with results, us, every warp
// both -> up to half -> up to three quarters: R-MAT-12, 4 queries 470, 385,
// 385; R-MAT-16, 16 queries 1962, 1821, 1821, 100 queries 4384, 4424, 3589;
// 20,000 vertices, 200 queries 3378, 2698, 2698; R-MAT-19, 40 queries 11322,
// 10239, 10252, 100 queries 20175, 20122, 20138.
__device__ __forceinline__ long long ppr_long_warps(const PprArgs &a, long long warps) {
  const long long n = (long long)a.nLong * ppr_slices(a.row);
  return 4 * n <= 3 * warps ? n : 0;
}

// The units [0, nLong), a slice of 32 queries each, a warp a slice.
__device__ __forceinline__ void ppr_long_units(const PprArgs &a, const PprRound &b, PprRing &ring) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  const long long gw = (long long)(threadIdx.x / 32) * gridDim.x + blockIdx.x;
  const int slices = ppr_slices(a.row);
  for (long long i = gw; i < (long long)a.nLong * slices; i += warps) {
    const int4 un = __ldg(a.unit + i / slices);
    const int sl = (int)(i % slices), q = 32 * sl + lane, v = un.x, slot = un.w;
    const bool act = (un.z >> 16) >= b.r;
    const int len = act ? un.z & 0xffff : 0;
    const bool mine = q < a.row;
    const int odeg = __ldg(a.outDegree + v);
    float acc = ppr_fold_ring(a.inSources + un.y, b.ct + 32 * sl, (size_t)a.row, min(a.row - 32 * sl, 32) / 4, len,
                              ring, lane);
    if (slot >= 0 &&
        !ppr_combine(a, slot, q, mine, (size_t)a.slotHub[slot] * slices + sl, kFullMask, 0, lane == 0, acc))
      continue;
    if (mine) ppr_finish(a, b, v, q, (size_t)v * a.row + q, act, acc, odeg);
  }
}

// Rows of QP floats whose long units go through the ring.  Rows of less than
// 16 bytes cannot, and of 32 floats the 32 rows that a warp's registers hold
// in flight are more than the ring's five stages of 8 (20 rounds, 32 queries,
// us, with the ring and without: R-MAT-12 860, 401, R-MAT-16 3020, 1732,
// R-MAT-18 6068, 5025).
__host__ __device__ constexpr bool ppr_ring_rows(int QP) { return QP >= 4 && QP < 32; }

// Round r of rows of QP <= 32 floats: long units through the ring, then
// groups of QP lanes take units (the groups of a warp neighbouring ones, so
// similar lengths).  Work is dealt block-first, so that the longest units
// spread over the SMs.  kL1: rows are read through L1, which pays where a line
// holds many and few sources have most of the edges (rows of 1 and 2; 20
// rounds, us, past L1 and through it: 2 queries, R-MAT-18 2788, 2245, lattice
// 500 x 500 243, 274; 4 queries 1808, 1841, 370, 452; 16 queries, 200,000
// vertices of 8 random edges 857, 1100).
template <int QP, bool kL1>
__device__ __forceinline__ void ppr_round_narrow(const PprArgs &a, int r, PprRing &ring) {
  constexpr int L = QP, G = 32 / L, M = 32 / L;
  const PprRound b = ppr_buffers(a, r);
  const int lane = threadIdx.x & 31;
  const int grp = lane / L, j = lane % L;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  const long long gw = (long long)(threadIdx.x / 32) * gridDim.x + blockIdx.x;
  const unsigned mask = L == 32 ? kFullMask : (((1u << (L & 31)) - 1u) << (grp * L));
  long long first = 0;
  if constexpr (ppr_ring_rows(QP)) {
    ppr_long_units(a, b, ring);
    first = a.nLong;
  }
  const long long busy = ppr_ring_rows(QP) ? ppr_long_warps(a, warps) : 0;
  for (long long base = first + (gw - busy) * G; gw >= busy && base < a.nUnits; base += (warps - busy) * G) {
    const long long u = base + grp;
    const int4 un = u < a.nUnits ? __ldg(a.unit + u) : make_int4(-1, 0, 0, -1);
    const int v = un.x, slot = un.w;
    const bool act = v >= 0 && (un.z >> 16) >= r;
    const int len = act ? un.z & 0xffff : 0;
    const int odeg = v >= 0 ? __ldg(a.outDegree + v) : 0;
    const int maxLen = __reduce_max_sync(kFullMask, len);
    const int32_t *src = a.inSources + un.y;
    float acc = 0.0f;
    int ids[M];
#pragma unroll
    for (int m = 0; m < M; ++m) ids[m] = m * L + j < len ? __ldg(src + m * L + j) : 0;
    for (int o = 0; o < maxLen; o += 32) {  // warp-uniform
      float c[32];
#pragma unroll
      for (int t = 0; t < 32; ++t) {
        const int s = __shfl_sync(kFullMask, ids[t / L], t % L, L);
        if constexpr (kL1)
          c[t] = t < len - o ? b.ct[(size_t)s * QP + j] : 0.0f;
        else
          c[t] = t < len - o ? __ldcg(b.ct + (size_t)s * QP + j) : 0.0f;
      }
#pragma unroll
      for (int m = 0; m < M; ++m) ids[m] = o + 32 + m * L + j < len ? __ldg(src + o + 32 + m * L + j) : 0;
#pragma unroll
      for (int t = 0; t < 32; ++t)
        if (t < len - o) acc = __fadd_rn(acc, c[t]);
    }
    if (v < 0) continue;
    if (slot >= 0 && !ppr_combine(a, slot, j, true, (size_t)a.slotHub[slot], mask, grp * L, j == 0, acc)) continue;
    ppr_finish(a, b, v, j, (size_t)v * QP + j, act, acc, odeg);
  }
}

// Round r of wider rows (a.row floats, a multiple of 8 up to QP).  Long
// units and hub chunks are taken a slice of 32 queries at a time, a lane per
// query, so that their chains run in parallel; the others a whole row at a
// time, four neighbouring queries a lane (one 16-byte load an edge and lane
// instead of four 4-byte ones).
template <int QP>
__device__ __forceinline__ void ppr_round_wide(const PprArgs &a, int r, PprRing &ring) {
  constexpr int L = QP / 4 < 32 ? QP / 4 : 32;  // lanes of a unit
  constexpr int G = 32 / L, NV = QP / (4 * L);  // units a warp, 16-byte words a lane
  constexpr int D = 8 / NV;                     // edges a step
  const PprRound b = ppr_buffers(a, r);
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  const long long gw = (long long)(threadIdx.x / 32) * gridDim.x + blockIdx.x;
  ppr_long_units(a, b, ring);
  const int grp = lane / L, j = lane % L;
  const long long busy = ppr_long_warps(a, warps);
  for (long long base = a.nLong + (gw - busy) * G; gw >= busy && base < a.nUnits; base += (warps - busy) * G) {
    const long long u = base + grp;
    const int4 un = u < a.nUnits ? __ldg(a.unit + u) : make_int4(-1, 0, 0, -1);
    const int v = un.x;
    const bool act = v >= 0 && (un.z >> 16) >= r;
    const int len = act ? un.z & 0xffff : 0;
    const int odeg = v >= 0 ? __ldg(a.outDegree + v) : 0;
    const int maxLen = __reduce_max_sync(kFullMask, len);
    float4 acc[NV];
    bool on[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      acc[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      on[k] = 4 * (j + L * k) < a.row;
    }
    const int32_t *src = a.inSources + un.y;
    int ids = j < len ? __ldg(src + j) : 0;
    for (int o = 0; o < maxLen; o += L) {  // warp-uniform
      const int next = o + L + j < len ? __ldg(src + o + L + j) : 0;
      for (int d = 0; d < L && o + d < maxLen; d += D) {
        const int n = len - o - d;  // edges from this step on (<= 0: none)
        float4 c[D][NV];
#pragma unroll
        for (int t = 0; t < D; ++t) {
          const int s = __shfl_sync(kFullMask, ids, d + t, L);
          const float4 *row = reinterpret_cast<const float4 *>(b.ct + (size_t)s * a.row) + j;
#pragma unroll
          for (int k = 0; k < NV; ++k)
            c[t][k] = t < n && on[k] ? row[L * k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int t = 0; t < D; ++t)
          if (t < n) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
              acc[k].x = __fadd_rn(acc[k].x, c[t][k].x);
              acc[k].y = __fadd_rn(acc[k].y, c[t][k].y);
              acc[k].z = __fadd_rn(acc[k].z, c[t][k].z);
              acc[k].w = __fadd_rn(acc[k].w, c[t][k].w);
            }
          }
      }
      ids = next;
    }
    if (v < 0) continue;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if (!on[k]) continue;
      const int q = 4 * (j + L * k);
      const size_t at = ((size_t)v * a.row + q) / 4;
      float4 nr, nc;
      if (act) {
        const int4 s = __ldg(reinterpret_cast<const int4 *>(a.sources) + q / 4);
        auto rank = [&](float x, int source, int qi) {
          const float tele = (qi < a.nQueries && source == v) ? a.teleport : 0.0f;
          return __fadd_rn(tele, __fmul_rn(a.damp, x));
        };
        nr = make_float4(rank(acc[k].x, s.x, q), rank(acc[k].y, s.y, q + 1), rank(acc[k].z, s.z, q + 2),
                         rank(acc[k].w, s.w, q + 3));
        nc = make_float4(ppr_contrib(nr.x, odeg), ppr_contrib(nr.y, odeg), ppr_contrib(nr.z, odeg),
                         ppr_contrib(nr.w, odeg));
      } else {
        nr = __ldcg(reinterpret_cast<const float4 *>(b.rk) + at);
        nc = __ldcg(reinterpret_cast<const float4 *>(b.ct) + at);
      }
      reinterpret_cast<float4 *>(b.rk2)[at] = nr;
      reinterpret_cast<float4 *>(b.ct2)[at] = nc;
    }
  }
}

template <int QP>
__device__ __forceinline__ void ppr_round(const PprArgs &a, int r) {
  __shared__ PprRing rings[8];  // a warp's each (256 threads)
  PprRing &ring = rings[threadIdx.x / 32];
  if constexpr (QP == 1)
    ppr_round_narrow<1, true>(a, r, ring);
  else if constexpr (QP == 2) {
    if (a.nLong > 0)
      ppr_round_narrow<2, true>(a, r, ring);
    else
      ppr_round_narrow<2, false>(a, r, ring);
  } else if constexpr (QP <= 32)
    ppr_round_narrow<QP, false>(a, r, ring);
  else
    ppr_round_wide<QP>(a, r, ring);
}

template <int QP>
__global__ void __launch_bounds__(256) ppr_round_kernel(const PprArgs a, int r) {
  ppr_round<QP>(a, r);
}

// Every round of a PPR batch in one cooperative launch (the batched engine,
// gas_batch_run): the served round body, rounds separated by bounded grid
// barriers.  *roundsOut receives the rounds completed.
template <int QP>
__global__ void __launch_bounds__(256) ppr_run_kernel(const PprArgs a, int rounds, unsigned *barrier,
                                                      unsigned *errWord, int32_t *roundsOut) {
  int r = 0;
  for (; r < rounds; ++r) {
    ppr_round<QP>(a, r);
    if (!grid_barrier(barrier, errWord)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *roundsOut = r;
}

}  // namespace detail
}  // namespace gas

// Batched multi-source BFS and SSSP: Q queries with independent sources on
// one resident graph, all rounds in one persistent cooperative launch.
//
// State is laid out vertex-major so a warp touches one vertex's queries
// with coalesced accesses:
//   value[V][Q]      BFS depth (-1 unreached) or SSSP distance (int32)
//   mask[3][V][W]    W = Q/32 words per vertex: the queries whose value at
//                    this vertex changed in a round (rotating: round r
//                    reads mask[r%3], writes mask[(r+1)%3] and clears
//                    mask[(r+2)%3], so no stamps and no extra barrier)
//   seen[V][W]       BFS: queries that have reached the vertex
//
// A round runs in one of two modes, chosen from the previous round's
// changed vertices (list L, with their out-degree total E_out):
//   push  (E_out * alpha <= E): a warp per list entry -- a changed vertex
//         u and one kPushChunk-edge chunk of its out-edges (hubs span
//         several entries, so no warp walks a hub alone) -- updates the
//         destinations for u's changed queries with atomics, a lane per
//         edge (or, for SSSP when u has more changed queries than the
//         chunk has edges, a lane per query); destinations that change are
//         appended to the next list (one atomic per warp and step);
//   pull  otherwise: one pass over work units (a vertex's in-edges, split
//         into chunks of at most `chunk` edges for high in-degree vertices),
//         lanes mapped to queries (lane l owns queries l + 32k), followed
//         by a compaction of the changed vertices into the list.
// The updates:
//   BFS   next(v) = OR of mask[u] over in-neighbours u, minus seen(v);
//         newly seen queries get depth = round + 1           (bfs.cu:54-66)
//   SSSP  for queries whose distance at in-neighbour u changed, relax
//         dist[u][q] + w with atomicMin on dist[v][q]        (sssp.cu:36-55)
// Every query's result equals its single-source result bit for bit: BFS
// depths and shortest-path distances are unique.  Rounds end when a round
// changes nothing (bounded waits, as in the single-query persistent kernel).
#pragma once

#include "persistent.cuh"

namespace gas {
namespace detail {

enum BatchKind { kBatchBFS = 1, kBatchSSSP = 2 };

struct BatchArgs {
  int32_t nVertices;
  int32_t nEdges;
  const int32_t *outOffsets;  // CSR (push rounds)
  const int32_t *outDests;
  const int32_t *weightsOut;  // CSR order (SSSP push rounds)
  int32_t *list[3];           // [listCap] changed vertices (rotating), one
  int32_t *listC[3];          //   entry per kPushChunk out-edges: (vertex, chunk)
  unsigned long long *listCnt;  // [3] (entries << 32) | out-degree total
  int32_t *inList;            // [V] round stamp of list membership
  int32_t alpha;              // push when out-degree total * alpha <= nEdges
  int32_t nQueries;       // padded to 32 * W
  int32_t nLive;          // queries among them
  const int32_t *inSources;
  const int32_t *weights;  // CSC order (SSSP)
  const int32_t *unitV;
  const int32_t *unitBeg;
  const int32_t *unitEnd;
  int32_t nUnits;
  int32_t *value;          // [V][Q]
  unsigned *mask[3];       // [V][W] each
  unsigned *seen;          // [V][W] (BFS)
  unsigned long long *cnt; // [3] changed (vertex, query) pairs per round
  unsigned *barrier;       // [2]
  unsigned *errWord;
  int32_t *roundsOut;
  int32_t maxRounds;       // 0 = until nothing changes
  // SSSP bucket order (delta-stepping; persistent kernel only): a changed
  // (u, q) is relaxed once dist[u][q] < thresh[q]; others wait in the
  // changed set.  A query's bound grows by delta after a round in which it
  // produced no value below the bound.  0 = every changed pair every round.
  int32_t delta;
  int32_t *thresh[2];      // [Q] by round parity
  unsigned *nearFlag[3];   // [W] queries with a new value below the bound (rotating)
  // Pair frontier (graphs of small out-degree, V * Q < 2^31): a thread per
  // changed (vertex, query) instead of a warp per vertex entry; state
  // query-major; every round pushes.  kPairsList: entries u * Q + q.
  int32_t pairMode;        // PairMode
  uint32_t *pairs[3];      // [V * Q] each (rotating, counts in listCnt >> 32)
};

// Shared-memory view of the bucket bounds for one round (null when off).
struct BatchBucket {
  const int32_t *bound;  // [Q] this round's thresh
  unsigned *near;        // [W] block-local near flags
};

constexpr int32_t kBatchInf = 0x7fffffff - 100000;  // SSSP gatherZero (sssp.cu:32-33)

// Out-edges per push-list entry; a list holds at most V + E / kPushChunk
// entries (each vertex once per round).
constexpr int kPushChunk = 512;

__host__ __device__ inline long long batch_list_capacity(long long nVertices, long long nEdges) {
  return nVertices + nEdges / kPushChunk + 32;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFullMask, x, o);
  return x;  // lane 0
}

// Appends, for each lane with `want`, vertex v of out-degree d to a list as
// ceil(d / kPushChunk) entries (at least one): one atomic per warp.
// Warp-uniform call.
__device__ __forceinline__ void warp_append(bool want, int v, int d, int32_t *list,
                                            int32_t *listC, unsigned long long *cnt) {
  const int lane = threadIdx.x & 31;
  const int ne = want ? max(1, (d + kPushChunk - 1) / kPushChunk) : 0;
  int incl = ne;
  unsigned dsum = want ? (unsigned)d : 0u;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFullMask, incl, o);
    const unsigned z = __shfl_up_sync(kFullMask, dsum, o);
    if (lane >= o) {
      incl += y;
      dsum += z;
    }
  }
  const int total = __shfl_sync(kFullMask, incl, 31);
  if (total == 0) return;
  const unsigned dtot = __shfl_sync(kFullMask, dsum, 31);
  unsigned long long base = 0ull;
  if (lane == 0) base = atomicAdd(cnt, ((unsigned long long)total << 32) | dtot);
  base = __shfl_sync(kFullMask, base, 0);
  const long long pos = (long long)(base >> 32) + incl - ne;
  for (int c = 0; c < ne; ++c) {
    list[pos + c] = v;
    listC[pos + c] = c;
  }
}

// Row i of W-word rows (16-byte aligned from W = 4 on, as the buffers are),
// zero unless ok.  Wide loads: past L1 every load is its own L2 request.
template <int W>
__device__ __forceinline__ void load_words(const unsigned *rows, int i, bool ok, unsigned (&m)[W]) {
  const unsigned *p = rows + (size_t)i * W;
#pragma unroll
  for (int k = 0; k < W; ++k) m[k] = 0u;
  if (!ok) return;
  if constexpr (W % 4 == 0) {
#pragma unroll
    for (int k = 0; k < W; k += 4) {
      const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(p + k));
      m[k] = x.x;
      m[k + 1] = x.y;
      m[k + 2] = x.z;
      m[k + 3] = x.w;
    }
  } else if constexpr (W == 2) {
    const uint2 x = __ldcg(reinterpret_cast<const uint2 *>(p));
    m[0] = x.x;
    m[1] = x.y;
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) m[k] = __ldcg(p + k);
  }
}

// Pull round of a BFS batch, a warp a unit: units u0, u0 + stride, ...  A
// lane looks up each of the next 32 (vertex, range, and whether the vertex
// still has a query to be reached: most have none from the third round on),
// then the warp walks those that do, the next one's first sources in flight,
// and ends a unit once every query has reached its vertex.  A vertex of one
// unit belongs to this warp alone: its seen row is read with the sources and
// written back plainly, where an atomic would be one more L2 round trip.
// Bound by L2: the masks of a round, one 32-byte sector an edge.  A run, with
// eight 4-byte loads an edge and every unit walked -> now: 256 queries on
// R-MAT-18 (6.1 M edges) 1.63 -> 0.69 ms, 64 queries 0.65 -> 0.36, 10 queries
// 0.29 -> 0.24; 200 queries on R-MAT-16 0.61 -> 0.28.
template <int W>
__device__ __forceinline__ void batch_bfs_pull(const BatchArgs &a, long long u0, long long stride, int round,
                                               const unsigned *cur, unsigned *nxt, unsigned long long &changed) {
  const int lane = threadIdx.x & 31;
  const int Q = W * 32;
  // this lane's word of a row: its live queries (lanes past W: none)
  const int liveBits = lane < W ? a.nLive - 32 * lane : 0;
  const unsigned live = liveBits >= 32 ? kFullMask : liveBits > 0 ? (1u << liveBits) - 1u : 0u;
  for (long long base = u0; base < a.nUnits; base += 32 * stride) {  // warp-uniform
    const long long u = base + lane * stride;
    int v = -1, beg = 0, end = 0;
    if (u < a.nUnits) {
      v = __ldg(a.unitV + u);
      beg = __ldg(a.unitBeg + u);
      end = __ldg(a.unitEnd + u);
      if ((u > 0 && __ldg(a.unitV + u - 1) == v) || (u + 1 < a.nUnits && __ldg(a.unitV + u + 1) == v))
        end = -end;  // (a unit's end is above 0) one of several of its vertex
    }
    unsigned row[W];
    load_words<W>(a.seen, v, v >= 0, row);
    bool need = false;
#pragma unroll
    for (int k = 0; k < W; ++k) need |= (~row[k] & __shfl_sync(kFullMask, live, k)) != 0u;
    unsigned work = __ballot_sync(kFullMask, need && v >= 0);
    if (!work) continue;
    int j = __ffs(work) - 1;
    int nb = __shfl_sync(kFullMask, beg, j), ne = __shfl_sync(kFullMask, end, j);
    int sn = nb + lane < abs(ne) ? __ldg(a.inSources + nb + lane) : -1;
    while (work) {
      work &= work - 1u;
      const int cv = __shfl_sync(kFullMask, v, j);
      const bool split = ne < 0;
      const int ce = abs(ne);
      int e0 = nb, s = sn;
      const unsigned seen = lane < W ? __ldcg(a.seen + (size_t)cv * W + lane) : 0u;
      if (work) {
        j = __ffs(work) - 1;
        nb = __shfl_sync(kFullMask, beg, j);
        ne = __shfl_sync(kFullMask, end, j);
        sn = nb + lane < abs(ne) ? __ldg(a.inSources + nb + lane) : -1;
      }
      unsigned acc[W], mine = 0u;
#pragma unroll
      for (int k = 0; k < W; ++k) acc[k] = 0u;
      for (;;) {  // 64 edges
        unsigned m[W];
        const int s1 = e0 + 32 + lane < ce ? __ldg(a.inSources + e0 + 32 + lane) : -1;
        load_words<W>(cur, s, s >= 0, m);
#pragma unroll
        for (int k = 0; k < W; ++k) acc[k] |= m[k];
        if (e0 + 32 < ce) {
          const int s2 = e0 + 64 + lane < ce ? __ldg(a.inSources + e0 + 64 + lane) : -1;
          load_words<W>(cur, s1, s1 >= 0, m);
#pragma unroll
          for (int k = 0; k < W; ++k) acc[k] |= m[k];
          s = s2;
        }
#pragma unroll
        for (int k = 0; k < W; ++k) {
          const unsigned all = __reduce_or_sync(kFullMask, acc[k]);
          if (lane == k) mine = all;
        }
        e0 += 64;
        if (e0 >= ce || __all_sync(kFullMask, (live & ~(mine | seen)) == 0u)) break;
      }
      unsigned fresh = mine & ~seen;
      if (split) {
        if (fresh) fresh &= ~atomicOr(a.seen + (size_t)cv * W + lane, fresh);
        if (fresh) atomicOr(nxt + (size_t)cv * W + lane, fresh);
      } else if (fresh) {
        a.seen[(size_t)cv * W + lane] = seen | fresh;
        nxt[(size_t)cv * W + lane] = fresh;
      }
      changed += __popc(fresh);
#pragma unroll
      for (int k = 0; k < W; ++k)
        if ((__shfl_sync(kFullMask, fresh, k) >> lane) & 1u) a.value[(size_t)cv * Q + k * 32 + lane] = round + 1;
    }
  }
}

// One unit of a pull round of an SSSP batch.
template <int W>
__device__ __forceinline__ void batch_sssp_unit(const BatchArgs &a, int u, const unsigned *cur, unsigned *nxt,
                                                unsigned long long &changed) {
  const int lane = threadIdx.x & 31;
  const int v = a.unitV[u];
  const int beg = a.unitBeg[u], end = a.unitEnd[u];
  const int Q = W * 32;
  int best[W];
#pragma unroll
  for (int k = 0; k < W; ++k) best[k] = kBatchInf;
  for (int e0 = beg; e0 < end; e0 += 32) {
    // lane j loads edge e0+j: source, weight and its changed-query mask
    const int e = e0 + lane;
    const bool ok = e < end;
    const int s = ok ? __ldg(a.inSources + e) : 0;
    const int w = ok ? __ldg(a.weights + e) : 0;
    unsigned m[W], any = 0u;
    load_words<W>(cur, s, ok, m);
#pragma unroll
    for (int k = 0; k < W; ++k) any |= m[k];
    unsigned work = __ballot_sync(kFullMask, any != 0u);  // edges with a changed query
    // warp-uniform; the values of T edges in flight a lane (32 loads at
    // most): a unit's time is one L2 round trip for each batch of them
    // (R-MAT-18: 10 queries 4.06 -> 1.99 ms a run, 64 queries 8.36 -> 3.75,
    // 256 queries 16.1 -> 13.6, from four edges in flight to T)
    constexpr int T = W == 1 ? 16 : 32 / W;
    while (work) {
      int d[T][W];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int js = work ? __ffs(work) - 1 : 0;
        const bool on = work != 0u;
        if (work) work &= work - 1;
        const int sj = __shfl_sync(kFullMask, s, js);
        const int wj = __shfl_sync(kFullMask, w, js);
#pragma unroll
        for (int k = 0; k < W; ++k) {
          const unsigned mk = __shfl_sync(kFullMask, m[k], js);
          d[t][k] = kBatchInf;
          if (on && ((mk >> lane) & 1u)) d[t][k] = __ldcg(a.value + (size_t)sj * Q + k * 32 + lane) + wj;
        }
      }
#pragma unroll
      for (int t = 0; t < T; ++t)
#pragma unroll
        for (int k = 0; k < W; ++k) best[k] = min(best[k], d[t][k]);
    }
  }
#pragma unroll
  for (int k = 0; k < W; ++k) {
    bool improved = false;
    if (best[k] < kBatchInf) {
      const int old = atomicMin(a.value + (size_t)v * Q + k * 32 + lane, best[k]);
      improved = best[k] < old;
    }
    const unsigned word = __ballot_sync(kFullMask, improved);
    if (lane == 0 && word) {
      atomicOr(nxt + (size_t)v * W + k, word);
      changed += __popc(word);
    }
  }
}

// A pull round: units u0, u0 + stride, ... (one warp).
template <int W, int KIND>
__device__ __forceinline__ void batch_pull_round(const BatchArgs &a, long long u0, long long stride, int round,
                                                 const unsigned *cur, unsigned *nxt, unsigned long long &changed) {
  if constexpr (KIND == kBatchBFS)
    batch_bfs_pull<W>(a, u0, stride, round, cur, nxt, changed);
  else
    for (long long u = u0; u < a.nUnits; u += stride) batch_sssp_unit<W>(a, (int)u, cur, nxt, changed);
}

// Push round: a warp per list entry (u, chunk), lanes over the chunk's
// out-edges (32 at a time).  Warp-uniform.
template <int W, int KIND>
__device__ __forceinline__ void batch_push_unit(const BatchArgs &a, int u, int chunk, int round,
                                                const unsigned *cur, unsigned *nxt,
                                                int32_t *listNext, int32_t *listNextC,
                                                unsigned long long *cntNext,
                                                unsigned long long &changed,
                                                const BatchBucket bk = BatchBucket{nullptr, nullptr}) {
  const int lane = threadIdx.x & 31;
  const int Q = W * 32;
  unsigned m[W];
  load_words<W>(cur, u, true, m);
  int du[W];
  if (KIND == kBatchSSSP) {
#pragma unroll
    for (int k = 0; k < W; ++k)
      du[k] = ((m[k] >> lane) & 1u) ? __ldcg(a.value + (size_t)u * Q + k * 32 + lane) : kBatchInf;
  }
  bool deferred = false;
  if (KIND == kBatchSSSP && bk.bound) {  // relax below the bound now, keep the rest
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const unsigned nearM =
          __ballot_sync(kFullMask, ((m[k] >> lane) & 1u) && du[k] < bk.bound[k * 32 + lane]);
      const unsigned far = m[k] & ~nearM;
      m[k] = nearM;
      if (far) {
        deferred = true;
        if (lane == 0) {
          atomicOr(nxt + (size_t)u * W + k, far);
          changed += __popc(far);
        }
      }
    }
  }
  int nbits = 0, nwords = 0;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    nbits += __popc(m[k]);
    nwords += m[k] != 0u;
  }
  unsigned nearW[W];
#pragma unroll
  for (int k = 0; k < W; ++k) nearW[k] = 0u;
  const int ub = a.outOffsets[u];
  const int eb = ub + chunk * kPushChunk;
  const int ee = min(eb + kPushChunk, a.outOffsets[u + 1]);
  // SSSP: a lane per edge costs ceil(deg/32) * nbits atomic steps, a lane
  // per query deg * nwords
  const bool perEdge =
      KIND == kBatchBFS || (long long)((ee - eb + 31) / 32) * nbits <= (long long)(ee - eb) * nwords;
  for (int e0 = eb; e0 < ee; e0 += 32) {
    const int e = e0 + lane;
    const bool ok = e < ee;
    const int v = ok ? __ldg(a.outDests + e) : 0;
    bool any = false;
    if (KIND == kBatchBFS) {
#pragma unroll
      for (int k = 0; k < W; ++k) {
        if (!m[k] || !ok) continue;
        const unsigned old = atomicOr(a.seen + (size_t)v * W + k, m[k]);
        unsigned fresh = m[k] & ~old;
        if (!fresh) continue;
        atomicOr(nxt + (size_t)v * W + k, fresh);
        any = true;
        changed += __popc(fresh);
        while (fresh) {
          const int b = __ffs(fresh) - 1;
          fresh &= fresh - 1u;
          a.value[(size_t)v * Q + k * 32 + b] = round + 1;
        }
      }
    } else if (perEdge) {
      const int w = ok ? __ldg(a.weightsOut + e) : 0;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        unsigned bits = m[k], imp = 0u;
        while (bits) {  // warp-uniform; up to four relaxations in flight
          int bs[4], ds[4], olds[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            bs[t] = bits ? __ffs(bits) - 1 : -1;
            if (bits) bits &= bits - 1u;
            ds[t] = __shfl_sync(kFullMask, du[k], bs[t] < 0 ? 0 : bs[t]);
          }
#pragma unroll
          for (int t = 0; t < 4; ++t)
            olds[t] = (ok && bs[t] >= 0)
                          ? atomicMin(a.value + (size_t)v * Q + k * 32 + bs[t], ds[t] + w)
                          : kBatchInf;
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (ok && bs[t] >= 0 && ds[t] + w < olds[t]) {
              imp |= 1u << bs[t];
              if (bk.bound && ds[t] + w < bk.bound[k * 32 + bs[t]]) nearW[k] |= 1u << bs[t];
            }
        }
        if (imp) {
          atomicOr(nxt + (size_t)v * W + k, imp);
          any = true;
          changed += __popc(imp);
        }
      }
    } else {  // lane per query, the 32 edges in turn
      const int w = ok ? __ldg(a.weightsOut + e) : 0;
      const int n = min(32, ee - e0);
      unsigned anyMask = 0u;
      for (int t = 0; t < n; ++t) {
        const int vt = __shfl_sync(kFullMask, v, t);
        const int wt = __shfl_sync(kFullMask, w, t);
#pragma unroll
        for (int k = 0; k < W; ++k) {
          bool imp = false;
          if ((m[k] >> lane) & 1u) {
            const int cand = du[k] + wt;
            const int old = atomicMin(a.value + (size_t)vt * Q + k * 32 + lane, cand);
            imp = cand < old;
            if (imp && bk.bound && cand < bk.bound[k * 32 + lane]) nearW[k] |= 1u << lane;
          }
          const unsigned word = __ballot_sync(kFullMask, imp);
          if (word) {
            if (lane == 0) {
              atomicOr(nxt + (size_t)vt * W + k, word);
              changed += __popc(word);
            }
            anyMask |= 1u << t;
          }
        }
      }
      any = (anyMask >> lane) & 1u;
    }
    bool want = false;
    if (any) want = atomicExch(a.inList + v, round + 1) != round + 1;
    warp_append(want, v, want ? a.outOffsets[v + 1] - a.outOffsets[v] : 0, listNext, listNextC,
                cntNext);
  }
  if (KIND == kBatchSSSP && bk.bound) {
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const unsigned nw = __reduce_or_sync(kFullMask, nearW[k]);
      if (lane == 0 && nw) atomicOr(bk.near + k, nw);
    }
    // u keeps its deferred queries: back on the next list (all its chunks)
    bool wantU = false;
    if (deferred && lane == 0) wantU = atomicExch(a.inList + u, round + 1) != round + 1;
    warp_append(wantU, u, wantU ? a.outOffsets[u + 1] - ub : 0, listNext, listNextC, cntNext);
  }
}

// ---- pair frontiers (graphs of small out-degree)
// State is query-major (value[q][v], mask and seen words [w][v]), so that
// the vertices of one query's wavefront touch neighbouring words.  The
// changed set is the round's mask, or a list as well (below).
//
// From the mask: activation is one reduction into the next round's mask,
// which also removes duplicates: no list, no counter that every warp contends
// for, and nothing to wait for.  Each block owns groups of 32 consecutive
// mask words (a warp reads one in a coalesced load), lists their set bits in
// shared memory, zeroes the words (so the mask is clean when it next collects
// bits) and relaxes a listed (vertex, query) a thread: a chain of four L2
// round trips a round (mask; value and row bounds; row; atomic) where list
// appends take seven.  64 SSSP queries, delta 512, from lists and from the
// mask: 256 x 256 lattice 6.9 -> 3.4 ms, 506 x 506 16.2 -> 9.4, 1000 x 1000
// 48 -> 35 (256 queries 193 -> 154); 64 BFS queries, 256 x 256 3.25 -> 2.06.
//
// From a list, for BFS over large masks: its rounds are short against the
// passes over the mask, the more so the fewer of a word's queries are live
// (lattices, from a list and from the mask, ms: 1000 x 1000, 1 M words, 4
// queries 12.4, 13.4, 16 12.6, 14.9, 32 13.0, 12.3; 700 x 700, 980,000 words,
// 33 queries 9.3, 9.8, 64 9.7, 9.5, but 490,000 words, 4 queries 8.1, 6.6; 500
// x 500, 500,000 words, 33 queries 6.3, 5.2).
constexpr long long kPairMaskWords = 3ll << 18;  // BFS: lists above
enum PairMode { kPairsOff = 0, kPairsMask = 1, kPairsList = 2 };
inline int pair_mode_of(bool bfs, long long nVertices, int W) {
  return bfs && nVertices * W > kPairMaskWords ? kPairsList : kPairsMask;
}
constexpr int kPairList = 1024;  // pairs a block lists at a time
constexpr int kPairWords = 8;    // mask words a thread reads a pass, half of them where that covers the mask

// Blocks of a persistent run over the mask.  A round is a chain of round trips
// and a grid barrier, which costs more the more blocks arrive: enough of them
// to read the mask in one pass and for a wavefront of about 5 sqrt(V)
// vertices a query, a pair a thread; whole blocks per SM (64 SSSP queries,
// 256 x 256 lattice: 3.65, 3.42 and 3.96 ms at 4, 2 and 1 an SM; 506 x 506:
// 9.4, 12.2, 19.6).
inline int batch_pair_blocks(int32_t nVertices, int W, int nQ, int sms) {
  double root = 1.0;
  while (root * root < (double)nVertices) root *= 1.1;
  const double words = (double)nVertices * W, front = 5.0 * root * nQ;
  const double want = (words / kPairWords > front ? words / kPairWords : front) / 256;
  const int perSM = (int)(want / (sms > 0 ? sms : 1) + 0.5);
  return (perSM > 1 ? perSM : 1) * (sms > 0 ? sms : 1);
}

struct PairSmem {
  uint32_t entry[kPairList];
  unsigned warpTot[8];
};

// Relaxes the out-edges of pair (u, q) for query q alone.
template <int W, int KIND>
__device__ __forceinline__ void batch_pair(const BatchArgs &a, int u, int q, int round, unsigned *nxt,
                                           unsigned long long &changed, const BatchBucket bk) {
  const unsigned bit = 1u << (q & 31);
  const int wq = q >> 5;
  const size_t V = (size_t)a.nVertices;
  const int eb = a.outOffsets[u], ee = a.outOffsets[u + 1];
  unsigned *nw = nxt + (size_t)wq * V;
  int du = 0;
  if (KIND == kBatchSSSP) {
    du = __ldcg(a.value + (size_t)q * V + u);
    if (bk.bound && du >= bk.bound[q]) {  // not this bucket: keep (u, q) for later
      atomicOr(nw + u, bit);
      ++changed;
      return;
    }
  }
  constexpr int J = 4;  // edges in flight
  for (int e0 = eb; e0 < ee; e0 += J) {
    int v[J], x[J];
#pragma unroll
    for (int t = 0; t < J; ++t) {
      v[t] = e0 + t < ee ? __ldg(a.outDests + e0 + t) : -1;
      if (KIND == kBatchSSSP) x[t] = e0 + t < ee ? du + __ldg(a.weightsOut + e0 + t) : 0;
    }
    int old[J];
#pragma unroll
    for (int t = 0; t < J; ++t)
      if (v[t] >= 0) {
        if (KIND == kBatchBFS)
          old[t] = (int)atomicOr(a.seen + (size_t)wq * V + v[t], bit);
        else
          old[t] = atomicMin(a.value + (size_t)q * V + v[t], x[t]);
      }
#pragma unroll
    for (int t = 0; t < J; ++t) {
      if (v[t] < 0) continue;
      if (KIND == kBatchBFS) {
        if ((unsigned)old[t] & bit) continue;
        a.value[(size_t)q * V + v[t]] = round + 1;
      } else {
        if (x[t] >= old[t]) continue;
        if (bk.bound && x[t] < bk.bound[q] && !(bk.near[wq] & bit)) atomicOr(bk.near + wq, bit);
      }
      atomicOr(nw + v[t], bit);  // result unused: a reduction
      ++changed;
    }
  }
}

// One round over the pairs of mask `cur`.  Every thread of a 256-thread block
// calls it.
template <int W, int KIND>
__device__ __forceinline__ void batch_pairs_round(const BatchArgs &a, int round, unsigned *cur, unsigned *nxt,
                                                  PairSmem &sm, unsigned long long &changed, const BatchBucket bk) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long words = (long long)a.nVertices * W;
  const long long half = (long long)gridDim.x * 32 * (kPairWords / 2) * 8;
  for (long long base = 0; base < words; base += 2 * half) {  // block-uniform
    const bool both = words - base > half;
    // warp k of the block takes groups blockIdx.x + grid * (k + 8 j)
    unsigned m[kPairWords];
    int n = 0;
#pragma unroll
    for (int j = 0; j < kPairWords; ++j) {
      const long long i = base + 32 * ((long long)blockIdx.x + (long long)gridDim.x * (warp + 8 * j)) + lane;
      m[j] = (j < kPairWords / 2 || both) && i < words ? __ldcg(cur + i) : 0u;
      if (m[j]) cur[i] = 0u;
      n += __popc(m[j]);
    }
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFullMask, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) sm.warpTot[warp] = (unsigned)incl;
    __syncthreads();
    int first = incl - n, total = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < warp) first += (int)sm.warpTot[k];
      total += (int)sm.warpTot[k];
    }
    for (int at = 0; at < total; at += kPairList) {  // block-uniform
      int pos = first - at;
      if (pos < kPairList && pos + n > 0) {
#pragma unroll
        for (int j = 0; j < kPairWords; ++j) {
          if (j >= kPairWords / 2 && !both) break;
          const uint32_t i =
              (uint32_t)(base + 32 * ((long long)blockIdx.x + (long long)gridDim.x * (warp + 8 * j)) + lane);
          unsigned rest = m[j];
          while (rest) {
            const int p = __ffs(rest) - 1;
            rest &= rest - 1u;
            if (pos >= 0 && pos < kPairList) sm.entry[pos] = (i << 5) | (uint32_t)p;  // V * Q < 2^31
            ++pos;
          }
        }
      }
      __syncthreads();
      const int here = min(total - at, kPairList);
      for (int k = threadIdx.x; k < here; k += 256) {
        const uint32_t e = sm.entry[k], i = e >> 5;
        const int w = W == 1 ? 0 : (int)(i / (uint32_t)a.nVertices);
        batch_pair<W, KIND>(a, (int)(i - (uint32_t)w * (uint32_t)a.nVertices), 32 * w + (int)(e & 31u), round, nxt,
                            changed, bk);
      }
      __syncthreads();  // the list is rewritten
    }
    __syncthreads();  // warpTot is rewritten
  }
}

// Appends each lane's entries out[k] with want[k] (k < K) to a pair list:
// one atomic per warp for all K.  Warp-uniform call.
template <int K>
__device__ __forceinline__ void warp_append_pairs(const bool (&want)[K], const uint32_t (&out)[K],
                                                  uint32_t *list, unsigned long long *cnt) {
  const int lane = threadIdx.x & 31;
  unsigned n = 0u;
#pragma unroll
  for (int k = 0; k < K; ++k) n += want[k] ? 1u : 0u;
  unsigned incl = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned o = __shfl_up_sync(kFullMask, incl, d);
    if (lane >= d) incl += o;
  }
  const unsigned total = __shfl_sync(kFullMask, incl, 31);
  if (total == 0u) return;
  unsigned long long base = 0ull;
  if (lane == 31) base = atomicAdd(cnt, (unsigned long long)total << 32);
  base = __shfl_sync(kFullMask, base, 31) >> 32;
  unsigned long long pos = base + (incl - n);
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (want[k]) list[pos++] = out[k];
}

// Pair-list push (BFS): lane i takes entry i of the current list (when
// `valid`), a changed (u, q), and marks u's out-neighbours for q; one seen for
// the first time is appended as (v, q).  Warp-uniform (lanes step through
// their edges together, up to the warp's largest out-degree).
template <int W>
__device__ __forceinline__ void batch_pair_unit(const BatchArgs &a, bool valid, uint32_t entry, int round,
                                                uint32_t *listNext, unsigned long long *cntNext,
                                                unsigned long long &changed) {
  constexpr int Q = 32 * W;
  constexpr int LOGQ = W == 1 ? 5 : W == 2 ? 6 : W == 4 ? 7 : 8;
  const int u = valid ? (int)(entry >> LOGQ) : 0;
  const int q = (int)(entry & (Q - 1));
  const unsigned bit = 1u << (q & 31);
  const int wq = q >> 5;
  const size_t V = (size_t)a.nVertices;
  const int eb = valid ? a.outOffsets[u] : 0;
  const int deg = valid ? a.outOffsets[u + 1] - eb : 0;
  // four out-edges a step, their appends to the next list in one atomic per
  // warp (the list counter is one word every warp of the grid contends for)
  constexpr int J = 4;
  const int maxDeg = __reduce_max_sync(kFullMask, deg);
  for (int j0 = 0; j0 < maxDeg; j0 += J) {
    bool want[J];
    uint32_t out[J];
#pragma unroll
    for (int t = 0; t < J; ++t) {
      const int j = j0 + t;
      want[t] = false;
      out[t] = 0u;
      if (j < deg) {
        const int v = __ldg(a.outDests + eb + j);
        const unsigned old = atomicOr(a.seen + (size_t)wq * V + v, bit);
        if (!(old & bit)) {
          a.value[(size_t)q * V + v] = round + 1;
          want[t] = true;
          changed += 1;
          out[t] = ((uint32_t)v << LOGQ) | (uint32_t)q;
        }
      }
    }
    warp_append_pairs<J>(want, out, listNext, cntNext);
  }
}

// One round over the pair list of round `round`, dealt to warps block-first.
template <int W>
__device__ __forceinline__ void batch_pair_list(const BatchArgs &a, int round, long long nList,
                                                unsigned long long *cntNext, unsigned long long &changed) {
  const uint32_t *pc = a.pairs[round % 3];
  uint32_t *pn = a.pairs[(round + 1) % 3];
  const long long threads = (long long)gridDim.x * blockDim.x;
  const long long gwl = (long long)(threadIdx.x / 32) * gridDim.x + blockIdx.x;
  for (long long base = gwl * 32; base < nList; base += threads) {
    const long long i = base + (threadIdx.x & 31);
    const bool valid = i < nList;
    batch_pair_unit<W>(a, valid, valid ? __ldcg(pc + i) : 0u, round, pn, cntNext, changed);
  }
}

// After a pull round: list the vertices with a changed query.
template <int W>
__device__ __forceinline__ void batch_compact(const BatchArgs &a, const unsigned *nxt,
                                              int32_t *listNext, int32_t *listNextC,
                                              unsigned long long *cntNext) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  const long long gw = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  for (long long base = gw * 32; base < a.nVertices; base += warps * 32) {
    const long long v = base + lane;
    unsigned any = 0u;
    unsigned m[W];
    load_words<W>(nxt, (int)v, v < a.nVertices, m);
#pragma unroll
    for (int k = 0; k < W; ++k) any |= m[k];
    const bool want = any != 0u;
    warp_append(want, (int)v, want ? a.outOffsets[v + 1] - a.outOffsets[v] : 0, listNext,
                listNextC, cntNext);
  }
}

// PAIRS: the instantiation for pair-frontier batches (a.pairMode), which
// holds only their rounds; from lists (BFS only) with at most 40 registers a
// thread, as more warps keep more of the latency-bound atomics in flight.  The
// others take at most 64, so that 4 CTAs fit an SM: pull and push rounds are
// latency-bound too (256 R-MAT-21 SSSP queries: 118 ms at 4 CTAs/SM, 170 ms
// at the 2 a 128-register build allows, before pull units kept more loads in
// flight).
template <int W, int KIND, int PAIRS = kPairsOff>
__global__ void __launch_bounds__(256, PAIRS == kPairsList ? 6 : 4) batch_run_kernel(const BatchArgs a) {
  __shared__ int32_t sBound[32 * W];
  __shared__ unsigned sNear[W];
  __shared__ typename std::conditional<PAIRS == kPairsMask, PairSmem, char>::type sPairs;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  const long long gw = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  // list entries are dealt to warps block-first (warp k of every block, then
  // warp k+1), so a short list spreads over every SM
  const long long gwl = (long long)(threadIdx.x / 32) * gridDim.x + blockIdx.x;
  const size_t maskWords = (size_t)a.nVertices * W;
  const bool buckets = KIND == kBatchSSSP && a.delta > 0;
  const BatchBucket bk{buckets ? sBound : nullptr, buckets ? sNear : nullptr};
  int r = 0;
  for (;; ++r) {
    if (a.maxRounds > 0 && r >= a.maxRounds) break;
    if (buckets) {
      // this round's bounds: last round's, plus delta for the queries that
      // produced no value below theirs (every block computes the same)
      const int32_t *tPrev = (r & 1) ? a.thresh[1] : a.thresh[0];
      int32_t *tNext = (r & 1) ? a.thresh[0] : a.thresh[1];
      const unsigned *nPrev = a.nearFlag[(r + 2) % 3];  // written in round r - 1
      for (int q = threadIdx.x; q < 32 * W; q += blockDim.x) {
        int32_t t = __ldcg(tPrev + q);
        if (r > 0 && !((__ldcg(nPrev + q / 32) >> (q % 32)) & 1u)) t += a.delta;
        sBound[q] = t;
        if (blockIdx.x == 0) tNext[q] = t;
      }
      if (threadIdx.x < W) sNear[threadIdx.x] = 0u;
      if (blockIdx.x == 0 && threadIdx.x < W) a.nearFlag[(r + 1) % 3][threadIdx.x] = 0u;
      __syncthreads();
    }
    unsigned *cur = a.mask[r % 3];
    unsigned *nxt = a.mask[(r + 1) % 3];
    unsigned *clr = a.mask[(r + 2) % 3];
    const int rc = r % 3, rn = (r + 1) % 3;
    const int32_t *listCur = a.list[rc];
    const int32_t *listCurC = a.listC[rc];
    int32_t *listNext = a.list[rn];
    int32_t *listNextC = a.listC[rn];
    unsigned long long *cntNext = a.listCnt + rn;
    const unsigned long long lc = a.listCnt[rc];
    const long long nList = (long long)(lc >> 32);
    const long long eOut = (long long)(lc & 0xffffffffull);
    const bool push = a.pairMode || buckets || eOut * a.alpha <= (long long)a.nEdges;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.cnt[rn] = 0ull;
      a.listCnt[(r + 2) % 3] = 0ull;  // input of round r-1, appended in round r+1
    }
    if (!PAIRS)  // pair rounds from the mask clear the words they read
      for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < maskWords;
           i += (size_t)gridDim.x * blockDim.x)
        clr[i] = 0u;
    unsigned long long changed = 0ull;
    if constexpr (PAIRS == kPairsMask) {
      batch_pairs_round<W, KIND>(a, r, cur, nxt, sPairs, changed, bk);
    } else if constexpr (PAIRS == kPairsList) {
      batch_pair_list<W>(a, r, nList, cntNext, changed);
    } else if (push) {
      for (long long i = gwl; i < nList; i += warps)
        batch_push_unit<W, KIND>(a, listCur[i], listCurC[i], r, cur, nxt, listNext, listNextC,
                                 cntNext, changed, bk);
    } else {
      batch_pull_round<W, KIND>(a, gw, warps, r, cur, nxt, changed);
    }
    (void)clr;
    changed = warp_sum_u64(changed);
    if ((threadIdx.x & 31) == 0 && changed) atomicAdd(a.cnt + rc, changed);
    if (buckets) {
      __syncthreads();
      if (threadIdx.x < W && sNear[threadIdx.x]) atomicOr(a.nearFlag[rc] + threadIdx.x, sNear[threadIdx.x]);
    }
    if (!grid_barrier(a.barrier, a.errWord)) break;
    if (a.cnt[rc] == 0ull) break;  // uniform: read after the barrier
    if (!PAIRS && !push) {
      batch_compact<W>(a, nxt, listNext, listNextC, cntNext);
      if (!grid_barrier(a.barrier, a.errWord)) break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.roundsOut = r;
}

// value[V][Q] := BFS -1 / SSSP gatherZero; sources get 0 and their bit.
// thresh0 (may be null): every query's first bucket bound, delta.
static __global__ void batch_init_kernel(int kind, int32_t nVertices, int32_t Q, int32_t *value,
                                         int32_t *thresh0 = nullptr, int32_t delta = 0) {
  const size_t n = (size_t)nVertices * Q;
  const int32_t fill = kind == kBatchBFS ? -1 : kBatchInf;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    value[i] = fill;
  if (thresh0)
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < (size_t)Q;
         q += (size_t)gridDim.x * blockDim.x)
      thresh0[q] = delta;
}

// Sources: value 0, their query bit, and the first list (each source
// vertex once; inList was reset to -1).
// Pair batches keep their state query-major (value[q][v], mask and seen words
// [w][v]); the first pair list is (s_q, q) per query.
static __global__ void batch_sources_kernel(int kind, int32_t nQueries, int32_t Q, int32_t W,
                                            int32_t nVertices, const int32_t *sources, int32_t *value,
                                            unsigned *mask0, unsigned *seen,
                                            const int32_t *outOffsets, int32_t *inList,
                                            int32_t *list0, int32_t *list0C,
                                            unsigned long long *listCnt0, int pairMode = kPairsOff,
                                            uint32_t *pairs0 = nullptr) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nQueries) return;
  const int s = sources[q];
  if (pairMode != kPairsOff) {
    value[(size_t)q * nVertices + s] = 0;
    atomicOr(mask0 + (size_t)(q / 32) * nVertices + s, 1u << (q % 32));
    if (kind == kBatchBFS) atomicOr(seen + (size_t)(q / 32) * nVertices + s, 1u << (q % 32));
    if (pairMode == kPairsList) {
      const unsigned long long pos = atomicAdd(listCnt0, 1ull << 32) >> 32;
      pairs0[pos] = (uint32_t)s * (uint32_t)Q + (uint32_t)q;
    }
    return;
  }
  value[(size_t)s * Q + q] = 0;
  atomicOr(mask0 + (size_t)s * W + q / 32, 1u << (q % 32));
  if (kind == kBatchBFS) atomicOr(seen + (size_t)s * W + q / 32, 1u << (q % 32));
  if (atomicExch(inList + s, 0) != 0) {
    const unsigned d = (unsigned)(outOffsets[s + 1] - outOffsets[s]);
    const unsigned ne = d > 0u ? (d + kPushChunk - 1) / kPushChunk : 1u;
    const unsigned long long pos = atomicAdd(listCnt0, ((unsigned long long)ne << 32) | d) >> 32;
    for (unsigned c = 0; c < ne; ++c) {
      list0[pos + c] = s;
      list0C[pos + c] = (int32_t)c;
    }
  }
}

// out[q][v] = value[v][q] for q < nQueries (32x32 tiles through shared memory)
static __global__ void batch_transpose_kernel(const int32_t *value, int32_t nVertices, int32_t Q,
                                       int32_t nQueries, int32_t *out) {
  __shared__ int32_t tile[32][33];
  const int v0 = blockIdx.x * 32, q0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int v = v0 + j, q = q0 + threadIdx.x;
    tile[j][threadIdx.x] = (v < nVertices && q < Q) ? value[(size_t)v * Q + q] : 0;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int q = q0 + j, v = v0 + threadIdx.x;
    if (q < nQueries && v < nVertices) out[(size_t)q * nVertices + v] = tile[threadIdx.x][j];
  }
}

}  // namespace detail
}  // namespace gas

// The leading dense (pull) rounds of a run that starts with every vertex
// active, in a kernel of their own (see dense.cuh for what a dense round is),
// on graphs that keep its layout: where pull_pays, and memory is to spare.  The
// others take run_dense_csc_kernel (persistent.cuh).
//
// dense.cuh's pass spends its time on instructions and L1 wavefronts, not on
// bytes: finding a vertex's share of unaligned quads, testing a frontier bit
// per edge and combining lanes cost about 80 instructions an edge on
// PageRank R-MAT-20, and a warp's 32 gathers hit up to 32 lines.  Here
//
//   * the in-edges are laid out in slices (pullIds): a slice is a warp's
//     work, 32 vertices of at most 64 in-edges (a lane each), 4 vertices of
//     65..1024 (8 lanes each) or one 1024-edge chunk of a larger one, and
//     each of its steps is 32 consecutive int4, lane l's next source ids.
//     Vertices of neighbouring degree share a slice, so little is padding;
//     a step is one coalesced load, four values, four folds: no search, no
//     alignment cases, no shuffles;
//   * the values of the graph's hot sources -- the vertices of highest
//     out-degree, which hold 59 % (R-MAT-22) to 76 % (R-MAT-20) of the edges
//     -- and their frontier bits are in shared memory, where 32 random reads
//     take about 4 cycles: one CTA of 768 to 1,024 threads per SM, filled from
//     a compact array at the start of a round (at most 20 MB from L2 over the
//     chip).
//     pullIds holds a hot source as its table slot;
//   * bits of cold sources are tested only for vertices that no hot
//     in-neighbour has made active (the wide form tests them all at once);
//   * Programs that say gatherFromSource have gatherMap evaluated once per
//     source and round instead of once per edge (PageRank: an IEEE division,
//     and 4 bytes a gather instead of 8), and their vertex data updated in
//     place: gathers read the messages, which alternate between two buffers;
//   * vertices without in-edges are left out once both value buffers hold
//     their final value (half of R-MAT-22's vertices).
//
// Active sets, counts and the order of every reduction are dense.cuh's, so
// results do not depend on which of the two ran a round: a lane here walks
// the shares of one or more of dense.cuh's lanes one after the other and
// combines them as that pass's shuffles do (pull_ordered).  Programs that say
// reduceAnyOrder are spared that order: a lane folds what it reads
// (pull_any; PageRank R-MAT-22 would take 10.0 ms instead of 12.7 so, but
// with sums, and so activations, of its own).
//
// Measured (run(), GB300): PageRank R-MAT-22 (4.0 M vertices, 62 M edges, 50
// rounds) 19.6 -> 12.7 ms, R-MAT-20 5.1 -> 4.3; CC R-MAT-22 (128 M edges)
// 1.93 -> 1.49; SSSP R-MAT-18 0.50 -> 0.46, R-MAT-21 2.71 -> 2.00.  No unit
// is at its limit then (PageRank: L2 53 % busy on R-MAT-22, 30 % on R-MAT-20,
// DRAM 27 and 19 %): a lane has four values in flight.  Table size (PageRank
// R-MAT-22, any order): 64 KB 11.0 ms, 96 KB 10.2, 128 KB 10.0, 160 KB 10.7,
// 192 KB 15.8: what the table takes, L1 lacks for loads in flight.
#pragma once

#include "dense.cuh"

namespace gas {
namespace detail {

constexpr int kPullBatch = 2;                 // work units a warp takes at a time

// Lanes of a vertex of in-degree 65..kChunkEdges and 9..64.  Few lanes a
// vertex cost the fewest instructions; a graph with too few units for every
// warp takes as many as dense.cuh's pass (WIDE), as its rounds last as long
// as the longest chain of steps (SSSP, 9,001 vertices: 252 us a run narrow,
// 207 with dense.cuh's pass).
__host__ __device__ constexpr int pull_mid_lanes(bool wide) { return wide ? 32 : 8; }
__host__ __device__ constexpr int pull_small_lanes(bool wide) { return wide ? kSmallLanes : 1; }
// What the choice of a kernel goes by.
struct PullShape {
  bool anyOrder, messages;  // the Program's declarations
  int entry;                // bytes of a source value
  bool carried;             // the slices carry the edge data (or there is none)
  long long nVertices, nEdges, maxOut;
  long long narrowUnits;    // chunks, mid / 4, small / 32
};
// Out-degrees of one size (random graphs, lattices): no few sources hold most
// of the edges.
inline bool pull_even(const PullShape &p) { return p.maxOut * p.nVertices < 16 * p.nEdges; }

// The wide form: fewer narrow units than two for each warp of the chip (152
// SMs of 28, the middle of 24 to 32), than one for Programs that reduce in any
// order, whose narrow units are the shorter chains.  Measured at one and at
// two (run(), us): SSSP, R-MAT of 300,000 vertices 414, 472, 200,000 332, 369,
// 100,000 281, 279; CC 300,000 144, 162; PageRank 400,000 1744, 1598, 200,000
// and 1,000,000 the same.  On even graphs the table answers little, the wide
// form's bit tests are gathers too, and a third of a unit is enough (random
// graphs, CSC, narrow, wide: CC, 70,000 vertices, 840,000 edges 126, 97, 140,
// 40,000, 640,000 74, 60, 66, 1,600,000 74, 74, 70, 20,000, 320,000 60, 56,
// 48; PageRank, 100,000, 1.6 M 484, 316, 500, 40,000, 1.6 M 406, 351, 287).
inline bool pull_wide(const PullShape &p) {
  return p.narrowUnits < (pull_even(p) ? 152ll * 10 : (p.anyOrder ? 1ll : 2ll) * 152 * 28);
}
// Whether the layout pays, `slices` slices of the form pull_wide chose.
//
// Programs that declare nothing pull whole vertices and keep dense.cuh's
// order: there only rounds short of units gain, on which a warp has few chains
// to run one after the other, and values that a lane can hold; edge data that
// the slices do not carry costs an access of its own an edge.  run() of ten
// rounds (PageRank thirty), CSC -> wide form, us, 8-byte values unless stated:
// PageRank R-MAT-14 570 -> 380, R-MAT-17 symmetric (20,688 slices) 1080 ->
// 1035, R-MAT-20 (108,595) 3011 -> 3973 (narrow form 4133), lattice 500 x 500
// (7,808) 304 -> 292, 700 x 700 (15,305) 420 -> 443; 256-byte values, R-MAT-17
// symmetric 1280 -> 1688; 8-byte edge data, R-MAT-14 (1,755) 234 -> 132,
// lattice 200 x 200 (1,250) 95 -> 72, 350 x 350 (3,827) 120 -> 124 to 131, 500
// x 500 154 -> 165.
//
// Minima on even graphs of 2 to 3.5 edges a vertex: the layout moves 48 bytes
// a vertex and round where the CSC moves 34, which shows once they leave L2
// (CC, 200 rounds, CSC -> layout, ms: lattice 1400 x 1400 9.9 -> 9.8, 1500 x
// 1500 10.5 -> 11.8, 2000 x 2000 19.9 -> 23.0; random, 2 edges a vertex, 2 M
// vertices 1.60 -> 1.72, 5 M 3.40 -> 3.84; 4 edges, 5 M 2.91 -> 2.71).  Sums
// have a division an edge to spare (PageRank 2000 x 2000 2.34 -> 2.32).
// Programs that gather vertex data are not even paid for smaller ones: a
// shortest-path run has one dense round there, after which L2 holds the layout
// in place of the CSC that the list rounds read (SSSP, random, 2 edges a vertex,
// 700,000 vertices 1172 -> 1230 us, 1 M 1285 -> 1395; 4 edges, 1 M 1473 ->
// 1524; 6 edges the same, lattice 1000 x 1000, 200 rounds, 922 -> 926).
inline bool pull_pays(const PullShape &p, bool wide, long long slices) {
  if (p.anyOrder && pull_even(p) &&
      (p.messages ? p.nVertices >= 2000000 && 2 * p.nEdges < 7 * p.nVertices
                  : p.nVertices >= 500000 && p.nEdges < 6 * p.nVertices))
    return false;
  if (p.anyOrder || p.messages) return true;
  return wide && p.entry <= 32 && slices <= (p.carried ? 4ll : 1ll) * 152 * 24;
}
constexpr int kHotBytes = GAS_PULL_HOT_BYTES; // shared memory for hot values
constexpr int kNoEdge = (int)0x80000000;      // stands for no edge: table slot 0, which no vertex has

// Programs whose gatherMap depends on the source's VertexData alone (neither
// on the destination nor on the edge) may declare
//   static constexpr bool gatherFromSource = true;
template <class P>
struct ProgramGatherFromSource {
  template <class Q>
  static auto test(int) -> std::integral_constant<bool, Q::gatherFromSource>;
  template <class Q>
  static std::false_type test(...);
  static constexpr bool value = decltype(test<P>(0))::value;
};

// Programs whose gatherReduce gives the same bits in any order (a minimum, a
// sum of whole numbers) may declare
//   static constexpr bool reduceAnyOrder = true;
template <class P>
struct ProgramReduceAnyOrder {
  template <class Q>
  static auto test(int) -> std::integral_constant<bool, Q::reduceAnyOrder>;
  template <class Q>
  static std::false_type test(...);
  static constexpr bool value = decltype(test<P>(0))::value;
};

// What a gather reads per source: the message (gatherMap's result) or the
// source's vertex data.  Messages use the two spare vertex buffers.
template <class P>
struct PullSource {
  typedef typename P::VertexData VD;
  typedef typename P::GatherResult GR;
  static constexpr bool kMessage = ProgramGatherFromSource<P>::value && sizeof(GR) <= sizeof(VD) &&
                                   alignof(GR) <= alignof(VD);
  typedef typename std::conditional<kMessage, GR, VD>::type type;
};

// Threads of the CTA, by the registers a thread needs (SSSP R-MAT-18 0.54 ms
// at 1,024 threads and 88 bytes of spills, 0.45 at 896 without; PageRank's 100
// bytes at 896 and CC's 40 at 1,024 cost less than the warps are worth:
// narrower blocks were up to 17 % slower).  The wide form keeps more: of 640, 768 and 896 threads (none spills at 768), 768 is 1 to 2 %
// ahead over R-MAT graphs of 4,096..150,000 vertices (PageRank 60,000: 644,
// 564, 619 us; 9,001: 386, 390, 416).
constexpr int kWideThreads = 768;
template <class P, bool WIDE>
struct PullThreads {
  static constexpr int value =
      WIDE ? kWideThreads : (ProgramReduceAnyOrder<P>::value ? 896 : 768) + (PullSource<P>::kMessage ? 128 : 0);
};

// The table's entries for values of `bytes` bytes: whole bitmap words.
__host__ __device__ constexpr int pull_hot_capacity(int bytes) { return kHotBytes / bytes / 128 * 128; }

// The hot vertices: as many whole degree classes of at least kHotMinOut as fit
// `most` slots.  deg(k): the out-degree of the k-th of nV vertices sorted by
// min(out-degree, kHotDegreeCap), the largest first (the sort's keys have 16
// bits; equal keys come by vertex id).  The cut is made on those capped
// degrees alone, so that the first `count` vertices are the ones of
// out-degree >= minOut: pull_finish tells a hot vertex by its degree.  Where
// more than `most` reach the cap, none is hot.
constexpr int kHotDegreeCap = 65535;
struct HotCut {
  int count, minOut;
};
template <class Deg>
__host__ __device__ inline HotCut hot_cut(const Deg &deg, int nV, int most, int least) {
  auto capped = [&](int k) {
    const int d = deg(k);
    return d < kHotDegreeCap ? d : kHotDegreeCap;
  };
  int minOut = nV > most ? capped(most) + 1 : 1;
  if (minOut > kHotDegreeCap) return {0, 0x7fffffff};
  if (minOut < least) minOut = least;
  int lo = 0, hi = nV < most ? nV : most;  // the first k of a smaller degree
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (capped(mid) >= minOut)
      lo = mid + 1;
    else
      hi = mid;
  }
  return {lo, minOut};
}

// Shared memory of a table of nHot slots (slot 0 included): the values, then
// their bits.  A launch takes what its graph's table needs; what it leaves is
// L1 for the other gathers.
template <class P>
__host__ __device__ constexpr size_t pull_table_bytes(int nHot) {
  return ((size_t)nHot * sizeof(typename PullSource<P>::type) + 15) / 16 * 16;
}
template <class P>
constexpr size_t pull_smem_bytes(int nHot) {
  return pull_table_bytes<P>(nHot) + (size_t)(nHot + 31) / 32 * 4;
}

// What changes from round to round, in shared memory: finishing a vertex
// reads it there (volatile), so that it takes no registers in the edge loops.
template <class P>
struct PullRound {
  typedef typename PullSource<P>::type Src;
  const Src *cur;   // source values of the previous round's end
  Src *next;
  Src *hotNext;     // the compact copy of the hot vertices' values
  const uint32_t *prevBits;
  uint32_t *curBits;
  uint32_t *hotBits;  // this round's bits of the hot vertices, by slot
  unsigned long long *cnt;
  int32_t iteration;
};

// The edge loops' own part.
template <class P>
struct PullCtx {
  typedef typename PullSource<P>::type Src;
  const Src *cur;
  const Src *hot;           // shared memory
  const uint32_t *hotPrev;  // shared memory
  const volatile PullRound<P> *round;
  bool allActive;
};

template <class P>
struct PullQuadEd {  // gatherMap reads 4-byte edge data
  static constexpr bool value = QuadEdgeData<P>::value && !PullSource<P>::kMessage;
};

template <class P>
__device__ __forceinline__ bool hot_bit(const PullCtx<P> &a, int s) {
  const int k = s & 0x7fffffff;
  return (a.hotPrev[k >> 5] >> (k & 31)) & 1u;
}

// The value of source s, from the table or from global memory: one generic
// load (a branch, or a predicated load from either space, costs more).
template <class P>
__device__ __forceinline__ typename PullSource<P>::type source_value(const PullCtx<P> &a, int s) {
  typedef typename PullSource<P>::type Src;
  const Src *p = (s < 0 ? a.hot : a.cur) + (s & 0x7fffffff);
  if constexpr (sizeof(Src) == 4) {
    uint32_t w;
    asm volatile("ld.u32 %0, [%1];" : "=r"(w) : "l"(p));
    Src v;
    memcpy(&v, &w, 4);
    return v;
  } else {
    return *p;
  }
}

// gatherMap of one in-edge of v whose source value is s.
template <class P>
__device__ __forceinline__ typename P::GatherResult
pull_map(const PullCtx<P> &a, int v, const typename PullSource<P>::type &s, const typename P::EdgeData *ep) {
  if constexpr (PullSource<P>::kMessage)
    return s;
  else
    return P::gatherMap(a.cur + v, &s, ep);
}

template <int W>
__device__ __forceinline__ bool group_any(bool p) {
  if constexpr (W == 32) {
    return __any_sync(kFullMask, p);
  } else {
    const unsigned b = __ballot_sync(kFullMask, p);
    return ((b >> ((threadIdx.x & 31) / W * W)) & ((1u << W) - 1u)) != 0u;
  }
}

// One work unit: its first int4, its longest vertex's aligned quads (in any
// order, and in the last class: its steps), and this lane's vertex.
struct PullUnit {
  int base, quads;
  int4 rec;  // vertex (-1: none), CSC begin, edges (of the chunk or vertex), out-degree
};

// The CSC range [beg, beg + len) as dense.cuh's group_edges splits it: `head`
// edges, `quads` aligned quads from quad `first` on, `tail` edges.
struct PullRange {
  int head, tail, first, quads;
};
__host__ __device__ __forceinline__ PullRange pull_range(int beg, int len) {
  PullRange r;
  const int end = beg + len;
  r.first = (beg + 3) >> 2;
  const int qe = end >> 2;
  r.quads = qe > r.first ? qe - r.first : 0;
  const int h = (4 - (beg & 3)) & 3;
  r.head = h < len ? h : len;
  r.tail = len - r.head - 4 * r.quads;
  return r;
}

// Steps of virtual lane k (of every real lane) in a unit of `quads` quads:
// quads k, k + LAYER, ... of its first real lane.
template <int LAYER>
__host__ __device__ __forceinline__ int pull_layers(int quads, int k) {
  return quads > k ? (quads - k + LAYER - 1) / LAYER : 0;
}

// Whether an in-neighbour of this lane's vertex has its bit set among the
// cold sources of the unit's `steps` steps (the ids again, from L2).
template <class P, int W>
__device__ __forceinline__ bool pull_cold(const PullCtx<P> &a, const gas_run_args &ra, const PullUnit &x, int steps,
                                          bool hit) {
  const int4 *ids = static_cast<const int4 *>(ra.pullIds) + x.base + (threadIdx.x & 31);
  const uint32_t *bits = a.round->prevBits;
  for (int t = 0; t < steps; ++t) {
    const int4 s4 = __ldg(ids + 32 * t);
    const int s[4] = {s4.x, s4.y, s4.z, s4.w};
    if (!hit) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (!hit && s[j] >= 0) hit = bit_test(bits, s[j]);
    }
    if constexpr (W > 1) hit = group_any<W>(hit);
    if (__all_sync(kFullMask, hit)) break;
  }
  return hit;
}

// One step of a lane: four ids, their values on the way, edge data, and the
// next step's ids in flight.
template <class P>
struct PullStep {
  typedef typename PullSource<P>::type Src;
  Src sv[4];
  int wt[PullQuadEd<P>::value ? 4 : 1];
};

// Loads the step whose ids are s4 (its values; its edge data from *eds),
// tests its hot sources' bits while some vertex of the warp is not known to
// be active, then fetches the next ids if there are any.
template <class P, int W, bool WIDE>
__device__ __forceinline__ void pull_step(const PullCtx<P> &a, const gas_run_args &ra, int4 &s4, const int4 *&ids,
                                          const int4 *&eds, bool more, bool &hit, bool &allHit, PullStep<P> &x) {
  const int s[4] = {s4.x, s4.y, s4.z, s4.w};
  if (ra.g.haveGather) {
#pragma unroll
    for (int j = 0; j < 4; ++j) x.sv[j] = source_value<P>(a, s[j]);
  }
  if constexpr (PullQuadEd<P>::value) {
    const int4 w4 = __ldg(eds);
    x.wt[0] = w4.x;
    x.wt[1] = w4.y;
    x.wt[2] = w4.z;
    x.wt[3] = w4.w;
    eds += 32;
  }
  if (!allHit) {
    if (!hit) {
      bool h = false;
      if constexpr (WIDE) {  // hot and cold ones alike, in flight with the values
        const uint32_t *bits = a.round->prevBits;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int k = s[j] & 0x7fffffff;
          h |= ((s[j] < 0 ? a.hotPrev : bits)[k >> 5] >> (k & 31)) & 1u;  // slot 0's bit is never set
        }
      } else if (ra.nHot > 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) h = h || (s[j] < 0 && hot_bit<P>(a, s[j]));
      } else {  // no hot sources (a lattice): pull_cold would find them all
        const uint32_t *bits = a.round->prevBits;
#pragma unroll
        for (int j = 0; j < 4; ++j) h |= s[j] >= 0 && bit_test(bits, s[j]);
      }
      hit = h;
    }
    if constexpr (W > 1) hit = group_any<W>(hit);
    allHit = __all_sync(kFullMask, hit);
  }
  ids += 32;
  if (more) s4 = __ldg(ids);
}

// gatherMap of edge j of a step; pos: its CSC position.
template <class P>
__device__ __forceinline__ typename P::GatherResult pull_edge(const PullCtx<P> &a, const gas_run_args &ra, int v,
                                                              const PullStep<P> &x, int j, int pos) {
  typedef typename P::EdgeData ED;
  if constexpr (PullQuadEd<P>::value) {
    ED e;
    memcpy(&e, &x.wt[j], sizeof(ED));
    return pull_map<P>(a, v, x.sv[j], &e);
  } else if constexpr (PullSource<P>::kMessage) {
    return pull_map<P>(a, v, x.sv[j], nullptr);
  } else {
    return pull_map<P>(a, v, x.sv[j], edge_ptr<P>(ra.g.edgeData, pos));
  }
}

// In-degree <= 8, one lane a vertex: a left fold from gatherZero.
template <class P, bool WIDE>
__device__ __forceinline__ bool pull_serial(const PullCtx<P> &a, const gas_run_args &ra, const PullUnit &u, int4 s4,
                                            EdgeAcc<typename P::GatherResult> &x) {
  const int lane = threadIdx.x & 31, v = u.rec.x;
  bool hit = a.allActive || v < 0;
  bool allHit = __all_sync(kFullMask, hit);
  const int4 *ids = static_cast<const int4 *>(ra.pullIds) + u.base + lane;
  const int4 *eds = static_cast<const int4 *>(ra.pullEds) + u.base + lane;
  for (int t = 0; t < u.quads; ++t) {  // warp-uniform
    PullStep<P> st;
    pull_step<P, 1, WIDE>(a, ra, s4, ids, eds, t + 1 < u.quads, hit, allHit, st);
    if (ra.g.haveGather) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (4 * t + j < u.rec.z)
          x.val = P::gatherReduce(x.val, pull_edge<P>(a, ra, v, st, j, u.rec.y + 4 * t + j));
    }
  }
  if (!WIDE && !allHit && ra.nHot > 1) hit = pull_cold<P, 1>(a, ra, u, u.quads, hit);
  return hit;
}

// W lanes a vertex, the quads of its in-edges dealt round-robin, folded as
// they come.
template <class P, int W, bool WIDE>
__device__ __forceinline__ bool pull_any(const PullCtx<P> &a, const gas_run_args &ra, const PullUnit &u, int sl,
                                         int4 s4, EdgeAcc<typename P::GatherResult> &x) {
  const int lane = threadIdx.x & 31, v = u.rec.x;
  bool hit = a.allActive || v < 0;
  bool allHit = __all_sync(kFullMask, hit);
  const int4 *ids = static_cast<const int4 *>(ra.pullIds) + u.base + lane;
  const int4 *eds = static_cast<const int4 *>(ra.pullEds) + u.base + lane;
  int rem = u.rec.z - 4 * sl;  // edges from the lane's next one on
  x.has = ra.g.haveGather && rem > 0 ? 1u : 0u;
  for (int t = 0; t < u.quads; ++t, rem -= 4 * W) {  // warp-uniform
    PullStep<P> st;
    pull_step<P, W, WIDE>(a, ra, s4, ids, eds, t + 1 < u.quads, hit, allHit, st);
    if (ra.g.haveGather) {
      const int pos = u.rec.y + u.rec.z - rem;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < rem) {
          const typename P::GatherResult m = pull_edge<P>(a, ra, v, st, j, pos + j);
          x.val = t == 0 && j == 0 ? m : P::gatherReduce(x.val, m);
        }
    }
  }
  if (!WIDE && !allHit && ra.nHot > 1) hit = pull_cold<P, W>(a, ra, u, u.quads, hit);
  return hit;
}

// W lanes a vertex, each taking VL consecutive ones of the W * VL lanes that
// group_edges gives it: per such lane its unaligned edge if it has one, then
// its quads, then the lanes' results combined in pairs, pairs of pairs, ...
// x: the lane's result; returns whether its vertex is active (group-uniform).
template <class P, int W, int VL, bool WIDE>
__device__ __forceinline__ bool pull_ordered(const PullCtx<P> &a, const gas_run_args &ra, const PullUnit &u, int sl,
                                             int4 s4, EdgeAcc<typename P::GatherResult> &x) {
  typedef typename P::GatherResult GR;
  constexpr int LAYER = W * VL;
  constexpr int ENDS = VL == 8 ? 2 : 1;
  const int lane = threadIdx.x & 31;
  const int v = u.rec.x;
  const PullRange rg = pull_range(u.rec.y, u.rec.z);
  bool hit = a.allActive || v < 0;
  bool allHit = __all_sync(kFullMask, hit);
  const int4 *ids = static_cast<const int4 *>(ra.pullIds) + u.base + lane;
  const int4 *eds = static_cast<const int4 *>(ra.pullEds) + u.base + lane;
  // the unaligned edges of this lane's share: VL 8 the head, then the tail
  // (its lanes 4..6); VL 4 the head for the first lane, the tail for the
  // second; VL 1 one edge of either
  GR ends[ENDS][VL == 1 ? 1 : 3];
  int nEnds[ENDS];
  const int tailPos = (u.rec.y + u.rec.z) & ~3;
#pragma unroll
  for (int h = 0; h < ENDS; ++h) {
    int pos;
    if constexpr (VL == 8) {
      nEnds[h] = h == 0 ? rg.head : rg.tail;
      pos = h == 0 ? u.rec.y : tailPos;
    } else if constexpr (VL == 4) {
      nEnds[h] = sl == 0 ? rg.head : sl == 1 ? rg.tail : 0;
      pos = sl == 0 ? u.rec.y : tailPos;
    } else {
      nEnds[h] = sl < 4 ? sl < rg.head : sl - 4 < rg.tail;
      pos = sl < 4 ? u.rec.y + sl : tailPos + sl - 4;
    }
    PullStep<P> st;
    pull_step<P, W, WIDE>(a, ra, s4, ids, eds, h + 1 < ENDS || u.quads > 0, hit, allHit, st);
    if (ra.g.haveGather) {
#pragma unroll
      for (int j = 0; j < (VL == 1 ? 1 : 3); ++j)
        if (j < nEnds[h]) ends[h][j] = pull_edge<P>(a, ra, v, st, j, pos + j);
    }
  }
  int left = 0;  // quad steps to come (warp-uniform)
#pragma unroll
  for (int k = 0; k < VL; ++k) left += pull_layers<LAYER>(u.quads, k);
  const int steps = ENDS + left;
  GR part[3];           // combined lanes waiting for their right neighbour
  unsigned parts = 0u;  // which of them hold a value
#pragma unroll
  for (int k = 0; k < VL; ++k) {
    GR acc;
    bool has = false;
    const int h = VL == 8 ? k / 4 : 0, j0 = VL == 8 ? k % 4 : k;
    if (j0 < (VL == 1 ? 1 : 3)) {
      has = j0 < nEnds[h] && ra.g.haveGather;
      if (has) acc = ends[h][j0 < 3 && VL != 1 ? j0 : 0];
    }
    const int layers = pull_layers<LAYER>(u.quads, k);
    int q = sl * VL + k;
#pragma unroll 1
    for (int l = 0; l < layers; ++l, q += LAYER) {  // warp-uniform
      PullStep<P> st;
      pull_step<P, W, WIDE>(a, ra, s4, ids, eds, --left > 0, hit, allHit, st);
      if (q < rg.quads && ra.g.haveGather) {
        const int pos = 4 * (rg.first + q);
        const GR m = pull_edge<P>(a, ra, v, st, 0, pos);
        acc = has ? P::gatherReduce(acc, m) : m;
        has = true;
#pragma unroll
        for (int j = 1; j < 4; ++j) acc = P::gatherReduce(acc, pull_edge<P>(a, ra, v, st, j, pos + j));
      }
    }
    // k's result joins those waiting on its left: one level per trailing 1 bit
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if ((1 << d) >= VL) break;
      if ((k >> d) & 1) {
        if ((parts >> d) & 1u) {
          acc = has ? P::gatherReduce(part[d], acc) : part[d];
          has = true;
        }
        parts &= ~(1u << d);
      } else {
        part[d] = acc;
        parts |= (has ? 1u : 0u) << d;
        break;
      }
    }
    if (k == VL - 1) {
      x.val = acc;
      x.has = has ? 1u : 0u;
    }
  }
  if (!WIDE && !allHit && ra.nHot > 1) hit = pull_cold<P, W>(a, ra, u, steps, hit);
  return hit;
}

// Ordered tree combine within aligned groups of W lanes, as dense.cuh's
// group_reduce; which lanes hold a value comes from one ballot.
template <class P, int W>
__device__ __forceinline__ void pull_combine(EdgeAcc<typename P::GatherResult> &x) {
  const int lane = threadIdx.x & 31;
  const unsigned has = __ballot_sync(kFullMask, x.has != 0u);
#pragma unroll
  for (int d = 1; d < W; d <<= 1) {
    const typename P::GatherResult ov = shfl_down_any_w(x.val, d, W);
    if ((lane & (2 * d - 1)) == 0 && ((has >> (lane + d)) & ((1u << d) - 1u)) != 0u) {
      x.val = x.has ? P::gatherReduce(x.val, ov) : ov;
      x.has = 1u;
    }
  }
}

template <class P>
__device__ __forceinline__ typename P::VertexData pull_own(const PullCtx<P> &a, const gas_run_args &ra, int v) {
  if constexpr (PullSource<P>::kMessage)
    return static_cast<const typename P::VertexData *>(ra.g.vertexData)[v];
  else
    return a.cur[v];
}

// apply() for vertex v (own: its vertex data) and its source value for the
// next round.
template <class P>
__device__ __forceinline__ void pull_finish(const PullCtx<P> &a, const gas_run_args &ra, int v, int inDeg,
                                            int outDeg, bool active, const typename P::GatherResult &g,
                                            typename P::VertexData own, DenseCounts &c) {
  typedef typename P::VertexData VD;
  typedef typename PullSource<P>::type Src;
  const bool isHot = outDeg >= ra.hotMinOut;
  const int slot = isHot ? __ldg(ra.slotOf + v) : 0;
  if (active) {
    const bool r = do_apply<P>(&own, g, a.round->iteration);
    ++c.active;
    c.inEdges += (unsigned)inDeg;
    if (r) {
      bit_set(a.round->curBits, v);
      if (isHot) bit_set(a.round->hotBits, slot);
      ++c.ret;
      c.outEdges += (unsigned)outDeg;
    }
  }
  if constexpr (PullSource<P>::kMessage) {
    if (active) static_cast<VD *>(ra.g.vertexData)[v] = own;
    if (outDeg == 0) return;  // nobody reads its message
    const Src s = active ? P::gatherMap(&own, &own, nullptr) : a.cur[v];
    a.round->next[v] = s;
    if (isHot) a.round->hotNext[slot] = s;
  } else {
    a.round->next[v] = own;
    if (isHot) a.round->hotNext[slot] = own;
  }
}

// Work units of a pass, heaviest first: chunks of large vertices, then slices
// of mid, small and tiny ones.
struct PullUnits {
  int chunks, mid, small, total;  // first unit past each class; below V + E / kChunkEdges
  int tiny;                       // vertices of the last class
};

template <bool WIDE>
__device__ __forceinline__ PullUnit pull_fetch(const gas_run_args &ra, const volatile PullUnits &n, int u) {
  const int lane = threadIdx.x & 31;
  PullUnit x;
  const int2 at = __ldg(reinterpret_cast<const int2 *>(ra.pullSlices) + u);
  x.base = at.x;
  x.quads = at.y;
  const int4 *rec = reinterpret_cast<const int4 *>(ra.pullRec) + ra.nChunkVertices;
  int i, count;
  if (u < n.chunks) {
    rec = reinterpret_cast<const int4 *>(ra.chunkRec);
    i = u;
    count = ra.nChunks;
  } else if (u < n.mid) {
    i = (u - n.chunks) * (32 / pull_mid_lanes(WIDE)) + lane / pull_mid_lanes(WIDE);
    count = ra.nMid;
  } else if (u < n.small) {
    rec += ra.nMid;
    i = (u - n.mid) * (32 / pull_small_lanes(WIDE)) + lane / pull_small_lanes(WIDE);
    count = ra.nSmall;
  } else {
    rec += ra.nMid + ra.nSmall;
    i = (u - n.small) * 32 + lane;
    count = n.tiny;
  }
  x.rec = i < count ? __ldg(rec + i) : make_int4(-1, 0, 0, 0);
  // its ids into L2 while the present unit runs (a step is 512 bytes; the
  // unit ends where the next begins)
  const int end = __ldg(reinterpret_cast<const int2 *>(ra.pullSlices) + u + 1).x;
  const int4 *ids = static_cast<const int4 *>(ra.pullIds);
  for (int k = x.base + 8 * lane; k < end; k += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(ids + k));
  return x;
}

template <class P, bool WIDE>
__device__ __forceinline__ void pull_unit(const PullCtx<P> &a, const gas_run_args &ra, const volatile PullUnits &n,
                                          int u, const PullUnit &pu, int4 s4, DenseCounts &c) {
  typedef typename P::GatherResult GR;
  constexpr bool kAny = ProgramReduceAnyOrder<P>::value;
  const int lane = threadIdx.x & 31;
  const GR gz = P::gatherZero;
  const int v = pu.rec.x, len = pu.rec.z, outDeg = pu.rec.w;
  EdgeAcc<GR> x;
  x.has = 0u;
  x.act = 0u;
  x.val = gz;
  if (u >= n.chunks) {
    bool act, mine = v >= 0;
    typename P::VertexData own;  // on its way while the edges are gathered
    if (mine) own = pull_own<P>(a, ra, v);
    if (u >= n.small) {
      act = pull_serial<P, WIDE>(a, ra, pu, s4, x);
    } else {
      constexpr int M = pull_mid_lanes(WIDE), S = pull_small_lanes(WIDE);
      if (u >= n.mid) {
        if constexpr (kAny)
          act = pull_any<P, S, WIDE>(a, ra, pu, lane % S, s4, x);
        else
          act = pull_ordered<P, S, kSmallLanes / S, WIDE>(a, ra, pu, lane % S, s4, x);
        if (S > 1 && ra.g.haveGather) pull_combine<P, S>(x);
        mine = mine && lane % S == 0;
      } else {
        if constexpr (kAny)
          act = pull_any<P, M, WIDE>(a, ra, pu, lane % M, s4, x);
        else
          act = pull_ordered<P, M, 32 / M, WIDE>(a, ra, pu, lane % M, s4, x);
        if (ra.g.haveGather) pull_combine<P, M>(x);
        mine = mine && lane % M == 0;
      }
      x.val = x.has ? P::gatherReduce(gz, x.val) : gz;
    }
    if (mine) pull_finish<P>(a, ra, v, len, outDeg, act, x.val, own, c);
    return;
  }
  {
    bool act;
    if constexpr (kAny)
      act = pull_any<P, 32, WIDE>(a, ra, pu, lane, s4, x);
    else
      act = pull_ordered<P, 32, 1, WIDE>(a, ra, pu, lane, s4, x);
    // a chunk publishes its partial; the vertex's last to arrive combines
    const int ch = u;
    if (ra.g.haveGather) pull_combine<P, 32>(x);
    unsigned last = 0u;
    if (lane == 0) {
      if (x.has) reinterpret_cast<GR *>(ra.chunkVal)[ch] = x.val;
      ra.chunkFlags[ch] = x.has | (act ? 2u : 0u);
      __threadfence();
      const unsigned prev = atomicAdd(ra.chunkArrive + ra.chunkSlot[ch], 1u);
      last = (prev + 1 == (unsigned)ra.chunkCount[ch]) ? 1u : 0u;
      if (last) __threadfence();
    }
    last = __shfl_sync(kFullMask, last, 0);
    if (!last) return;
    const int first = ra.chunkFirst[ch], count = ra.chunkCount[ch];
    EdgeAcc<GR> tot;
    tot.has = 0u;
    tot.act = 0u;
    tot.val = gz;
    for (int c0 = 0; c0 < count; c0 += 32) {
      EdgeAcc<GR> y;
      y.has = 0u;
      y.act = 0u;
      y.val = gz;
      if (c0 + lane < count) {
        const unsigned f = __ldcg(ra.chunkFlags + first + c0 + lane);
        y.has = f & 1u;
        y.act = (f >> 1) & 1u;
        if (y.has) y.val = load_cg(reinterpret_cast<const GR *>(ra.chunkVal) + first + c0 + lane);
      }
      group_reduce<P, 32>(y);
      if (lane == 0) {
        tot.act |= y.act;
        if (y.has) {
          tot.val = tot.has ? P::gatherReduce(tot.val, y.val) : y.val;
          tot.has = 1u;
        }
      }
    }
    if (lane == 0) {
      ra.chunkArrive[ra.chunkSlot[ch]] = 0u;  // ready for the next dense round
      const GR g = (ra.g.haveGather && tot.has) ? P::gatherReduce(gz, tot.val) : gz;
      pull_finish<P>(a, ra, v, ra.g.inOffsets[v + 1] - ra.g.inOffsets[v], outDeg, tot.act != 0u || a.allActive, g,
                     pull_own<P>(a, ra, v), c);
    }
  }
}

// The units of a pass over the first nTiny vertices of the last class.
template <bool WIDE>
__host__ __device__ __forceinline__ PullUnits pull_units(const gas_run_args &ra, int nTiny) {
  constexpr int M = 32 / pull_mid_lanes(WIDE), S = 32 / pull_small_lanes(WIDE);
  PullUnits n;
  n.chunks = ra.nChunks;
  n.mid = n.chunks + (ra.nMid + M - 1) / M;
  n.small = n.mid + (ra.nSmall + S - 1) / S;
  n.total = n.small + (nTiny + 31) / 32;
  n.tiny = nTiny;
  return n;
}

// A warp's first unit and its ids.  They are the same in every round; the
// wide form, whose rounds are a chain of few loads, keeps them in shared
// memory (in registers they were spilled, and local memory is an L2 round
// trip once a barrier has invalidated L1).
struct PullFirst {
  PullUnit unit;
  int4 ids;
};
template <int NT>
struct PullKept {
  int4 rec[NT], ids[NT];
  int2 at[NT];
};
template <int NT>
__device__ __forceinline__ void keep_first(PullKept<NT> &k, const PullFirst &f) {
  k.rec[threadIdx.x] = f.unit.rec;
  k.ids[threadIdx.x] = f.ids;
  k.at[threadIdx.x] = make_int2(f.unit.base, f.unit.quads);
}
template <int NT>
__device__ __forceinline__ PullFirst kept_first(const PullKept<NT> &k) {
  const int2 at = k.at[threadIdx.x];
  return {{at.x, at.y, k.rec[threadIdx.x]}, k.ids[threadIdx.x]};
}
template <bool WIDE>
__device__ __forceinline__ PullFirst pull_first(const gas_run_args &ra, const volatile PullUnits &n, int u) {
  PullFirst f = {{0, 0, make_int4(-1, 0, 0, 0)}, make_int4(kNoEdge, kNoEdge, kNoEdge, kNoEdge)};
  if (u < n.total) {
    f.unit = pull_fetch<WIDE>(ra, n, u);
    // (every unit but those of vertices without in-edges has a first step)
    if (u < n.small || f.unit.quads > 0)
      f.ids = __ldg(static_cast<const int4 *>(ra.pullIds) + f.unit.base + (threadIdx.x & 31));
  }
  return f;
}
__device__ __forceinline__ int pull_first_unit() {
  return (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x;
}

// One dense pass, heaviest units first.  The first three quarters are dealt
// round-robin, block-first (neighbouring units, of similar weight, to
// different SMs), the rest taken kPullBatch at a time from a counter; the
// next unit and its first ids, and the next batch, are fetched one unit
// ahead.
template <class P, bool WIDE>
__device__ DenseCounts pull_pass(const PullCtx<P> &a, const gas_run_args &ra, const volatile PullUnits &n,
                                 const PullKept<WIDE ? kWideThreads : 1> &kept) {
  DenseCounts c = {0u, 0u, 0u, 0u};
  const int lane = threadIdx.x & 31;
  const int warps = (int)(gridDim.x * (blockDim.x / 32));
  // units below it are dealt; all, where the warps have few each: their
  // requests to one counter would take longer than the imbalance costs (CC
  // on a 400 x 400 lattice, one unit a warp: 11.9 us a round with them)
  const int dealt = n.total < 4 * warps ? 4 * warps : n.total / 4 * 3 / warps * warps;
  int u = pull_first_unit();
  const PullUnit noUnit = {0, 0, make_int4(-1, 0, 0, 0)};
  PullFirst f;
  if constexpr (WIDE)
    f = kept_first(kept);
  else
    f = pull_first<WIDE>(ra, n, u);
  PullUnit pu = f.unit;
  int4 s4 = f.ids;
  int next = n.total;  // lane 0: the next batch, asked for one unit early
  if (lane == 0 && u + warps >= dealt && dealt < n.total)
    next = dealt + kPullBatch * (int)atomicAdd(a.round->cnt + 2, 1ull);
  while (u < n.total) {
    int un;
    if (u + warps < dealt) {
      un = u + warps;
      if (lane == 0 && un + warps >= dealt && dealt < n.total)
        next = dealt + kPullBatch * (int)atomicAdd(a.round->cnt + 2, 1ull);
    } else if (u >= dealt && (u - dealt) % kPullBatch != kPullBatch - 1) {
      un = u + 1;
    } else {
      un = __shfl_sync(kFullMask, next, 0);
      if (lane == 0 && un < n.total) next = dealt + kPullBatch * (int)atomicAdd(a.round->cnt + 2, 1ull);
    }
    const PullUnit pn = un < n.total ? pull_fetch<WIDE>(ra, n, un) : noUnit;
    pull_unit<P, WIDE>(a, ra, n, u, pu, s4, c);
    if (un < n.total && (un < n.small || pn.quads > 0))
      s4 = __ldg(static_cast<const int4 *>(ra.pullIds) + pn.base + lane);
    pu = pn;
    u = un;
  }
  return c;
}

}  // namespace detail
}  // namespace gas

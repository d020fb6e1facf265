// Internal helpers shared by the translation units of libgas_gb300.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "gas_gb300.h"

namespace gas {
namespace internal {

// Records a one-line message for gas_last_error() and returns `code`.
gas_status fail(gas_status code, const char *fmt, ...);
// Maps a CUDA error to GAS_ERR_OOM / GAS_ERR_CUDA with a message.
gas_status cuda_fail(cudaError_t e, const char *what);

// Stable counting sort of an edge list by `key` on the host: off[V+1],
// adj[E] and optionally perm[p] = edge index placed at position p.
void build_adjacency(int32_t nV, int32_t nE, const int32_t *key, const int32_t *other,
                     std::vector<int32_t> &off, std::vector<int32_t> &adj,
                     std::vector<int32_t> *perm);

// The same on the device (gas_graph_build.cu).  Working memory of its
// sorts, for max(nV, nE) elements: sort_scratch_bytes sizes it, and with a
// base address lays it out in *x.
struct SortScratch {
  uint32_t *keys[2];
  uint32_t *spare;
  uint32_t *hist;
  uint32_t *sums;
};
size_t sort_scratch_bytes(int32_t nV, int32_t nE, SortScratch *x, void *base);
// dOff[V+1], dAdj[E], optional dPerm[E] of a stable sort of the edges by
// dKey.  `sorted`: the keys already ascend.  Device arrays, stream-ordered
// on `s`.
gas_status device_build_adjacency(cudaStream_t s, int32_t nV, int32_t nE, const int32_t *dKey,
                                  const int32_t *dOther, bool sorted, int32_t *dOff, int32_t *dAdj,
                                  uint32_t *dPerm, const SortScratch &x);
// The first edge with an id outside [0, nV), or -1, and whether the edges
// come by ascending source / destination (waits; 16 bytes of scratch).
struct EdgeCheck {
  long long firstBad = -1;
  bool srcSorted = true, dstSorted = true;
};
gas_status device_check_edges(cudaStream_t s, int32_t nV, int32_t nE, const int32_t *dSrcs,
                              const int32_t *dDsts, void *scratch, EdgeCheck *out);
// In-degree classes of the pull passes (dense.cuh): bins[V] = hubs (more
// than kChunkEdges in-edges) | 65..kChunkEdges | 9..64 | 1..8 | 0, the
// second and third by falling degree, ties and the others by vertex id; the
// hubs' chunks; counts (zero before the call) and the largest degrees.
struct DegreeBins {
  int32_t nHub, nMid, nSmall, nTiny, nZero, nChunks, maxIn, maxOut;
};
struct HubChunks {
  int32_t *vertex, *begin, *first, *count, *slot;
};
gas_status device_degree_bins(cudaStream_t s, int32_t nV, const int32_t *inOff, const int32_t *outOff,
                              int32_t maxHubs, int32_t *bins, const HubChunks &hubs, DegreeBins *dCounts,
                              const SortScratch &x);
// The layout of the leading dense rounds' kernel (gas_run_args::pullIds and
// the fields after it).  First, from the CSC, the out-degrees and the bins:
// the vertices' and chunks' records and the hot vertices, `capacity` at most;
// *info (device) receives their number and their smallest out-degree.
struct HotInfo {
  int32_t nHot, minOut;
};
struct PullLayout {
  int32_t *slotOf, *hotVertex;
  int4 *rec, *chunkRec;
  bool anyOrder;  // steps as pull_any walks them, else as pull_ordered does
  bool wide;      // more lanes a vertex (pull_mid_lanes)
};
gas_status device_pull_records(cudaStream_t s, int32_t nV, const int32_t *inOff, const int32_t *outOff,
                               const int32_t *bins, const HubChunks &hubs, const DegreeBins *dCounts,
                               int32_t maxChunks, int32_t capacity, const PullLayout &out, HotInfo *info,
                               const SortScratch &x);
// Then, with the counts on the host: the number n of slices, their first int4
// and quads (slices[n + 1]) and *quads, the int4 they take together (waits);
// and their ids and 4-byte edge data (eds null: none).
int32_t pull_slice_count(const DegreeBins &n, bool wide);
gas_status device_pull_slices(cudaStream_t s, const DegreeBins &n, const PullLayout &l, int2 *slices,
                              long long *quads, const SortScratch &x);
gas_status device_pull_fill(cudaStream_t s, const DegreeBins &n, const PullLayout &l, const int2 *slices,
                            const int32_t *inSrc, const int32_t *ed, int4 *ids, int4 *eds);
// out[q] = CSC position of the edge at CSR position q.
gas_status device_csr_to_csc(cudaStream_t s, int32_t n, const uint32_t *cscPerm,
                             const uint32_t *csrPerm, int32_t *out);
// out[p] = in[perm[p]] / out[perm[p]] = in[p] for n elements of `bytes`.
gas_status device_gather_bytes(cudaStream_t s, const void *dIn, const uint32_t *dPerm, int32_t n,
                               int32_t bytes, void *dOut);
gas_status device_scatter_bytes(cudaStream_t s, const void *dIn, const uint32_t *dPerm, int32_t n,
                                int32_t bytes, void *dOut);

// Device graph of a gas_core (CSC, CSR, edge data in CSC order), for the
// other engines of the library that share its graph build.
struct CoreGraph {
  int device;
  cudaStream_t stream;
  int32_t nV, nE;
  const int32_t *inOff, *inSrc, *outOff, *outDst;
  const void *edgeData;
  int32_t edgeBytes;
  const std::vector<int32_t> *hInOff;
  const std::vector<int32_t> *hOutOff;
  int32_t maxOutDeg;
};
bool core_graph(struct gas_core_s *c, CoreGraph *out);
// Keep the CSR permutation at the next set_graph (false also frees a kept
// one), and gather host values (one int32 per edge, edge-list order) into a
// new device array in CSR order (the caller frees it).
void core_keep_csr_perm(struct gas_core_s *c, bool keep);
gas_status core_permute_csr(struct gas_core_s *c, const int32_t *hostVals, int32_t **devOut);

// A gas_batch's graph with its batched-run extras: out-edge weights in CSR
// order and the pull work units (a vertex's in-edges, hubs in chunks).
struct BatchGraph {
  CoreGraph g;
  const int32_t *weightsOut;
  const int32_t *unitV, *unitBeg, *unitEnd;
  int32_t nUnits;
};
bool batch_graph(struct gas_batch_s *b, BatchGraph *out);

// Personalised PageRank structures of a graph (gas_serve.cu): out-degrees
// and the pull work units (a vertex's in-edges, hubs cut into
// gas::detail::kPprChunk-edge chunks with partial-sum slots), hub chunks
// first, then longest first, each with the last of `rounds` rounds in which
// its vertex is active.
struct PprGraph {
  int32_t *outDegree = nullptr;  // [V]
  int32_t *mem = nullptr;        // unit records (4 words) | slotFirst | slotCount | slotHub
  int32_t units = 0, slots = 0, hubs = 0;
  int32_t nLong[2] = {0, 0};     // units that are hub chunks or over kPprLong[k] edges
};
gas_status build_ppr_graph(const CoreGraph &g, int sms, int rounds, PprGraph *out);
void free_ppr_graph(PprGraph *p);

}  // namespace internal
}  // namespace gas

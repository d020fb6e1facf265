// Device graph builder: CSR / CSC from an edge list on the GPU, and the
// degree bins of the pull passes.
//
// The reference builds both adjacencies on the host (util.h:44-121,
// edgeListToCSR/CSC; gpugas.h:212-322 copies them up).  Here the edge list
// is copied to the device once and each adjacency is a stable LSD radix
// sort of (key, payload) pairs with digits of at most 8 bits (the key bits
// divided evenly over the passes: fewer digits, longer runs):
//
//   per pass:  block histograms of the digit (4096 edges per block)
//              -> exclusive scan in digit-major order (a digit's blocks in
//                 order after every smaller digit)
//              -> scatter: each warp ranks 512 consecutive edges per digit
//                 in edge order (warp match + per-warp counts), the block
//                 stages its edges in shared memory in digit order and
//                 writes each digit's run with consecutive threads
//
// which gives the same order as build_adjacency's stable counting sort
// (in-edges of a vertex in edge-list order).  The payload is the adjacency
// itself, or the edge index where the permutation is wanted (edge data).
// Offsets are binary searches in the sorted keys (counters per key are
// contended by every SM at a power-law graph's hubs).  An edge list already in key order -- files list edges by
// source -- needs no sort on that side.
//
// A scatter moves 8 bytes in and 8 out an edge and pass.  On 128 M edges
// (R-MAT-22, three passes) it takes 1.36 / 1.37 / 1.13 ms, about 1.5 TB/s,
// bound by the ranking (match, shared-memory counts) rather than by HBM; a
// block that wrote its edges unstaged, one 256-edge step at a time with
// four block barriers a step, took 2.81 / 2.80 / 1.60 ms.  The offsets'
// searches take 0.12 ms a side there (per-key counters 1.46 and 2.15 ms).
// Degree bins: 0.14 ms (a host loop with std::stable_sort took about 12 ms
// on R-MAT-20).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "gas_gb300/detail/pull.cuh"
#include "gas_internal.h"

using gas::internal::cuda_fail;
using gas::internal::fail;

namespace {

constexpr int kBins = 256;  // at most 8 bits a digit
constexpr int kRThreads = 256;
constexpr int kRItems = 16;
constexpr int kRTile = kRThreads * kRItems;  // edges per sort block
constexpr int kRWarps = kRThreads / 32;
constexpr int kSThreads = 1024;
constexpr int kSItems = 8;
constexpr int kSTile = kSThreads * kSItems;  // elements per scan block

__global__ void radix_hist_kernel(const uint32_t *keys, long long n, int shift, uint32_t digitMask,
                                  int nBlocks, uint32_t *hist) {
  __shared__ uint32_t h[kBins];
  h[threadIdx.x] = 0u;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kRTile;
#pragma unroll 4
  for (int i = 0; i < kRItems; ++i) {
    const long long idx = base + (long long)i * kRThreads + threadIdx.x;
    if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & digitMask], 1u);
  }
  __syncthreads();
  if (threadIdx.x <= digitMask) hist[(size_t)threadIdx.x * nBlocks + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of one pass.  vals == null stands for the identity
// (edge index), the first pass's payload; keysOut == null drops the keys.
__global__ void __launch_bounds__(kRThreads)
    radix_scatter_kernel(const uint32_t *keysIn, const uint32_t *valsIn, uint32_t *keysOut,
                         uint32_t *valsOut, long long n, int shift, uint32_t digitMask, int nBlocks,
                         const uint32_t *histScan) {
  __shared__ uint32_t cnt[kRWarps][kBins];  // per warp and digit: edges so far, then first slot
  __shared__ uint32_t start[kBins];         // the digit's first slot in the tile
  __shared__ uint32_t gbase[kBins];         // its global position minus that slot
  __shared__ uint32_t buf[kRTile];
  __shared__ uint32_t warpTot[kRWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned ltMask = (1u << lane) - 1u;
#pragma unroll
  for (int w = 0; w < kRWarps; ++w) cnt[w][tid] = 0u;
  const long long base = (long long)blockIdx.x * kRTile;
  const int count = (int)min((long long)kRTile, n - base);
  const int first = warp * (32 * kRItems) + lane;  // this thread's edges: first + 32 j
  uint32_t key[kRItems], pos[kRItems];
#pragma unroll
  for (int j = 0; j < kRItems; ++j)
    key[j] = first + 32 * j < count ? keysIn[base + first + 32 * j] : 0u;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRItems; ++j) {
    const bool valid = first + 32 * j < count;
    const uint32_t d = (key[j] >> shift) & digitMask;
    const unsigned peers = __match_any_sync(gas::detail::kFullMask, valid ? d : 0xffffffffu);
    const uint32_t before = cnt[warp][d];
    __syncwarp();
    if (valid && (peers & ltMask) == 0u) cnt[warp][d] = before + (uint32_t)__popc(peers);
    __syncwarp();
    pos[j] = before + (uint32_t)__popc(peers & ltMask);
  }
  __syncthreads();
  {  // digit tid: the warps' first slots, then the digit's own
    uint32_t run = 0u;
#pragma unroll
    for (int w = 0; w < kRWarps; ++w) {
      const uint32_t c = cnt[w][tid];
      cnt[w][tid] = run;
      run += c;
    }
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(gas::detail::kFullMask, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) warpTot[warp] = incl;
    __syncthreads();
    uint32_t excl = incl - run;
#pragma unroll
    for (int w = 0; w < kRWarps; ++w)
      if (w < warp) excl += warpTot[w];
    start[tid] = excl;
    gbase[tid] = (tid <= (int)digitMask ? histScan[(size_t)tid * nBlocks + blockIdx.x] : 0u) - excl;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRItems; ++j)
    if (first + 32 * j < count) {
      const uint32_t d = (key[j] >> shift) & digitMask;
      pos[j] += start[d] + cnt[warp][d];
      buf[pos[j]] = key[j];
    }
  __syncthreads();
  uint32_t dst[kRItems];
#pragma unroll
  for (int j = 0; j < kRItems; ++j) {
    const int i = tid + kRThreads * j;
    if (i < count) {
      const uint32_t k = buf[i];
      dst[j] = gbase[(k >> shift) & digitMask] + (uint32_t)i;
      if (keysOut) keysOut[dst[j]] = k;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRItems; ++j)
    if (first + 32 * j < count)
      buf[pos[j]] = valsIn ? valsIn[base + first + 32 * j] : (uint32_t)(base + first + 32 * j);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRItems; ++j) {
    const int i = tid + kRThreads * j;
    if (i < count) valsOut[dst[j]] = buf[i];
  }
}

// Block-wide exclusive scan of kSTile elements (in place); the block's
// total goes to sums[blockIdx.x] when sums is non-null.
__global__ void scan_block_kernel(uint32_t *data, long long n, uint32_t *sums) {
  __shared__ uint32_t warpTot[kSThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long base = (long long)blockIdx.x * kSTile + (long long)tid * kSItems;
  uint32_t v[kSItems];
  uint32_t t = 0u;
#pragma unroll
  for (int k = 0; k < kSItems; ++k) {
    v[k] = base + k < n ? data[base + k] : 0u;
    t += v[k];
  }
  uint32_t incl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(gas::detail::kFullMask, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warpTot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = warpTot[lane];
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(gas::detail::kFullMask, wi, o);
      if (lane >= o) wi += y;
    }
    warpTot[lane] = wi - w;  // exclusive
    if (lane == 31 && sums) sums[blockIdx.x] = wi;
  }
  __syncthreads();
  uint32_t run = warpTot[warp] + incl - t;
#pragma unroll
  for (int k = 0; k < kSItems; ++k) {
    if (base + k < n) data[base + k] = run;
    run += v[k];
  }
}

__global__ void scan_add_kernel(uint32_t *data, long long n, const uint32_t *offs) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) data[i] += offs[i / kSTile];
}

// Words exclusive_scan needs for n elements (its block sums, level by level).
size_t scan_words(long long n) {
  size_t w = 0;
  for (long long b = (n + kSTile - 1) / kSTile; b > 1; b = (b + kSTile - 1) / kSTile) w += (size_t)b;
  return w + 1;
}

// In place; `sums` holds scan_words(n) words.
gas_status exclusive_scan(uint32_t *data, long long n, uint32_t *sums, cudaStream_t s) {
  if (n <= 0) return GAS_OK;
  const long long blocks = (n + kSTile - 1) / kSTile;
  scan_block_kernel<<<(unsigned)blocks, kSThreads, 0, s>>>(data, n, blocks > 1 ? sums : nullptr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "graph build scan");
  if (blocks == 1) return GAS_OK;
  gas_status st = exclusive_scan(sums, blocks, sums + blocks, s);
  if (st) return st;
  scan_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(data, n, sums);
  e = cudaGetLastError();
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "graph build scan");
}

// off[v] = first position of a key >= v in the sorted keys, v = 0..nV.
__global__ void offsets_kernel(const uint32_t *keys, long long n, int32_t nV, int32_t *off) {
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v <= nV;
       v += (long long)gridDim.x * blockDim.x) {
    long long lo = 0, hi = n;
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (keys[mid] < (uint32_t)v)
        lo = mid + 1;
      else
        hi = mid;
    }
    off[v] = (int32_t)lo;
  }
}

__global__ void iota_kernel(uint32_t *out, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = (uint32_t)i;
}

__global__ void gather_kernel(const int32_t *src, const uint32_t *perm, long long n, int32_t *dst) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[perm[i]];
}

// out[p] = in[perm[p]] for elements of `bytes` bytes (word copies when the
// size is a multiple of 4).
__global__ void gather_bytes_kernel(const unsigned char *in, const uint32_t *perm, long long n,
                                    int bytes, unsigned char *out) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x) {
    const size_t s = (size_t)perm[p] * bytes, d = (size_t)p * bytes;
    if ((bytes & 3) == 0) {
      for (int k = 0; k < bytes; k += 4)
        *reinterpret_cast<uint32_t *>(out + d + k) = *reinterpret_cast<const uint32_t *>(in + s + k);
    } else {
      for (int k = 0; k < bytes; ++k) out[d + k] = in[s + k];
    }
  }
}

// out[perm[p]] = in[p]: back to edge-list order.
__global__ void scatter_bytes_kernel(const unsigned char *in, const uint32_t *perm, long long n,
                                     int bytes, unsigned char *out) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x) {
    const size_t d = (size_t)perm[p] * bytes, s = (size_t)p * bytes;
    for (int k = 0; k < bytes; ++k) out[d + k] = in[s + k];
  }
}

// Ids in [0, nV)?  *firstBad = the first edge with one outside; also
// whether each end's ids come in ascending order (unsorted[0]: a,
// unsorted[1]: b).
__global__ void check_ids_kernel(const int32_t *a, const int32_t *b, long long n, int32_t nV,
                                 unsigned long long *firstBad, unsigned *unsorted) {
  bool ua = false, ub = false;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int32_t x = a[i], y = b[i];
    if ((unsigned)x >= (unsigned)nV || (unsigned)y >= (unsigned)nV)
      atomicMin(firstBad, (unsigned long long)i);
    if (i > 0) {
      ua |= a[i - 1] > x;
      ub |= b[i - 1] > y;
    }
  }
  // one store per warp that saw a descent (every writer stores the same)
  if (__any_sync(gas::detail::kFullMask, ua) && (threadIdx.x & 31) == 0) unsorted[0] = 1u;
  if (__any_sync(gas::detail::kFullMask, ub) && (threadIdx.x & 31) == 0) unsorted[1] = 1u;
}

// Sort key of each vertex's degree class, in the order the pull pass hands
// its work out: hubs (in-degree > kChunkEdges) first, then in-degree 65..
// kChunkEdges and 9..64 by falling degree, then 1..8, then no in-edges.
// Adds the class counts, the hubs' chunks and the largest degrees to *c.
__global__ void degree_class_kernel(const int32_t *inOff, const int32_t *outOff, int32_t nV,
                                    uint32_t *key, gas::internal::DegreeBins *c) {
  using gas::detail::kChunkEdges;
  __shared__ int sums[8];
  if (threadIdx.x < 8) sums[threadIdx.x] = 0;
  __syncthreads();
  int n[5] = {0, 0, 0, 0, 0}, chunks = 0, maxIn = 0, maxOut = 0;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nV;
       v += (long long)gridDim.x * blockDim.x) {
    const int d = inOff[v + 1] - inOff[v];
    maxIn = max(maxIn, d);
    maxOut = max(maxOut, outOff[v + 1] - outOff[v]);
    uint32_t k;
    if (d > kChunkEdges) {
      k = 0u;
      ++n[0];
      chunks += (d + kChunkEdges - 1) / kChunkEdges;
    } else if (d > 64) {
      k = 1u + (uint32_t)(kChunkEdges - d);
      ++n[1];
    } else if (d > GAS_TPV_MAX_DEGREE) {
      k = 1u + kChunkEdges + (uint32_t)(64 - d);
      ++n[2];
    } else {
      k = 65u + kChunkEdges + (d == 0 ? 1u : 0u);
      ++n[d == 0 ? 4 : 3];
    }
    key[v] = k;
  }
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int w = __reduce_add_sync(gas::detail::kFullMask, n[i]);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(&sums[i], w);
  }
  const int wc = __reduce_add_sync(gas::detail::kFullMask, chunks);
  const int wi = __reduce_max_sync(gas::detail::kFullMask, maxIn);
  const int wo = __reduce_max_sync(gas::detail::kFullMask, maxOut);
  if ((threadIdx.x & 31) == 0) {
    if (wc) atomicAdd(&sums[5], wc);
    atomicMax(&sums[6], wi);
    atomicMax(&sums[7], wo);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (sums[0]) atomicAdd(&c->nHub, sums[0]);
    if (sums[1]) atomicAdd(&c->nMid, sums[1]);
    if (sums[2]) atomicAdd(&c->nSmall, sums[2]);
    if (sums[3]) atomicAdd(&c->nTiny, sums[3]);
    if (sums[4]) atomicAdd(&c->nZero, sums[4]);
    if (sums[5]) atomicAdd(&c->nChunks, sums[5]);
    atomicMax(&c->maxIn, sums[6]);
    atomicMax(&c->maxOut, sums[7]);
  }
}

// Chunks of each hub (hubs: the first c->nHub entries of `bins`), 0 past them.
__global__ void hub_count_kernel(const int32_t *bins, const int32_t *inOff,
                                 const gas::internal::DegreeBins *c, int32_t maxHubs, uint32_t *count) {
  const int n = c->nHub;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < maxHubs; i += gridDim.x * blockDim.x) {
    const int v = i < n ? bins[i] : 0;
    count[i] = i < n ? (uint32_t)((inOff[v + 1] - inOff[v] + gas::detail::kChunkEdges - 1) /
                                  gas::detail::kChunkEdges)
                     : 0u;
  }
}

// The hubs' chunk entries (a warp per hub); first[i] = hub i's first chunk.
__global__ void hub_chunks_kernel(const int32_t *bins, const int32_t *inOff,
                                  const gas::internal::DegreeBins *c, const uint32_t *first,
                                  gas::internal::HubChunks out) {
  const int n = c->nHub, lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n;
       i += (gridDim.x * blockDim.x) >> 5) {
    const int v = bins[i], b = inOff[v];
    const int nch = (inOff[v + 1] - b + gas::detail::kChunkEdges - 1) / gas::detail::kChunkEdges;
    const int f = (int)first[i];
    for (int k = lane; k < nch; k += 32) {
      out.vertex[f + k] = v;
      out.begin[f + k] = b + k * gas::detail::kChunkEdges;
      out.first[f + k] = f;
      out.count[f + k] = nch;
      out.slot[f + k] = i;
    }
  }
}

// Sort key of the out-degrees, the largest first.
__global__ void out_degree_key_kernel(const int32_t *outOff, int32_t nV, uint32_t *key) {
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nV;
       v += (long long)gridDim.x * blockDim.x)
    key[v] = (uint32_t)(gas::detail::kHotDegreeCap -
                        min(outOff[v + 1] - outOff[v], gas::detail::kHotDegreeCap));
}

// The least out-degree of a hot vertex.  Each slot costs every SM its share of
// the table's fill in every round, and saves an SM outDeg / 152 gathers.
// Without a least degree, 10, 32, 64, 128, 256 (run(), us): CC 200 x 200
// lattice 2910, 1920 and the same from there on (its degree-4 half was hot);
// CC, 60,000 vertices, 1.7 M edges 133, 123, 115, 115, 113, 111; PageRank of
// 30,000 and 150,000 vertices 515, 525, 496, 496, 492, 488 and 1016, 998,
// 961, 957, 957, 955, of 9,001 240, 263, 257, 257, 257, 257; SSSP of 60,000
// 275, 261, 250, 248, 248, 250.  Graphs of a million vertices fill the table
// with higher degrees than these.
constexpr int kHotMinOut = 64;

// order: the vertices by falling out-degree (out_degree_key_kernel).  The hot
// ones (hot_cut) take the slots below `capacity`, of which the first stays
// unused (one block).
__global__ void hot_pick_kernel(const uint32_t *order, const int32_t *outOff, int32_t nV, int32_t capacity,
                                gas::internal::HotInfo *info, int32_t *hotVertex) {
  __shared__ int sHot;
  if (threadIdx.x == 0) {
    const gas::detail::HotCut cut = gas::detail::hot_cut(
        [&](int k) { return outOff[order[k] + 1] - outOff[order[k]]; }, nV, capacity - 1, kHotMinOut);
    sHot = cut.count;
    info->nHot = cut.count + 1;
    info->minOut = cut.minOut;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < sHot; k += blockDim.x) hotVertex[k + 1] = (int32_t)order[k];
}

__global__ void hot_slots_kernel(const gas::internal::HotInfo *info, const int32_t *hotVertex, int32_t *slotOf) {
  const int n = info->nHot;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x + 1; k < n; k += gridDim.x * blockDim.x)
    slotOf[hotVertex[k]] = k;
}

__global__ void pull_records_kernel(const int32_t *bins, const int32_t *inOff, const int32_t *outOff, int32_t nV,
                                    int4 *rec) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nV;
       i += (long long)gridDim.x * blockDim.x) {
    const int v = bins[i], b = inOff[v];
    rec[i] = make_int4(v, b, inOff[v + 1] - b, outOff[v + 1] - outOff[v]);
  }
}

__global__ void chunk_records_kernel(const gas::internal::DegreeBins *c, gas::internal::HubChunks hubs,
                                     const int32_t *inOff, const int32_t *outOff, int4 *rec) {
  const int n = c->nChunks;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int v = hubs.vertex[i], b = hubs.begin[i];
    rec[i] = make_int4(v, b, min(gas::detail::kChunkEdges, inOff[v + 1] - b), outOff[v + 1] - outOff[v]);
  }
}

// A slice's class and first record (pull.cuh: chunks, mid, small, tiny).
struct SliceAt {
  const int4 *rec;
  int count;  // vertices
  int lanes;  // of each
  int virt;   // of dense.cuh's lanes in each (0: quads dealt round-robin)
};
__device__ __forceinline__ SliceAt slice_at(const gas::internal::DegreeBins &n, const gas::internal::PullLayout &l,
                                            int u) {
  const int ml = gas::detail::pull_mid_lanes(l.wide), sl = gas::detail::pull_small_lanes(l.wide);
  const int M = 32 / ml, S = 32 / sl;
  if (u < n.nChunks) return {l.chunkRec + u, 1, 32, l.anyOrder ? 0 : 1};
  u -= n.nChunks;
  const int4 *rec = l.rec + n.nHub;
  const int mid = (n.nMid + M - 1) / M, small = (n.nSmall + S - 1) / S;
  if (u < mid) return {rec + u * M, min(M, n.nMid - u * M), ml, l.anyOrder ? 0 : 32 / ml};
  u -= mid;
  rec += n.nMid;
  if (u < small) return {rec + u * S, min(S, n.nSmall - u * S), sl, l.anyOrder ? 0 : gas::detail::kSmallLanes / sl};
  u -= small;
  rec += n.nSmall;
  return {rec + u * 32, min(32, n.nTiny + n.nZero - u * 32), 1, 0};
}

__device__ __forceinline__ int slice_layers(const SliceAt &s, int quads, int k) {
  return s.lanes * s.virt == 8 ? gas::detail::pull_layers<8>(quads, k) : gas::detail::pull_layers<32>(quads, k);
}

// Per slice its longest vertex's quads, or its steps where quads are dealt
// round-robin, and the int4 it takes: 32 a step.
__global__ void slice_steps_kernel(const gas::internal::DegreeBins n, const gas::internal::PullLayout l, int nSlices,
                                   uint32_t *size, int2 *slices) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u > nSlices) return;
  if (u == nSlices) {
    size[u] = 0u;
    slices[u] = make_int2(0, 0);
    return;
  }
  const SliceAt s = slice_at(n, l, u);
  int quads = 0;
  for (int k = 0; k < s.count; ++k)
    quads = max(quads, s.virt == 0 ? ((s.rec[k].z + 3) / 4 + s.lanes - 1) / s.lanes
                                   : gas::detail::pull_range(s.rec[k].y, s.rec[k].z).quads);
  int steps = s.virt == 0 ? quads : s.virt == 8 ? 2 : 1;
  for (int k = 0; k < s.virt; ++k) steps += slice_layers(s, quads, k);
  size[u] = 32u * (uint32_t)steps;
  slices[u].y = quads;
}

__global__ void slice_extents_kernel(const uint32_t *base, int nSlices, int2 *slices) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u <= nSlices) slices[u].x = (int)base[u];
}

// A warp per slice writes its steps in the order pull.cuh walks them.
__global__ void slice_fill_kernel(const gas::internal::DegreeBins n, const gas::internal::PullLayout l,
                                  const int2 *slices, int nSlices, const int32_t *inSrc, const int32_t *ed, int4 *ids,
                                  int4 *eds) {
  const int lane = threadIdx.x & 31;
  for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < nSlices; u += (gridDim.x * blockDim.x) >> 5) {
    const SliceAt s = slice_at(n, l, u);
    const int2 at = slices[u];
    const int g = lane / s.lanes, sl = lane % s.lanes;
    const int4 rec = g < s.count ? s.rec[g] : make_int4(-1, 0, 0, 0);
    size_t pos = (size_t)at.x + lane;
    // one step: edges [e, e + count) of the CSC, count <= 4
    auto put = [&](int e, int count) {
      int id[4], w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        id[j] = gas::detail::kNoEdge;
        w[j] = 0;
        if (j < count) {
          const int32_t src = inSrc[e + j], slot = l.slotOf[src];
          id[j] = slot >= 0 ? (int32_t)(0x80000000u | (uint32_t)slot) : src;
          if (eds) w[j] = ed[e + j];
        }
      }
      ids[pos] = make_int4(id[0], id[1], id[2], id[3]);
      if (eds) eds[pos] = make_int4(w[0], w[1], w[2], w[3]);
      pos += 32;
    };
    if (s.virt == 0) {
      for (int t = 0; t < at.y; ++t) {
        const int e = 4 * (t * s.lanes + sl);
        put(rec.y + e, min(4, rec.z - e));
      }
      continue;
    }
    const gas::detail::PullRange r = gas::detail::pull_range(rec.y, rec.z);
    const int tail = (rec.y + rec.z) & ~3;
    if (s.virt == 8) {
      put(rec.y, r.head);
      put(tail, r.tail);
    } else if (s.virt == 1) {
      if (sl < 4)
        put(rec.y + sl, sl < r.head ? 1 : 0);
      else
        put(tail + sl - 4, sl - 4 < r.tail ? 1 : 0);
    } else {
      put(sl == 0 ? rec.y : tail, sl == 0 ? r.head : sl == 1 ? r.tail : 0);
    }
    for (int k = 0; k < s.virt; ++k) {
      const int layers = slice_layers(s, at.y, k);
      for (int j = 0; j < layers; ++j) {
        const int q = sl * s.virt + k + s.lanes * s.virt * j;
        put(4 * (r.first + q), q < r.quads ? 4 : 0);
      }
    }
  }
}

__global__ void invert_kernel(const uint32_t *perm, long long n, uint32_t *inv) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (long long)gridDim.x * blockDim.x)
    inv[perm[p]] = (uint32_t)p;
}

__global__ void compose_kernel(const uint32_t *inv, const uint32_t *perm, long long n, int32_t *out) {
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x)
    out[q] = (int32_t)inv[perm[q]];
}

int grid_for(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 152 * 16)); }

}  // namespace

namespace gas {
namespace internal {

gas_status device_check_edges(cudaStream_t s, int32_t nV, int32_t nE, const int32_t *dSrcs,
                              const int32_t *dDsts, void *scratch, EdgeCheck *out) {
  *out = EdgeCheck();
  if (nE <= 0) return GAS_OK;
  struct {
    unsigned long long bad;
    unsigned unsorted[2];
  } h = {~0ull, {0u, 0u}};
  cudaError_t e = cudaMemcpyAsync(scratch, &h, sizeof(h), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    unsigned long long *d = static_cast<unsigned long long *>(scratch);
    check_ids_kernel<<<grid_for(nE), 256, 0, s>>>(dSrcs, dDsts, nE, nV, d,
                                                  reinterpret_cast<unsigned *>(d + 1));
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, scratch, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "edge id check");
  if (h.bad != ~0ull) out->firstBad = (long long)h.bad;
  out->srcSorted = h.unsorted[0] == 0u;
  out->dstSorted = h.unsorted[1] == 0u;
  return GAS_OK;
}

namespace {

// Passes of a sort of `bits`-bit keys and the digit width of each.
struct Digits {
  int passes, bits;
};
Digits digits_for(int bits) {
  Digits d;
  d.passes = (bits + 7) / 8;
  d.bits = (bits + d.passes - 1) / d.passes;
  return d;
}

// Stable sort of n (key, payload) pairs by `bits`-bit keys; payload null:
// the index.  The sorted payload goes to valsOut, the sorted keys to
// *sortedKeys (inside the scratch) unless sortedKeys is null.
gas_status radix_sort(cudaStream_t s, long long n, const uint32_t *keys, const uint32_t *vals, int bits,
                      uint32_t *valsOut, const uint32_t **sortedKeys, const SortScratch &x) {
  const Digits dg = digits_for(bits);
  const uint32_t mask = (1u << dg.bits) - 1u;
  const int nBlocks = (int)((n + kRTile - 1) / kRTile);
  const uint32_t *kin = keys, *vin = vals;
  for (int p = 0; p < dg.passes; ++p) {
    const bool lastPass = p + 1 == dg.passes;
    uint32_t *kout = x.keys[p & 1];
    // the last pass writes valsOut; before it the payload alternates
    // between valsOut and the spare so that it never reads what it writes
    uint32_t *vout = ((dg.passes - 1 - p) & 1) ? x.spare : valsOut;
    radix_hist_kernel<<<nBlocks, kRThreads, 0, s>>>(kin, n, p * dg.bits, mask, nBlocks, x.hist);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "graph build sort");
    gas_status st = exclusive_scan(x.hist, (long long)(mask + 1) * nBlocks, x.sums, s);
    if (st) return st;
    radix_scatter_kernel<<<nBlocks, kRThreads, 0, s>>>(
        kin, vin, lastPass && !sortedKeys ? nullptr : kout, vout, n, p * dg.bits, mask, nBlocks, x.hist);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "graph build sort");
    kin = kout;
    vin = vout;
  }
  if (sortedKeys) *sortedKeys = kin;
  return GAS_OK;
}

}  // namespace

size_t sort_scratch_bytes(int32_t nV, int32_t nE, SortScratch *x, void *base) {
  const long long n = std::max<long long>(std::max(nE, nV), 1);
  const long long hist = (long long)kBins * ((n + kRTile - 1) / kRTile);
  unsigned char *p = static_cast<unsigned char *>(base);
  size_t used = 0;
  auto take = [&](size_t words) {
    uint32_t *r = reinterpret_cast<uint32_t *>(p + used);
    used += (words * 4 + 255) & ~(size_t)255;
    return r;
  };
  uint32_t *k0 = take(n), *k1 = take(n), *sp = take(n), *h = take(hist);
  uint32_t *su = take(scan_words(std::max<long long>(hist, n)));
  if (x) *x = SortScratch{{k0, k1}, sp, h, su};
  return used;
}

gas_status device_build_adjacency(cudaStream_t s, int32_t nV, int32_t nE, const int32_t *dKey,
                                  const int32_t *dOther, bool sorted, int32_t *dOff, int32_t *dAdj,
                                  uint32_t *dPermOut, const SortScratch &x) {
  const long long n = nE;
  const uint32_t *keys = reinterpret_cast<const uint32_t *>(dKey);
  cudaError_t e = cudaSuccess;
  if (n > 0 && sorted) {
    e = cudaMemcpyAsync(dAdj, dOther, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess && dPermOut) {
      iota_kernel<<<grid_for(n), 256, 0, s>>>(dPermOut, n);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) return cuda_fail(e, "graph build");
  } else if (n > 0) {
    int bits = 1;
    while (bits < 31 && (1ll << bits) < nV) ++bits;
    gas_status st = radix_sort(s, n, keys, dPermOut ? nullptr : reinterpret_cast<const uint32_t *>(dOther),
                               bits, dPermOut ? dPermOut : reinterpret_cast<uint32_t *>(dAdj), &keys, x);
    if (st) return st;
    if (dPermOut) {
      gather_kernel<<<grid_for(n), 256, 0, s>>>(dOther, dPermOut, n, dAdj);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "graph build");
    }
  }
  offsets_kernel<<<grid_for((long long)nV + 1), 256, 0, s>>>(keys, n, nV, dOff);
  e = cudaGetLastError();
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "graph build");
}

gas_status device_degree_bins(cudaStream_t s, int32_t nV, const int32_t *inOff, const int32_t *outOff,
                              int32_t maxHubs, int32_t *bins, const HubChunks &hubs, DegreeBins *dCounts,
                              const SortScratch &x) {
  if (nV <= 0) return GAS_OK;
  int32_t *first = reinterpret_cast<int32_t *>(x.spare);
  degree_class_kernel<<<std::min(grid_for(nV), 152 * 8), 256, 0, s>>>(inOff, outOff, nV, x.keys[1], dCounts);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "degree bins");
  // keys below 2^11 (66 + kChunkEdges): two passes; keys[1] is free again
  // when the second pass, whose keys are dropped, would write it
  static_assert(gas::detail::kChunkEdges + 66 < (1 << 11), "degree class keys");
  gas_status st = radix_sort(s, nV, x.keys[1], nullptr, 11, reinterpret_cast<uint32_t *>(bins), nullptr, x);
  if (st) return st;
  if (maxHubs > 0) {
    uint32_t *cnt = reinterpret_cast<uint32_t *>(first);
    hub_count_kernel<<<grid_for(maxHubs), 256, 0, s>>>(bins, inOff, dCounts, maxHubs, cnt);
    st = exclusive_scan(cnt, maxHubs, x.sums, s);
    if (st) return st;
    hub_chunks_kernel<<<grid_for(32ll * maxHubs), 256, 0, s>>>(bins, inOff, dCounts, cnt, hubs);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "degree bins");
  }
  return GAS_OK;
}

gas_status device_pull_records(cudaStream_t s, int32_t nV, const int32_t *inOff, const int32_t *outOff,
                               const int32_t *bins, const HubChunks &hubs, const DegreeBins *dCounts,
                               int32_t maxChunks, int32_t capacity, const PullLayout &out, HotInfo *info,
                               const SortScratch &x) {
  if (nV <= 0) return GAS_OK;
  out_degree_key_kernel<<<grid_for(nV), 256, 0, s>>>(outOff, nV, x.keys[1]);
  // the order is needed only until the hot vertices are listed: it stands
  // where their slots go
  uint32_t *order = reinterpret_cast<uint32_t *>(out.slotOf);
  gas_status st = radix_sort(s, nV, x.keys[1], nullptr, 16, order, nullptr, x);
  if (st) return st;
  hot_pick_kernel<<<1, 1024, 0, s>>>(order, outOff, nV, capacity, info, out.hotVertex);
  cudaError_t e = cudaMemsetAsync(out.slotOf, 0xff, 4 * (size_t)nV, s);
  if (e != cudaSuccess) return cuda_fail(e, "pull layout");
  hot_slots_kernel<<<grid_for(capacity), 256, 0, s>>>(info, out.hotVertex, out.slotOf);
  pull_records_kernel<<<grid_for(nV), 256, 0, s>>>(bins, inOff, outOff, nV, out.rec);
  if (maxChunks > 0)
    chunk_records_kernel<<<grid_for(maxChunks), 256, 0, s>>>(dCounts, hubs, inOff, outOff, out.chunkRec);
  e = cudaGetLastError();
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "pull layout");
}

int32_t pull_slice_count(const DegreeBins &n, bool wide) {
  const int M = 32 / gas::detail::pull_mid_lanes(wide), S = 32 / gas::detail::pull_small_lanes(wide);
  return n.nChunks + (n.nMid + M - 1) / M + (n.nSmall + S - 1) / S + (n.nTiny + n.nZero + 31) / 32;
}

gas_status device_pull_slices(cudaStream_t s, const DegreeBins &n, const PullLayout &l, int2 *slices,
                              long long *quads, const SortScratch &x) {
  const int32_t k = pull_slice_count(n, l.wide);
  *quads = 0;
  if (k == 0) return GAS_OK;
  uint32_t *base = x.spare;
  slice_steps_kernel<<<(k + 256) / 256, 256, 0, s>>>(n, l, k, base, slices);
  gas_status st = exclusive_scan(base, (long long)k + 1, x.sums, s);
  if (st) return st;
  slice_extents_kernel<<<(k + 256) / 256, 256, 0, s>>>(base, k, slices);
  uint32_t total = 0;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&total, base + k, 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  *quads = total;
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "pull layout");
}

gas_status device_pull_fill(cudaStream_t s, const DegreeBins &n, const PullLayout &l, const int2 *slices,
                            const int32_t *inSrc, const int32_t *ed, int4 *ids, int4 *eds) {
  const int32_t k = pull_slice_count(n, l.wide);
  if (k == 0) return GAS_OK;
  slice_fill_kernel<<<grid_for(32ll * k), 256, 0, s>>>(n, l, slices, k, inSrc, ed, ids, eds);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "pull layout");
}

gas_status device_csr_to_csc(cudaStream_t s, int32_t n, const uint32_t *cscPerm,
                             const uint32_t *csrPerm, int32_t *out) {
  if (n <= 0) return GAS_OK;
  uint32_t *inv = nullptr;
  cudaError_t e = cudaMallocAsync(&inv, sizeof(uint32_t) * n, s);
  if (e == cudaSuccess) {
    invert_kernel<<<grid_for(n), 256, 0, s>>>(cscPerm, n, inv);
    compose_kernel<<<grid_for(n), 256, 0, s>>>(inv, csrPerm, n, out);
    e = cudaGetLastError();
    cudaFreeAsync(inv, s);
  }
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "CSR to CSC edge map");
}

gas_status device_gather_bytes(cudaStream_t s, const void *dIn, const uint32_t *dPerm, int32_t n,
                               int32_t bytes, void *dOut) {
  if (n <= 0 || bytes <= 0) return GAS_OK;
  gather_bytes_kernel<<<grid_for(n), 256, 0, s>>>(reinterpret_cast<const unsigned char *>(dIn),
                                                  dPerm, n, bytes,
                                                  reinterpret_cast<unsigned char *>(dOut));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "edge data permutation");
}

gas_status device_scatter_bytes(cudaStream_t s, const void *dIn, const uint32_t *dPerm, int32_t n,
                                int32_t bytes, void *dOut) {
  if (n <= 0 || bytes <= 0) return GAS_OK;
  scatter_bytes_kernel<<<grid_for(n), 256, 0, s>>>(reinterpret_cast<const unsigned char *>(dIn),
                                                   dPerm, n, bytes,
                                                   reinterpret_cast<unsigned char *>(dOut));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GAS_OK : cuda_fail(e, "edge data un-permutation");
}

}  // namespace internal
}  // namespace gas

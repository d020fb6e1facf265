// Programs that declare nothing (no gatherFromSource, no reduceAnyOrder) and
// one of minima in any order, from every vertex active: run() with the leading dense rounds in their own
// kernel, and with every round in the main kernel.  Vertex data of 8 bytes,
// of 256 bytes, and edge data of 8 bytes; sums in an order that shows.
#include <cstdio>
#include <cstring>
#include <vector>

#include "gas_gb300/gpugas.cuh"

template <int N>
struct Values {
  float x[N];
};

// N floats a vertex; EXTRA: 8 bytes of edge data.
template <int N, bool EXTRA>
struct Smooth {
  typedef Values<N> VertexData;
  struct None {};
  struct Pair {
    float scale;
    int add;
  };
  typedef typename std::conditional<EXTRA, Pair, None>::type EdgeData;
  typedef float GatherResult;
  static constexpr float gatherZero = 0.0f;
  __host__ __device__ static float gatherMap(const VertexData *dst, const VertexData *src, const EdgeData *e) {
    float v = src->x[0] * 0.3f + src->x[N - 1] + dst->x[1] * 0.01f;
    if constexpr (EXTRA) v = v * e->scale + (float)e->add;
    return v;
  }
  __host__ __device__ static float gatherReduce(const float &l, const float &r) { return l + r; }
  __host__ __device__ static bool apply(VertexData *v, const float &g) {
    const float next = 0.2f + 0.6f * (g - floorf(g));  // keeps moving: every round is dense
    const bool more = next != v->x[0];
    v->x[N - 1] = 0.5f * v->x[0];
    v->x[0] = next;
    v->x[1] += 1e-3f;
    return more;
  }
  __host__ __device__ static void scatter(const VertexData *, const VertexData *, EdgeData *) {}
};

// 256 bytes a vertex, minima in any order.
struct Least {
  struct VertexData {
    int x[64];
  };
  struct EdgeData {};
  typedef int GatherResult;
  static constexpr int gatherZero = 0x7fffffff;
  static constexpr bool reduceAnyOrder = true;
  __host__ __device__ static int gatherMap(const VertexData *, const VertexData *src, const EdgeData *) {
    return src->x[0] ^ src->x[63];
  }
  __host__ __device__ static int gatherReduce(const int &l, const int &r) { return l < r ? l : r; }
  __host__ __device__ static bool apply(VertexData *v, const int &g) {
    v->x[63] = v->x[0];
    v->x[0] = (int)((unsigned)(g + v->x[5]) * 2654435761u >> 3);  // keeps moving
    return true;
  }
  __host__ __device__ static void scatter(const VertexData *, const VertexData *, EdgeData *) {}
};

template <class P>
int run(int nV, int nE, const std::vector<int32_t> &s, const std::vector<int32_t> &d, FILE *out) {
  typedef typename P::VertexData VD;
  typedef typename P::EdgeData ED;
  std::vector<ED> ed;
  if constexpr (!std::is_empty<ED>::value) {
    ed.resize(nE);
    for (int i = 0; i < nE; ++i) ed[i] = {0.5f + (float)(i % 7) * 0.125f, i % 3};
  }
  for (int main_only = 0; main_only < 2; ++main_only) {
    std::vector<VD> vd(nV);
    for (int v = 0; v < nV; ++v)
      for (int k = 0; k < (int)(sizeof(VD) / 4); ++k)
        vd[v].x[k] = std::is_same<P, Least>::value ? (v * 31 + k) % 100003 : 0.001f * (float)((v * 7 + k) % 1013);
    GASEngineGPU<P> engine;
    if (main_only) engine.setRunBlocksPerSM(4);  // a launch shape of its own
    engine.setGraph(nV, vd.data(), nE, ed.empty() ? nullptr : ed.data(), s.data(), d.data());
    gas_core_set_dense_policy(engine.core(), 1 << 20);  // dense while any vertex returned true
    engine.setActive(0, nV);
    const int32_t rounds = engine.runFor(6);
    engine.getResults();
    const int32_t head[2] = {(int32_t)engine.lastStatus(), rounds};
    if (head[0]) fprintf(stderr, "%s\n", engine.lastError());
    fwrite(head, 4, 2, out);
    fwrite(vd.data(), sizeof(VD), nV, out);
    if (head[0]) return 1;
  }
  return 0;
}

// pull_forms IN OUT: {nV, nE, which, 0}, sources, destinations.
int main(int argc, char **argv) {
  if (argc != 3) return 2;
  FILE *f = fopen(argv[1], "rb");
  if (!f) return 2;
  int32_t h[4];
  if (fread(h, 4, 4, f) != 4) return 2;
  std::vector<int32_t> s(h[1]), d(h[1]);
  if (fread(s.data(), 4, h[1], f) != (size_t)h[1] || fread(d.data(), 4, h[1], f) != (size_t)h[1]) return 2;
  fclose(f);
  FILE *out = fopen(argv[2], "wb");
  if (!out) return 2;
  const int rc = h[2] == 0   ? run<Smooth<64, false>>(h[0], h[1], s, d, out)
                 : h[2] == 1 ? run<Smooth<2, false>>(h[0], h[1], s, d, out)
                 : h[2] == 3 ? run<Least>(h[0], h[1], s, d, out)
                             : run<Smooth<2, true>>(h[0], h[1], s, d, out);
  fclose(out);
  return rc;
}

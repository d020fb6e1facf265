// A download after a round that set a device error bit, behind the C ABI: it
// reports the error and leaves the caller's array as it is; the next one,
// with the error reported, copies.
#include <cstdio>
#include <vector>

#include "gas_gb300_core.h"

__global__ void fail_round(gas_gather_args a) { atomicOr(a.errWord, GAS_DEVERR_CAPACITY); }
__global__ void fail_run(const gas_run_args ra) {
  atomicOr(ra.g.errWord, GAS_DEVERR_CAPACITY);
  *ra.roundsOut = 1;
}

static gas_status launch_round(void *, const gas_gather_args *a, void *stream) {
  fail_round<<<1, 1, 0, (cudaStream_t)stream>>>(*a);
  return GAS_OK;
}
static gas_status launch_run(void *, const gas_run_args *ra, void *stream) {
  fail_run<<<1, 1, 0, (cudaStream_t)stream>>>(*ra);
  return GAS_OK;
}

int main() {
  const int nV = 100000;
  std::vector<int32_t> s(nV), d(nV), vd(nV), mine(nV, -7);
  for (int v = 0; v < nV; ++v) s[v] = vd[v] = v, d[v] = (v + 1) % nV;
  gas_core *c = nullptr;
  int32_t it = 0;
  if (gas_core_create(0, nullptr, &c) != GAS_OK) return 2;
  if (gas_core_set_graph(c, nV, nV, s.data(), d.data(), nullptr, 0, 4, 4) != GAS_OK) return 2;
  if (gas_core_upload_vertex_data(c, vd.data()) != GAS_OK) return 2;
  if (gas_core_set_active(c, 0, nV) != GAS_OK) return 2;
  if (gas_core_gather_apply(c, 1, &launch_round, nullptr) != GAS_OK) return 2;
  const gas_status first = gas_core_download_vertex_data(c, mine.data());
  int touched = 0, wrong = 0;
  for (int v = 0; v < nV; ++v) touched += mine[v] != -7;
  const gas_status second = gas_core_download_vertex_data(c, mine.data());
  for (int v = 0; v < nV; ++v) wrong += mine[v] != v;
  // run() reports its own error
  if (gas_core_set_active(c, 0, nV) != GAS_OK) return 2;
  const gas_status run = gas_core_run_persistent(c, 1, 1, &launch_run, &launch_round, nullptr, &it);
  const gas_status after = gas_core_download_vertex_data(c, mine.data());
  printf("%d %d %d %d %d %d\n", (int)first, touched, (int)second, wrong, (int)run, (int)after);
  gas_core_destroy(c);
  return 0;
}

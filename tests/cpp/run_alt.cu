// A run kernel that leaves its result in the alternate vertex buffer and says
// so in vcurOut, behind the C ABI: the result is what a download gives.
#include <cstdio>
#include <vector>

#include "gas_gb300_core.h"

__global__ void triple(const gas_run_args ra) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < ra.g.nVertices) static_cast<int *>(ra.vertexAlt)[v] = 3 * static_cast<int *>(ra.g.vertexData)[v];
  if (v == 0) {
    *ra.roundsOut = 1;
    *ra.vcurOut = 1;
  }
}

static gas_status launch_run(void *, const gas_run_args *ra, void *stream) {
  triple<<<(ra->g.nVertices + 255) / 256, 256, 0, (cudaStream_t)stream>>>(*ra);
  return cudaGetLastError() == cudaSuccess ? GAS_OK : GAS_ERR_CUDA;
}
static gas_status no_launch(void *, const gas_gather_args *, void *) { return GAS_ERR_STATE; }

int main() {
  const int nV = 1000;
  std::vector<int32_t> s(nV), d(nV), vd(nV);
  for (int v = 0; v < nV; ++v) s[v] = vd[v] = v, d[v] = (v + 1) % nV;
  gas_core *c = nullptr;
  int32_t it = 0, bad = 0;
  gas_status st = gas_core_create(0, nullptr, &c);
  if (st == GAS_OK) st = gas_core_set_graph(c, nV, nV, s.data(), d.data(), nullptr, 0, 4, 4);
  if (st == GAS_OK) st = gas_core_upload_vertex_data(c, vd.data());
  for (int k = 1; k <= 2 && st == GAS_OK; ++k) {  // 3x, then 9x
    st = gas_core_set_active(c, 0, nV);
    if (st == GAS_OK) st = gas_core_run_persistent(c, 0, 1, &launch_run, &no_launch, nullptr, &it);
    if (st == GAS_OK) st = gas_core_download_vertex_data(c, vd.data());
    for (int v = 0; v < nV; ++v) bad += vd[v] != (k == 1 ? 3 : 9) * v;
  }
  printf("%d %d %d\n", (int)st, it, bad);
  gas_core_destroy(c);
  return st == GAS_OK && it == 1 && bad == 0 ? 0 : 1;
}

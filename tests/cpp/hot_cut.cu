// hot_cut (pull.cuh) on the host: reads nV, most, least and nV out-degrees,
// orders the vertices as the builder's sort does (capped degree, falling;
// ties by id), writes minOut and the hot vertices.
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <vector>

#include "gas_gb300/detail/pull.cuh"

int main() {
  int nV, most, least;
  if (scanf("%d %d %d", &nV, &most, &least) != 3) return 2;
  std::vector<int> deg(nV), order(nV);
  for (int &d : deg)
    if (scanf("%d", &d) != 1) return 2;
  std::iota(order.begin(), order.end(), 0);
  auto key = [&](int v) { return std::min(deg[v], gas::detail::kHotDegreeCap); };
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return key(x) > key(y); });
  const gas::detail::HotCut cut =
      gas::detail::hot_cut([&](int k) { return deg[order[k]]; }, nV, most, least);
  printf("%d", cut.minOut);
  for (int k = 0; k < cut.count; ++k) printf(" %d", order[k]);
  printf("\n");
  return 0;
}

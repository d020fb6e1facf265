// The choice between the kernels of the leading dense rounds (pull.cuh) for a
// shape read from standard input: csc, narrow or wide.
#include <cstdio>

#include "gas_gb300/detail/pull.cuh"

int main() {
  gas::detail::PullShape p;
  int any, messages, carried;
  long long narrowSlices, wideSlices;
  if (scanf("%d %d %d %d %lld %lld %lld %lld %lld %lld", &any, &messages, &p.entry, &carried, &p.nVertices, &p.nEdges,
            &p.maxOut, &p.narrowUnits, &narrowSlices, &wideSlices) != 10)
    return 2;
  p.anyOrder = any != 0;
  p.messages = messages != 0;
  p.carried = carried != 0;
  const bool wide = gas::detail::pull_wide(p);
  puts(!gas::detail::pull_pays(p, wide, wide ? wideSlices : narrowSlices) ? "csc" : wide ? "wide" : "narrow");
  return 0;
}

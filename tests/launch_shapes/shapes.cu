// Prints launch shapes and index maps of the kernels for every grid length the
// library dispatches (les_engine.cuh with_small); host code only, checked by
// tests/test_launch_shapes.py.
//   clip_walls <NSX> <row transforms' threads> <block>
#include <cstdio>
#include "les_kernels.cuh"
using namespace les;

template <int NSX> void clip_walls() {
  using C = RowCfg<3 * NSX / 2>;
  printf("clip_walls %d %d %d\n", NSX, C::THREADS, C::SUM_THREADS);
}
template <int N> void one() { clip_walls<N>(); }
int main() {
  one<16>(); one<32>(); one<64>(); one<96>(); one<128>(); one<192>(); one<256>(); one<384>(); one<512>();
  return 0;
}

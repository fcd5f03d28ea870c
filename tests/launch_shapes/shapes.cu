// Prints launch shapes and index maps of the kernels for every grid length the
// library dispatches (les_engine.cuh with_small); host code only, checked by
// tests/test_launch_shapes.py.
//   clip_walls <NSX> <row transforms' threads> <block>
//   row <real bytes> <NSX> <thread of the team> <written by the next level's
//       pass 1> : <read by the forward transform's last pass>
//       (elements of the row's buffer in k_row_fused)
//   tile <real bytes> <NS> <rows> <columns> <boxes> <rows of a box>
//       (TMA prefetches of k_y_inverse, k_y_forward)
//   rows <real bytes> <NX> <bytes>    (bulk prefetches of k_row_fused, k_lgrad_x)
#include <cstdio>
#include <vector>
#include "les_fused.cuh"
#include "les_learned.cuh"
using namespace les;

template <int NSX> void clip_walls() {
  using C = RowCfg<3 * NSX / 2>;
  printf("clip_walls %d %d %d\n", NSX, C::THREADS, C::SUM_THREADS);
}
// a row of shared memory that notes what is read
template <class T> struct Noted {
  std::vector<int>* at;
  int base;
  cx<T> operator[](int i) const {
    at->push_back(base + i);
    return mk((T)0, (T)0);
  }
};
template <class T, int NSX> void row() {
  using C = FusedCfg<T, NSX>;
  for (int t = 0; t < C::TP; t++) {
    int j, partner;
    mirror_lanes<C::M1, C::TP>(t, t & 31, j, partner);
    const bool act = j < C::M1;
    std::vector<int> read;
    cx<T> v[12];
    own_elements<C::SB>(Noted<T>{&read, C::off(act ? j : 0)}, act, v);
    printf("row %d %d %d", (int)sizeof(T), NSX, t);
    for (int b = 0; act && b < 12; b++) printf(" %d", C::off(j) + b * C::SB);
    printf(" :");
    for (int e : read) printf(" %d", e);
    printf("\n");
  }
}
template <class T, int ROWS, int TC, int NS> void tile() {
  using B = ColBox<T, ROWS, TC>;
  printf("tile %d %d %d %d %d %d\n", (int)sizeof(T), NS, ROWS, TC, B::ok ? B::NB : 0, B::BR);
}
template <class T, int N> void prefetches() {
  constexpr int M = 3 * N / 2, TC = ColPlan<T, M>::TC;
  tile<T, N, TC, N>();
  tile<T, M, TC, N>();
  printf("rows %d %d %d\n", (int)sizeof(T), N, (int)(FusedCfg<T, N>::ROWS * FusedCfg<T, N>::KX * sizeof(cx<T>)));
  printf("rows %d %d %d\n", (int)sizeof(T), N, (int)(LgxCfg<T, N>::RB * (N / 2) * sizeof(cx<T>)));
}
template <int N> void one() {
  clip_walls<N>();
  row<float, N>();
  row<double, N>();
  prefetches<float, N>();
  prefetches<double, N>();
}
int main() {
  one<16>(); one<32>(); one<64>(); one<96>(); one<128>(); one<192>(); one<256>(); one<384>(); one<512>();
  return 0;
}

// les_ops.cu -- operator-level transforms on caller-owned device buffers:
// xderiv, yderiv, expand, compress, deal (filter_fftw.f90:138-329).
#include "les_engine.cuh"

namespace les {
cudaError_t upload_twiddles_ops() { return upload_tu_twiddles(); }

template <class T>
void op_xderiv(const T* in, T* out, int n1, int n2, int howmany, double len, cudaStream_t s) {
  const cx<T>* tw = (const cx<T>*)twiddles(-1, sizeof(T) == 8);
  const double pi = 4.0 * std::atan(1.0);
  int nrows = n2 * howmany;
  bool ok = with_any(n1, [&](auto cn) {
    constexpr int N = decltype(cn)::value;
    using C = RowCfg<N>;
    launch(k_op_xderiv<T, N>, dim3(cdiv((nrows + 1) / 2, C::NT)), dim3(C::THREADS), C::template smem<T>(), s, in,
           out, nrows, (T)(2.0 * pi / len), tw);
  });
  if (!ok) throw CudaError("xderiv: unsupported length", LES_EINVAL);
}

template <class T>
void op_yderiv(const T* in, T* out, int n1, int n2, int howmany, double len, cudaStream_t s) {
  const cx<T>* tw = (const cx<T>*)twiddles(-1, sizeof(T) == 8);
  const double pi = 4.0 * std::atan(1.0);
  bool ok = with_any(n2, [&](auto cn) {
    constexpr int N = decltype(cn)::value;
    using C = ColCfg<N, T>;
    launch(k_op_yderiv<T, N>, dim3(cdiv((n1 + 1) / 2, C::TC), howmany), dim3(C::THREADS), C::buf(), s, in, out, n1,
           (T)(2.0 * pi / len), tw);
  });
  if (!ok) throw CudaError("yderiv: unsupported length", LES_EINVAL);
}

// The three kernels of expand, compress and deal: rows of length NR forward
// (the first KX modes, layout la of x-spectral rows at `a`), columns, rows
// back from layout lb at `b`.
template <class T, int N, int KX>
static void rows_forward(const T* in, cx<T>* a, int nrows, RowLayout la, const cx<T>* tw, cudaStream_t s) {
  using C = RowCfg<N>;
  launch(k_op_row_r2c<T, N, KX>, dim3(cdiv(nrows / 2, C::NT)), dim3(C::THREADS), C::template smem<T>(), s, in, a, nrows / 2,
         la, tw);
}
template <class T, int N>
static void rows_back(const cx<T>* b, T* out, int nrows, int KX, RowLayout lb, const cx<T>* tw, cudaStream_t s) {
  using C = RowCfg<N>;
  launch(k_op_row_c2r<T, N>, dim3(cdiv((nrows + 1) / 2, C::NT)), dim3(C::THREADS), C::template smem<T>(), s, b, out, nrows,
         KX, lb, tw);
}
template <class T, bool FROM_PAD, bool TO_PAD>
static void columns(const cx<T>* a, cx<T>* b, int ny, int KX, int howmany, RowLayout la, RowLayout lb, double scale,
                    const cx<T>* tw, cudaStream_t s) {
  with_small(ny, [&](auto cn) {
    constexpr int N = decltype(cn)::value;
    using C = ColPlan<T, 3 * N / 2>;
    launch(k_col_resize<T, N, FROM_PAD, TO_PAD>, dim3(cdiv(KX, C::TC), howmany), dim3(C::THREADS), C::smem() / 2, s, a, b,
           KX, la, lb, (T)scale, tw);
  });
}
static RowLayout layout(int ny, long long rs) { return RowLayout{ny, rs, rs * ny}; }

// expand: r2c rows (nx) -> forward y (ny, scaled, Nyquist dropped), pad and
// inverse y (3ny/2) -> c2r rows (3nx/2).  Without scratch (t1 = t2 = null) the
// x-spectral rows live in `out`, the modes of row y at the start of out's row
// y (3nx/4 complex values apart): out must be aligned to a complex value and
// must not overlap `in`.
template <class T>
void op_expand(const T* in, T* out, int nx, int ny, int howmany, cudaStream_t s, cx<T>* t1, cx<T>* t2) {
  const cx<T>* tw = (const cx<T>*)twiddles(-1, sizeof(T) == 8);
  const int KX = nx / 2, MY = 3 * ny / 2;
  if (!supported_small(nx) || !supported_small(ny)) throw CudaError("expand: unsupported size", LES_EINVAL);
  const long long rs = t1 ? KX : 3 * nx / 4;
  RowLayout l1 = layout(ny, rs), l2 = layout(MY, rs);
  if (!t1) {
    t1 = t2 = reinterpret_cast<cx<T>*>(out);
    l1.ps = l2.ps;
  }
  with_small(nx, [&](auto cn) {
    constexpr int N = decltype(cn)::value;
    rows_forward<T, N, N / 2>(in, t1, howmany * ny, l1, tw, s);
  });
  columns<T, false, true>(t1, t2, ny, KX, howmany, l1, l2, 1.0 / ((double)nx * ny), tw, s);
  with_small(nx, [&](auto cn) { rows_back<T, 3 * decltype(cn)::value / 2>(t2, out, howmany * MY, KX, l2, tw, s); });
}

// compress: r2c rows (3nx/2, keep nx/2) -> forward y (3ny/2), truncate,
// scale, inverse y (ny) -> c2r rows (nx).  t2: howmany*(3ny/2)*nx/2; without
// t1 the small spectral rows live in `out` (aligned to a complex value).
template <class T>
void op_compress(const T* in, T* out, int nx, int ny, int howmany, cudaStream_t s, cx<T>* t1, cx<T>* t2) {
  const cx<T>* tw = (const cx<T>*)twiddles(-1, sizeof(T) == 8);
  const int KX = nx / 2, MX = 3 * nx / 2, MY = 3 * ny / 2;
  if (!supported_small(nx) || !supported_small(ny)) throw CudaError("compress: unsupported size", LES_EINVAL);
  if (!t1) t1 = reinterpret_cast<cx<T>*>(out);
  const RowLayout l1 = layout(ny, KX), l2 = layout(MY, KX);
  with_small(nx, [&](auto cn) {
    constexpr int N = decltype(cn)::value;
    rows_forward<T, 3 * N / 2, N / 2>(in, t2, howmany * MY, l2, tw, s);
  });
  columns<T, true, false>(t2, t1, ny, KX, howmany, l2, l1, 1.0 / ((double)MX * MY), tw, s);
  with_small(nx, [&](auto cn) { rows_back<T, decltype(cn)::value>(t1, out, howmany * ny, KX, l1, tw, s); });
}

// deal in place; without t1 the spectral rows live in x (aligned to a complex
// value).
template <class T>
void op_deal(T* x, int nx, int ny, int howmany, cudaStream_t s, cx<T>* t1) {
  const cx<T>* tw = (const cx<T>*)twiddles(-1, sizeof(T) == 8);
  const int KX = nx / 2;
  if (!supported_small(nx) || !supported_small(ny)) throw CudaError("deal: unsupported size", LES_EINVAL);
  if (!t1) t1 = reinterpret_cast<cx<T>*>(x);
  const RowLayout l = layout(ny, KX);
  with_small(nx, [&](auto cn) {
    constexpr int N = decltype(cn)::value;
    rows_forward<T, N, N / 2>(x, t1, howmany * ny, l, tw, s);
  });
  columns<T, false, false>(t1, t1, ny, KX, howmany, l, l, 1.0 / ((double)nx * ny), tw, s);
  with_small(nx, [&](auto cn) { rows_back<T, decltype(cn)::value>(t1, x, howmany * ny, KX, l, tw, s); });
}

template void op_xderiv<double>(const double*, double*, int, int, int, double, cudaStream_t);
template void op_xderiv<float>(const float*, float*, int, int, int, double, cudaStream_t);
template void op_yderiv<double>(const double*, double*, int, int, int, double, cudaStream_t);
template void op_yderiv<float>(const float*, float*, int, int, int, double, cudaStream_t);
template void op_expand<double>(const double*, double*, int, int, int, cudaStream_t, cx<double>*, cx<double>*);
template void op_expand<float>(const float*, float*, int, int, int, cudaStream_t, cx<float>*, cx<float>*);
template void op_compress<double>(const double*, double*, int, int, int, cudaStream_t, cx<double>*, cx<double>*);
template void op_compress<float>(const float*, float*, int, int, int, cudaStream_t, cx<float>*, cx<float>*);
template void op_deal<double>(double*, int, int, int, cudaStream_t, cx<double>*);
template void op_deal<float>(float*, int, int, int, cudaStream_t, cx<float>*);

}  // namespace les

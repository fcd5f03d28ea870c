// les_kernels.cuh -- device kernels of one RK3 stage on a device-resident
// channel domain.
//
// State (spectral on the small grid, which represents exactly the
// Nyquist-free fields the reference carries after deal()):
//   uh, vh, wh        small spectra u^ = FFT2(u)/(nx*ny), [z][ky][kx], kx < nx/2
//   ruo, rvo, rwo     tendencies of the previous stage (spectral)
//   mu, mv, mru, mrv  FP64 shadows of the kx=ky=0 modes (mean profiles)
//   e, re             SGS TKE and its tendency in physical space (the e
//                     update clips at emin, comp2.f90:38)
// Work arrays on the 3/2-padded grid (nxb = 3nx/2, nyb = 3ny/2):
//   "mixed" arrays    x-spectral, y-physical  [z][y][kx]  (kx < nx/2)
//   "padded" arrays   physical                [z][y][x]
//
// One stage (les.F90:254-285) is:
//   k_e_prep                    e ghosts, x spectrum of e
//   k_y_inverse, k_x_inverse    expand() of u, v, w, e fused with the
//                               spectral derivatives ux..ey (derivs1/2)
//   k_clip_y, k_clip_x          derivatives of max(E, emin) - E
//   k_wall_sums, k_wall_final   plane means for sufsim / sufsim_upper
//   k_flux                      compadv1, complen, compsgs1, compsgs3
//                               pointwise, written as flux fields
//   k_x_forward, k_y_forward    compress() fused with -d/dx, -d/dy of the
//                               fluxes; the e part also inverts re in y
//   k_e_update                  e = max(e + dtab1*re, emin)
//   k_press                     comprhs + press (tridv) per (kx, ky) and
//                               comp2 in spectral space, FP64
// The x kernels, the clip kernels, k_wall_sums and k_flux are the unfused
// middle (Smagorinsky, shear production); les_fused.cuh holds the fused one.
#pragma once
#include "fft_core.cuh"
#include "fft_inplace.cuh"
#include "les_tma.cuh"

namespace les {

// ---------------------------------------------------------------------------
// launch shapes
// ---------------------------------------------------------------------------
template <int N> struct RowCfg {
  static constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  static constexpr int NT = (128 / N2) > 0 ? (128 / N2) : 1;  // row transforms per CTA
  static constexpr int THREADS = NT * N2;
  // THREADS rounded up to whole warps, for a kernel that also sums over its block
  static constexpr int SUM_THREADS = (THREADS + 31) / 32 * 32;
  template <class T> static constexpr size_t smem() { return (size_t)smem_fft_elems<N, false>(NT) * sizeof(cx<T>); }
};
template <int N, class T> struct ColCfg {
  static constexpr int N2 = Split<N>::N2;
  static constexpr int TCB = (sizeof(T) == 8) ? 4 : 8;  // 64-byte row segments
  static constexpr int TC = (TCB * N2 >= 64) ? TCB : (64 / N2);
  static constexpr int THREADS = TC * N2;
  static constexpr size_t buf() { return (size_t)TC * N * sizeof(cx<T>); }
};

// Scalars of one stage (double; kernels cast).
struct StageArgs {
  int NX, NY, NZ, MX, MY, KX;
  int imodel, isurface, tke_production, zeta;
  int mnout_sgs;  // record the SGS means (mnout and istage == 1)
  double dz, dzm, dzm2, todzm, kx0, ky0;
  double emin, ceps, dsl, forcing, nu, xkmax;
  double dtab1, dtab2, dtabm;
  double zl, ugal, vgal;
};

// Wall-model scalars for one wall (lowerbc.f90:56-124 / upperbc.f90:63-122).
struct WallSide {
  double u1xy, v1xy, vsfc, utau, windm, ufluc2mroot, vfluc2mroot, suflucm, svflucm;
  double moengu2mroot, moengv2mroot, auuwm, auvwm, denom;
};
struct WallParams {
  WallSide w[2];  // 0 = lower (level 1), 1 = upper (level nnz)
  double dudt, dvdt, utau_s;
};

// Device error word bits.
constexpr int ERR_NAN = 1, ERR_UTAU = 2;

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
template <class T> __device__ __forceinline__ T tmax(T a, T b) { return a > b ? a : b; }
template <class T> __device__ __forceinline__ T tmin(T a, T b) { return a < b ? a : b; }

// Element n of the length-N sequence A + iB of two real rows, from the K <= N/2 + 1
// modes of A and B that are kept (the others are zero, the imaginary parts of
// modes 0 and N/2 ignored): the mode to read, and what to make of it.  The loads
// need no branch, so a thread's go out together; behind branches they were a chain
// (expand of 384x384x64 FP64 230 -> 215 us, k_e_update of 512x512x64 147 -> 123,
// k_clip_walls 110 -> 90).
struct PairMode {
  int k;
  bool mirror, zero, real;
  template <class T> __device__ __forceinline__ cx<T> join(cx<T> a, cx<T> b) const {
    if (real) a.y = b.y = (T)0;
    const cx<T> v = mirror ? mk(a.x + b.y, b.x - a.y) : mk(a.x - b.y, a.y + b.x);
    return zero ? zero_cx<T>() : v;
  }
};
template <int N> __device__ __forceinline__ PairMode pair_mode(int n, int K) {
  const bool direct = n < K, mirror = !direct && N - n < K;
  const int k = direct ? n : mirror ? N - n : 0;
  return {k, mirror, !direct && !mirror, k == 0 || 2 * k == N};
}
// d/dx of a transformed row or column, with the 1/N of the inverse transform
// (the Nyquist mode dropped), at the inverse transform's loads: a pass over shared
// memory, a barrier and a division per mode less.  Mode k = n2 + m with m known at
// compile time: one conversion a thread, and only m = 0 and N/2 can be mode 0 or
// Nyquist.  The kernels' registers are bounded (168 FP64, 128 FP32): unbounded, 512
// points in FP64 lose a third of their blocks.  FP64 k_op_xderiv 576x576x27 66 us with
// the factor in a pass of its own, 57 with a conversion per mode, 45 so; k_op_yderiv 92,
// 62, 61; FP32 192x144x24 k_op_yderiv 5.2, 5.4, 3.6.
template <class T, int N> struct Derivative {
  T k1;
  __device__ __forceinline__ explicit Derivative(T k0) : k1(k0 / (T)N) {}
  __device__ __forceinline__ cx<T> operator()(int n2, int m, cx<T> v) const {
    const cx<T> d = mul_i(v) * (k1 * ((T)n2 + (T)(2 * m >= N ? m - N : m)));
    return ((m == 0 || 2 * m == N) && n2 == 0) ? zero_cx<T>() : d;
  }
};
// ---------------------------------------------------------------------------
// Generic small-grid transforms (upload, download, deal, expand, compress)
// ---------------------------------------------------------------------------

// Rows of real planes -> first KOUT complex modes of each row (unscaled).
// in: nrows rows of length N (row r at in + r*N); out: row r at out + r*KOUT.
template <class T, int N>
__global__ void __launch_bounds__(RowCfg<N>::THREADS)
k_row_r2c(const T* __restrict__ in, cx<T>* __restrict__ out, int nrows, int KOUT, const cx<T>* __restrict__ tw) {
  using C = RowCfg<N>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int p0 = blockIdx.x * C::NT;
  const int npair = (nrows + 1) / 2;
  if (p0 >= npair) return;
  fft_core<N, -1, false, false, true>(C::NT, sm, tw, [&](int t, int n) {
    int p = p0 + t;
    cx<T> v = zero_cx<T>();
    if (p < npair) v = mk(in[(size_t)(2 * p) * N + n], (2 * p + 1 < nrows) ? in[(size_t)(2 * p + 1) * N + n] : (T)0);
    return v;
  }, NoStore{});
  for (int i = threadIdx.x; i < C::NT * KOUT; i += blockDim.x) {
    int t = i / KOUT, k = i - t * KOUT, p = p0 + t;
    if (p >= npair) continue;
    cx<T> zk = sm[t * N + k], zm = conj(sm[t * N + (N - k) % N]);
    cx<T> a = (zk + zm) * (T)0.5;
    cx<T> d = zk - zm;
    out[(size_t)(2 * p) * KOUT + k] = a;
    if (2 * p + 1 < nrows) out[(size_t)(2 * p + 1) * KOUT + k] = mk(d.y * (T)0.5, -d.x * (T)0.5);
  }
}

// First KIN complex modes of each row (higher modes zero, imaginary parts of
// mode 0 ignored as in a c2r transform) -> real rows of length N.
// FP32 rows with a radix-16 first pass: six blocks per SM, or the twiddles asked for
// with the data take 106 registers (384x192x40 10.2 us, 8.1 bounded; 9.4 with the
// twiddles asked for after the data).
template <class T, int N>
__global__ void __launch_bounds__(RowCfg<N>::THREADS, sizeof(T) == 4 && Split<N>::N1 == 16 ? 6 : 0)
k_row_c2r(const cx<T>* __restrict__ in, T* __restrict__ out, int nrows, int KIN, const cx<T>* __restrict__ tw) {
  using C = RowCfg<N>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int p0 = blockIdx.x * C::NT;
  const int npair = (nrows + 1) / 2;
  if (p0 >= npair) return;
  const int row = 2 * (p0 + (int)(threadIdx.x / Split<N>::N2));  // of the transform this thread loads
  const cx<T>* ra = in + (size_t)(row < nrows ? row : 2 * p0) * KIN;
  const bool two = row + 1 < nrows;
  fft_core<N, +1, false, false, false>(C::NT, sm, tw, [&](int, int n) {
    const PairMode m = pair_mode<N>(n, KIN);
    return m.join(ra[m.k], two ? ra[KIN + m.k] : zero_cx<T>());
  }, [&](int t, int n, cx<T> v) {
    int p = p0 + t;
    if (p >= npair) return;
    out[(size_t)(2 * p) * N + n] = v.x;
    if (2 * p + 1 < nrows) out[(size_t)(2 * p + 1) * N + n] = v.y;
  });
}

// Where an operator keeps the x-spectral rows of its planes: row r of plane p
// at p ps + r rs complex values (rows per plane: ny).
struct RowLayout {
  int ny;
  long long rs, ps;
  __device__ __forceinline__ long long at(int row) const { return (long long)(row / ny) * ps + (long long)(row % ny) * rs; }
};

// k_row_r2c and k_row_c2r with the spectral rows in a given layout, which may
// lie inside the real rows' own buffer (row r's modes at the start of row r):
// a block reads its rows before it writes them, and no other block touches
// them.  So expand and deal need no scratch.  Planes have an even number of
// rows, so a pair lies in one; the first K modes are kept, K known at compile
// time (with K and a row's plane divided out for every value, 96 rows of 768
// points took 5.8 us in FP32 and 6.7 in FP64, now 4.4 and 5.1).
template <class T, int N, int K>
__global__ void __launch_bounds__(RowCfg<N>::THREADS)
k_op_row_r2c(const T* in, cx<T>* out, int npair, RowLayout lo, const cx<T>* __restrict__ tw) {
  using C = RowCfg<N>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int p0 = blockIdx.x * C::NT;
  if (p0 >= npair) return;
  fft_core<N, -1, false, false, true>(C::NT, sm, tw, [&](int t, int n) {
    const int p = p0 + t;
    if (p >= npair) return zero_cx<T>();
    return mk(in[(size_t)(2 * p) * N + n], in[(size_t)(2 * p + 1) * N + n]);
  }, NoStore{});
  for (int i = threadIdx.x; i < C::NT * K; i += C::THREADS) {
    const int t = i / K, k = i - t * K, p = p0 + t;
    if (p >= npair) continue;
    const cx<T> zk = sm[t * N + k], zm = conj(sm[t * N + (N - k) % N]);
    const cx<T> d = zk - zm;
    cx<T>* o = out + lo.at(2 * p) + k;
    o[0] = (zk + zm) * (T)0.5;
    o[lo.rs] = mk(d.y * (T)0.5, -d.x * (T)0.5);
  }
}
template <class T, int N>
__global__ void __launch_bounds__(RowCfg<N>::THREADS)
k_op_row_c2r(const cx<T>* in, T* out, int nrows, int K, RowLayout li, const cx<T>* __restrict__ tw) {
  using C = RowCfg<N>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int p0 = blockIdx.x * C::NT, npair = (nrows + 1) / 2;
  if (p0 >= npair) return;
  const int row = 2 * (p0 + (int)(threadIdx.x / Split<N>::N2));  // of the transform this thread loads
  const cx<T>* ra = in + li.at(row < nrows ? row : 2 * p0);
  const bool two = row + 1 < nrows;
  const cx<T>* rb = two ? in + li.at(row + 1) : ra;
  fft_core<N, +1, false, false, false>(C::NT, sm, tw, [&](int, int n) {
    const PairMode m = pair_mode<N>(n, K);
    return m.join(ra[m.k], two ? rb[m.k] : zero_cx<T>());
  }, [&](int t, int n, cx<T> v) {
    const int p = p0 + t;
    if (p >= npair) return;
    out[(size_t)(2 * p) * N + n] = v.x;
    if (2 * p + 1 < nrows) out[(size_t)(2 * p + 1) * N + n] = v.y;
  });
}

// Columns of x-spectral planes [plane][N][KX] (KX columns) -> forward DFT
// along y, times `scale`, Nyquist row N/2 dropped (deal semantics).
// With INV = true: inverse DFT, no scaling.
template <class T, int N, bool INV, bool DROP = !INV>
__global__ void __launch_bounds__(ColCfg<N, T>::THREADS)
k_col_small(const cx<T>* __restrict__ in, cx<T>* __restrict__ out, int KX, T scale, const cx<T>* __restrict__ tw) {
  using C = ColCfg<N, T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const size_t plane = (size_t)blockIdx.y * N * KX;
  const int kx0 = blockIdx.x * C::TC;
  // in-place use (in == out) is safe: every load of the tile precedes the
  // __syncthreads() inside fft_core that precedes every store
  fft_core<N, INV ? +1 : -1, true, false, false>(C::TC, sm, tw, [&](int t, int n) {
    int kx = kx0 + t;
    return (kx < KX) ? in[plane + (size_t)n * KX + kx] : zero_cx<T>();
  }, [&](int t, int k, cx<T> v) {
    int kx = kx0 + t;
    if (kx >= KX) return;
    if (!INV) v = (DROP && k == N / 2) ? zero_cx<T>() : v * scale;
    out[plane + (size_t)k * KX + kx] = v;
  });
}

// ---------------------------------------------------------------------------
// Stage kernels
// ---------------------------------------------------------------------------
// lower/upper ghosts of e (lowerbc.f90:13-17, upperbc.f90:20-24), with `zeta`
// the zeta part of the stage for e (comp1.f90:131; the fused stage leaves it
// to k_e_update), and the x-transform of e (first half of expand,
// filter_fftw.f90:262-263).  e has levels 0..NZ+1.  Also clears the level's
// clip flag (when given) for k_clip_walls.
template <class T, int NX>
__global__ void __launch_bounds__(RowCfg<NX>::THREADS)
k_e_prep(T* __restrict__ e, const T* __restrict__ re, cx<T>* __restrict__ Xe, int NY, int NZ, T dtab2, int zeta,
         int* __restrict__ clipflag, const cx<T>* __restrict__ tw) {
  using C = RowCfg<NX>;
  constexpr int KX = NX / 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int z = blockIdx.y + 1;  // 1..NZ-1
  const int p0 = blockIdx.x * C::NT;
  const size_t plane = (size_t)NY * NX;
  T* ez = e + (size_t)z * plane;
  if (clipflag && blockIdx.x == 0 && threadIdx.x == 0) clipflag[z - 1] = 0;
  fft_core<NX, -1, false, false, true>(C::NT, sm, tw, [&](int t, int n) {
    int p = p0 + t;
    return (p < NY / 2) ? mk(ez[(size_t)(2 * p) * NX + n], ez[(size_t)(2 * p + 1) * NX + n]) : zero_cx<T>();
  }, NoStore{});
  cx<T>* out = Xe + (size_t)(z - 1) * NY * KX;
  for (int i = threadIdx.x; i < C::NT * KX; i += blockDim.x) {
    int t = i / KX, k = i - t * KX, p = p0 + t;
    if (p >= NY / 2) continue;
    cx<T> zk = sm[t * NX + k], zm = conj(sm[t * NX + (NX - k) % NX]);
    cx<T> d = zk - zm;
    out[(size_t)(2 * p) * KX + k] = (zk + zm) * (T)0.5;
    out[(size_t)(2 * p + 1) * KX + k] = mk(d.y * (T)0.5, -d.x * (T)0.5);
  }
  if (!zeta && z != 1 && z != NZ - 1) return;
  for (int i = threadIdx.x; i < C::NT * NX; i += blockDim.x) {
    int t = i / NX, n = i - t * NX, p = p0 + t;
    if (p >= NY / 2) continue;
#pragma unroll
    for (int r = 0; r < 2; r++) {
      size_t off = (size_t)(2 * p + r) * NX + n;
      T val = ez[off];
      if (z == 1) e[off] = val;
      if (z == NZ - 1) {
        e[(size_t)NZ * plane + off] = val;
        e[(size_t)(NZ + 1) * plane + off] = val;
      }
      if (zeta) ez[off] = val - dtab2 * re[(size_t)(z - 1) * plane + off];
    }
  }
}

struct Ptr8 { void* p[8]; };
struct Ptr12 { void* p[12]; };

// Column transforms along y on the padded grid (M = 3 NS/2 = 12 M1, small
// length NS = 8 M1): a CTA owns TC columns (64-byte row segments) and M1
// threads per column, thread = (column t, j).  In place (fft_inplace.cuh),
// two shared-memory tiles (two transforms side by side, one pair of barriers
// for both).  Element n sits at row b SB + r SR + i of its tile; SR is odd,
// so that neighbouring threads' rows alternate between the two halves of the
// banks in every pass, and every address is a base plus a constant.  The
// pointer arrays are __grid_constant__: indexed by blockIdx.z, a plain struct
// parameter was copied to local memory by every thread (a quarter of the
// kernels' time).  Per stage at 512x512x256, against one two-pass transform
// per CTA: k_y_inverse FP32 1.09 -> 0.92 ms, FP64 2.03 -> 1.89 (0.96 and 1.95
// now that e's forward transform, a kernel of its own then, is in it too);
// k_y_forward 1.87 -> 1.21, 3.43 -> 2.34 ms (HBM floors 0.66 and 1.31); at
// 64x64x64 FP64 18 -> 11 and 28 -> 12 us.  Bound by load latency and the
// load/store path (64-byte rows) at 0.54-0.68 of the copy rate.
template <class T, int M> struct ColPlan {
  using P = InPlace<M>;
  static constexpr int M1 = P::M1, R2 = P::R2, R3 = P::R3, NS = 8 * M1;
  static constexpr int TCB = sizeof(T) == 8 ? 4 : 8;
  static constexpr int TC = TCB * ((64 + TCB * M1 - 1) / (TCB * M1));  // at least 64 threads
  static constexpr int THREADS = TC * M1;
  static constexpr int SR = R3 > 1 ? R3 + 1 : 1, SB = R3 > 1 ? R2 * SR : (M1 | 1);
  static constexpr int BUF = 12 * SB * TC;
  static constexpr size_t smem() { return (size_t)2 * BUF * sizeof(cx<T>); }
  // CTAs per SM the register budget aims at (both tiles' shared memory allows it)
  static constexpr int CTAS = (sizeof(T) == 8 ? 512 : 1024) / THREADS;
  static __device__ __forceinline__ int off(int m) { return R3 > 1 ? (m / R3) * SR + m % R3 : m; }
  // this thread's pass 2 twiddles W_M1^(r i), r = 1..3
  static __device__ __forceinline__ void twiddles2(const cx<T>* tw, int q, cx<T> (&w)[4]) {
    if constexpr (R3 > 1) {
      const cx<T>* g = tw + tw_off(M);
#pragma unroll
      for (int r = 1; r < 4; r++) w[r] = g[12 * r * (q % R3)];
    }
  }
  // pass 2 of NB blocks b (12 padded, 8 small) of a tile, R3 > 1
  template <int NB, bool INV> static __device__ __forceinline__ void pass2(cx<T>* buf, const cx<T> (&w)[4], int q) {
    static_assert(R3 == 1 || R2 == 4, "rounds of M1 threads");
    cx<T>* p = buf + (size_t)((q / R3) * SB + q % R3) * TC;
#pragma unroll
    for (int jj = 0; jj < NB / 4; jj++) {
      cx<T> v[4];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        v[r] = p[(4 * jj * SB + r * SR) * TC];
        if (!INV && r > 0) v[r] = cmul(v[r], w[r]);
      }
      Dft<4, INV ? +1 : -1, T>::run(v);
#pragma unroll
      for (int r = 0; r < 4; r++) p[(4 * jj * SB + r * SR) * TC] = (INV && r > 0) ? cmul(v[r], conj(w[r])) : v[r];
    }
  }
  // last pass of an inverse transform of NB blocks: store(row, value); rows in
  // the order of the padded map (NB = 12) or b + NB (r + R2 i)
  template <int NB, class StoreF> static __device__ __forceinline__ void last(const cx<T>* buf, int q, StoreF store) {
    constexpr int R = R3 > 1 ? R3 : R2, ITEMS = R3 > 1 ? NB * R2 : NB;
#pragma unroll
    for (int it = 0; it < (ITEMS + M1 - 1) / M1; it++) {
      const int u = q + it * M1;
      if (ITEMS % M1 != 0 && u >= ITEMS) break;
      const int b = R3 > 1 ? u / R2 : u, r = R3 > 1 ? u % R2 : 0;
      const cx<T>* p = buf + (size_t)(b * SB + r * SR) * TC;
      cx<T> v[R];
#pragma unroll
      for (int i = 0; i < R; i++) v[i] = p[i * TC];
      Dft<R, +1, T>::run(v);
      const int x0 = NB == 12 ? P::x_of(b * M1 + r * R3) : b + NB * r;
#pragma unroll
      for (int i = 0; i < R; i++) {
        int x = x0 + NB * (R3 > 1 ? R2 : 1) * i;
        if (NB == 12 && P::PFA) x = x >= M ? x - M : x;
        store(x, v[i]);
      }
    }
  }
  // first pass of a forward transform of NB blocks, rows load(row)
  template <int NB, class LoadF> static __device__ __forceinline__ void first(cx<T>* buf, int q, LoadF load) {
    constexpr int R = R3 > 1 ? R3 : R2, ITEMS = R3 > 1 ? NB * R2 : NB;
#pragma unroll
    for (int it = 0; it < (ITEMS + M1 - 1) / M1; it++) {
      const int u = q + it * M1;
      if (ITEMS % M1 != 0 && u >= ITEMS) break;
      const int b = R3 > 1 ? u / R2 : u, r = R3 > 1 ? u % R2 : 0;
      cx<T>* p = buf + (size_t)(b * SB + r * SR) * TC;
      const int x0 = NB == 12 ? P::x_of(b * M1 + r * R3) : b + NB * r;
      cx<T> v[R];
#pragma unroll
      for (int i = 0; i < R; i++) {
        int x = x0 + NB * (R3 > 1 ? R2 : 1) * i;
        if (NB == 12 && P::PFA) x = x >= M ? x - M : x;
        v[i] = load(x);
      }
      Dft<R, -1, T>::run(v);
#pragma unroll
      for (int i = 0; i < R; i++) p[i * TC] = v[i];
    }
  }
  // Forward transform of length NS of the rows load(row): thread j ends with
  // the modes ky = j + M1 m, m = 0..7, times scale, Nyquist removed.  One or
  // two barriers; the caller may then write the elements (b, j) without one.
  template <class LoadF>
  static __device__ __forceinline__ void forward_small(cx<T>* buf, const cx<T>* tw, const cx<T> (&w2)[4], int j, T scale,
                                                       LoadF load, cx<T> (&R)[8]) {
    first<8>(buf, j, load);
    __syncthreads();
    if constexpr (R3 > 1) {
      pass2<8, false>(buf, w2, j);
      __syncthreads();
    }
    const cx<T>* g = tw + tw_off(NS);
    const cx<T>* p = buf + off(j) * TC;
#pragma unroll
    for (int b = 0; b < 8; b++) R[b] = b ? cmul(p[b * SB * TC], g[b * j]) : p[0];
    Dft<8, -1, T>::run(R);
#pragma unroll
    for (int m = 0; m < 8; m++) R[m] = (m == 4 && j == 0) ? zero_cx<T>() : R[m] * scale;
  }
  // Inverse of it: the modes in registers to rows store(row, value).
  template <class StoreF>
  static __device__ __forceinline__ void inverse_small(cx<T>* buf, const cx<T>* tw, const cx<T> (&w2)[4], int j,
                                                       cx<T> (&R)[8], StoreF store) {
    Dft<8, +1, T>::run(R);
    const cx<T>* g = tw + tw_off(NS);
    cx<T>* p = buf + off(j) * TC;
#pragma unroll
    for (int b = 0; b < 8; b++) p[b * SB * TC] = b ? cmul(R[b], conj(g[b * j])) : R[b];
    __syncthreads();
    if constexpr (R3 > 1) {
      pass2<8, true>(buf, w2, j);
      __syncthreads();
    }
    last<8>(buf, j, store);
  }
};

// Pass 1 twiddles of thread j: W_(M/3)^(k j), k = 1..3 (PFA), or W_M^(b j).
template <class T, int M> struct ColTw1 {
  static constexpr int NT = InPlace<M>::PFA ? 3 : 11;
  cx<T> w[NT];
  __device__ __forceinline__ ColTw1(const cx<T>* tw, int j) {
    const cx<T>* g = tw + tw_off(M);
#pragma unroll
    for (int k = 0; k < NT; k++) w[k] = g[(InPlace<M>::PFA ? 3 : 1) * (k + 1) * j];
  }
  __device__ __forceinline__ cx<T> of(int b) const { return InPlace<M>::PFA ? w[(b & 3) ? (b & 3) - 1 : 0] : w[b ? b - 1 : 0]; }
  static __device__ __forceinline__ bool one(int b) { return InPlace<M>::PFA ? (b & 3) == 0 : b == 0; }
};

// Pass 1 of the padded inverse transform of thread j's modes x (ky = j + M1 m)
// into a tile.
template <class T, int M>
__device__ __forceinline__ void col_pad_pass1(cx<T>* buf, int j, const cx<T> (&x)[8], const ColTw1<T, M>& tw1,
                                              const cx<T> (&w3)[3]) {
  using C = ColPlan<T, M>;
  cx<T> v[12];
  if constexpr (InPlace<M>::PFA) Dft12Pfa<T, C::M1>::padded(x, w3, v);
  else dft12_padded<T>(x, v);
  cx<T>* p = buf + C::off(j) * C::TC;
#pragma unroll
  for (int b = 0; b < 12; b++) p[b * C::SB * C::TC] = ColTw1<T, M>::one(b) ? v[b] : cmul(v[b], conj(tw1.of(b)));
}
// Last pass of the padded forward transform: thread j's kept modes.
template <class T, int M>
__device__ __forceinline__ void col_trunc_pass1(const cx<T>* buf, int j, const ColTw1<T, M>& tw1, const cx<T> (&w3)[3],
                                                cx<T> (&o)[8]) {
  using C = ColPlan<T, M>;
  const cx<T>* p = buf + C::off(j) * C::TC;
  cx<T> v[12];
#pragma unroll
  for (int b = 0; b < 12; b++)
    v[b] = ColTw1<T, M>::one(b) ? p[b * C::SB * C::TC] : cmul(p[b * C::SB * C::TC], tw1.of(b));
  if constexpr (InPlace<M>::PFA) Dft12Pfa<T, C::M1>::forward(v, w3, o);
  else {
    cx<T> y[12];
    dft12_forward<T>(v, y);
#pragma unroll
    for (int m = 0; m < 4; m++) { o[m] = y[m]; o[4 + m] = y[8 + m]; }
  }
}

// expand() of u, v, w, e in y fused with d/dy: for field f = blockIdx.z
// (u, v, w, e), out[2f] = IFFT_M(pad(s)) and out[2f+1] = IFFT_M(i*ky*pad(s)),
// TC columns per block, both from one load of the columns (8 values a
// thread).  u, v, w come as spectra; e as the x-spectral rows of k_e_prep,
// whose y transform (times `scale`) is the block's first step: it ends with
// the modes in the registers where the others are loaded.  Thread 0 first has the TMA prefetch into L2 the columns of the
// block `pdist` blocks ahead (les_tma.cuh; maps: tensor maps of src[0..3] as
// [NZ*NS][KX] rows; pdist 0 prefetches nothing).
template <class T, int NS>
__global__ void __launch_bounds__(ColPlan<T, 3 * NS / 2>::THREADS, ColPlan<T, 3 * NS / 2>::CTAS)
k_y_inverse(const __grid_constant__ Ptr8 src, const __grid_constant__ Ptr8 dst, int KX, int NZ, T ky0, T scale,
            const cx<T>* __restrict__ tw,
            const __grid_constant__ ColMaps maps, unsigned pdist) {
  constexpr int M = 3 * NS / 2;
  using C = ColPlan<T, M>;
  constexpr int TC = C::TC, M1 = C::M1;
  prefetch_tile_ahead<T, NS, TC>(maps, pdist, [&](unsigned bx, unsigned by, unsigned bz, int& q, int& cg, int& row0) {
    q = (int)bz; cg = (int)bx; row0 = (int)by * NS;
    return !(bz >= 2 && (int)by + 1 == NZ);
  });
  extern __shared__ __align__(16) unsigned char smraw[];
  const int f = blockIdx.z, z = blockIdx.y + 1;
  if (f >= 2 && z == NZ) return;
  const int t = threadIdx.x % TC, j = threadIdx.x / TC;
  const int kx = blockIdx.x * TC + t;
  const bool in = kx < KX;
  cx<T>* buf = reinterpret_cast<cx<T>*>(smraw) + t;
  const cx<T>* s = reinterpret_cast<const cx<T>*>(src.p[f]) + (size_t)(z - 1) * NS * KX + (in ? kx : 0);
  cx<T> x[8], w2[4];
  if (f < 3) {
#pragma unroll
    for (int m = 0; m < 8; m++) x[m] = (m == 4 && j == 0) ? zero_cx<T>() : s[(j + M1 * m) * KX];  // no Nyquist mode
  }
  const ColTw1<T, M> tw1(tw, j);
  C::twiddles2(tw, j, w2);
  cx<T> w3[3];
  InPlace<M>::rotations(j, w3);
  if (f == 3) C::forward_small(buf, tw, w2, j, scale, [&](int row) { return s[row * KX]; }, x);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if (h) {
#pragma unroll
      for (int m = 0; m < 8; m++) x[m] = mul_i(x[m]) * (ky0 * (T)(m < 4 ? j + M1 * m : j + M1 * m - NS));
    }
    col_pad_pass1<T, M>(buf + h * C::BUF, j, x, tw1, w3);
  }
  __syncthreads();
  if constexpr (C::R3 > 1) {
    C::template pass2<12, true>(buf, w2, j);
    C::template pass2<12, true>(buf + C::BUF, w2, j);
    __syncthreads();
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    cx<T>* out = reinterpret_cast<cx<T>*>(dst.p[2 * f + h]) + (size_t)(z - 1) * M * KX + kx;
    C::template last<12>(buf + h * C::BUF, j, [&](int row, cx<T> v) {
      if (in) out[row * KX] = v;
    });
  }
}

// expand() in x fused with d/dx: six paired inverse row transforms give
// U,UX | V,VX | W,WX | UY,VY | E,EX | EY,WY on the padded grid.  A pair's members
// share their rounding: E goes with its own derivative (beside WY it took WY's
// rounding: in FP32 at 256x256x4, two stages, e off by 5e-5 of its maximum, 3e-7
// so), and EY, which only meets twice the viscosity, with WY.
// src: Um, UYm, Vm, VYm, Wm, WYm, Em, EYm; dst: U, UX, UY, V, VX, VY, W, WX,
// WY, E, EX, EY.  blockIdx.z = group.
template <class T, int NSX>
__global__ void __launch_bounds__(RowCfg<3 * NSX / 2>::THREADS)
k_x_inverse(const __grid_constant__ Ptr8 src, const __grid_constant__ Ptr12 dst, int MY, int NZ, T kx0, const cx<T>* __restrict__ tw) {
  constexpr int MX = 3 * NSX / 2;
  constexpr int KX = NSX / 2;
  using C = RowCfg<MX>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int g = blockIdx.z, z = blockIdx.y + 1;
  if (z == NZ && (g == 2 || g == 4 || g == 5)) return;
  // (source A, ikx on A, source B, ikx on B, output A, output B)
  const int sA[6] = {0, 2, 4, 1, 6, 7}, mA[6] = {0, 0, 0, 0, 0, 0};
  const int sB[6] = {0, 2, 4, 3, 6, 5}, mB[6] = {1, 1, 1, 0, 1, 0};
  const int oA[6] = {0, 3, 6, 2, 9, 11}, oB[6] = {1, 4, 7, 5, 10, 8};
  const size_t zoff = (size_t)(z - 1) * MY;
  const cx<T>* A = reinterpret_cast<const cx<T>*>(src.p[sA[g]]) + zoff * KX;
  const cx<T>* B = reinterpret_cast<const cx<T>*>(src.p[sB[g]]) + zoff * KX;
  const bool ma = mA[g], mb = mB[g];
  const int y0 = blockIdx.x * C::NT;
  T* outA = reinterpret_cast<T*>(dst.p[oA[g]]) + zoff * MX;
  T* outB = reinterpret_cast<T*>(dst.p[oB[g]]) + zoff * MX;
  const int yl = y0 + (int)(threadIdx.x / Split<MX>::N2);  // the row this thread loads
  const size_t ro = (size_t)(yl < MY ? yl : y0) * KX;
  fft_core<MX, +1, false, false, false>(C::NT, sm, tw, [&](int, int n) {
    const PairMode m = pair_mode<MX>(n, KX);
    cx<T> a = A[ro + m.k], b = B[ro + m.k];
    const T kk = kx0 * (T)m.k;
    if (ma) a = mul_i(a) * kk;
    if (mb) b = mul_i(b) * kk;
    return m.join(a, b);
  }, [&](int t, int n, cx<T> v) {
    int y = y0 + t;
    if (y >= MY) return;
    outA[(size_t)y * MX + n] = v.x;
    outB[(size_t)y * MX + n] = v.y;
  });
}

// yderiv of delta = max(emin - E, 0) on padded planes (column pairs),
// added to EY.  This and k_clip_x make EX, EY the derivatives of the
// clipped ebuf = max(expand(e), emin) (comp1.f90:109,121; derivs2.f90:20-21).
// Blocks whose points are all above emin stop once they are loaded: clipped or not,
// E is read once (k_clip_y and k_clip_x of 512x512x32 FP64, unclipped 102 and 26 us,
// clipped 307 and 429; with a scan of E before the transform's own loads 120 and
// 249, 355 and 877; always transforming 322 and 559).  Registers of the 768-point
// blocks: 168 (FP64) and, in k_clip_x, 96 (FP32), a block per SM more than unbounded
// (k_clip_y FP64 440 -> 307, k_clip_x FP32 274 -> 237).
template <class T, int NSY>
__global__ void __launch_bounds__(ColCfg<3 * NSY / 2, T>::THREADS, NSY == 512 && sizeof(T) == 8 ? 3 : 0)
k_clip_y(const T* __restrict__ E, T* __restrict__ EY, int MX, T emin, T ky0, const cx<T>* __restrict__ tw) {
  constexpr int M = 3 * NSY / 2;
  using C = ColCfg<M, T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const size_t zoff = (size_t)blockIdx.y * M * MX;
  const int c0 = blockIdx.x * C::TC, ncp = MX / 2;
  const cx<T>* Ez = reinterpret_cast<const cx<T>*>(E + zoff);
  bool below = false;
  const bool any = fft_core<M, -1, true, false, true>(C::TC, sm, tw, [&](int t, int n) {
    int c = c0 + t;
    cx<T> v = zero_cx<T>();
    if (c < ncp) {
      cx<T> ev = Ez[(size_t)n * ncp + c];
      v = mk(tmax(emin - ev.x, (T)0), tmax(emin - ev.y, (T)0));
    }
    below |= (v.x > (T)0) | (v.y > (T)0);
    return v;
  }, NoStore{}, [&] { return __syncthreads_or(below) != 0; });
  if (!any) return;  // delta is zero: so are its derivatives
  cx<T>* EYz = reinterpret_cast<cx<T>*>(EY + zoff);
  fft_core<M, +1, true, true, false>(C::TC, sm, tw, Derivative<T, M>(ky0), [&](int t, int n, cx<T> d) {
    int c = c0 + t;
    if (c >= ncp) return;
    cx<T> o = EYz[(size_t)n * ncp + c];
    EYz[(size_t)n * ncp + c] = mk(o.x + d.x, o.y + d.y);
  });
}

// xderiv of delta (row pairs), added to EX; E <- max(E, emin).
template <class T, int NSX>
__global__ void __launch_bounds__(RowCfg<3 * NSX / 2>::THREADS, NSX == 512 ? (sizeof(T) == 8 ? 3 : 5) : 0)
k_clip_x(T* __restrict__ E, T* __restrict__ EX, int MY, T emin, T kx0, const cx<T>* __restrict__ tw) {
  constexpr int MX = 3 * NSX / 2;
  using C = RowCfg<MX>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const size_t zoff = (size_t)blockIdx.y * MY * MX;
  const int p0 = blockIdx.x * C::NT, np = MY / 2;
  T* Ez = E + zoff;
  T* EXz = EX + zoff;
  bool below = false;
  const bool any = fft_core<MX, -1, false, false, true>(C::NT, sm, tw, [&](int t, int n) {
    int p = p0 + t;
    cx<T> v = zero_cx<T>();
    if (p < np) {
      T a = Ez[(size_t)(2 * p) * MX + n], b = Ez[(size_t)(2 * p + 1) * MX + n];
      v = mk(tmax(emin - a, (T)0), tmax(emin - b, (T)0));
      below |= !(a >= emin) | !(b >= emin);
    }
    return v;
  }, NoStore{}, [&] { return __syncthreads_or(below) != 0; });
  if (!any) return;  // nothing to raise, delta is zero
  fft_core<MX, +1, false, true, false>(C::NT, sm, tw, Derivative<T, MX>(kx0), [&](int t, int n, cx<T> d) {
    int p = p0 + t;
    if (p >= np) return;
#pragma unroll
    for (int r = 0; r < 2; r++) {
      size_t off = (size_t)(2 * p + r) * MX + n;
      EXz[off] += r ? d.y : d.x;
      Ez[off] = tmax(Ez[off], emin);
    }
  });
}

// Block-wide sum of NV doubles per thread, written (not accumulated) to
// out[q] by thread 0: a fixed reduction order, so results are reproducible.
// The block has THREADS threads, whole warps: a shuffle from a lane that does
// not exist has no defined value.
template <int NV, int THREADS>
__device__ __forceinline__ void block_sum_store(double (&v)[NV], double* out) {
  static_assert(THREADS % 32 == 0 && THREADS <= 1024, "the shuffles name every lane of every warp");
  __shared__ double red[32][NV];
#pragma unroll
  for (int q = 0; q < NV; q++)
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; q++) red[warp][q] = v[q];
  __syncthreads();
  if (warp == 0) {
    constexpr int nw = THREADS / 32;
#pragma unroll
    for (int q = 0; q < NV; q++) {
      double s = (lane < nw) ? red[lane][q] : 0.0;
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) out[q] = s;
    }
  }
}

// Per-level totals of partial sums: one block per level z, out[z*ostride + q] =
// sum over p < nparts of part[(z*nparts + p)*NQ + q], in a fixed order.
// Neighbouring threads take neighbouring values (kSumThreads is a multiple of
// NQ: a thread's are all of quantity t % NQ), several loads in flight, so that a
// level's partials (one per warp of k_row_fused or k_flux, 442 KB of SGS means
// at 768x768 points) arrive at the block's bandwidth and not one latency after
// the other: 32 levels of 512x512 25 -> 8 us (SGS) and 20 -> 4 us (divz) against
// 256 threads that each took a whole row of NQ values.
constexpr int kSumThreads = 960;
template <int NQ>
__global__ void __launch_bounds__(kSumThreads) k_sum_parts(const double* __restrict__ part, int nparts,
                                                           double* __restrict__ out, int ostride) {
  static_assert(kSumThreads % NQ == 0 && kSumThreads % 32 == 0 && NQ <= kSumThreads / 32, "a warp per quantity");
  __shared__ double red[kSumThreads];
  const int t = threadIdx.x, n = nparts * NQ;
  const double* p = part + (size_t)blockIdx.x * n;
  double s = 0.0;
#pragma unroll 8
  for (int i = t; i < n; i += kSumThreads) s += p[i];
  red[t] = s;
  __syncthreads();
  const int q = t >> 5;
  if (q >= NQ) return;
  s = 0.0;
  for (int i = t & 31; i < kSumThreads / NQ; i += 32) s += red[i * NQ + q];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((t & 31) == 0) out[(size_t)blockIdx.x * ostride + q] = s;
}

// Raw sums over the padded planes U, V at level 1 (blockIdx.y = 0) and nnz
// (blockIdx.y = 1): sum U, V, wind, U^2, V^2, wind^2, wind*U, wind*V, one
// partial per block in part[side][block][8] (summed in order by k_wall_final).
template <class T>
__global__ void __launch_bounds__(256) k_wall_sums(const T* __restrict__ U, const T* __restrict__ V, int NZ, size_t P, double* part) {
  const int side = blockIdx.y;
  const size_t off = side == 0 ? 0 : (size_t)(NZ - 1) * P;
  double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < P; i += (size_t)gridDim.x * blockDim.x) {
    double u = (double)U[off + i], v = (double)V[off + i];
    double wd = (double)sqrt((T)(U[off + i] * U[off + i] + V[off + i] * V[off + i]));
    s[0] += u; s[1] += v; s[2] += wd; s[3] += u * u; s[4] += v * v; s[5] += wd * wd; s[6] += wd * u; s[7] += wd * v;
  }
  block_sum_store<8, 256>(s, part + ((size_t)side * gridDim.x + blockIdx.x) * 8);
}

// As k_wall_sums, straight from the mixed rows of u and v (x-spectral, y
// physical): block `blk` of `nblk` transforms C::NT rows of U + iV of level 1
// (side 0) or nnz (one complex transform for both) and sums its points, without
// storing them.  Part of k_clip_walls, which has blocks of the same shape; the
// threads that fill the last warp (THREADS is 126 or 120 at six of the nine
// lengths) transform nothing and add zeros.
template <class T, int NSX>
__device__ __forceinline__ void wall_rows_block(const cx<T>* __restrict__ Um, const cx<T>* __restrict__ Vm, int side,
                                                int blk, int nblk, int MY, int NZ, double* part, cx<T>* sm,
                                                const cx<T>* __restrict__ tw) {
  constexpr int MX = 3 * NSX / 2, KX = NSX / 2;
  using C = RowCfg<MX>;
  const int y0 = blk * C::NT;
  const size_t off = side == 0 ? 0 : (size_t)(NZ - 1) * MY * KX;
  double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int yl = y0 + (int)(threadIdx.x / Split<MX>::N2);  // the row this thread loads
  const size_t ro = off + (size_t)(yl < MY ? yl : y0) * KX;
  fft_core<MX, +1, false, false, false>(C::NT, sm, tw, [&](int, int n) {
    const PairMode m = pair_mode<MX>(n, KX);
    return m.join(Um[ro + m.k], Vm[ro + m.k]);
  }, [&](int t, int, cx<T> uv) {
    if (y0 + t >= MY) return;
    const double u = (double)uv.x, v = (double)uv.y, wd = (double)sqrt((T)(uv.x * uv.x + uv.y * uv.y));
    s[0] += u; s[1] += v; s[2] += wd; s[3] += u * u; s[4] += v * v; s[5] += wd * wd; s[6] += wd * u; s[7] += wd * v;
  });
  block_sum_store<8, C::SUM_THREADS>(s, part + ((size_t)side * nblk + blk) * 8);
}

// Wall-model scalars for both walls (lowerbc.f90:56-124, upperbc.f90:63-122)
// and the global dudt, dvdt (lowerbc.f90:70-72) from the FP64 mean shadows.
// One block of 18 warps: a warp per sum (16 plane sums, then mru, mrv), each
// in a fixed order, then one lane per wall.  (One thread for everything: 55
// us per stage at any size; this 8-10 us.)
constexpr int kWallFinalThreads = 18 * 32;
static __global__ void __launch_bounds__(kWallFinalThreads)
k_wall_final(const double* __restrict__ part, int nblk, const double* __restrict__ mru,
             const double* __restrict__ mrv, StageArgs a, double P, double vk, double zody,
             double ufree, WallParams* wp, int* err) {
  __shared__ double acc[18];
  {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
    if (w < 16)
      for (int b = lane; b < nblk; b += 32) s += part[((size_t)(w >> 3) * nblk + b) * 8 + (w & 7)];
    else
      for (int z = lane; z < a.NZ; z += 32) s += w == 16 ? mru[z] : mrv[z];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) acc[w] = s;
  }
  __syncthreads();
  if (threadIdx.x > 1) return;
  const double su = acc[16], sv = acc[17];
  if (threadIdx.x == 0) {
    wp->dudt = su / a.NZ;
    wp->dvdt = sv / a.NZ;
    wp->utau_s = sqrt(a.zl / 2 * sqrt(wp->dvdt * wp->dvdt + (a.forcing - wp->dudt) * (a.forcing - wp->dudt)));
  }
  {
    const int side = threadIdx.x;
    const double* s = acc + side * 8;
    WallSide& w = wp->w[side];
    double mU = s[0] / P, mV = s[1] / P;
    w.u1xy = mU + (side ? a.ugal : 0.0);
    w.v1xy = mV + (side ? a.vgal : 0.0);
    double windm = s[2] / P;
    w.vsfc = sqrt(w.u1xy * w.u1xy + w.v1xy * w.v1xy);
    windm = fmax(windm, ufree);
    windm = fmax(windm, 0.01);
    w.windm = windm;
    w.vsfc = fmax(w.vsfc, 0.01);
    w.utau = w.vsfc * vk / zody;
    if (w.utau > 10.0) atomicOr(err, ERR_UTAU);
    double tep = fmin(fmax(w.u1xy / w.vsfc, -1.0), 1.0);
    double ut2 = w.utau * w.utau;
    double sg = copysign(1.0, w.v1xy);
    double sgn_wall = side ? 1.0 : -1.0;
    // theta = acos(tep): cos(theta) = tep, sin(theta) >= 0
    w.auuwm = sgn_wall * ut2 * tep;
    w.auvwm = sgn_wall * ut2 * sqrt((1.0 - tep) * (1.0 + tep)) * sg;
    // fluctuation moments: ufluc = U + ugal - u1xy = U - cu
    double cu = w.u1xy - a.ugal, cv = w.v1xy - a.vgal;
    double Suu = s[3] - 2 * cu * s[0] + P * cu * cu;
    double Svv = s[4] - 2 * cv * s[1] + P * cv * cv;
    double Sss = s[5] - 2 * windm * s[2] + P * windm * windm;
    double Sus = s[6] - windm * s[0] - cu * s[2] + P * cu * windm;
    double Svs = s[7] - windm * s[1] - cv * s[2] + P * cv * windm;
    w.ufluc2mroot = sqrt(Suu / P);
    w.vfluc2mroot = sqrt(Svv / P);
    w.suflucm = Sus / P;
    w.svflucm = Svs / P;
    double Smu = w.u1xy * w.u1xy * Sss + 2 * w.u1xy * windm * Sus + windm * windm * Suu;
    w.moengu2mroot = sqrt(Smu / P);
    w.moengv2mroot = w.moengu2mroot;  // moengv2m = sum(moengu2) in the reference (lowerbc.f90:121)
    w.denom = sqrt((windm * w.u1xy + w.suflucm) * (windm * w.u1xy + w.suflucm) +
                   (windm * w.v1xy + w.svflucm) * (windm * w.v1xy + w.svflucm));
  }
}

// Wall stress tau13, tau23 at one point (lowerbc.f90:126-161, upperbc.f90:124-158).
template <class T>
__device__ __forceinline__ void wall_stress(const WallSide& w, const WallParams& wp, const StageArgs& a, int side,
                                            T U, T V, T& tu, T& tv) {
  const double sg = side ? 1.0 : -1.0;
  const double ut2 = w.utau * w.utau;
  double Ud = (double)U + a.ugal, Vd = (double)V + a.vgal;
  double uf = Ud - w.u1xy, vf = Vd - w.v1xy;
  double wind = (double)sqrt(U * U + V * V);
  double ru, rv;
  switch (a.isurface) {
    case 1: ru = sg * ut2 / w.vsfc * Ud; rv = sg * ut2 / w.vsfc * Vd; break;
    case 2:
      ru = sg * ut2 / (w.windm * w.vsfc) * (w.windm * uf + wind * w.u1xy);
      rv = sg * ut2 / (w.windm * w.vsfc) * (w.windm * vf + wind * w.v1xy);
      break;
    case 3:
      ru = w.auuwm - sg * 0.35 * uf * ut2 / w.ufluc2mroot;
      rv = w.auvwm - sg * 0.35 * vf * ut2 / w.vfluc2mroot;
      break;
    case 4: ru = sg * ut2 * (wind * Ud) / w.denom; rv = sg * ut2 * (wind * Vd) / w.denom; break;
    case 5: {
      double sf = wind - w.windm;
      double mu = sf * w.u1xy + w.windm * uf, mv = sf * w.v1xy + w.windm * vf;
      ru = w.auuwm - sg * 0.35 * ut2 * mu / w.moengu2mroot;
      rv = w.auvwm - sg * 0.35 * ut2 * mv / w.moengv2mroot;
      break;
    }
    default: {  // 6
      double au = -a.zl / 2 * (a.forcing - wp.dudt), av = -a.zl / 2 * (-wp.dvdt);
      ru = -sg * au + sg * w.utau * wp.utau_s * uf / w.vsfc;
      rv = -sg * av + sg * w.utau * wp.utau_s * vf / w.vsfc;
      break;
    }
  }
  tu = (T)ru;
  tv = (T)rv;
}

// Padded-grid pointwise part of comp1 for level z (blockIdx.y + 1):
// compadv1 + complen + compsgs1 + compsgs3 written as the fields whose x/y
// derivatives and values the compress step needs:
//   u: A=UU+tuu (-d/dx), B=UV+tuv (-d/dy), Pu (value)
//   v: B (-d/dx), C=VV+tvv (-d/dy), Pv
//   w: D=0.5(U0+U1)W0+tuw (-d/dx), G=0.5(V0+V1)W0+tvw (-d/dy), Pw
//   e: F=0.5E0(U0+U1)-2xkk EX (-d/dx), H=0.5E0(V0+V1)-2xkk EY (-d/dy), Pe
// in: U,UX,UY,V,VX,VY,W,WX,WY,E,EX,EY   out: A,B,C,D,G,F,H,Pu,Pv,Pw,Pe
// stats: divz[z] (comp1.f90:145) and the SGS means (compsgs3.f90:71-78), one
// partial sum per (level, warp).
//
// What bounds it: the twelve fields in and eleven out, in HBM or L2.  A thread
// walks up `zchunk` levels of one point and keeps its window of levels z-1 to
// z+2 in registers, so each input is loaded once, one square root is taken per
// level instead of three and the strain of a level is summed once (96x128x45
// FP64, Smagorinsky: 102 -> 63 us; the fields take 45 us at 5 TB/s).
struct Ptr11 { void* p[11]; };
constexpr int kFluxThreads = 128;
template <class T>
__global__ void __launch_bounds__(kFluxThreads, sizeof(T) == 8 ? 4 : 6)
k_flux(const __grid_constant__ Ptr12 in, const __grid_constant__ Ptr11 out, const __grid_constant__ StageArgs a,
       const WallParams* __restrict__ wpp, double* __restrict__ divpart, double* __restrict__ sgspart, int zchunk) {
  const int NZ = a.NZ;
  const int za = blockIdx.y * zchunk + 1, zb = min(za + zchunk - 1, NZ);
  const size_t P = (size_t)a.MX * a.MY;
  const size_t idx = (size_t)blockIdx.x * kFluxThreads + threadIdx.x;
  const bool valid = idx < P;
  const size_t q = valid ? idx : 0;
  auto at = [&](int f, int L, int hi) -> T {  // zero outside levels 1..hi
    return (L >= 1 && L <= hi) ? reinterpret_cast<const T*>(in.p[f])[(size_t)(L - 1) * P + q] : (T)0;
  };
  auto Eat = [&](int L) { return at(9, L < 1 ? 1 : (L > NZ - 1 ? NZ - 1 : L), NZ - 1); };
  const T dzm = (T)a.dzm, todzm = (T)a.todzm, xkmax = (T)a.xkmax, nu = (T)a.nu, c01 = (T)0.1 * (T)a.dsl;
  const bool smag = a.imodel == 4, strain = smag || a.tke_production;
  const WallParams& wp = *wpp;

  // U, V, W of levels z-1, z, z+1, z+2; E of z-1, z, z+1; ux, vy, uy + vx and
  // the diagonal part of the strain of z, z+1, z+2; viscosity of z-1, z, z+1
  T U[4], V[4], W[4], E[3], ux[3], vy[3], sxy[3], g[3], xk[3];
  T shz = (T)0, sh1 = (T)0;  // strain of z and z+1
  T wx0, wy0, wx1, wy1;      // WX, WY of z and z+1
  auto diag = [&](int L, T uxL, T vyL, T sL, T wL, T wb) {
    const T wz = (L >= 1 && L <= NZ) ? (wL - wb) * dzm : (T)0;
    return uxL * uxL + vyL * vyL + wz * wz + (T)0.5 * sL * sL;
  };
  // loads level L into slot 3 of U, V, W and slot 2 of the derivatives
  auto fetch = [&](int L) {
    U[3] = at(0, L, NZ); V[3] = at(3, L, NZ); W[3] = at(6, L, NZ - 1);
    ux[2] = at(1, L, NZ); vy[2] = at(5, L, NZ); sxy[2] = at(2, L, NZ) + at(4, L, NZ);
    g[2] = diag(L, ux[2], vy[2], sxy[2], W[3], W[2]);
  };
  auto shift = [&]() {
#pragma unroll
    for (int i = 0; i < 3; i++) { U[i] = U[i + 1]; V[i] = V[i + 1]; W[i] = W[i + 1]; }
#pragma unroll
    for (int i = 0; i < 2; i++) { ux[i] = ux[i + 1]; vy[i] = vy[i + 1]; sxy[i] = sxy[i + 1]; g[i] = g[i + 1]; }
  };
  // strain of level L from the velocities of L and L+1 (of NZ-1 and NZ at the
  // top, of 1 and 2 at the bottom: UZ and VZ take the nearest interior face)
  auto shear = [&](T gl, T gu, T uz, T vz, T wx, T wy) {
    const T c = uz + wx, d = vz + wy;
    return gl + gu + c * c + d * d;
  };
  auto visc = [&](T sh, T e) { return (smag ? tmin(c01 * c01 * sqrt(sh), xkmax) : tmin(c01 * sqrt(e), xkmax)) + nu; };
  auto tau = [&](T x, T uz, T vz, T wx, T wy, T& tu, T& tv) {  // interior faces
    tu = -x * (uz + wx);
    tv = -x * (vz + wy);
  };

  // window of z = za: levels za-1 .. za+1
  T tum, tvm;
  {
    U[1] = U[2] = V[1] = V[2] = W[1] = ux[1] = vy[1] = sxy[1] = g[1] = (T)0;
    W[2] = at(6, za - 2, NZ - 1);
    fetch(za - 1);
    shift();
    fetch(za);
    shift();
    const T gm = g[0];
    fetch(za + 1);
    shift();
    E[0] = Eat(za - 1);
    E[1] = Eat(za);
    const T wxm = at(7, za - 1, NZ - 1), wym = at(8, za - 1, NZ - 1);
    wx1 = at(7, za, NZ - 1); wy1 = at(8, za, NZ - 1);
    T shm = (T)0;
    // faces: UZ of za-1 (of 1 when za = 1) and of za (of NZ-1 when za = NZ)
    const T uzm = za > 1 ? (U[1] - U[0]) * dzm : (U[2] - U[1]) * dzm, vzm = za > 1 ? (V[1] - V[0]) * dzm : (V[2] - V[1]) * dzm;
    const T uz = za < NZ ? (U[2] - U[1]) * dzm : uzm, vz = za < NZ ? (V[2] - V[1]) * dzm : vzm;
    if (strain) {
      shm = shear(gm, g[0], uzm, vzm, wxm, wym);
      sh1 = shear(g[0], g[1], uz, vz, wx1, wy1);
    }
    xk[1] = visc(shm, E[0]);
    xk[2] = visc(sh1, E[1]);
    if (za == 1) wall_stress<T>(wp.w[0], wp, a, 0, U[1], V[1], tum, tvm);
    else tau(xk[1], uzm, vzm, wxm, wym, tum, tvm);
  }
  for (int z = za; z <= zb; z++) {
    // slots 0..2: levels z-1, z, z+1; slot 3 / 2: z+2
    fetch(z + 2);
    xk[0] = xk[1]; xk[1] = xk[2];
    shz = sh1; wx0 = wx1; wy0 = wy1;
    E[2] = Eat(z + 1);
    wx1 = at(7, z + 1, NZ - 1); wy1 = at(8, z + 1, NZ - 1);
    const T uz = (U[2] - U[1]) * dzm, vz = (V[2] - V[1]) * dzm;
    if (z < NZ) {
      const T uz1 = z + 1 < NZ ? (U[3] - U[2]) * dzm : uz, vz1 = z + 1 < NZ ? (V[3] - V[2]) * dzm : vz;
      if (strain) sh1 = shear(g[1], g[2], uz1, vz1, wx1, wy1);
      xk[2] = visc(sh1, E[2]);
    }
    const T xkm = xk[0], xk0 = xk[1], xkp = xk[2];
    const T U0 = U[1], U1 = U[2], Um = U[0], V0 = V[1], V1 = V[2], Vm = V[0], W0 = W[1], W1 = W[2], Wm = W[0];
    const T s = xkm + xk0;
    const T tuu = -s * ux[0], tvv = -s * vy[0], tuv = -s * sxy[0] * (T)0.5;
    T tuw0, tvw0;
    if (z == NZ) wall_stress<T>(wp.w[1], wp, a, 1, U0, V0, tuw0, tvw0);
    else tau(xk0, uz, vz, wx0, wy0, tuw0, tvw0);
    const T wz0 = (W0 - Wm) * dzm;
    const T tww0 = -s * wz0;
    const size_t o = (size_t)(z - 1) * P + q;
    auto put = [&](int i, T v) { reinterpret_cast<T*>(out.p[i])[o] = v; };
    if (valid) {
      put(0, U0 * U0 + tuu);
      put(1, U0 * V0 + tuv);
      put(2, V0 * V0 + tvv);
      put(7, -((U1 + U0) * W0 - (Um + U0) * Wm) * todzm + (T)a.forcing - (tuw0 - tum) * dzm);
      put(8, -((V1 + V0) * W0 - (Vm + V0) * Wm) * todzm - (tvw0 - tvm) * dzm);
      if (z < NZ) {
        const T wz1 = (W1 - W0) * dzm;
        const T tww1 = -(xk0 + xkp) * wz1;
        put(3, (T)0.5 * (U0 + U1) * W0 + tuw0);
        put(4, (T)0.5 * (V0 + V1) * W0 + tvw0);
        const T hp = (T)0.5 * (W1 + W0), hm = (T)0.5 * (W0 + Wm);
        put(9, -(hp * hp - hm * hm) * dzm - (tww1 - tww0) * dzm);
        const int le = z < NZ - 2 ? z : NZ - 2;
        const T ex = at(10, le, NZ - 1), ey = at(11, le, NZ - 1);
        const T E0 = E[1], E1 = E[2], Em = E[0];
        put(5, (T)0.5 * E0 * (U0 + U1) - (T)2 * xk0 * ex);
        put(6, (T)0.5 * E0 * (V0 + V1) - (T)2 * xk0 * ey);
        T pe = -(W1 * E1 - Wm * Em) * todzm + ((xkp + xk0) * (E1 - E0) - (xk0 + xkm) * (E0 - Em)) * (T)a.dzm2 -
               (T)a.ceps * E0 * sqrt(E0);
        if (a.tke_production) pe += xk0 * shz;
        put(10, pe);
      } else {
        put(4, (T)0);  // G at the top level (pairs with C in the forward transform)
      }
    }
    const size_t slot = ((size_t)(z - 1) * gridDim.x + blockIdx.x) * (kFluxThreads / 32) + (threadIdx.x >> 5);
    const T d = ux[0] + vy[0] + wz0;
    double dd = valid ? (double)(d * d) : 0.0;
    for (int m = 16; m > 0; m >>= 1) dd += __shfl_xor_sync(0xffffffffu, dd, m);
    if ((threadIdx.x & 31) == 0) divpart[slot] = dd;
    if (a.mnout_sgs) {
      const T st[6] = {tuu, tvv, tuv, tww0, tuw0, tvw0};
#pragma unroll
      for (int i = 0; i < 6; i++) {
        double v = valid ? (double)st[i] : 0.0;
        for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
        if ((threadIdx.x & 31) == 0) sgspart[slot * 6 + i] = v;
      }
    }
    tum = tuw0; tvm = tvw0;
    shift();
    E[0] = E[1]; E[1] = E[2];
  }
}

// compress() in x fused with -d/dx: six paired forward row transforms of the
// flux fields, keep kx < nx/2, combine:
//   g0 (A, Pu) -> Xu1 = -ikx A^ + Pu^      g1 (B, Pv) -> Xv1 = -ikx B^ + Pv^, Xu2 = B^
//   g2 (C, G)  -> Xv2 = C^, Xw2 = G^       g3 (D, Pw) -> Xw1 = -ikx D^ + Pw^
//   g4 (F, Pe) -> Xe1 = -ikx F^ + Pe^      g5 (H, -)  -> Xe2 = H^
// in: A,B,C,D,G,F,H,Pu,Pv,Pw,Pe; out: Xu1,Xu2,Xv1,Xv2,Xw1,Xw2,Xe1,Xe2
template <class T, int NSX>
__global__ void __launch_bounds__(RowCfg<3 * NSX / 2>::THREADS)
k_x_forward(const __grid_constant__ Ptr11 in, const __grid_constant__ Ptr8 out, int MY, int NZ, T kx0, const cx<T>* __restrict__ tw) {
  constexpr int MX = 3 * NSX / 2;
  constexpr int KX = NSX / 2;
  using C = RowCfg<MX>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int g = blockIdx.z, z = blockIdx.y + 1;
  if (z == NZ && g >= 3) return;
  const int sA[6] = {0, 1, 2, 3, 5, 6}, sB[6] = {7, 8, 4, 9, 10, -1};
  const size_t zoff = (size_t)(z - 1) * MY;
  const T* A = (const T*)in.p[sA[g]] + zoff * MX;
  const T* B = sB[g] >= 0 ? (const T*)in.p[sB[g]] + zoff * MX : nullptr;
  const int y0 = blockIdx.x * C::NT;
  const int yl = y0 + (int)(threadIdx.x / Split<MX>::N2);  // the row this thread loads
  const size_t ro = (size_t)(yl < MY ? yl : y0) * MX;
  fft_core<MX, -1, false, false, true>(C::NT, sm, tw, [&](int, int n) { return mk(A[ro + n], B ? B[ro + n] : (T)0); },
                                       NoStore{});
  auto O = [&](int j) { return (cx<T>*)out.p[j] + zoff * KX; };
  for (int i = threadIdx.x; i < C::NT * KX; i += blockDim.x) {
    int t = i / KX, k = i - t * KX, y = y0 + t;
    if (y >= MY) continue;
    cx<T> zk = sm[t * MX + k], zm = conj(sm[t * MX + (MX - k) % MX]);
    cx<T> ah = (zk + zm) * (T)0.5;
    cx<T> d = zk - zm;
    cx<T> bh = mk(d.y * (T)0.5, -d.x * (T)0.5);
    T kk = kx0 * (T)k;
    cx<T> dxa = mk(kk * ah.y, -kk * ah.x);  // -i kx a^
    size_t o = (size_t)y * KX + k;
    switch (g) {
      case 0: O(0)[o] = dxa + bh; break;
      case 1: O(2)[o] = dxa + bh; O(1)[o] = ah; break;
      case 2: O(3)[o] = ah; if (z < NZ) O(5)[o] = bh; break;
      case 3: O(4)[o] = dxa + bh; break;
      case 4: O(6)[o] = dxa + bh; break;
      default: O(7)[o] = ah; break;
    }
  }
}

// compress() in y fused with -d/dy: for field f (u, v, w, e)
//   R^(ky) = (FFT_M(X1) - i ky FFT_M(X2)) / (MX*MY) at the kept ky,
// rw's plane mean removed (comp1.f90:172).  R^ of u, v, w is written to
// rnew[f]; for e, re = IFFT_NS(R^) (x-spectral) is written to rnew[3].
// TC columns per block (ColPlan); X1 and X2 go through the two tiles, the
// rows loaded in the permuted order, and meet in the registers of thread j,
// whose eight kept outputs are ky = j + M1 m: for e these are also the inputs
// of the inverse transform's radix-8 first pass.  Thread 0 first has the TMA
// prefetch into L2 the columns of the block `pdist` blocks ahead (les_tma.cuh;
// maps: tensor maps of X[0..7] as [NZ*M][KX] rows; pdist 0 prefetches nothing).
template <class T, int NS>
__global__ void __launch_bounds__(ColPlan<T, 3 * NS / 2>::THREADS, ColPlan<T, 3 * NS / 2>::CTAS)
k_y_forward(const __grid_constant__ Ptr8 X, const __grid_constant__ Ptr8 rnew, int KX, int NZ, T ky0, T scale, const cx<T>* __restrict__ tw,
            const __grid_constant__ ColMaps maps, unsigned pdist) {
  constexpr int M = 3 * NS / 2;
  using C = ColPlan<T, M>;
  constexpr int TC = C::TC, M1 = C::M1;
#pragma unroll
  for (int h = 0; h < 2; h++)
    prefetch_tile_ahead<T, M, TC>(maps, pdist, [&](unsigned bx, unsigned by, unsigned bz, int& q, int& cg, int& row0) {
      q = 2 * (int)bz + h; cg = (int)bx; row0 = (int)by * M;
      return !(bz >= 2 && (int)by + 1 == NZ);
    });
  extern __shared__ __align__(16) unsigned char smraw[];
  const int f = blockIdx.z, z = blockIdx.y + 1;
  if (f >= 2 && z == NZ) return;
  const int t = threadIdx.x % TC, j = threadIdx.x / TC;
  const int kx = blockIdx.x * TC + t;
  const bool in = kx < KX;
  cx<T>* buf = reinterpret_cast<cx<T>*>(smraw) + t;
  cx<T> w2[4];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const cx<T>* s = reinterpret_cast<const cx<T>*>(X.p[2 * f + h]) + (size_t)(z - 1) * M * KX + (in ? kx : 0);
    C::template first<12>(buf + h * C::BUF, j, [&](int row) { return s[row * KX]; });
  }
  C::twiddles2(tw, j, w2);
  __syncthreads();
  if constexpr (C::R3 > 1) {
    C::template pass2<12, false>(buf, w2, j);
    C::template pass2<12, false>(buf + C::BUF, w2, j);
    __syncthreads();
  }
  const ColTw1<T, M> tw1(tw, j);
  cx<T> w3[3], R[8];
  InPlace<M>::rotations(j, w3);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    cx<T> o[8];
    col_trunc_pass1<T, M>(buf + h * C::BUF, j, tw1, w3, o);
#pragma unroll
    for (int m = 0; m < 8; m++) {
      if (h == 0) R[m] = o[m];
      else {
        const T kk = ky0 * (T)(m < 4 ? j + M1 * m : j + M1 * m - NS);
        R[m] = mk(R[m].x + kk * o[m].y, R[m].y - kk * o[m].x) * scale;
      }
    }
  }
  if (j == 0) {
    R[4] = zero_cx<T>();  // Nyquist
    if (f == 2 && kx == 0) R[0] = zero_cx<T>();
  }
  cx<T>* dst = reinterpret_cast<cx<T>*>(rnew.p[f]) + (size_t)(z - 1) * NS * KX + kx;
  if (f < 3) {
#pragma unroll
    for (int m = 0; m < 8; m++)
      if (in) dst[(j + M1 * m) * KX] = R[m];
    return;
  }
  // e: inverse transform of length NS in the first tile (thread j writes the
  // elements it has just read)
  C::inverse_small(buf, tw, w2, j, R, [&](int row, cx<T> v) {
    if (in) dst[row * KX] = v;
  });
}

// Columns of the operator entry points (x-spectral planes, one per
// blockIdx.y), TC columns per block: forward y transform of length NS (times
// `scale`, Nyquist dropped) or of the padded rows cut to the kept modes
// (FROM_PAD), then the inverse transform back, padded (TO_PAD) or not, without
// leaving the block: expand, compress and deal in one column kernel each (src
// may be dst: a block reads its columns before it writes them).
template <class T, int NS, bool FROM_PAD, bool TO_PAD>
__global__ void __launch_bounds__(ColPlan<T, 3 * NS / 2>::THREADS, ColPlan<T, 3 * NS / 2>::CTAS)
k_col_resize(const cx<T>* src, cx<T>* dst, int KX, RowLayout ls, RowLayout ld, T scale, const cx<T>* __restrict__ tw) {
  constexpr int M = 3 * NS / 2;
  using C = ColPlan<T, M>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int t = threadIdx.x % C::TC, j = threadIdx.x / C::TC;
  const int kx = blockIdx.x * C::TC + t;
  const bool in = kx < KX;
  cx<T>* buf = reinterpret_cast<cx<T>*>(smraw) + t;
  src += blockIdx.y * ls.ps + (in ? kx : 0);
  dst += blockIdx.y * ld.ps + kx;
  const int rs = (int)ls.rs, rd = (int)ld.rs;
  auto load = [&](int row) { return src[row * rs]; };
  auto store = [&](int row, cx<T> v) {
    if (in) dst[row * rd] = v;
  };
  cx<T> w2[4], R[8];
  C::twiddles2(tw, j, w2);
  if constexpr (FROM_PAD) {
    C::template first<12>(buf, j, load);
    __syncthreads();
    if constexpr (C::R3 > 1) {
      C::template pass2<12, false>(buf, w2, j);
      __syncthreads();
    }
    const ColTw1<T, M> tw1(tw, j);
    cx<T> w3[3];
    InPlace<M>::rotations(j, w3);
    col_trunc_pass1<T, M>(buf, j, tw1, w3, R);
#pragma unroll
    for (int m = 0; m < 8; m++) R[m] = (m == 4 && j == 0) ? zero_cx<T>() : R[m] * scale;
  } else {
    C::forward_small(buf, tw, w2, j, scale, load, R);
  }
  if constexpr (TO_PAD) {
    const ColTw1<T, M> tw1(tw, j);
    cx<T> w3[3];
    InPlace<M>::rotations(j, w3);
    col_pad_pass1<T, M>(buf, j, R, tw1, w3);
    __syncthreads();
    if constexpr (C::R3 > 1) {
      C::template pass2<12, true>(buf, w2, j);
      __syncthreads();
    }
    C::template last<12>(buf, j, store);
  } else {
    C::inverse_small(buf, tw, w2, j, R, store);
  }
}

// The stage's e update (comp1.f90:131, comp2.f90:38) with re from its
// x-spectral rows: e = max(e - dtab2*re_old + dtab1*re, emin), re = c2r(rem),
// levels 1..nnz-1 (nrows = ny (nnz-1) rows; dtab2 = 0 in the first stage).
// The transform leaves its rows in shared memory; the elementwise pass then
// reads and writes whole rows, four values a thread, so the loads of e and
// re are not chained to the transform's stores.
template <class T, int NX>
__global__ void __launch_bounds__(RowCfg<NX>::THREADS)
k_e_update(const cx<T>* __restrict__ rem, T* __restrict__ re, T* __restrict__ e, int nrows, T dtab1, T dtab2, T emin,
           const cx<T>* __restrict__ tw) {
  using C = RowCfg<NX>;
  constexpr int KX = NX / 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int p0 = blockIdx.x * C::NT, np = nrows / 2;
  const int pl = p0 + (int)(threadIdx.x / Split<NX>::N2);  // the pair this thread loads
  const cx<T>* ra = rem + (size_t)(2 * (pl < np ? pl : p0)) * KX;
  fft_core<NX, +1, false, false, true>(C::NT, sm, tw, [&](int, int n) {
    const PairMode m = pair_mode<NX>(n, KX);
    return m.join(ra[m.k], ra[KX + m.k]);
  }, NoStore{});
  struct alignas(4 * sizeof(T)) V4 { T v[4]; };
  constexpr int ITEMS = C::NT * NX / 4;
#pragma unroll 2
  for (int i = threadIdx.x; i < ITEMS; i += C::THREADS) {
    const int t = i / (NX / 4), n = 4 * (i - t * (NX / 4)), p = p0 + t;
    if (p >= np) continue;
    const cx<T>* s = sm + t * NX + n;
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const size_t o = ((size_t)(2 * p + r) * NX + n) / 4;
      V4* ev = reinterpret_cast<V4*>(e) + o;
      V4* rv = reinterpret_cast<V4*>(re) + o;
      V4 x = *ev, nr;
      if (dtab2 != (T)0) {
        const V4 old = *rv;
#pragma unroll
        for (int q = 0; q < 4; q++) x.v[q] = x.v[q] - dtab2 * old.v[q];
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        nr.v[q] = r ? s[q].y : s[q].x;
        x.v[q] = tmax(x.v[q] + dtab1 * nr.v[q], emin);
      }
      *ev = x;
      *rv = nr;
    }
  }
}

// comprhs + press + tridv for every (kx, ky) column in z, in FP64, and (with
// UPDATE) comp2's update of u, v, w and their tendencies from the new p
// (comprhs.f90:17-35, press.F90:37-101, tridv.f90:29-53, comp2.f90:15-43).
//   rhs = ikx (Ru + u*/dtab1) + iky (Rv + v*/dtab1) + (Q(z) - Q(z-1))/dz,
//   Q = w*/dtab1 + Rw, u* = u - dtab2*Ru_old (comp1.f90:127);
//   Ru' = Ru - ikx p, Rv' = Rv - iky p, Rw' = Rw - (p(z+1)-p(z))/dz (mean 0),
//   u = u* + dtab1 Ru', ..., w plane mean removed.  The kx=ky=0 modes of u, v
//   and their tendencies live in the FP64 shadows mu, mv, mru, mrv.
// A block owns MODES modes; MODES consecutive threads take one chunk of L
// levels each, so a column is solved by blockDim/MODES threads: every thread
// sweeps its chunk with a zero inflow, the chunks' inflows come from a scan
// of (product of -d, last value) over the chunks, and r, d, p stay in shared
// memory.  The pivots d = 1/(b - d_prev) depend on the grid alone; a chunk
// starts from their closed form, d_n = -cosh((n-1/2)t)/cosh((n+1/2)t) with
// 2 cosh t - 2 = dz^2 (kx^2 + ky^2) (the determinants of the constant band
// with the wall's first row).  Bound by HBM on large grids (r and d never go
// there, and the update's second read of the inputs mostly hits L2), by the
// chain of levels on small ones, which the chunks cut to L + chunks / warp
// steps: 64x64x64 FP64 120 -> 10 us, 128x128x96 FP64 232 -> 46 us, 512x512x256
// mixed 1402 -> 1264 us against one thread per column and a separate update.
// Shared memory goes with the threads and levels of the launch (tables for 16
// warps in every block left 512x512x8 mixed at 44 us instead of 31).
template <class T, int MODES, bool RHS_IN_PH, bool UPDATE>
__global__ void __launch_bounds__(512)
k_press(cx<T>* __restrict__ uh, cx<T>* __restrict__ vh, cx<T>* __restrict__ wh, cx<T>* __restrict__ ruo,
        cx<T>* __restrict__ rvo, cx<T>* __restrict__ rwo, const cx<T>* __restrict__ run, const cx<T>* __restrict__ rvn,
        const cx<T>* __restrict__ rwn, cx<double>* __restrict__ ph, double* mu, double* mv, double* mru, double* mrv,
        StageArgs a, int L, int* err) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int KX = a.KX, NY = a.NY, NZ = a.NZ;
  const int nm = KX * NY, nt = blockDim.x, tid = threadIdx.x;
  cx<double>* const R = reinterpret_cast<cx<double>*>(smraw) + tid;                        // R[l nt]: r, then p
  double* const D = reinterpret_cast<double*>(smraw + (size_t)L * nt * sizeof(cx<double>)) + tid;  // D[l nt]
  const int md = tid % MODES, c = tid / MODES;
  const int lane = tid & 31, warp = tid >> 5, nwarp = nt >> 5;
  // totals of a warp's chunks: [forward, backward][warp][product, re, im][mode]
  double* const tots = D - tid + (size_t)L * nt + md;
  auto tot = [&](int dir, int w, int q) -> double& { return tots[((dir * nwarp + w) * 3 + q) * MODES]; };
  const int m = blockIdx.x * MODES + md;
  const int ky = m / KX, kx = m - ky * KX;
  const bool live = ky != NY / 2 && m != 0;
  const double xk = a.kx0 * kx, yk = a.ky0 * signed_k(ky, NY);
  const double dzdz = a.dz * a.dz, kap = dzdz * (xk * xk + yk * yk);
  const double dtabm = a.dtabm, dtab1 = a.dtab1, dtab2 = a.zeta ? a.dtab2 : 0.0;
  const int zs = c * L + 1, n = min(L, NZ - zs + 1);  // levels zs .. zs + n - 1 (n <= 0: none)
  auto at = [&](int z) { return (size_t)(z - 1) * nm + m; };
  auto ld = [](cx<T> v) { return mk((double)v.x, (double)v.y); };
  // LB levels' loads in flight at a time
  constexpr int LB = sizeof(T) == 4 ? 4 : 2;
  cx<T> u[LB], v[LB], w[LB], uo[LB], vo[LB], wo[LB], un[LB], vn[LB], wn[LB];
  auto fetch = [&](int l0) {
#pragma unroll
    for (int i = 0; i < LB; i++) {
      const int z = zs + l0 + i;
      if (l0 + i >= n) break;
      const size_t o = at(z);
      u[i] = uh[o]; v[i] = vh[o]; uo[i] = ruo[o]; vo[i] = rvo[o]; un[i] = run[o]; vn[i] = rvn[o];
      const bool inw = z < NZ;
      w[i] = inw ? wh[o] : zero_cx<T>(); wo[i] = inw ? rwo[o] : zero_cx<T>(); wn[i] = inw ? rwn[o] : zero_cx<T>();
    }
  };
  // forward sweep of the chunk with zero inflow; pr: product of -d of the
  // levels zs - 1 .. zs + n - 2
  double din = -1.0, pr = 1.0;
  cx<double> rl = mk(0.0, 0.0);
  if (live && n > 0) {
    cx<double> qprev = mk(0.0, 0.0);
    if (!RHS_IN_PH && c > 0) {
      const size_t o = at(zs - 1);
      qprev = (ld(wh[o]) - ld(rwo[o]) * dtab2) * dtabm + ld(rwn[o]);
    }
    if (c > 0) {
      const double t = 2.0 * asinh(0.5 * sqrt(kap)), e = exp(-t), n2 = 2.0 * (zs - 1);
      din = -e * (1.0 + exp(-(n2 - 1.0) * t)) / (1.0 + exp(-(n2 + 1.0) * t));
    }
    double dprev = din;
    for (int l0 = 0; l0 < n; l0 += LB) {
      if (!RHS_IN_PH) fetch(l0);
#pragma unroll
      for (int i = 0; i < LB; i++) {
        const int l = l0 + i, z = zs + l;
        if (l >= n) break;
        cx<double> rhs;
        if constexpr (RHS_IN_PH) rhs = ph[at(z)];
        else {
          const cx<double> gu = ld(un[i]) + (ld(u[i]) - ld(uo[i]) * dtab2) * dtabm;
          const cx<double> gv = ld(vn[i]) + (ld(v[i]) - ld(vo[i]) * dtab2) * dtabm;
          const cx<double> q = (ld(w[i]) - ld(wo[i]) * dtab2) * dtabm + ld(wn[i]);
          rhs = mul_i(gu) * xk + mul_i(gv) * yk + (q - qprev) * a.dzm;
          qprev = q;
        }
        pr *= -dprev;
        const double d = 1.0 / (-kap - (z == NZ ? 1.0 : 2.0) - dprev);
        rl = rhs * dzdz - rl * dprev;
        D[l * nt] = d;
        R[l * nt] = rl;
        dprev = d;
      }
    }
  }
  // inflow of each chunk: exclusive scan of y -> val + pr y over the chunks
  // below (forward) or above (backward)
  auto inflow = [&](int dir, double ip, cx<double> iv) -> cx<double> {
#pragma unroll
    for (int o = MODES; o < 32; o *= 2) {
      const int src = dir ? lane + o : lane - o;
      const double p2 = __shfl_sync(0xffffffffu, ip, src & 31);
      const cx<double> v2 = mk(__shfl_sync(0xffffffffu, iv.x, src & 31), __shfl_sync(0xffffffffu, iv.y, src & 31));
      if (src >= 0 && src < 32) {
        iv = iv + v2 * ip;
        ip *= p2;
      }
    }
    if (dir ? lane < MODES : lane >= 32 - MODES) {
      tot(dir, warp, 0) = ip;
      tot(dir, warp, 1) = iv.x;
      tot(dir, warp, 2) = iv.y;
    }
    __syncthreads();
    cx<double> y = mk(0.0, 0.0);
    for (int k = 0; k < (dir ? nwarp - 1 - warp : warp); k++) {
      const int w = dir ? nwarp - 1 - k : k;
      y = mk(tot(dir, w, 1), tot(dir, w, 2)) + y * tot(dir, w, 0);
    }
    if (MODES == 32) return y;
    // this chunk's inflow: the neighbour chunk's inclusive value applied to y
    const int src = dir ? lane + MODES : lane - MODES;
    const double p2 = __shfl_sync(0xffffffffu, ip, src & 31);
    const cx<double> v2 = mk(__shfl_sync(0xffffffffu, iv.x, src & 31), __shfl_sync(0xffffffffu, iv.y, src & 31));
    return (src >= 0 && src < 32) ? v2 + y * p2 : y;
  };
  const cx<double> rin = inflow(0, pr, rl);
  // backward sweep: the forward inflow added on the way (r = r_local + P rin,
  // P the product of -d down to the chunk's first level), zero p above
  cx<double> p = mk(0.0, 0.0);
  double pb = 1.0;
  if (live && n > 0) {
    double P = -din;
    for (int l = 0; l < n; l++) {  // forward products
      R[l * nt] = R[l * nt] + rin * P;
      P *= -D[l * nt];
    }
    for (int l = n - 1; l >= 0; l--) {
      const double d = D[l * nt];
      p = (R[l * nt] - p) * d;
      R[l * nt] = p;
      pb *= -d;
    }
  }
  const cx<double> pin = inflow(1, pb, p);  // p of level zs + n
  if (live && n > 0) {
    double P = 1.0;
    for (int l = n - 1; l >= 0; l--) {
      P *= -D[l * nt];
      R[l * nt] = R[l * nt] + pin * P;
    }
  }
  bool bad = false;
  auto t2 = [](cx<double> v) { return mk((T)v.x, (T)v.y); };
  for (int l0 = 0; l0 < n; l0 += LB) {
    if (UPDATE && live) fetch(l0);
#pragma unroll
    for (int i = 0; i < LB; i++) {
      const int l = l0 + i, z = zs + l;
      if (l >= n) break;
      const size_t o = at(z);
      const cx<double> p0 = live ? R[l * nt] : mk(0.0, 0.0);
      ph[o] = p0;
      if constexpr (UPDATE) {
        if (live) {
          const cx<double> rpu = ld(un[i]) - mul_i(p0) * xk, rpv = ld(vn[i]) - mul_i(p0) * yk;
          const cx<double> nu = ld(u[i]) - ld(uo[i]) * dtab2 + rpu * dtab1;
          const cx<double> nv = ld(v[i]) - ld(vo[i]) * dtab2 + rpv * dtab1;
          uh[o] = t2(nu); vh[o] = t2(nv); ruo[o] = t2(rpu); rvo[o] = t2(rpv);
          bad = bad || !isfinite(nu.x + nu.y + nv.x + nv.y);
          if (z < NZ) {
            const cx<double> p1 = l + 1 < n ? R[(l + 1) * nt] : pin;
            const cx<double> rpw = ld(wn[i]) - (p1 - p0) * a.dzm;
            const cx<double> nw = ld(w[i]) - ld(wo[i]) * dtab2 + rpw * dtab1;
            wh[o] = t2(nw); rwo[o] = t2(rpw);
            bad = bad || !isfinite(nw.x + nw.y);
          }
        } else if (m == 0) {
          const double rpu = (double)run[o].x, rpv = (double)rvn[o].x;
          const double nu = mu[z - 1] - dtab2 * mru[z - 1] + dtab1 * rpu, nv = mv[z - 1] - dtab2 * mrv[z - 1] + dtab1 * rpv;
          mu[z - 1] = nu; mv[z - 1] = nv; mru[z - 1] = rpu; mrv[z - 1] = rpv;
          uh[o] = t2(mk(nu, 0.0)); vh[o] = t2(mk(nv, 0.0));
          ruo[o] = t2(mk(rpu, 0.0)); rvo[o] = t2(mk(rpv, 0.0));
          if (z < NZ) { wh[o] = t2(mk(0.0, 0.0)); rwo[o] = t2(mk(0.0, 0.0)); }
          bad = bad || !isfinite(nu) || !isfinite(nv);
        }
      }
    }
  }
  if (UPDATE && bad) atomicOr(err, ERR_NAN);
}

// The pressure solve of k_press with one thread per column, for more levels
// than k_press's chunks hold: Thomas sweeps through scratch d[z][mode],
// r[z][mode].
template <class T, bool RHS_IN_PH>
__global__ void k_press_long(const cx<T>* __restrict__ uh, const cx<T>* __restrict__ vh, const cx<T>* __restrict__ wh,
                        const cx<T>* __restrict__ ruo, const cx<T>* __restrict__ rvo, const cx<T>* __restrict__ rwo,
                        const cx<T>* __restrict__ run, const cx<T>* __restrict__ rvn, const cx<T>* __restrict__ rwn,
                        cx<double>* __restrict__ ph, double* __restrict__ dscr, cx<double>* __restrict__ rscr,
                        StageArgs a) {
  const int KX = a.KX, NY = a.NY, NZ = a.NZ;
  const int nm = KX * NY;
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= nm) return;
  const int ky = m / KX, kx = m - ky * KX;
  if (ky == NY / 2 || (kx == 0 && ky == 0)) {
    for (int z = 0; z < NZ; z++) ph[(size_t)z * nm + m] = mk(0.0, 0.0);
    return;
  }
  const double xk = a.kx0 * kx, yk = a.ky0 * signed_k(ky, NY);
  const double k2 = xk * xk + yk * yk, dzdz = a.dz * a.dz;
  const double dtabm = a.dtabm, dtab2 = a.zeta ? a.dtab2 : 0.0;
  auto ld = [&](const cx<T>* f, int z) -> cx<double> {
    cx<T> v = f[(size_t)(z - 1) * nm + m];
    return mk((double)v.x, (double)v.y);
  };
  cx<double> qprev = mk(0.0, 0.0), rprev = mk(0.0, 0.0);
  double dprev = 0.0;
  for (int z = 1; z <= NZ; z++) {
    cx<double> us = ld(uh, z) - ld(ruo, z) * dtab2;
    cx<double> vs = ld(vh, z) - ld(rvo, z) * dtab2;
    cx<double> q = mk(0.0, 0.0);
    if (z < NZ) q = (ld(wh, z) - ld(rwo, z) * dtab2) * dtabm + ld(rwn, z);
    cx<double> gu = ld(run, z) + us * dtabm, gv = ld(rvn, z) + vs * dtabm;
    cx<double> rhs = mul_i(gu) * xk + mul_i(gv) * yk + (q - qprev) * a.dzm;
    if (RHS_IN_PH) rhs = ph[(size_t)(z - 1) * nm + m];
    cx<double> r = rhs * dzdz;
    double b = -dzdz * k2 - ((z == 1 || z == NZ) ? 1.0 : 2.0);
    double d;
    if (z == 1) d = 1.0 / b;
    else {
      double fac = dprev;
      d = 1.0 / (b - fac);
      r = r - rprev * fac;
    }
    dscr[(size_t)(z - 1) * nm + m] = d;
    rscr[(size_t)(z - 1) * nm + m] = r;
    dprev = d; rprev = r; qprev = q;
  }
  cx<double> p = rprev * dprev;
  ph[(size_t)(NZ - 1) * nm + m] = p;
  for (int z = NZ - 1; z >= 1; z--) {
    double d = dscr[(size_t)(z - 1) * nm + m];
    cx<double> r = rscr[(size_t)(z - 1) * nm + m];
    p = (r - p) * d;
    ph[(size_t)(z - 1) * nm + m] = p;
  }
}

// comp2 (comp2.f90:15-43) in spectral space, FP64 arithmetic:
//   Ru' = Ru - ikx p, Rv' = Rv - iky p, Rw' = Rw - (p(z+1)-p(z))/dz (mean 0),
//   u = u* + dtab1 Ru', ..., w plane mean removed.  The kx=ky=0 modes of u, v
//   and their tendencies live in the FP64 shadows mu, mv, mru, mrv.
template <class T>
__global__ void k_update(cx<T>* uh, cx<T>* vh, cx<T>* wh, const cx<T>* ruo, const cx<T>* rvo, const cx<T>* rwo,
                         const cx<T>* run, const cx<T>* rvn, const cx<T>* rwn, cx<T>* ruout, cx<T>* rvout,
                         cx<T>* rwout, const cx<double>* __restrict__ ph, double* __restrict__ mu,
                         double* __restrict__ mv, double* __restrict__ mru, double* __restrict__ mrv, StageArgs a,
                         int* err) {
  const int KX = a.KX, NY = a.NY, NZ = a.NZ;
  const int nm = KX * NY;
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int z = blockIdx.y + 1;
  if (m >= nm) return;
  const int ky = m / KX, kx = m - ky * KX;
  if (ky == NY / 2) return;
  const double xk = a.kx0 * kx, yk = a.ky0 * signed_k(ky, NY);
  const double dtab1 = a.dtab1, dtab2 = a.zeta ? a.dtab2 : 0.0;
  const size_t o = (size_t)(z - 1) * nm + m;
  auto d2 = [](cx<T> v) { return mk((double)v.x, (double)v.y); };
  auto t2 = [](cx<double> v) { return mk((T)v.x, (T)v.y); };
  const cx<double> p = ph[o];
  bool bad = false;
  if (m == 0) {
    double us = mu[z - 1] - dtab2 * mru[z - 1];
    double vs = mv[z - 1] - dtab2 * mrv[z - 1];
    double rpu = (double)run[o].x, rpv = (double)rvn[o].x;
    double un = us + dtab1 * rpu, vn = vs + dtab1 * rpv;
    mu[z - 1] = un; mv[z - 1] = vn; mru[z - 1] = rpu; mrv[z - 1] = rpv;
    uh[o] = t2(mk(un, 0.0)); vh[o] = t2(mk(vn, 0.0));
    ruout[o] = t2(mk(rpu, 0.0)); rvout[o] = t2(mk(rpv, 0.0));
    if (z < NZ) { wh[o] = t2(mk(0.0, 0.0)); rwout[o] = t2(mk(0.0, 0.0)); }
    bad = !isfinite(un) || !isfinite(vn);
  } else {
    cx<double> rpu = d2(run[o]) - mul_i(p) * xk;
    cx<double> rpv = d2(rvn[o]) - mul_i(p) * yk;
    cx<double> un = d2(uh[o]) - d2(ruo[o]) * dtab2 + rpu * dtab1;
    cx<double> vn = d2(vh[o]) - d2(rvo[o]) * dtab2 + rpv * dtab1;
    uh[o] = t2(un); vh[o] = t2(vn); ruout[o] = t2(rpu); rvout[o] = t2(rpv);
    bad = !isfinite(un.x + un.y + vn.x + vn.y);
    if (z < NZ) {
      cx<double> p1 = ph[o + nm];
      cx<double> rpw = d2(rwn[o]) - (p1 - p) * a.dzm;
      cx<double> wn = d2(wh[o]) - d2(rwo[o]) * dtab2 + rpw * dtab1;
      wh[o] = t2(wn); rwout[o] = t2(rpw);
      bad = bad || !isfinite(wn.x + wn.y);
    }
  }
  if (bad) atomicOr(err, ERR_NAN);
}

// comprhs (comprhs.f90:17-35) alone: ph = rhs in the small-spectrum
// convention (used by the split entry points; k_press recomputes it inline).
template <class T>
__global__ void k_rhs(const cx<T>* __restrict__ uh, const cx<T>* __restrict__ vh, const cx<T>* __restrict__ wh,
                      const cx<T>* __restrict__ ru, const cx<T>* __restrict__ rv, const cx<T>* __restrict__ rw,
                      cx<double>* __restrict__ ph, StageArgs a) {
  const int KX = a.KX, NY = a.NY, NZ = a.NZ;
  const int nm = KX * NY;
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int z = blockIdx.y + 1;
  if (m >= nm) return;
  const int ky = m / KX, kx = m - ky * KX;
  const size_t o = (size_t)(z - 1) * nm + m;
  if (ky == NY / 2) { ph[o] = mk(0.0, 0.0); return; }
  const double xk = a.kx0 * kx, yk = a.ky0 * signed_k(ky, NY);
  auto d2 = [](cx<T> v) { return mk((double)v.x, (double)v.y); };
  cx<double> q = mk(0.0, 0.0), qm = mk(0.0, 0.0);
  if (z < NZ) q = d2(wh[o]) * a.dtabm + d2(rw[o]);
  if (z > 1) qm = d2(wh[o - nm]) * a.dtabm + d2(rw[o - nm]);
  cx<double> gu = d2(ru[o]) + d2(uh[o]) * a.dtabm, gv = d2(rv[o]) + d2(vh[o]) * a.dtabm;
  ph[o] = mul_i(gu) * xk + mul_i(gv) * yk + (q - qm) * a.dzm;
}

// The zeta part of the stage on u, v, w (comp1.f90:126-133) as a separate
// pass, for the split entry points: u -= dtab2*ru (spectral + FP64 shadows).
template <class T>
__global__ void k_zeta(cx<T>* uh, cx<T>* vh, cx<T>* wh, const cx<T>* ruo, const cx<T>* rvo, const cx<T>* rwo,
                       double* mu, double* mv, const double* mru, const double* mrv, StageArgs a) {
  const int nm = a.KX * a.NY;
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int z = blockIdx.y + 1;
  if (m >= nm) return;
  const size_t o = (size_t)(z - 1) * nm + m;
  const T d = (T)a.dtab2;
  if (m == 0) {
    mu[z - 1] -= a.dtab2 * mru[z - 1];
    mv[z - 1] -= a.dtab2 * mrv[z - 1];
    uh[o] = mk((T)mu[z - 1], (T)0);
    vh[o] = mk((T)mv[z - 1], (T)0);
  } else {
    uh[o] = uh[o] - ruo[o] * d;
    vh[o] = vh[o] - rvo[o] * d;
  }
  if (z < a.NZ) wh[o] = wh[o] - rwo[o] * d;
}

// SplitMix64 (Steele, Lea & Flood 2014) as a counter-based stream: output n
// of the stream seeded with s is mix(s + (n+1)*0x9e3779b97f4a7c15).
static __device__ __forceinline__ uint64_t splitmix64_at(uint64_t s, uint64_t n) {
  uint64_t z = s + (n + 1) * 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

// Seeded initial condition on the small grid (levels 1..nnz): parabolic mean
// plus uniform(-amp, amp)*utau perturbations for field f (0 u, 1 v, 2 w).
template <class T>
__global__ void k_ic_fill(T* __restrict__ out, int f, unsigned long long seed, int NX, int NY, int NZ, double dz,
                          double hh, double ub, double amp, double utau) {
  const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t tot = (size_t)NX * NY * NZ;
  if (n >= tot) return;
  const int iz = (int)(n / ((size_t)NX * NY)) + 1;
  double mean = 0.0;
  if (f == 0) {
    double zm = ((double)iz - 0.5) * dz;
    double eta = (zm - hh) / hh;
    mean = 1.5 * ub * (1.0 - eta * eta);
  }
  uint64_t r = splitmix64_at((uint64_t)seed + (uint64_t)f, (uint64_t)n);
  double u01 = (double)(r >> 11) * (1.0 / 9007199254740992.0);
  double val = mean + (2.0 * u01 - 1.0) * amp * utau;
  if (f == 2 && iz == NZ) val = 0.0;
  out[n] = (T)val;
}

// Per-level plane sums (FP64) of up to 4 small-grid fields: acc[z*8 + q].
// One block per level (blockIdx.y), so the sums are reproducible.
template <class T>
__global__ void __launch_bounds__(1024) k_plane_sums(const T* __restrict__ f0, const T* __restrict__ f1, const T* __restrict__ f2,
                             const T* __restrict__ f3, size_t P, double* acc) {
  const size_t off = (size_t)blockIdx.y * P;
  double s[4] = {0, 0, 0, 0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < P; i += (size_t)gridDim.x * blockDim.x) {
    if (f0) s[0] += (double)f0[off + i];
    if (f1) s[1] += (double)f1[off + i];
    if (f2) s[2] += (double)f2[off + i];
    if (f3) s[3] += (double)f3[off + i];
  }
  block_sum_store<4, 1024>(s, acc + (size_t)blockIdx.y * 8);
}

// Moments of compmn (compmn.F90:29-62) at level iz = blockIdx.y + 1:
// u, v, w are small-grid physical fields on levels 1..nnz (u, v at nnz+1 are
// zero); means[z*8 + 0/1] hold the plane means of u and v.  One block per
// level, as k_plane_sums.
template <class T>
__global__ void __launch_bounds__(1024) k_moments(const T* __restrict__ u, const T* __restrict__ v, const T* __restrict__ w, size_t P, int NZ,
                          const double* __restrict__ means, double* acc) {
  const int iz = blockIdx.y + 1;
  const size_t off = (size_t)(iz - 1) * P;
  const T um = (T)means[(size_t)(iz - 1) * 8 + 0], vm = (T)means[(size_t)(iz - 1) * 8 + 1];
  const T um1 = iz < NZ ? (T)means[(size_t)iz * 8 + 0] : (T)0;
  const T vm1 = iz < NZ ? (T)means[(size_t)iz * 8 + 1] : (T)0;
  double s[6] = {0, 0, 0, 0, 0, 0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < P; i += (size_t)gridDim.x * blockDim.x) {
    T u1 = iz < NZ ? u[off + P + i] : (T)0;
    T v1 = iz < NZ ? v[off + P + i] : (T)0;
    T ul = (T)0.5 * ((u[off + i] - um) + u1 - um1);
    T vl = (T)0.5 * ((v[off + i] - vm) + v1 - vm1);
    T w0 = w[off + i];
    s[0] += (double)(ul * ul); s[1] += (double)(vl * vl); s[2] += (double)(w0 * w0);
    s[3] += (double)(ul * w0); s[4] += (double)(vl * w0); s[5] += (double)(ul * vl);
  }
  block_sum_store<6, 1024>(s, acc + (size_t)(iz - 1) * 8);
}

// Max |u|, |v|, |w| for the CFL time step (les.F90:205-207).
template <class T>
__global__ void k_absmax3(const T* __restrict__ u, const T* __restrict__ v, const T* __restrict__ w, size_t n,
                          unsigned long long* out) {
  T m[3] = {0, 0, 0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    m[0] = tmax(m[0], (T)fabs(u[i])); m[1] = tmax(m[1], (T)fabs(v[i])); m[2] = tmax(m[2], (T)fabs(w[i]));
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    double d = (double)m[q];
    for (int o = 16; o > 0; o >>= 1) d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out + q, (unsigned long long)__double_as_longlong(d));
  }
}

// comp2's e update in physical space (split entry points).
template <class T>
__global__ void k_e_update_phys(T* __restrict__ e, const T* __restrict__ re, size_t n, T dtab1, T emin) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) e[i] = tmax(e[i] + dtab1 * re[i], emin);
}

// Elementwise helpers.
template <class T>
__global__ void k_fill(T* p, size_t n, T v) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}
template <class S, class D>
__global__ void k_convert(const S* __restrict__ in, D* __restrict__ out, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (D)in[i];
}
// Set the kx=ky=0 mode of every level of a spectral array from FP64 values.
template <class T>
__global__ void k_set_mean(cx<T>* __restrict__ sp, const double* __restrict__ mean, size_t nm, int NZ) {
  int z = blockIdx.x * blockDim.x + threadIdx.x;
  if (z < NZ) sp[(size_t)z * nm] = mk((T)mean[z], (T)0);
}

// Batched 1D spectral derivative (xderiv/yderiv of filter_fftw.f90:138-248)
// along rows or columns of real planes, pairing rows/columns.
template <class T, int N>
__global__ void __launch_bounds__(RowCfg<N>::THREADS, sizeof(T) == 8 ? 3 : 4)
k_op_xderiv(const T* __restrict__ in, T* __restrict__ out, int nrows, T k0, const cx<T>* __restrict__ tw) {
  using C = RowCfg<N>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int p0 = blockIdx.x * C::NT;
  const int npair = (nrows + 1) / 2;
  if (p0 >= npair) return;
  fft_core<N, -1, false, false, true>(C::NT, sm, tw, [&](int t, int n) {
    int p = p0 + t;
    return (p < npair) ? mk(in[(size_t)(2 * p) * N + n], (2 * p + 1 < nrows) ? in[(size_t)(2 * p + 1) * N + n] : (T)0)
                       : zero_cx<T>();
  }, NoStore{});
  fft_core<N, +1, false, true, false>(C::NT, sm, tw, Derivative<T, N>(k0), [&](int t, int n, cx<T> v) {
    int p = p0 + t;
    if (p >= npair) return;
    out[(size_t)(2 * p) * N + n] = v.x;
    if (2 * p + 1 < nrows) out[(size_t)(2 * p + 1) * N + n] = v.y;
  });
}
template <class T, int N>
__global__ void __launch_bounds__(ColCfg<N, T>::THREADS, (sizeof(T) == 8 ? 384 : 512) / ColCfg<N, T>::THREADS)
k_op_yderiv(const T* __restrict__ in, T* __restrict__ out, int n1, T k0, const cx<T>* __restrict__ tw) {
  using C = ColCfg<N, T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const size_t plane = (size_t)blockIdx.y * N * n1;
  const int ncp = (n1 + 1) / 2, c0 = blockIdx.x * C::TC;
  const int cl = c0 + (int)(threadIdx.x % C::TC);  // the column pair this thread loads
  const T* col = in + plane + 2 * (cl < ncp ? cl : c0);
  const int second = 2 * (cl < ncp ? cl : c0) + 1 < n1 ? 1 : 0;
  fft_core<N, -1, true, false, true>(C::TC, sm, tw, [&](int, int n) {
    const T* r = col + (size_t)n * n1;
    const T b = r[second];
    return mk(r[0], second ? b : (T)0);
  }, NoStore{});
  fft_core<N, +1, true, true, false>(C::TC, sm, tw, Derivative<T, N>(k0), [&](int t, int n, cx<T> v) {
    int c = c0 + t;
    if (c >= ncp) return;
    out[plane + (size_t)n * n1 + 2 * c] = v.x;
    if (2 * c + 1 < n1) out[plane + (size_t)n * n1 + 2 * c + 1] = v.y;
  });
}

// tridv (tridv.f90:1-55) for one right-hand side per thread; bdar is
// (ny, n, 4) column-major.
static __global__ void k_op_tridv(double* bdar, int ny, int n) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ny) return;
  double* b = bdar;
  double* d = bdar + (size_t)ny * n;
  double* a = bdar + (size_t)2 * ny * n;
  double* r = bdar + (size_t)3 * ny * n;
  auto I = [ny, j](int i) { return (size_t)(i - 1) * ny + j; };
  if (n <= 1) { r[I(1)] = r[I(1)] / d[I(1)]; return; }
  d[I(1)] = 1.0 / d[I(1)];
  for (int i = 2; i <= n; i++) {
    double fac = b[I(i)] * d[I(i - 1)];
    d[I(i)] = 1.0 / (d[I(i)] - fac * a[I(i - 1)]);
    r[I(i)] = r[I(i)] - fac * r[I(i - 1)];
  }
  r[I(n)] = r[I(n)] * d[I(n)];
  for (int i = n - 1; i >= 1; i--) r[I(i)] = d[I(i)] * (r[I(i)] - a[I(i)] * r[I(i + 1)]);
}

}  // namespace les

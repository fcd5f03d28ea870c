// fft_inplace.cuh -- in-place transforms of the 3/2-padded lengths N = 12 M1.
//
// The inverse runs decimation in frequency, natural order in, permuted order
// out; the forward transform runs the same passes backwards, permuted in,
// natural out.  Neither the pointwise phase of the fused row kernel nor the
// y-column kernels (whose rows are loaded and stored one by one) care about
// the order of the padded points, so nothing is ever reordered: every pass
// reads and writes the same elements, and a pass needs one barrier instead of
// the two of an autosorting pass.
//   element n = b M1 + r R3 + i   (M1 = R2 R3, b < 12, r < R2, i < R3)
//   pass 1 (radix 12, over b): thread j = r R3 + i
//   pass 2 (radix R2, over r): thread (b, i), twiddle W_M1^(r i)
//   pass 3 (radix R3, over i): thread (b, r); none when R3 = 1
// The first factor is 12 because a padded line has modes |k| < N/3 only: of
// pass 1's 12 inputs (outputs, forward) the middle 4 are zero (unwanted) at
// compile time.
// Pass 1's twiddles: for N = 3 * 2^m (PFA) the factor 3 is split off by the
// prime-factor map (no twiddles; thread j's 3-point transforms are rotated by
// W_3^s, s = s(j), which costs two real factors per term) and the factor 4
// needs W_(N/3)^(j k), k = 1..3: three table values a thread instead of
// eleven.  Else (N = 9 * 2^m) W_N^(b j).  With R2 = 4 pass 2 is exactly three
// rounds of M1 threads with one i each, again three table values.
#pragma once
#include "fft_core.cuh"

namespace les {

template <int MX> struct RowPlan;
template <> struct RowPlan<24> { static constexpr int R2 = 2, R3 = 1; };
template <> struct RowPlan<48> { static constexpr int R2 = 4, R3 = 1; };
template <> struct RowPlan<96> { static constexpr int R2 = 8, R3 = 1; };
template <> struct RowPlan<144> { static constexpr int R2 = 12, R3 = 1; };
template <> struct RowPlan<192> { static constexpr int R2 = 16, R3 = 1; };
template <> struct RowPlan<288> { static constexpr int R2 = 4, R3 = 6; };
template <> struct RowPlan<384> { static constexpr int R2 = 4, R3 = 8; };
template <> struct RowPlan<576> { static constexpr int R2 = 4, R3 = 12; };
template <> struct RowPlan<768> { static constexpr int R2 = 4, R3 = 16; };

// a + s b, one packed instruction in FP32
template <class T> __device__ __forceinline__ cx<T> axpy(cx<T> a, T s, cx<T> b) { return mk(a.x + s * b.x, a.y + s * b.y); }
template <> __device__ __forceinline__ cx<float> axpy<float>(cx<float> a, float s, cx<float> b) {
  cx<float> r;
  asm("{\n\t.reg .b64 a, b, s, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 s, {%6, %6};\n\t"
      "fma.rn.f32x2 r, b, s, a;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(s));
  return r;
}
// a + s i b
template <class T> __device__ __forceinline__ cx<T> axipy(cx<T> a, T s, cx<T> b) { return mk(a.x - s * b.y, a.y + s * b.x); }

// 12-point DFTs as 3 x 4 without inner twiddles (prime-factor maps: input
// n = 4 a + 3 c, output k = 4 k3 + 9 k4, both mod 12).
// Inverse with inputs 4..7 zero: x[0..3] inputs 0..3, x[4..7] inputs 8..11.
template <class T> __device__ __forceinline__ void dft12_padded(const cx<T> (&x)[8], cx<T> (&y)[12]) {
  constexpr T h = (T)0.5, s3 = (T)0.86602540378443864676372317075293618;
  cx<T> g[3][4];  // [k3][c]
  // c = 0: inputs 0, 4, 8;  c = 1: 3, 7, 11 (the second is zero)
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const cx<T> p = c == 0 ? x[0] : x[3], q = c == 0 ? x[4] : x[7];
    const cx<T> t = axpy<T>(p, -h, q);
    g[0][c] = p + q;
    g[1][c] = axipy<T>(t, -s3, q);
    g[2][c] = axipy<T>(t, s3, q);
  }
  {  // c = 2: inputs 6, 10, 2 (the first is zero)
    const cx<T> s = x[6] + x[2], d = x[6] - x[2], t = s * (-h);
    g[0][2] = s;
    g[1][2] = axipy<T>(t, s3, d);
    g[2][2] = axipy<T>(t, -s3, d);
  }
  {  // c = 3: inputs 9, 1, 5 (the third is zero)
    const cx<T> t = axpy<T>(x[5], -h, x[1]);
    g[0][3] = x[5] + x[1];
    g[1][3] = axipy<T>(t, s3, x[1]);
    g[2][3] = axipy<T>(t, -s3, x[1]);
  }
#pragma unroll
  for (int k3 = 0; k3 < 3; k3++) {
    Dft<4, +1, T>::run(g[k3]);
#pragma unroll
    for (int k4 = 0; k4 < 4; k4++) y[(4 * k3 + 9 * k4) % 12] = g[k3][k4];
  }
}
// Forward with all inputs; the caller leaves outputs 4..7 unused.
template <class T> __device__ __forceinline__ void dft12_forward(const cx<T> (&x)[12], cx<T> (&y)[12]) {
  constexpr T h = (T)0.5, s3 = (T)0.86602540378443864676372317075293618;
  cx<T> g[3][4];
#pragma unroll
  for (int a = 0; a < 3; a++) {
#pragma unroll
    for (int c = 0; c < 4; c++) g[a][c] = x[(4 * a + 3 * c) % 12];
    Dft<4, -1, T>::run(g[a]);
  }
#pragma unroll
  for (int k4 = 0; k4 < 4; k4++) {
    const cx<T> s = g[1][k4] + g[2][k4], d = g[1][k4] - g[2][k4], t = axpy<T>(g[0][k4], -h, s);
    y[(9 * k4) % 12] = g[0][k4] + s;
    y[(4 + 9 * k4) % 12] = axipy<T>(t, -s3, d);
    y[(8 + 9 * k4) % 12] = axipy<T>(t, s3, d);
  }
}

// Rotated 12-point DFT of pass 1 for N = 3 * 2^m: 3-point transforms over a
// (input n = j + M1 (c + 4 a), rotated by W_3^(s_c x3), s_c = s + c M1 u mod 3
// with u = (N/3)^-1 mod 3), then 4-point transforms over c; output b = 4 x3 + k4.
// w[s] = W_3^(s(j) + s) for s = 0..2.
template <class T, int M1> struct Dft12Pfa {
  static constexpr int U = (4 * M1) % 3, STEP = (U * M1) % 3;  // u = Q^-1 = Q mod 3
  // inverse, inputs 4..7 zero: x[0..3] inputs 0..3, x[4..7] inputs 8..11
  static __device__ __forceinline__ void padded(const cx<T> (&x)[8], const cx<T> (&w)[3], cx<T> (&y)[12]) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const cx<T> p = x[c], q = x[4 + c], al = w[(c * STEP) % 3], be = w[(c * STEP + 2) % 3];
      const cx<T> re = axpy<T>(p * al.x, be.x, q), im = axpy<T>(p * al.y, be.y, q);
      y[c] = p + q;
      y[4 + c] = mk(re.x - im.y, re.y + im.x);
      y[8 + c] = mk(re.x + im.y, re.y - im.x);
    }
#pragma unroll
    for (int k3 = 0; k3 < 3; k3++) Dft<4, +1, T>::run(y + 4 * k3);
  }
  // forward, outputs 0..3 and 8..11 (z[0..3], z[4..7])
  static __device__ __forceinline__ void forward(cx<T> (&y)[12], const cx<T> (&w)[3], cx<T> (&z)[8]) {
#pragma unroll
    for (int k3 = 0; k3 < 3; k3++) Dft<4, -1, T>::run(y + 4 * k3);
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const cx<T> s = y[4 + c] + y[8 + c], d = y[4 + c] - y[8 + c], al = w[(c * STEP) % 3], be = w[(c * STEP + 2) % 3];
      z[c] = axipy<T>(axpy<T>(y[c], al.x, s), -al.y, d);
      z[4 + c] = axipy<T>(axpy<T>(y[c], be.x, s), -be.y, d);
    }
  }
};

// Index maps of a padded length.
template <int N> struct InPlace {
  static constexpr int R2 = RowPlan<N>::R2, R3 = RowPlan<N>::R3, M1 = N / 12;
  static_assert(R2 * R3 == M1, "row plan");
  static constexpr bool PFA = M1 % 3 != 0;
  // x of the point at element n: b = 4 x3 + k4 and kappa = k4 + 4 (r + R2 i)
  // stand for x mod 3 = x3, x mod N/3 = 3 kappa (PFA); else b + 12 (r + R2 i)
  static __device__ __forceinline__ int x_of(int n) {
    const int b = n / M1, m = n - b * M1, o = m / R3 + R2 * (m % R3);
    if (!PFA) return b + 12 * o;
    constexpr int Q = 4 * M1, U = Q % 3 == 1 ? Q : 2 * Q;  // U = 1 mod 3, 0 mod Q
    return ((b >> 2) * U + 3 * ((b & 3) + 4 * o)) % N;
  }
  // W_3^(s(j) + 0, 1, 2), s(j) = j (N/3)^-1 mod 3: thread j's rotations (PFA)
  template <class T> static __device__ __forceinline__ void rotations(int j, cx<T> (&w)[3]) {
#pragma unroll
    for (int s = 0; s < 3; s++) {
      const int e = (j * ((4 * M1) % 3) + s) % 3;
      w[s] = mk(e ? (T)-0.5 : (T)1,
                e == 0 ? (T)0 : (e == 1 ? (T)1 : (T)-1) * (T)0.86602540378443864676372317075293618);
    }
  }
};

template <class T> __device__ __forceinline__ cx<T> shfl_cx(unsigned mask, cx<T> v, int src) {
  return mk(__shfl_sync(mask, v.x, src), __shfl_sync(mask, v.y, src));
}

// A row's team of TP threads (M1 rounded up to a power of two): thread t's
// pass 1 index j (M1: none) and the lane of its mirror partner M1 - j.  A
// team of two warps splits j so that both are in the same warp.
template <int M1, int TP> __host__ __device__ __forceinline__ void mirror_lanes(int t, int lane, int& j, int& partner) {
  if (TP <= 32) {
    j = t;
    partner = (lane & ~(TP - 1)) | (t == 0 || t >= M1 ? t : M1 - t);
  } else {
    constexpr int H = M1 / 4;
    const int l = t & 31;
    if (t < 32) {
      j = l < H ? l : (l == H ? 2 * H : l + 2 * H);
      partner = (l == 0 || l == H || l >= 2 * H) ? l : 2 * H - l;
    } else {
      j = l < H ? H + l : l + H + 1;
      partner = l >= 2 * H ? l : 2 * H - 1 - l;
    }
    if (l >= 2 * H) j = M1;
  }
}
// The elements (b, j), b < 12, of the forward transform's last pass; p points
// at (0, j).  A thread without a j reads none: whatever element it named would
// be another thread's, which may already be writing the next row's pass 1.
template <int SB, class T, class P> __host__ __device__ __forceinline__ void own_elements(P p, bool act, cx<T> (&v)[12]) {
#pragma unroll
  for (int b = 0; b < 12; b++) v[b] = act ? p[b * SB] : mk((T)0, (T)0);
}

}  // namespace les

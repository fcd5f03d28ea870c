// les_fused.cuh -- the padded-grid part of comp1 as one kernel per (padded
// y rows, z chunk): inverse x transforms of the mixed arrays, the pointwise
// advection / SGS fluxes, and the forward x transforms with -d/dx folded in,
// without ever writing the padded physical fields to HBM.
//
// The CTA walks up its z chunk with the sliding window of comp1.f90:91-121 /
// 179-184 along ROWS rows of the padded plane.  Each row has six teams of TP
// threads and six shared-memory buffers; team w owns transform w of both
// phases and buffer w:
//   phase I   (inverse)  w0: U+iV (z+1)   w1: W+iE (z+1)   w2: UX+iVX (z)
//                        w3: UY+iVY (z)   w4: WX+iWY (z)   w5: EX+iEY (le)
//             (when the learned closure supplies the interior momentum
//             stresses only ux and vy are needed, for the divergence
//             diagnostic: w2 transforms UX+iVY, w3 and w4 idle)
//   phase II  (pointwise, all threads) the eleven flux rows of k_flux,
//             written over the six rows it read
//   phase III (forward)  w0: A+iPu  w1: B+iPv  w2: C+iG  w3: D+iPw
//                        w4: F+iPe  w5: H
// Each thread keeps its own points of the window (levels z-1 and z) in
// registers, so a row needs six buffers instead of eleven.
#pragma once
#include "les_kernels.cuh"

namespace les {

// Row transforms of the fused kernel: fft_inplace.cuh, a team of TP threads
// per row.
// Element (b, r, i) sits at b SB + r SR + i; SR and SB come from counting the
// wavefronts of every pass over a warp's lanes (FP32: 16 lanes a wavefront,
// FP64: 8): with them all passes but pass 1 are conflict-free for R3 >= 8, and
// every address is a per-thread base plus a constant.  (One pad element per
// 128 bytes instead took 2.2 times the minimum at 576 points in FP32, 1.7 times
// in FP64, 1.3 at 384 and 1.7 at 288.)
template <class T, int NSX> struct FusedCfg {
  static constexpr int MX = 3 * NSX / 2, KX = NSX / 2;
  static constexpr int R2 = RowPlan<MX>::R2, R3 = RowPlan<MX>::R3, M1 = MX / 12;
  static_assert(R2 * R3 == M1 && 4 * M1 == KX, "row plan");
  // threads of a team: M1 rounded up to a power of two
  static constexpr int TP = M1 <= 2 ? 2 : M1 <= 4 ? 4 : M1 <= 8 ? 8 : M1 <= 16 ? 16 : M1 <= 32 ? 32 : 64;
  static constexpr int TR = 6 * TP;                      // threads of a row
  static constexpr int ROWS = TR >= 96 ? 1 : 96 / TR;    // rows of a CTA (divides every padded ny)
  static constexpr int THREADS = TR * ROWS;
  static constexpr int WARPS = THREADS / 32;
  static constexpr int PPT = (MX + TR - 1) / TR;         // points of a thread in phase II
  static constexpr bool PFA = InPlace<MX>::PFA;
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int SR = R3 == 16 ? 17 : R3 == 12 ? 15 : R3 == 8 ? 9 : R3 == 6 ? (F32 ? 7 : 6) : 1;
  static constexpr int SB = R3 == 1 ? (M1 | 1) : R2 * SR + (R3 == 6 && !F32 ? 1 : 0);
  static constexpr int BUF = 12 * SB + (TP == 8 ? 12 : TP == 2 ? 14 : 0);
  static constexpr int NT1 = PFA ? 3 : 11;               // pass 1 twiddles of a thread
  static constexpr int NTW = NT1 * M1 + (R3 > 1 ? (R2 - 1) * R3 : 0);
  static __device__ __forceinline__ int x_of(int n) { return InPlace<MX>::x_of(n); }
  static constexpr size_t smem() { return ((size_t)6 * ROWS * BUF + NTW) * sizeof(cx<T>); }
  // Resident CTAs per SM the register budget aims at: 24 warps of <= 80
  // registers in FP32, 12 of <= 168 in FP64.  Tighter budgets spill (FP64 at
  // 18 warps: 64-point grids 47 -> 60 us per launch), looser ones leave the
  // passes' shared-memory latency uncovered (FP32 at 12 warps: 512x512x32
  // 719 -> 885 us).
  static constexpr int CTAS = (sizeof(T) == 4 ? 768 : 384) / THREADS;
  // offset of r R3 + i within b, address of element n
  static __device__ __forceinline__ constexpr int off(int m) { return R3 == 1 ? m : (m / R3) * SR + m % R3; }
  static __device__ __forceinline__ int at(int n) { return (n / M1) * SB + off(n % M1); }
  // element of the pointwise phase's point p: in FP32 four neighbouring b run
  // fastest (SB = 4 mod 16 8-byte banks), else natural order
  static __device__ __forceinline__ int elem(int p) {
    if (!F32 || R3 == 1) return p;
    const int q = p >> 2, i = q % R3, r = (q / R3) % R2, bh = q / M1;
    return ((p & 3) + 4 * bh) * M1 + r * R3 + i;
  }
};

// Passes 2 and 3 of a team's transform in its buffer.  t = thread of the
// team.  INV: pass 2 then 3; else 3 then 2, with the conjugate twiddles.
template <class T, int NSX, bool INV> struct RowPasses {
  using C = FusedCfg<T, NSX>;
  static constexpr int R2 = C::R2, R3 = C::R3, TP = C::TP, M1 = C::M1;
  static __device__ __forceinline__ void pass2(cx<T>* buf, const cx<T>* tw2, int t) {
    if constexpr (R3 > 1) {
      static_assert(R2 == 4, "three rounds of M1 threads");
      if (TP > M1 && t >= M1) return;
      // FP32: b runs fastest
      const int i = C::F32 ? t / 4 : t % R3;
      cx<T>* p = buf + (C::F32 ? t % 4 : t / R3) * C::SB + i;
      cx<T> w[R2];
#pragma unroll
      for (int r = 1; r < R2; r++) w[r] = INV ? conj(tw2[(r - 1) * R3 + i]) : tw2[(r - 1) * R3 + i];
#pragma unroll
      for (int jj = 0; jj < 3; jj++) {
        cx<T> v[R2];
#pragma unroll
        for (int r = 0; r < R2; r++) {
          v[r] = p[4 * jj * C::SB + r * C::SR];
          if (!INV && r > 0) v[r] = cmul(v[r], w[r]);
        }
        Dft<R2, INV ? +1 : -1, T>::run(v);
#pragma unroll
        for (int r = 0; r < R2; r++) p[4 * jj * C::SB + r * C::SR] = (INV && r > 0) ? cmul(v[r], w[r]) : v[r];
      }
    } else {
      constexpr int J = (12 + TP - 1) / TP;
#pragma unroll
      for (int jj = 0; jj < J; jj++) {
        const int b = t + TP * jj;
        if (J * TP > 12 && b >= 12) break;
        cx<T>* p = buf + b * C::SB;
        cx<T> v[R2];
#pragma unroll
        for (int r = 0; r < R2; r++) v[r] = p[r];
        Dft<R2, INV ? +1 : -1, T>::run(v);
#pragma unroll
        for (int r = 0; r < R2; r++) p[r] = v[r];
      }
    }
  }
  static __device__ __forceinline__ void pass3(cx<T>* buf, int t) {
    constexpr int ITEMS = 12 * R2, J = (ITEMS + TP - 1) / TP;
#pragma unroll
    for (int jj = 0; jj < J; jj++) {
      const int it = t + TP * jj;
      if (J * TP > ITEMS && it >= ITEMS) break;
      const int b = it / R2, r = it - b * R2;
      cx<T>* p = buf + b * C::SB + r * C::SR;
      cx<T> v[R3];
#pragma unroll
      for (int i = 0; i < R3; i++) v[i] = p[i];
      Dft<R3, INV ? +1 : -1, T>::run(v);
#pragma unroll
      for (int i = 0; i < R3; i++) p[i] = v[i];
    }
  }
};

// Barrier of one team: the lanes `mask` of a warp, or the named barrier of a
// team of two warps.
template <int TP> __device__ __forceinline__ void team_sync(int bar, unsigned mask) {
  if (TP <= 32) __syncwarp(mask);
  else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(TP) : "memory");
}

struct FusedArgs {
  // mixed inputs (x-spectral, y physical on the padded grid): Um, UYm, Vm,
  // VYm, Wm, WYm, Em, EYm; outputs Xu1, Xu2, Xv1, Xv2, Xw1, Xw2, Xe1, Xe2
  Ptr8 in, out;
  const void* dEX;       // clip corrections (padded physical, levels 1..nnz-1)
  const void* dEY;
  const int* clipflag;   // per level 1..nnz-1 (index z-1)
  const unsigned char* rowclip;  // per level and block of k_clip_walls: its rows of dEX are set
  const WallParams* wp;
  double* divpart;  // [level][CTA][warp] partial sums of divz, one writer each
  double* sgspart;  // [level][CTA][warp][6] partial SGS means (stage 1 with mnout)
  // learned closure: when lflag is set and *lflag != 0 the interior momentum
  // stresses are left to the network (the wall-model rows stay)
  const int* lflag;
  int zchunk;
};

// Square root of the TKE in the FP32 form: the hardware approximation
// (sqrt.approx.f32) instead of the correctly rounded sequence, 3% of the
// fused kernel (the mixed-form tolerances against the oracle bound its
// effect); FP64 keeps sqrt().
template <class T> __device__ __forceinline__ T tke_sqrt(T e) { return sqrt(e); }
template <> __device__ __forceinline__ float tke_sqrt<float>(float e) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(e));
  return r;
}

// What bounds it: shared-memory wavefronts and issue slots, not HBM (15% of
// its peak).  At 512x512x32 (768-point rows) FP32 runs the load/store data
// path at 70% and issues 0.56 per scheduler and cycle, FP64 62% and 0.36 with
// the FP64 pipe at 41%.  Before, autosorted rows of one warp per transform
// and the window in shared memory left 6 (FP64) or 12 (FP32) warps per SM:
// 1939 -> 1283 us (FP64), 887 -> 643 us (FP32), 827 -> 586 us (FP32, learned);
// 64x64x64 FP64 168 -> 47 us.
template <class T, int NSX>
__global__ void __launch_bounds__(FusedCfg<T, NSX>::THREADS, FusedCfg<T, NSX>::CTAS)
k_row_fused(const __grid_constant__ FusedArgs f, const __grid_constant__ StageArgs a, const cx<T>* __restrict__ tw) {
  using C = FusedCfg<T, NSX>;
  constexpr int MX = C::MX, KX = C::KX, M1 = C::M1, R2 = C::R2, R3 = C::R3, TP = C::TP, TR = C::TR;
  constexpr int BUF = C::BUF, SB = C::SB, PPT = C::PPT;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  cx<T>* tw1 = sm + (size_t)6 * C::ROWS * BUF;  // [k - 1][j]: W_(N/3)^(k j) (PFA) or W_N^(k j)
  cx<T>* tw2 = tw1 + C::NT1 * M1;               // [r - 1][i]: W_M1^(r i)
  {
    const cx<T>* twg = tw + tw_off(MX);
    for (int i = threadIdx.x; i < C::NT1 * M1; i += C::THREADS)
      tw1[i] = twg[(C::PFA ? 3 : 1) * (i / M1 + 1) * (i % M1)];
    if (R3 > 1)
      for (int i = threadIdx.x; i < (R2 - 1) * R3; i += C::THREADS) tw2[i] = twg[12 * (i / R3 + 1) * (i % R3)];
  }
  __syncthreads();

  const int NZ = a.NZ, MY = a.MY;
  const int row = C::ROWS > 1 ? (int)threadIdx.x / TR : 0;
  const int tr = C::ROWS > 1 ? (int)threadIdx.x % TR : (int)threadIdx.x;  // thread of the row
  const int team = tr / TP, t = tr % TP;
  const int y = blockIdx.x * C::ROWS + row;
  const int z0 = blockIdx.y * f.zchunk + 1;
  const int z1 = min(z0 + f.zchunk - 1, NZ);
  if (z0 > NZ) return;
  const int lane = threadIdx.x & 31;
  cx<T>* rowbuf = sm + (size_t)row * 6 * BUF;
  cx<T>* buf = rowbuf + team * BUF;
  const int bar = 1 + team;
  const unsigned mask = TP >= 32 ? 0xffffffffu : ((1u << (TP & 31)) - 1u) << (lane & ~(TP - 1));

  int j, partner;
  mirror_lanes<M1, TP>(t, lane, j, partner);
  const bool act = (TP == M1) || j < M1;
  if (!act) j = 0;
  cx<T>* pj = buf + C::off(j);
  const cx<T>* twj = tw1 + j;
  cx<T> w3[3];
  InPlace<MX>::rotations(j, w3);

  const T dzm = (T)a.dzm, todzm = (T)a.todzm, emin = (T)a.emin;
  const T xkmax = (T)a.xkmax, nu = (T)a.nu, c01 = (T)0.1 * (T)a.dsl;
  const WallParams& wp = *f.wp;
  // weight of the interior momentum stresses: 0 when the learned closure
  // supplies them (the wall rows stay)
  const bool learned = (f.lflag && f.lflag[0]);
  const T mom = learned ? (T)0 : (T)1;
  auto xkk = [&](T sq) { return tmin(c01 * sq, xkmax) + nu; };  // from the square root of e

  const size_t zstride = (size_t)MY * KX;
  auto mix = [&](int q, int z) -> const cx<T>* {
    return reinterpret_cast<const cx<T>*>(f.in.p[q]) + (size_t)(z - 1) * zstride + (size_t)y * KX;
  };
  // this team's inputs A + iB (array, i kx on A and on B) and outputs:
  // -i kx a^ + b^ to array o1, a^ to o2, b^ to o3 (8: none)
  auto pick = [&](unsigned table) { return (int)((table >> (4 * team)) & 15u); };
  const int qa = pick(0x641040), qb = pick(learned ? 0x753362 : 0x753262);
  const bool ma = 0x34 >> team & 1, mb = !learned && team == 2;
  const int o1 = pick(0x864820), o2 = pick(0x788318), o3 = pick(0x888588);

  // the window at this thread's points: level z - 1 and level z
  // (s: the square roots of e; FP32 takes them again, cheaper than the registers)
  constexpr bool KEEP = sizeof(T) == 8;
  T Um[PPT], Vm[PPT], Wm[PPT], Em[PPT], sm1[KEEP ? PPT : 1], tum[PPT], tvm[PPT];
  T U0[PPT], V0[PPT], W0[PPT], E0[PPT], s0[KEEP ? PPT : 1];

  // iteration z0 - 1 fills the window (levels z0 - 1 and z0)
  for (int z = z0 - 1; z <= z1; z++) {
    const bool pre = z < z0, top = z == NZ;
    const int le = z < NZ - 2 ? z : NZ - 2;
    // ---- phase I: inverse transforms ----
    {
      // team 0: U + iV at z + 1; 1: W + iE at z + 1 (w = 0 above nnz - 1, e
      // clamped to level nnz - 1); 2: UX + iVX (learned: UX + iVY); 3: UY +
      // iVY; 4: WX + iWY; 5: EX + iEY at le.  While filling the window teams
      // 2 and 3 take U + iV and W + iE at z = z0 - 1.
      const bool fill = pre && (team == 2 || team == 3);
      const int ja = fill ? 4 * (team - 2) : qa, jb = fill ? 4 * (team - 2) + 2 : qb;
      const bool ia = ma && !fill, ib = mb && !fill;
      const int za = team < 2 ? z + 1 : (team == 5 ? le : z), zb = (jb == 6) ? min(za, NZ - 1) : za;
      const bool on = team < 2 ? !top
                               : team == 2 ? z >= 1
                                           : team == 3 ? (pre ? z >= 1 : !learned)
                                                       : team == 4 ? (!learned && z >= 1 && !top) : (!pre && !top);
      const bool hasA = !(ja == 4 && za > NZ - 1);
      if (on) {
        const cx<T>* A = mix(ja, hasA ? za : 1) + j;
        const cx<T>* B = mix(jb, zb) + j;
        // modes k = j + M1 m of Z = A + iB and their mirror images
        cx<T> x[8], mir[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const int k = j + M1 * m;
          cx<T> av = hasA ? A[M1 * m] : zero_cx<T>(), bv = B[M1 * m];
          const T kk = (T)a.kx0 * (T)k;
          if (ia) av = mul_i(av) * kk;
          if (ib) bv = mul_i(bv) * kk;
          if (m == 0 && j == 0) { av.y = 0; bv.y = 0; }
          x[m] = mk(av.x - bv.y, av.y + bv.x);
          mir[m] = mk(av.x + bv.y, bv.x - av.y);
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const cx<T> r = shfl_cx(mask, mir[m], partner), own = m < 3 ? mir[m + 1] : zero_cx<T>();
          x[7 - m] = j == 0 ? own : r;
        }
        if (act) {
          cx<T> v[12];
          if constexpr (C::PFA) {
            Dft12Pfa<T, M1>::padded(x, w3, v);
#pragma unroll
            for (int k = 0; k < 4; k++) {
              const cx<T> w = k ? conj(twj[(k - 1) * M1]) : zero_cx<T>();
#pragma unroll
              for (int b = k; b < 12; b += 4) pj[b * SB] = k ? cmul(v[b], w) : v[b];
            }
          } else {
            dft12_padded<T>(x, v);
            pj[0] = v[0];
#pragma unroll
            for (int b = 1; b < 12; b++) pj[b * SB] = cmul(v[b], conj(twj[(b - 1) * M1]));
          }
        }
        team_sync<TP>(bar, mask);
        RowPasses<T, NSX, true>::pass2(buf, tw2, t);
        if (R3 > 1) {
          team_sync<TP>(bar, mask);
          RowPasses<T, NSX, true>::pass3(buf, t);
        }
      }
    }
    __syncthreads();
    if (pre) {
#pragma unroll
      for (int q = 0; q < PPT; q++) {
        const int n = tr + TR * q;
        if (PPT * TR > MX && n >= MX) break;
        const cx<T>* p = rowbuf + C::at(C::elem(n));
        const cx<T> uv = p[0], we = p[BUF];
        U0[q] = uv.x; V0[q] = uv.y; W0[q] = we.x; E0[q] = tmax(we.y, emin);
        if (KEEP) s0[q] = tke_sqrt(E0[q]);
        if (z == 0) {  // w(0) = 0, e(0) = e(1)
          Um[q] = Vm[q] = Wm[q] = (T)0;
          Em[q] = E0[q];
          if (KEEP) sm1[q] = s0[q];
          wall_stress<T>(wp.w[0], wp, a, 0, uv.x, uv.y, tum[q], tvm[q]);
        } else {
          const cx<T> uvm = p[2 * BUF], wem = p[3 * BUF];
          const cx<T> wxy = learned ? zero_cx<T>() : p[4 * BUF];
          Um[q] = uvm.x; Vm[q] = uvm.y; Wm[q] = wem.x; Em[q] = tmax(wem.y, emin);
          const T sq = tke_sqrt(Em[q]), xk = xkk(sq);
          if (KEEP) sm1[q] = sq;
          tum[q] = -mom * xk * ((uv.x - uvm.x) * dzm + wxy.x);
          tvm[q] = -mom * xk * ((uv.y - uvm.y) * dzm + wxy.y);
        }
      }
      __syncthreads();
      continue;
    }
    // L2 prefetch (one thread, nothing waits on it) of the rows the next
    // level's phase I reads from DRAM: U, V, W, E at z+2 and VY, UY, WY, EY at
    // z+1 (U, V, W, E at z+1 were this level's window rows and are in L2)
    if (threadIdx.x == 0 && z + 1 <= z1) {
      constexpr unsigned RB = C::ROWS * KX * sizeof(cx<T>);
      if (z + 2 <= NZ) { tma::prefetch_l2(mix(0, z + 2), RB); tma::prefetch_l2(mix(2, z + 2), RB); }
      if (z + 2 <= NZ - 1) { tma::prefetch_l2(mix(4, z + 2), RB); tma::prefetch_l2(mix(6, z + 2), RB); }
      tma::prefetch_l2(mix(3, z + 1), RB);
      if (!learned) tma::prefetch_l2(mix(1, z + 1), RB);
      if (z + 1 <= NZ - 1) {
        if (!learned) tma::prefetch_l2(mix(5, z + 1), RB);
        tma::prefetch_l2(mix(7, min(z + 1, NZ - 2)), RB);
      }
    }
    // ---- phase II: fluxes (k_flux) ----
    double divz_part = 0.0;
    double sgs_part[6] = {0, 0, 0, 0, 0, 0};
    // the clip corrections: dEY on a flagged level, dEX where the row's block
    // of k_clip_walls clipped (2 NT rows each)
    constexpr int BR = 2 * RowCfg<MX>::NT;
    const bool clip = (!top) && f.clipflag[le - 1];
    const bool clipx = clip && f.rowclip[(size_t)(le - 1) * ((MY + BR - 1) / BR) + y / BR];
#pragma unroll
    for (int q = 0; q < PPT; q++) {
      const int n = tr + TR * q;
      if (PPT * TR > MX && n >= MX) break;
      cx<T>* p = rowbuf + C::at(C::elem(n));
      // learned: buffer 2 holds (ux, vy); the other gradients are not needed
      const cx<T> d2 = p[2 * BUF];
      const cx<T> d3 = learned ? mk((T)0, d2.y) : p[3 * BUF];
      const T ux = d2.x, vx = learned ? (T)0 : d2.y, uy = d3.x, vy = d3.y;
      const T sq0 = KEEP ? s0[q] : tke_sqrt(E0[q]), sqm = KEEP ? sm1[q] : tke_sqrt(Em[q]);
      const T xkm = xkk(sqm), xk0 = xkk(sq0);
      const T s = mom * (xkm + xk0);
      const T tuu = -s * ux, tvv = -s * vy, tuv = -s * (uy + vx) * (T)0.5;
      const T wz0 = (W0[q] - Wm[q]) * dzm;
      const T tww0 = -s * wz0;
      const T A = U0[q] * U0[q] + tuu, B = U0[q] * V0[q] + tuv, Cc = V0[q] * V0[q] + tvv;
      T tuw0, tvw0, U1 = (T)0, V1 = (T)0;
      const T d = ux + vy + wz0;
      divz_part += (double)(d * d);
      if (!top) {
        const cx<T> uv1 = p[0], we1 = p[BUF];
        const cx<T> wxy = learned ? zero_cx<T>() : p[4 * BUF];
        cx<T> exy = p[5 * BUF];
        if (clip) {
          const size_t o = ((size_t)(le - 1) * MY + y) * MX + C::x_of(C::elem(n));
          if (clipx) exy.x += reinterpret_cast<const T*>(f.dEX)[o];
          exy.y += reinterpret_cast<const T*>(f.dEY)[o];
        }
        U1 = uv1.x; V1 = uv1.y;
        const T W1 = we1.x, E1 = tmax(we1.y, emin), sq1 = tke_sqrt(E1), xkp = xkk(sq1);
        tuw0 = -mom * xk0 * ((U1 - U0[q]) * dzm + wxy.x);
        tvw0 = -mom * xk0 * ((V1 - V0[q]) * dzm + wxy.y);
        const T wz1 = (W1 - W0[q]) * dzm;
        const T tww1 = -mom * (xk0 + xkp) * wz1;
        const T D = (T)0.5 * (U0[q] + U1) * W0[q] + tuw0;
        const T G = (T)0.5 * (V0[q] + V1) * W0[q] + tvw0;
        const T hp = (T)0.5 * (W1 + W0[q]), hm = (T)0.5 * (W0[q] + Wm[q]);
        const T Pw = -(hp * hp - hm * hm) * dzm - (tww1 - tww0) * dzm;
        const T F = (T)0.5 * E0[q] * (U0[q] + U1) - (T)2 * xk0 * exy.x;
        const T H = (T)0.5 * E0[q] * (V0[q] + V1) - (T)2 * xk0 * exy.y;
        const T Pe = -(W1 * E1 - Wm[q] * Em[q]) * todzm +
                     ((xkp + xk0) * (E1 - E0[q]) - (xk0 + xkm) * (E0[q] - Em[q])) * (T)a.dzm2 -
                     (T)a.ceps * E0[q] * sq0;
        p[2 * BUF] = mk(Cc, G);
        p[3 * BUF] = mk(D, Pw);
        p[4 * BUF] = mk(F, Pe);
        p[5 * BUF] = mk(H, (T)0);
        const T Pu = -((U1 + U0[q]) * W0[q] - (Um[q] + U0[q]) * Wm[q]) * todzm + (T)a.forcing - (tuw0 - tum[q]) * dzm;
        const T Pv = -((V1 + V0[q]) * W0[q] - (Vm[q] + V0[q]) * Wm[q]) * todzm - (tvw0 - tvm[q]) * dzm;
        p[0] = mk(A, Pu);
        p[BUF] = mk(B, Pv);
        if (a.mnout_sgs) {
          sgs_part[0] += (double)tuu; sgs_part[1] += (double)tvv; sgs_part[2] += (double)tuv;
          sgs_part[3] += (double)tww0; sgs_part[4] += (double)tuw0; sgs_part[5] += (double)tvw0;
        }
        Um[q] = U0[q]; Vm[q] = V0[q]; Wm[q] = W0[q]; Em[q] = E0[q]; tum[q] = tuw0; tvm[q] = tvw0;
        if (KEEP) { sm1[q] = sq0; s0[q] = sq1; }
        U0[q] = U1; V0[q] = V1; W0[q] = W1; E0[q] = E1;
      } else {
        wall_stress<T>(wp.w[1], wp, a, 1, U0[q], V0[q], tuw0, tvw0);
        p[2 * BUF] = mk(Cc, (T)0);
        const T Pu = (Um[q] + U0[q]) * Wm[q] * todzm + (T)a.forcing - (tuw0 - tum[q]) * dzm;
        const T Pv = (Vm[q] + V0[q]) * Wm[q] * todzm - (tvw0 - tvm[q]) * dzm;
        p[0] = mk(A, Pu);
        p[BUF] = mk(B, Pv);
        if (a.mnout_sgs) {
          sgs_part[0] += (double)tuu; sgs_part[1] += (double)tvv; sgs_part[2] += (double)tuv;
          sgs_part[3] += (double)tww0; sgs_part[4] += (double)tuw0; sgs_part[5] += (double)tvw0;
        }
      }
    }
    // statistics of this level: one partial sum per warp
    {
      const size_t slot = ((size_t)(z - 1) * gridDim.x + blockIdx.x) * C::WARPS + (threadIdx.x >> 5);
      for (int o = 16; o > 0; o >>= 1) divz_part += __shfl_xor_sync(0xffffffffu, divz_part, o);
      if (lane == 0) f.divpart[slot] = divz_part;
      if (a.mnout_sgs) {
#pragma unroll
        for (int q = 0; q < 6; q++) {
          for (int o = 16; o > 0; o >>= 1) sgs_part[q] += __shfl_xor_sync(0xffffffffu, sgs_part[q], o);
          if (lane == 0) f.sgspart[slot * 6 + q] = sgs_part[q];
        }
      }
    }
    __syncthreads();
    // ---- phase III: forward transforms, -d/dx, truncation to kx < nx/2 ----
    if (!(top && team >= 3)) {
      if (R3 > 1) {
        RowPasses<T, NSX, false>::pass3(buf, t);
        team_sync<TP>(bar, mask);
      }
      RowPasses<T, NSX, false>::pass2(buf, tw2, t);
      team_sync<TP>(bar, mask);
      cx<T> zf[8];  // outputs 0..3 and 8..11
      {
        cx<T> v[12];
        own_elements<SB>((const cx<T>*)pj, act, v);
        if constexpr (C::PFA) {
#pragma unroll
          for (int k = 1; k < 4; k++) {
            const cx<T> w = twj[(k - 1) * M1];
#pragma unroll
            for (int b = k; b < 12; b += 4) v[b] = cmul(v[b], w);
          }
          Dft12Pfa<T, M1>::forward(v, w3, zf);
        } else {
#pragma unroll
          for (int b = 1; b < 12; b++) v[b] = cmul(v[b], twj[(b - 1) * M1]);
          cx<T> o[12];
          dft12_forward<T>(v, o);
#pragma unroll
          for (int m = 0; m < 4; m++) { zf[m] = o[m]; zf[4 + m] = o[8 + m]; }
        }
      }
      const size_t orow = (size_t)(z - 1) * zstride + (size_t)y * KX + j;
      auto O = [&](int q) { return reinterpret_cast<cx<T>*>(f.out.p[q & 7]) + orow; };
      cx<T>* const p1 = O(o1);
      cx<T>* const p2 = O(o2);
      cx<T>* const p3 = O(o3);
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const cx<T> zk = zf[m];
        const cx<T> other = shfl_cx(mask, zf[7 - m], partner);
        const cx<T> zmr = conj(j == 0 ? zf[m ? 8 - m : 0] : other);
        if (!act) continue;
        const int k = j + M1 * m;
        const cx<T> ah = (zk + zmr) * (T)0.5;
        const cx<T> dd = zk - zmr;
        const cx<T> bh = mk(dd.y * (T)0.5, -dd.x * (T)0.5);
        const T kk = (T)a.kx0 * (T)k;
        const cx<T> dxa = mk(kk * ah.y, -kk * ah.x);  // -i kx a^
        if (o1 < 8) p1[M1 * m] = dxa + bh;
        if (o2 < 8) p2[M1 * m] = ah;
        if (o3 < 8 && !top) p3[M1 * m] = bh;
      }
    }
    // no barrier here: the next level's pass 1 writes the elements this
    // thread's last pass read, in the same buffer, and no other thread read
    // them (own_elements)
  }
}

// A clipping block of k_clip_walls: the row pairs p0.. again, E and dEX.  A call
// of its own, so that its three transforms' registers leave the scan of the
// unclipped blocks alone (inlined: 512x512x32 FP64 unclipped 52 us, 59 with
// Derivative as it is now, clipped 203; called: 50 and 190).
template <class T, int NSX>
__device__ __noinline__ void clip_rows(const cx<T>* ra, T* E, T* dEX, int z, int p0, int MY, T emin, T kx0,
                                       const cx<T>* tw) {
  constexpr int MX = 3 * NSX / 2;
  constexpr int KX = NSX / 2;
  using C = RowCfg<MX>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const int np = MY / 2;
  fft_core<MX, +1, false, false, true>(C::NT, sm, tw, [&](int, int n) {
    const PairMode m = pair_mode<MX>(n, KX);
    return m.join(ra[m.k], ra[KX + m.k]);
  }, NoStore{});
  const size_t zoff = (size_t)(z - 1) * MY * MX;
  for (int i = threadIdx.x; i < C::NT * MX; i += C::SUM_THREADS) {
    const int t = i / MX, n = i - t * MX, p = p0 + t;
    const cx<T> v = sm[i];
    if (p < np) {
      E[zoff + (size_t)(2 * p) * MX + n] = v.x;
      E[zoff + (size_t)(2 * p + 1) * MX + n] = v.y;
    }
    sm[i] = mk(tmax(emin - v.x, (T)0), tmax(emin - v.y, (T)0));
  }
  __syncthreads();
  fft_core<MX, -1, false, true, true>(C::NT, sm, tw, NoLoad{}, NoStore{});
  fft_core<MX, +1, false, true, false>(C::NT, sm, tw, Derivative<T, MX>(kx0), [&](int t, int n, cx<T> d) {
    const int p = p0 + t;
    if (p >= np) return;
    dEX[zoff + (size_t)(2 * p) * MX + n] = d.x;
    dEX[zoff + (size_t)(2 * p + 1) * MX + n] = d.y;
  });
}

// Does max(expand(e), emin) clip, and if so dEX = xderiv(delta), delta =
// max(emin - E, 0).  A block inverts C::NT row pairs of Em.  rowclip[z-1][block]
// says whether one of its points lies below emin; only then does it store its
// rows of E (for k_clipd_y) and dEX and set the level's flag: elsewhere delta
// and its x derivative are zero.  One kernel instead of a flag pass, a pass
// for E and one for dEX; a clipping block transforms its rows again, so that
// the common case keeps nothing (with the first transform's rows kept in
// shared memory an unclipped 512x512x256 stage took 418 us instead of 134).
// The first four block rows sum the wall rows, two block rows a side: a launch
// less (a 32x32x16 FP64 stage 79.5 -> 74.0 us, 64x64x64 135 -> 126).
// Registers: 168 (FP64) and 128 (FP32); unbounded, the 768-point FP32 rows take 190
// and an unclipped 512x512x64 launch 66 us instead of 47.
template <class T, int NSX>
__global__ void __launch_bounds__(RowCfg<3 * NSX / 2>::SUM_THREADS, sizeof(T) == 8 ? 3 : 4)
k_clip_walls(const cx<T>* __restrict__ Em, T* __restrict__ E, T* __restrict__ dEX, int* __restrict__ flags,
             unsigned char* __restrict__ rowclip, const cx<T>* __restrict__ Um, const cx<T>* __restrict__ Vm,
             double* __restrict__ wpart, int nwall, int MY, int NZ, T emin, T kx0, const cx<T>* __restrict__ tw) {
  constexpr int MX = 3 * NSX / 2;
  constexpr int KX = NSX / 2;
  using C = RowCfg<MX>;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  if (blockIdx.y < 4) {
    const int blk = (blockIdx.y & 1) * gridDim.x + blockIdx.x;
    if (blk < nwall) wall_rows_block<T, NSX>(Um, Vm, blockIdx.y >> 1, blk, nwall, MY, NZ, wpart, sm, tw);
    return;
  }
  const int z = (int)blockIdx.y - 3;
  const int p0 = blockIdx.x * C::NT, np = MY / 2;
  const cx<T>* in = Em + (size_t)(z - 1) * MY * KX;
  const int pl = p0 + (int)(threadIdx.x / Split<MX>::N2);  // the pair this thread loads
  const cx<T>* ra = in + (size_t)(2 * (pl < np ? pl : p0)) * KX;
  bool below = false;
  fft_core<MX, +1, false, false, false>(C::NT, sm, tw, [&](int, int n) {
    const PairMode m = pair_mode<MX>(n, KX);
    return m.join(ra[m.k], ra[KX + m.k]);
  }, [&](int t, int, cx<T> v) {
    below = below || (p0 + t < np && (v.x < emin || v.y < emin));
  });
  const bool any = __syncthreads_or(below);
  if (threadIdx.x == 0) {
    rowclip[(size_t)(z - 1) * gridDim.x + blockIdx.x] = any;
    if (any) atomicOr(flags + (z - 1), 1);
  }
  if (!any) return;
  clip_rows<T, NSX>(ra, E, dEX, z, p0, MY, emin, kx0, tw);
}

// dEY = yderiv(delta), delta = max(emin - E, 0), flagged levels only; rowclip
// (one byte per brows rows) says where E was stored, delta is zero elsewhere.
template <class T, int NSY>
__global__ void __launch_bounds__(ColCfg<3 * NSY / 2, T>::THREADS)
k_clipd_y(const T* __restrict__ E, T* __restrict__ dEY, const int* __restrict__ flags,
          const unsigned char* __restrict__ rowclip, int brows, int MX, T emin, T ky0, const cx<T>* __restrict__ tw) {
  constexpr int M = 3 * NSY / 2;
  using C = ColCfg<M, T>;
  if (!flags[blockIdx.y]) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
  const size_t zoff = (size_t)blockIdx.y * M * MX;
  const int c0 = blockIdx.x * C::TC, ncp = MX / 2;
  const cx<T>* Ez = reinterpret_cast<const cx<T>*>(E + zoff);
  __shared__ unsigned char clipped[M];
  for (int n = threadIdx.x; n < M; n += blockDim.x)
    clipped[n] = rowclip[(size_t)blockIdx.y * ((M + brows - 1) / brows) + n / brows];
  __syncthreads();
  fft_core<M, -1, true, false, true>(C::TC, sm, tw, [&](int t, int n) {
    int c = c0 + t;
    cx<T> v = zero_cx<T>();
    if (c < ncp) {  // load first, select after: the loads stay independent
      const cx<T> ev = Ez[(size_t)n * ncp + c];
      const bool on = clipped[n];
      v = mk(on ? tmax(emin - ev.x, (T)0) : (T)0, on ? tmax(emin - ev.y, (T)0) : (T)0);
    }
    return v;
  }, NoStore{});
  cx<T>* out = reinterpret_cast<cx<T>*>(dEY + zoff);
  fft_core<M, +1, true, true, false>(C::TC, sm, tw, Derivative<T, M>(ky0), [&](int t, int n, cx<T> d) {
    int c = c0 + t;
    if (c < ncp) out[(size_t)n * ncp + c] = d;
  });
}

}  // namespace les

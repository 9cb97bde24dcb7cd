// wave_cell.cuh -- the 2D wave stages (RHS, RK4 and Fehlberg stages; every kind and
// precision of wave2d.cuh) with one short-lived CTA per 32 x 8 cell of the grid.
//
// The persistent stage kernels (wave_stage_kernel, wave_fixed_kernel) keep HBM busy on
// large grids but take 8 (FP32) to 13 us (FP64) for a stage whose SMs get one tile each:
// tensor-map fetch, TMA load, conversion by six warps, computation and the x-face pass
// follow one another on one tile of 64 x 12..32 points. Here a CTA of 256 threads owns
// 32 x 8 points: all its loads are in flight at once, every thread converts
// the values it loaded, and several CTAs per SM overlap their phases. The same operations
// in the same order as the persistent kernels in FP32 (bit for bit); in FP64 the same
// fixed-point stencils, box units being those of this cell.
//
// A CTA:
//   1. loads p (x and y halo), u (x halo), v (y halo) into registers, and the operands of
//      the stage update (u^n, acc, ..., coefficients) of its own points;
//   2. closure columns: their x-closure sums go to all threads of the CTA, one sum per
//      thread (in the row warps, four to six lanes of every warp would hold GB300's narrow
//      FP64 pipe for the whole sequence), kept in shared memory. Their lines come from L2
//      (from a copy of the box in shared memory instead: nothing gained at 65^2, 17 %
//      slower at 1025^2, where the copy and its registers cost CTAs per SM);
//   3. FP64: conversion to words, or to int64 in units of the cell's largest exponent
//      (fx_fine); the boxes to shared memory;
//   4. stencils, SAT and update per point; points on an x face only leave their RHS in
//      shared memory, and the first warp finishes them, one point per lane.
// Launched with programmatic stream serialization: the next stage's CTAs may start while
// this one's last ones run, and wait (griddepcontrol.wait) before they touch memory. For
// that reason arrays that a stage writes are read through L2 (ld.cg), never the
// non-coherent cache.
//
// AOS (RHS only): source and destination in the reference's AoS FP64 layout, so that an
// RHS evaluation on device arrays is one kernel without the conversions to and from planes.
#pragma once

#include "wave2d.cuh"

namespace sbp {

constexpr int kCellTX = 32, kCellTY = 8, kCellThreads = 256;  // one point per thread

template <int ORD> struct WaveCell {
  static constexpr int R = OpShape<ORD>::W / 2, CS = OpShape<ORD>::CS;
  static constexpr int WARPS = kCellThreads / 32, TY = kCellTY;
  static constexpr int PW = kCellTX + 2 * R, PH = TY + 2 * R;
  static constexpr int NP = PH * PW, NU = TY * PW, NV = PH * kCellTX, N = NP + NU + NV;
  static constexpr int PER = (N + kCellThreads - 1) / kCellThreads;  // values a thread loads
};

template <typename T> __device__ __forceinline__ T ld_l2(const T* p) { return __ldcg(p); }

// Closure row of D1 through an accessor: closure_line's operations in its order.
template <typename T, int ORD, typename Ld>
__device__ __forceinline__ T closure_by(const Ld& ld, int n, int i, const T (&cls)[6][9]) {
  constexpr int CW = OpShape<ORD>::CW;
  T s;
  if (i < OpShape<ORD>::CS) {
    s = cls[i][0] * ld(0);
#pragma unroll
    for (int k = 1; k < CW; k++) s = fma(cls[i][k], ld(k), s);
  } else {
    const int r = n - 1 - i;
    s = -cls[r][CW - 1] * ld(n - CW);
#pragma unroll
    for (int k = 1; k < CW; k++) s = fma(-cls[r][CW - 1 - k], ld(n - CW + k), s);
  }
  return s;
}

// Interior taps through an accessor around index i, in the persistent kernels' order.
template <typename T, int ORD, typename Ld>
__device__ __forceinline__ T taps_by(const Ld& ld, int i, const T (&taps)[7]) {
  constexpr int W = OpShape<ORD>::W, R = (W - 1) / 2;
  T s = taps[0] * ld(i - R);
#pragma unroll
  for (int k = 1; k < W; k++)
    if (k != R) s = fma(taps[k], ld(i - R + k), s);
  return s;
}

// CTAs per SM the registers are sized for: the late Fehlberg stages hold a point's
// earlier derivatives in registers.
template <int STAGE> constexpr int wave_cell_ctas() { return STAGE >= ST_RKF1 + 2 ? 2 : 3; }

template <typename T, int ORD, int KIND, int STAGE, bool AOS>
__global__ void __launch_bounds__(kCellThreads, wave_cell_ctas<STAGE>())
    wave_cell_kernel(const __grid_constant__ WaveParams<T> prm) {
  static_assert(!AOS || STAGE == ST_RHS, "AoS arrays: RHS only");
  using C = WaveCell<ORD>;
  constexpr bool FIX = sizeof(T) == 8, COMP = IsCompensated<T>::value, RKF = is_rkf_stage(STAGE);
  constexpr int R = C::R, CS = C::CS, W = OpShape<ORD>::W, TY = C::TY, PW = C::PW, PER = C::PER, TX = kCellTX;
  constexpr int RKS = RKF ? STAGE - ST_RKF1 + 1 : 1;
  constexpr bool LOAD_UN = STAGE == ST_MID || (STAGE == ST_LAST && COMP), LOAD_ACC = STAGE == ST_MID || STAGE == ST_LAST;
  constexpr bool LOAD_CEN = STAGE == ST_FIRST && FIX;  // FP64: the box holds integers, u^n comes again
  constexpr int NK = KIND == WK_VAR ? 2 : (KIND == WK_MMS ? 3 : 0);
  __shared__ union {
    T f[C::N];
    long long i[FIX ? C::N : 1];
  } box;
  __shared__ T s_cls[2][TY][2 * CS];  // x-closure sums of p and u: [.][row][closure column]
  __shared__ T s_def[2][TY][3];       // RHS of x-face points: [west, east][row][u, v, p]
  __shared__ int s_max[C::WARPS][2];
  __shared__ double s_err[C::WARPS];
  __shared__ double s_ct;
  (void)s_max;
  (void)s_err;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nx = prm.nx, ny = prm.ny;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const long long pitch = prm.pitch, plane = prm.plane;
  const int i = i0 + lane;
  const int ys = KIND == WK_VAR ? prm.ysplit : 0;
  const auto interface_row = [&](int jj) { return KIND == WK_VAR && ys > 0 && (jj == ys - 1 || jj == ys); };
  grid_dependency_wait();
  if (prm.skip && *reinterpret_cast<const volatile int*>(prm.skip)) return;  // uniform over the grid

  // one value of the stage input
  const auto in_at = [&](int comp, int gj, int gi) -> T {
    if constexpr (AOS) return (T)ld_l2(prm.aos_in + 3 * ((long long)gj * nx + gi) + comp);
    else return ld_l2(prm.in + comp * plane + (long long)gj * pitch + gi);
  };

  // ---- 1. loads
  T val[PER];
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int e = tid + c * kCellThreads;
    val[c] = T(0);
    int comp, r, x;
    if (e < C::NP) {
      comp = 2, r = e / PW - R, x = e % PW - R;
    } else if (e < C::NP + C::NU) {
      comp = 0, r = (e - C::NP) / PW, x = (e - C::NP) % PW - R;
    } else {
      comp = 1, r = (e - C::NP - C::NU) / TX - R, x = (e - C::NP - C::NU) % TX;
    }
    const int gj = j0 + r, gi = i0 + x;
    if (e < C::N && gj >= 0 && gj < ny && gi >= 0 && gi < nx) val[c] = in_at(comp, gj, gi);
  }
  const int y = warp, j = j0 + y;  // this thread's point (i, j)
  const bool live = i < nx && j < ny;
  T un[3], ac[3], cm[3], co[NK > 0 ? NK : 1];
  double pre[3][RKS];
  if (live) {
    const long long q = (long long)j * pitch + i;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const long long o = c * plane + q;
      if constexpr (LOAD_UN) un[c] = ld_l2(prm.un + o);
      if constexpr (LOAD_CEN) un[c] = ld_l2(prm.in + o);
      if constexpr (LOAD_ACC) ac[c] = ld_l2(prm.acc + o);
      if constexpr (STAGE == ST_LAST && COMP) cm[c] = ld_l2(prm.comp + o);
      if constexpr (RKF) {
#pragma unroll
        for (int s = 0; s < RKS - 1; s++)
          if (RKS < 6 || s != 1) pre[c][s] = ld_l2(prm.rkk[s] + o);
        pre[c][RKS - 1] = ld_l2(prm.rku + o);
      }
    }
#pragma unroll
    for (int c = 0; c < NK; c++) co[c] = __ldg(prm.rinv + c * plane + q);
  }
  (void)un;
  (void)ac;
  (void)cm;
  (void)co;
  (void)pre;
  if constexpr (KIND == WK_MMS) {
    if (tid == 32)
      s_ct = prm.tctl ? cos(5 * 3.14159265358979323846264 *
                            __dadd_rn(ld_l2(prm.tctl), __dmul_rn(prm.tc, ld_l2(prm.tctl + 1))))
                      : (prm.ctp ? ld_l2(prm.ctp) : prm.ct);
  }

  // ---- 2. x-closure columns of this cell: [0, CS) and [nx - CS, nx), one sum per thread
  const int wcols = i0 == 0 ? CS : 0;
  const int e0 = i0 > nx - CS ? i0 : nx - CS, e1 = i0 + TX < nx ? i0 + TX : nx;
  const int ncol = wcols + (e1 > e0 ? e1 - e0 : 0);
  for (int t = tid; t < 2 * TY * ncol; t += kCellThreads) {
    const int col = t % ncol, yr = (t / ncol) % TY, d = t / (ncol * TY), jr = j0 + yr;
    const int I = col < wcols ? col : e0 + col - wcols;
    if (jr >= ny) continue;
    T s = closure_by<T, ORD>([&](int k) { return in_at(d == 0 ? 2 : 0, jr, k); }, nx, I, prm.dx.cls);
    if constexpr (FIX) s *= prm.fx_isig[0];
    s_cls[d][yr][col] = s;
  }

  // ---- 3. boxes to shared memory
  constexpr bool FINE = fx_fine<KIND, STAGE>();
  int ebp = 0, ebuv = 0;
  bool taps = false;  // the cell's values leave the fixed-point range: FP64 taps
  if constexpr (FIX && FINE) {
    bool out = false;
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int e = tid + c * kCellThreads;
      const long long w = fx_pack((double)val[c], out);
      if (e < C::N) box.i[e] = w;
    }
    taps = __syncthreads_or(out);
  } else if constexpr (FIX) {
    unsigned mp = 0, muv = 0;
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const unsigned h = (unsigned)__double2hiint((double)val[c]) & 0x7FF00000u;
      if (tid + c * kCellThreads < C::NP) mp = max(mp, h);
      else muv = max(muv, h);
    }
    mp = __reduce_max_sync(0xffffffffu, mp);
    muv = __reduce_max_sync(0xffffffffu, muv);
    if (lane == 0) {
      s_max[warp][0] = (int)(mp >> 20);
      s_max[warp][1] = (int)(muv >> 20);
    }
    __syncthreads();
    int ep, euv;
    fx_tile_emax<C::WARPS, true>(&s_max[0][0], ep, euv, taps);
    ebp = fx_base<false>(ep);
    ebuv = fx_base<false>(euv);
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int e = tid + c * kCellThreads;
      const double v = (double)val[c];
      if (e < C::N)
        box.i[e] = fx_from<false>((unsigned)__double2loint(v), (unsigned)__double2hiint(v), e < C::NP ? ep : euv);
    }
    __syncthreads();
  } else {
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int e = tid + c * kCellThreads;
      if (e < C::N) box.f[e] = val[c];
    }
    __syncthreads();
  }

  // ---- 4. points
  const bool xfaces = prm.bc != BC_NONE && (i0 == 0 || (nx - 1 >= i0 && nx - 1 < i0 + TX));
  const double h = RKF ? ld_l2(prm.tctl + 1) : 0.0;
  double errsq = 0.0;
  (void)h;
  // RK stage update of one point: the RHS k (FIX && scaled: in units of sigma), the
  // operands of the update; all in the persistent kernels' operations
  const auto store = [&](int jj, int ii, const T (&k)[3], bool scaled, const T* cen, const T* u0, const T* a0,
                         const T* c0, const double (*p0)[RKS]) {
    const long long q = (long long)jj * pitch + ii;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const long long o = c * plane + q;
      T kt = k[c], ca = prm.c_acc, cw = prm.c_w;
      if constexpr (FIX) {
        if (scaled) {
          if constexpr (STAGE == ST_RHS || RKF) {
            kt *= c == 0 ? prm.fx_sig[0] : (c == 1 ? prm.fx_sig[1] : prm.fx_sigp);
          } else {
            ca = prm.fx_ca[c];
            cw = prm.fx_cw[c];
          }
        }
      }
      if constexpr (STAGE == ST_RHS) {
        if constexpr (AOS) prm.aos_out[3 * ((long long)jj * nx + ii) + c] = (double)kt;
        else prm.kout[o] = kt;
      } else if constexpr (RKF) {
        const double kS = kt;
        if constexpr (RKS < 6) {
          prm.rkk[RKS - 1][o] = kS;
          double s = kRkfA[RKS][0] * (RKS == 1 ? kS : p0[c][0]);
#pragma unroll
          for (int s2 = 1; s2 < RKS; s2++) s = fma(kRkfA[RKS][s2], s2 == RKS - 1 ? kS : p0[c][s2], s);
          prm.wout[o] = fma(h, s, p0[c][RKS - 1]);
        } else {
          double u5, u4;
          rkf_candidate(p0[c][5], h, p0[c][0], p0[c][2], p0[c][3], p0[c][4], kS, u5, u4);
          prm.rkunew[o] = u5;
          errsq += rkf_err_term(u5, u4, prm.rkatol, prm.rkrtol);
        }
      } else if constexpr (STAGE == ST_FIRST) {
        prm.acc[o] = COMP ? ca * kt : fma(ca, kt, cen[c]);
        prm.wout[o] = fma(cw, kt, cen[c]);
      } else if constexpr (STAGE == ST_MID) {
        prm.acc[o] = fma(ca, kt, a0[c]);
        prm.wout[o] = fma(cw, kt, u0[c]);
      } else {
        const T d = fma(ca, kt, a0[c]);
        if constexpr (COMP) {
          // Kahan summation of the step increment into the FP32 state
          const T yv = d - c0[c];
          const T tv = u0[c] + yv;
          prm.comp[o] = (tv - u0[c]) - yv;
          prm.un[o] = tv;
        } else {
          prm.un[o] = d;
        }
      }
    }
  };

  const auto point = [&]() {
    const int jb0 = (ys > 0 && j >= ys) ? ys : 0;
    const int nyb = ys > 0 ? (j >= ys ? ny - ys : ys) : ny;
    const bool xint = i >= CS && i < nx - CS, yint = j - jb0 >= CS && j - jb0 < nyb - CS;
    const int ccol = i < CS ? i : wcols + (i - e0);  // this column's closure sums
    const int cp = (y + R) * PW + lane + R, cu = C::NP + y * PW + lane + R, cv = C::NP + C::NU + (y + R) * TX + lane;
    const auto y_closure = [&](int comp) {
      return closure_by<T, ORD>([&](int k) { return in_at(comp, jb0 + k, i); }, nyb, j - jb0, prm.dy.cls);
    };
    T k[3], cen[3];
    if constexpr (FIX) {
      const bool xfx = xint && !taps, yfx = yint && !taps;
      const auto other_x = [&](int d, int comp) -> T {
        if (!xint) return s_cls[d][y][ccol];
        return taps_by<T, ORD>([&](int q) { return in_at(comp, j, q); }, i, prm.dx.taps) * prm.fx_isig[0];
      };
      const auto other_y = [&](int comp) -> T {
        if (!yint) return y_closure(comp) * prm.fx_isig[1];
        return taps_by<T, ORD>([&](int q) { return in_at(comp, q, i); }, j, prm.dy.taps) * prm.fx_isig[1];
      };
      const auto d1 = [&](int at, int st, int eb) {
        if constexpr (FINE) return fx_d1<ORD>(box.i + at, st);
        else return fx_to<false>(fx_stencil<ORD>(box.i + at, st), eb);
      };
      k[0] = xfx ? d1(cp, 1, ebp) : other_x(0, 2);
      k[1] = yfx ? d1(cp, PW, ebp) : other_y(2);
      if (xfx && yfx && prm.fx_square) {
        if constexpr (FINE) k[2] = fx_d1_sum<ORD>(box.i + cu, 1, box.i + cv, TX);
        else k[2] = fx_to<false>(fx_stencil<ORD>(box.i + cu, 1) + fx_stencil<ORD>(box.i + cv, TX), ebuv);
      } else {
        const double ax = xfx ? d1(cu, 1, ebuv) : other_x(1, 0);
        const double ay = yfx ? d1(cv, TX, ebuv) : other_y(1);
        k[2] = fma(prm.fx_rho, ay, ax);
      }
      if constexpr (KIND == WK_VAR) {
        k[0] *= co[0];
        k[1] *= co[0];
        k[2] *= co[1];
      } else if constexpr (KIND == WK_MMS) {
        k[0] = fma(s_ct, co[1], co[0] * k[0]);
        k[1] = fma(s_ct, co[2], co[0] * k[1]);
      }
      if constexpr (LOAD_CEN) {
#pragma unroll
        for (int c = 0; c < 3; c++) cen[c] = un[c];
      }
    } else {
      const T* f = box.f;
      const auto chain = [&](int at, int st, const T (&tp)[7], T s, bool first) {
#pragma unroll
        for (int q = 0; q < W; q++)
          if (q != R) {
            const T v = f[at + (q - R) * st];
            s = (first && q == 0) ? tp[0] * v : fma(tp[q], v, s);
          }
        return s;
      };
      const T dxp = xint ? chain(cp, 1, prm.dx.taps, T(0), true) : s_cls[0][y][ccol];
      const T dyp = yint ? chain(cp, PW, prm.dy.taps, T(0), true) : y_closure(2);
      T kp = xint ? chain(cu, 1, prm.dx.taps, T(0), true) : s_cls[1][y][ccol];
      if (yint) kp = chain(cv, TX, prm.dy.taps, kp, false);
      else kp += y_closure(1);
      if constexpr (KIND == WK_VAR) {
        k[0] = co[0] * dxp;
        k[1] = co[0] * dyp;
        k[2] = co[1] * kp;
      } else {
        k[0] = dxp;
        k[1] = dyp;
        k[2] = kp;
      }
      cen[0] = f[cu];
      cen[1] = f[cv];
      cen[2] = f[cp];
    }
    const bool edge = i == 0 || j == 0 || i == nx - 1 || j == ny - 1 || interface_row(j);
    bool scaled = true;
    if (prm.bc != BC_NONE && edge) {
      T kt[3] = {k[0], k[1], k[2]};
      if constexpr (FIX) {  // true units
        kt[0] *= prm.fx_sig[0];
        kt[1] *= prm.fx_sig[1];
        kt[2] *= prm.fx_sigp;
      }
      if (j != 0 && j != ny - 1 && !interface_row(j)) {  // an x-face point only: the first warp's
        T* d = s_def[i == 0 ? 0 : 1][y];
        d[0] = kt[0];
        d[1] = kt[1];
        d[2] = kt[2];
        return;
      }
      const Rhs3<T> r = apply_sat<T, KIND>(prm, prm.in, i, j, in_at(2, j, i), in_at(0, j, i),
                                           in_at(1, j, i), Rhs3<T>{kt[0], kt[1], kt[2]});
      k[0] = r.u;
      k[1] = r.v;
      k[2] = r.p;
      scaled = false;
    }
    store(j, i, k, scaled, cen, un, ac, cm, pre);
  };
  if (live) point();
  if (xfaces) {  // uniform over the CTA
    __syncthreads();
    for (int e = lane; warp == 0 && e < 2 * TY; e += 32) {
      const int side = e / TY, jf = j0 + e % TY, ii = side == 0 ? 0 : nx - 1;
      if (ii < i0 || ii >= i0 + TX || jf >= ny || jf == 0 || jf == ny - 1 || interface_row(jf)) continue;
      const T* d = s_def[side][e % TY];
      const T cen[3] = {in_at(0, jf, ii), in_at(1, jf, ii), in_at(2, jf, ii)};
      const Rhs3<T> r =
          apply_sat<T, KIND>(prm, prm.in, ii, jf, cen[2], cen[0], cen[1], Rhs3<T>{d[0], d[1], d[2]});
      const T k[3] = {r.u, r.v, r.p};
      T u0[3], a0[3], c0[3];
      double p0[3][RKS];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const long long o = c * plane + (long long)jf * pitch + ii;
        if constexpr (LOAD_UN) u0[c] = ld_l2(prm.un + o);
        if constexpr (LOAD_ACC) a0[c] = ld_l2(prm.acc + o);
        if constexpr (STAGE == ST_LAST && COMP) c0[c] = ld_l2(prm.comp + o);
        if constexpr (RKF) {
#pragma unroll
          for (int s = 0; s < RKS - 1; s++)
            if (RKS < 6 || s != 1) p0[c][s] = ld_l2(prm.rkk[s] + o);
          p0[c][RKS - 1] = ld_l2(prm.rku + o);
        }
      }
      store(jf, ii, k, false, cen, u0, a0, c0, p0);
    }
  }
  if constexpr (STAGE == ST_RKF6) {
    // fixed-order sum over the CTA's threads -> one partial per CTA
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) errsq += __shfl_down_sync(0xffffffffu, errsq, off);
    if (lane == 0) s_err[warp] = errsq;
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
      for (int q = 0; q < C::WARPS; q++) s += s_err[q];
      prm.rkpart[blockIdx.y * gridDim.x + blockIdx.x] = s;
    }
  }
}

}  // namespace sbp

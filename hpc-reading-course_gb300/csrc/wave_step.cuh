// wave_step.cuh -- whole RK4 steps of small FP64 2D wave grids, one launch per step.
//
// On grids of one or two hundred points per side a stage is shorter than what surrounds it:
// launch, the wait for the previous kernel's memory, loads from L2 and the tail take most of
// the 6 to 8 us of a stage in its cell form (wave_cell.cuh). Here a CTA computes all four
// stages of TC x TC points: it loads u^n on the points the first stage reads for them (the
// cell, and per stage and side one stencil reach R), computes stage 1 on the points stage 2
// reads, and so on; stage inputs stay in shared memory. Neighbouring CTAs repeat each other's
// halo points (16 x 16 at order 4: 2016 point-stages for 1024), and the FP64 pipe bounds a
// CTA, so the form pays while every SM has at most one. u^{n+1} goes to another buffer, since
// neighbours read u^n; two buffers alternate.
// Measured, us per stage (a step's quarter), cells / this: rho=K=1 129^2 6.0 / 3.1, 6.9 / 4.1 and
// 7.8 / 5.9 at orders 2, 4 and 6, 257^2 6.8 / 4.9 and 7.9 / 6.3 (order 6: 217^2 8.6 / 7.0); variable
// 129^2 6.6 / 3.9, 7.8 / 4.9, 8.4 / 6.7; forced 6.5 / 3.6, 7.4 / 4.6, 7.8 / 6.6; grids of 20:1 and
// 1:9 the same gains. With more cells than SMs it loses: some SM then takes two, one after the
// other (order 4 289^2 9.6 against 7.2).
//
// Per stage: the closure sums and the SAT of face points, one per thread (a row of the cell
// has one to six such points; in the point loop each would hold its warp's FP64 pipe); the
// points of the stage's rectangle (fixed-point stencils on words, wave2d_fixed.cuh), their next
// stage input in registers; conversion to words in place, which hold the values whole: closure
// rows and SAT take them back. A rectangle with a value that has no word is kept as doubles,
// and its stencils are FP64 taps.
#pragma once

#include "wave_cell.cuh"

namespace sbp {

constexpr int kStepThreads = 512;
// Cell sides: 16, and the largest whose box fits a CTA's shared memory.
constexpr int kStepSmall = 16;
constexpr int step_large(int order) { return order == 6 ? 20 : 24; }

// TC: the cell's side.
template <int ORD, int TC> struct WaveStep {
  static constexpr int R = OpShape<ORD>::W / 2, CS = OpShape<ORD>::CS, CW = OpShape<ORD>::CW;
  // How far the four stages' reads extend beyond a cell, both sides together: a reach per
  // stage and side, where a closure row asks for its whole block instead (a grid edge on one
  // or both sides, or the interface of two blocks).
  static constexpr int M = 3 * R + (R > CS - 1 ? R : CS - 1);
  static constexpr int GROW = 2 * M > 7 * R + CW ? 2 * M : 7 * R + CW;
  static constexpr int P = TC + GROW, N = P * P;  // box side, points
  static constexpr int CR = 4 * CS;               // closure rows a rectangle can have
  static constexpr int PER = (N + kStepThreads - 1) / kStepThreads;
  // u^n, the stage input (words), coefficient planes, acc, y-closure sums
  static constexpr int smem(int planes) { return ((6 + planes) * N + 3 * TC * TC + 2 * CR * P) * 8; }
};

// The interval of a stage input that the points [lo, hi) of a line read: closure rows of
// [b, e) (the block the points are in) read its first or last CW points.
template <int ORD> __host__ __device__ inline void step_reads(int& lo, int& hi, int n, int ysplit) {
  constexpr int R = OpShape<ORD>::W / 2, CS = OpShape<ORD>::CS, CW = OpShape<ORD>::CW;
  int l = lo - R, h = hi + R;
  const int edges[2][2] = {{0, ysplit > 0 ? ysplit : n}, {ysplit > 0 ? ysplit : 0, n}};
  for (int q = 0; q < (ysplit > 0 ? 2 : 1); q++) {
    const int b = edges[q][0], e = edges[q][1];
    if (lo < b + CS && hi > b) h = h > b + CW ? h : b + CW, l = l < b ? l : b;
    if (hi > e - CS && lo < e) l = l < e - CW ? l : e - CW, h = h > e ? h : e;
  }
  lo = l > 0 ? l : 0;
  hi = h < n ? h : n;
}

// The RK4 coefficients times each component's scale (set_fixed_scales): ca dt/6 and dt/3, cw
// dt/2 and dt.
struct WaveStepCoef {
  double ca[2][3], cw[2][3];
};

// SAT of a face point, to be added to its RHS (the terms of apply_sat, one direction each).
template <int KIND>
__device__ __forceinline__ void sat_coefficients(const WaveParams<double>& prm, int i, int j, double& hr, double& z,
                                                 double& hc, double& hk) {
  hr = 0.5, z = 1.0, hc = 0.5, hk = 0.5;
  if constexpr (KIND == WK_VAR) {
    const double2* t = reinterpret_cast<const double2*>(prm.satc) + 2 * sat_point(prm.nx, prm.ny, prm.ysplit, i, j);
    const double2 a = __ldg(t), b = __ldg(t + 1);
    hr = a.x, z = a.y, hc = b.x, hk = b.y;
  }
}
// On the lower (lo) or upper face of a direction with weight bw: the terms of the normal
// velocity (.u) and of p (.p).
template <int KIND>
__device__ __forceinline__ Rhs3<double> face_sat(const WaveParams<double>& prm, int i, int j, bool lo, double bw,
                                                 double p, double un) {
  double hr, z, hc, hk;
  sat_coefficients<KIND>(prm, i, j, hr, z, hc, hk);
  const double sg = lo ? -1.0 : 1.0;
  if (prm.bc == BC_FREE_SURFACE) return Rhs3<double>{sg * (2.0 * hr) * (bw * p), 0.0, 0.0};
  const double g = bw * (p - sg * (z * un));
  return Rhs3<double>{sg * (hr * g), 0.0, -(hc * g)};
}
// A row on a y face or an interface line: the terms of v (.u) and of p (.p); po, vo: p and v on
// the other block's copy of the line.
template <int KIND>
__device__ __forceinline__ Rhs3<double> row_sat(const WaveParams<double>& prm, int i, int j, double p, double v,
                                                double po, double vo) {
  Rhs3<double> r{0.0, 0.0, 0.0};
  if (j == 0 || j == prm.ny - 1) r = face_sat<KIND>(prm, i, j, j == 0, prm.bwy, p, v);
  if constexpr (KIND == WK_VAR) {
    const int ys = prm.ysplit;
    if (ys > 0 && (j == ys - 1 || j == ys)) {
      double hr, z, hc, hk;
      sat_coefficients<KIND>(prm, i, j, hr, z, hc, hk);
      const double sg = j == ys - 1 ? 1.0 : -1.0;
      r.u += sg * hr * (prm.bwy * (p - po));
      r.p += sg * hk * (prm.bwy * (v - vo));
    }
  }
  return r;
}

template <int ORD, int KIND, int TC>
__global__ void __launch_bounds__(kStepThreads, 1) wave_step_kernel(const __grid_constant__ WaveParams<double> prm,
                                                                    const __grid_constant__ WaveStepCoef cf) {
  using S = WaveStep<ORD, TC>;
  constexpr int CS = S::CS, P = S::P, N = S::N, PER = S::PER, NT = kStepThreads;
  constexpr int NK = KIND == WK_VAR ? 2 : (KIND == WK_MMS ? 3 : 0);
  extern __shared__ __align__(16) unsigned char step_smem[];
  double* const su = reinterpret_cast<double*>(step_smem);         // u^n: [3][N]
  long long* const si = reinterpret_cast<long long*>(su + 3 * N);  // stage input, as words: [3][N]
  double* const sk = reinterpret_cast<double*>(si + 3 * N);        // coefficients: [NK][N]
  double* const sacc = sk + NK * N;                                // acc: [3][TC * TC]
  double* const scy = sacc + 3 * TC * TC;                          // y-closure sums of p and v: [2][CR][P]
  __shared__ double s_cls[2][P][2 * CS];  // x-closure sums of p and u, units of sigma: [.][row][column]
  __shared__ double s_sat[2][P][2];       // x-face SAT of u and p, units of sigma: [west, east][row]
  __shared__ double s_saty[4][P][2];      // SAT of v and p on rows 0, ny - 1, ys - 1, ys
  const int tid = threadIdx.x;
  const int nx = prm.nx, ny = prm.ny, ys = KIND == WK_VAR ? prm.ysplit : 0;
  const long long pitch = prm.pitch, plane = prm.plane;
  const int ci = blockIdx.x * TC, cj = blockIdx.y * TC;
  const int ce = ci + TC < nx ? ci + TC : nx, cn = cj + TC < ny ? cj + TC : ny;
  // rectangle s: the points stage s + 1 computes (s = 0..3); their reads are rectangle s - 1;
  // box: what stage 1 reads
  int x0[4], x1[4], y0[4], y1[4], bx0, bx1, by0, by1;
  x0[3] = ci, x1[3] = ce, y0[3] = cj, y1[3] = cn;
#pragma unroll
  for (int s = 2; s >= 0; s--) {
    x0[s] = x0[s + 1], x1[s] = x1[s + 1], y0[s] = y0[s + 1], y1[s] = y1[s + 1];
    step_reads<ORD>(x0[s], x1[s], nx, 0);
    step_reads<ORD>(y0[s], y1[s], ny, ys);
  }
  bx0 = x0[0], bx1 = x1[0], by0 = y0[0], by1 = y1[0];
  step_reads<ORD>(bx0, bx1, nx, 0);
  step_reads<ORD>(by0, by1, ny, ys);
  const int bw = bx1 - bx0, bn = bw * (by1 - by0);
  if (bw > P || by1 - by0 > P) {  // the box is sized for every position (tests/test_wave_step.py)
    if (tid == 0) atomicOr(prm.err, ERR_BAD_LAUNCH);
    return;
  }
  const auto interface_row = [&](int j) { return ys > 0 && (j == ys - 1 || j == ys); };
  const auto at = [&](int i, int j) { return (j - by0) * P + (i - bx0); };
  const auto div = [](int e, int w) {  // e / w for e, w below 2^15
    return (int)(((float)e + 0.5f) * __frcp_rn((float)w));
  };
  grid_dependency_wait();

  // u^n and the coefficients on the box
  double v[PER][3];  // this thread's values of the next stage input
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int e = tid + c * NT;
    if (e < bn) {
      const int r = div(e, bw), i = bx0 + e - r * bw, j = by0 + r;
      const long long q = (long long)j * pitch + i;
#pragma unroll
      for (int m = 0; m < 3; m++) {
        v[c][m] = ld_l2(prm.in + m * plane + q);
        su[m * N + at(i, j)] = v[c][m];
      }
#pragma unroll
      for (int m = 0; m < NK; m++) sk[m * N + at(i, j)] = __ldg(prm.rinv + m * plane + q);
    }
  }
  double ct[3] = {0, 0, 0};
  if constexpr (KIND == WK_MMS) {
#pragma unroll
    for (int m = 0; m < 3; m++) ct[m] = ld_l2(prm.ctp + m);  // the forcing's factor at t, t + dt/2, t + dt
  }
  int px0 = bx0, px1 = bx1, py0 = by0;  // the rectangle the values v belong to

#pragma unroll 1
  for (int s = 0; s < 4; s++) {
    // ---- the stage input to shared memory
    const int pw = px1 - px0, pn = s == 0 ? bn : (x1[s - 1] - x0[s - 1]) * (y1[s - 1] - y0[s - 1]);
    long long word[PER][3];
    bool out = false;
#pragma unroll
    for (int c = 0; c < PER; c++)
      if (tid + c * NT < pn) {
#pragma unroll
        for (int m = 0; m < 3; m++) word[c][m] = fx_pack(v[c][m], out);
      }
    const bool taps = __syncthreads_or(out);  // and every thread has read the previous stage input
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int e = tid + c * NT;
      if (e < pn) {
        const int r = div(e, pw), o = at(px0 + e - r * pw, py0 + r);
#pragma unroll
        for (int m = 0; m < 3; m++) si[m * N + o] = taps ? __double_as_longlong(v[c][m]) : word[c][m];
      }
    }
    __syncthreads();
    // a value of the stage input
    const auto val = [&](int m, int i, int j) {
      const long long q = si[m * N + at(i, j)];
      return taps ? __longlong_as_double(q) : fx_unpack(q);
    };
    // ---- x-closure sums and x-face SAT, one per thread
    const int ax0 = x0[s], ax1 = x1[s], ay0 = y0[s], ay1 = y1[s], rows = ay1 - ay0;
    const int wc = ax0 < CS ? CS - ax0 : 0;                                      // columns [ax0, ax0 + wc) and
    const int e0 = ax0 > nx - CS ? ax0 : nx - CS, ec = ax1 > e0 ? ax1 - e0 : 0;  // [e0, e0 + ec)
    const int nc = wc + ec;
    // closure rows of the rectangle: of [0, CS), [ys - CS, ys + CS), [ny - CS, ny)
    const int w = ax1 - ax0;
    const int r0 = ay0, l0 = ay1 < CS ? rows : (CS > ay0 ? CS - ay0 : 0);
    int r1 = 0, l1 = 0;
    if (ys > 0) {
      r1 = ay0 > ys - CS ? ay0 : ys - CS;
      l1 = (ay1 < ys + CS ? ay1 : ys + CS) - r1;
      if (l1 < 0) l1 = 0;
    }
    const int r2 = ay0 > ny - CS ? ay0 : ny - CS, l2 = ay1 > r2 ? ay1 - r2 : 0;
    const int ncr = l0 + l1 + l2;
    const auto up = [](int n) { return (n + 31) & ~31; };  // task kinds start at whole warps
    const bool sat = prm.bc != BC_NONE;
    const bool sat_x = sat && (ax0 == 0 || ax1 == nx);
    const bool sat_y = sat && (ay0 == 0 || ay1 == ny || (ys > 0 && ay0 <= ys && ay1 >= ys));
    const int tx = up(2 * rows * nc), ty = tx + up(2 * w * ncr), tsx = ty + (sat_x ? up(2 * rows) : 0),
              total = tsx + (sat_y ? up(4 * w) : 0);
    if (total > 0) {  // uniform
      for (int t = tid; t < total; t += NT) {
        if (t < tx) {
          if (t >= 2 * rows * nc) continue;
          const int q = div(t, nc), col = t - q * nc, d = q >= rows, yr = q - d * rows;
          const int i = col < wc ? ax0 + col : e0 + col - wc;
          s_cls[d][yr][col] = prm.fx_isig[0] *
              closure_by<double, ORD>([&](int k) { return val(d == 0 ? 2 : 0, k, ay0 + yr); }, nx, i, prm.dx.cls);
        } else if (t < ty) {
          if (t - tx >= 2 * w * ncr) continue;
          const int q = div(t - tx, w), i = ax0 + t - tx - q * w, d = q >= ncr, cr = q - d * ncr;
          const int j = cr < l0 ? r0 + cr : (cr < l0 + l1 ? r1 + cr - l0 : r2 + cr - l0 - l1);
          const int jb0 = (ys > 0 && j >= ys) ? ys : 0, nyb = ys > 0 ? (j >= ys ? ny - ys : ys) : ny;
          scy[(d * S::CR + cr) * P + i - ax0] = prm.fx_isig[1] *
              closure_by<double, ORD>([&](int k) { return val(d == 0 ? 2 : 1, i, jb0 + k); }, nyb, j - jb0, prm.dy.cls);
        } else if (t < tsx) {
          const int q = t - ty, side = q >= rows, yr = q - side * rows, i = side == 0 ? 0 : nx - 1, j = ay0 + yr;
          if (yr >= rows || i < ax0 || i >= ax1) continue;
          const Rhs3<double> z = face_sat<KIND>(prm, i, j, side == 0, prm.bwx, val(2, i, j), val(0, i, j));
          s_sat[side][yr][0] = z.u * prm.fx_isig[0];
          s_sat[side][yr][1] = z.p * prm.fx_isig[0];
        } else {
          const int q = div(t - tsx, w), i = ax0 + t - tsx - q * w;
          const int j = q == 0 ? 0 : (q == 1 ? ny - 1 : (q == 2 ? ys - 1 : ys));
          if (q > 3 || (q > 1 && ys == 0) || j < ay0 || j >= ay1) continue;
          const double vo = q > 1 ? val(1, i, q == 2 ? ys : ys - 1) : 0.0, po = q > 1 ? val(2, i, q == 2 ? ys : ys - 1) : 0.0;
          const Rhs3<double> z = row_sat<KIND>(prm, i, j, val(2, i, j), val(1, i, j), po, vo);
          s_saty[q][i - ax0][0] = z.u * prm.fx_isig[1];
          s_saty[q][i - ax0][1] = z.p * prm.fx_isig[0];
        }
      }
      __syncthreads();
    }
    // ---- points
    const int n = w * rows;
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const int e = tid + c * NT;
      if (e >= n) continue;
      const int r = div(e, w), i = ax0 + e - r * w, j = ay0 + r, o = at(i, j);
      const int jb0 = (ys > 0 && j >= ys) ? ys : 0;
      const int nyb = ys > 0 ? (j >= ys ? ny - ys : ys) : ny;
      const bool xint = i >= CS && i < nx - CS, yint = j - jb0 >= CS && j - jb0 < nyb - CS;
      const long long *cp = si + 2 * N + o, *cu = si + o, *cv = si + N + o;
      const int col = i < CS ? i - ax0 : wc + (i - e0);
      // this row's place among the closure rows
      const int cr = j < CS ? j - r0 : (j >= ny - CS ? l0 + l1 + j - r2 : l0 + j - r1);
      const auto d_y = [&](int m) {
        if (!yint) return scy[((m == 2 ? 0 : 1) * S::CR + cr) * P + i - ax0];
        return prm.fx_isig[1] * taps_by<double, ORD>([&](int k) { return val(m, i, k); }, j, prm.dy.taps);
      };
      const auto x_taps = [&](int m) {
        return prm.fx_isig[0] * taps_by<double, ORD>([&](int k) { return val(m, k, j); }, i, prm.dx.taps);
      };
      double k[3];
      const bool xfx = xint && !taps, yfx = yint && !taps;
      if (xfx) k[0] = fx_d1<ORD>(cp, 1);
      else k[0] = xint ? x_taps(2) : s_cls[0][r][col];
      if (yfx) k[1] = fx_d1<ORD>(cp, P);
      else k[1] = d_y(2);
      if (xfx && yfx && prm.fx_square) {
        k[2] = fx_d1_sum<ORD>(cu, 1, cv, P);
      } else {
        const double ax = xfx ? fx_d1<ORD>(cu, 1) : (xint ? x_taps(0) : s_cls[1][r][col]);
        const double ay = yfx ? fx_d1<ORD>(cv, P) : d_y(1);
        k[2] = fma(prm.fx_rho, ay, ax);
      }
      if constexpr (KIND == WK_VAR) {
        const double ri = sk[o];
        k[0] *= ri;
        k[1] *= ri;
        k[2] *= sk[N + o];
      } else if constexpr (KIND == WK_MMS) {
        const double ri = sk[o], cts = s == 0 ? ct[0] : (s == 3 ? ct[2] : ct[1]);
        k[0] = fma(cts, sk[N + o], ri * k[0]);
        k[1] = fma(cts, sk[2 * N + o], ri * k[1]);
      }
      if (sat) {
        if (j == 0 || j == ny - 1 || interface_row(j)) {
          const double* z = s_saty[j == 0 ? 0 : (j == ny - 1 ? 1 : (j == ys - 1 ? 2 : 3))][i - ax0];
          k[1] += z[0];
          k[2] += z[1];
        }
        if (i == 0 || i == nx - 1) {
          const double* z = s_sat[i == 0 ? 0 : 1][r];
          k[0] += z[0];
          k[2] += z[1];
        }
      }
      const bool own = i >= ci && i < ce && j >= cj && j < cn;
      const int oa = (j - cj) * TC + i - ci;
#pragma unroll
      for (int m = 0; m < 3; m++) {
        const double u0 = su[m * N + o];
        if (s < 3) {
          if (own) {
            double& a = sacc[m * TC * TC + oa];
            a = fma(cf.ca[s == 0 ? 0 : 1][m], k[m], s == 0 ? u0 : a);
          }
          v[c][m] = fma(cf.cw[s == 2 ? 1 : 0][m], k[m], u0);
        } else {
          prm.wout[m * plane + (long long)j * pitch + i] = fma(cf.ca[0][m], k[m], sacc[m * TC * TC + oa]);
        }
      }
    }
    px0 = ax0, px1 = ax1, py0 = ay0;
  }
}

}  // namespace sbp

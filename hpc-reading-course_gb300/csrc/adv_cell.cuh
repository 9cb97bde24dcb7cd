// adv_cell.cuh -- FP64 stages of 2D advection with one short CTA per cell of 32 x 8 or
// 32 x 16 points.
//
// line_stage_kernel's form (one thread per point, every tap a global load) issues eight FP64
// FMAs of taps per point at order 4 on a pipe that takes 19 clocks per warp instruction and SM:
// 5.8 clocks per point. Here the cell's box of u is loaded once and converted to words
// (wave2d_fixed.cuh), the interior stencils are integer sums, and the FP64 pipe keeps the two
// scalings and the update. A thread takes ROWS rows of a column. x-closure sums: one per thread,
// as in wave_cell.cuh, whose notes on overlapped launches and ld.cg apply here. Measured, us per
// stage, line form -> this: 2049^2 70 -> 44, 103 -> 50 and 137 -> 59 at orders 2, 4 and 6, with
// velocity fields 89 -> 68, 122 -> 73, 154 -> 77; 801^2 order 4 19.9 -> 10.4. The FP64 pipe (four
// instructions per point: 2.4 of 3.5 clocks at 2049^2 order 4) and the integer instructions
// bound it together.
#pragma once

#include "line_kernels.cuh"
#include "wave_cell.cuh"

namespace sbp {

// FIELDS: a velocity at every point (one kernel for both would execute both forms' FP64
// instructions, seven per point instead of four).
template <int ORD, int STAGE, bool FIELDS, int ROWS>
__global__ void __launch_bounds__(kCellThreads, 4) adv_cell_kernel(const __grid_constant__ LineParams<double> prm) {
  constexpr int R = OpShape<ORD>::W / 2, CS = OpShape<ORD>::CS, TX = kCellTX, TY = kCellThreads / 32 * ROWS;
  constexpr int PW = TX + 2 * R, N = (TY + 2 * R) * PW, PER = (N + kCellThreads - 1) / kCellThreads;
  __shared__ long long box[N];
  __shared__ double s_cls[TY][2 * CS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nx = prm.nx, ny = prm.ny, i0 = blockIdx.x * TX, j0 = blockIdx.y * TY, i = i0 + lane;
  const int y0 = warp * ROWS;  // this thread's points: column i, rows j0 + y0 ..
  const long long pitch = prm.pitch;
  grid_dependency_wait();
  if (prm.skip && *reinterpret_cast<const volatile int*>(prm.skip)) return;  // uniform over the grid
  const auto in_at = [&](int gj, int gi) { return ld_l2(prm.in + (long long)gj * pitch + gi); };
  double val[PER];
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int e = tid + c * kCellThreads, gj = j0 + e / PW - R, gi = i0 + e % PW - R;
    val[c] = e < N && gj >= 0 && gj < ny && gi >= 0 && gi < nx ? in_at(gj, gi) : 0.0;
  }
  double u0[ROWS], a0[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    const int j = j0 + y0 + r;
    const long long q = (long long)j * pitch + i;
    u0[r] = a0[r] = 0.0;
    if (i < nx && j < ny) {
      if (STAGE == ST_FIRST) u0[r] = in_at(j, i);
      if (STAGE == ST_MID) u0[r] = ld_l2(prm.un + q);
      if (STAGE == ST_MID || STAGE == ST_LAST) a0[r] = ld_l2(prm.acc + q);
    }
  }
  // x-closure columns of this cell: [0, CS) and [nx - CS, nx), one sum per thread
  const int wcols = i0 == 0 ? CS : 0;
  const int e0 = i0 > nx - CS ? i0 : nx - CS, e1 = i0 + TX < nx ? i0 + TX : nx;
  const int ncol = wcols + (e1 > e0 ? e1 - e0 : 0);
  for (int t = tid; t < TY * ncol; t += kCellThreads) {
    const int col = t % ncol, yr = t / ncol, jr = j0 + yr;
    const int I = col < wcols ? col : e0 + col - wcols;
    if (jr < ny) s_cls[yr][col] = closure_by<double, ORD>([&](int k) { return in_at(jr, k); }, nx, I, prm.dx.cls);
  }
  bool out = false;
#pragma unroll
  for (int c = 0; c < PER; c++) {
    const int e = tid + c * kCellThreads;
    const long long w = fx_pack(val[c], out);
    if (e < N) box[e] = w;
  }
  const bool taps = __syncthreads_or(out);  // a value without a word: FP64 taps
  if (i >= nx) return;
  const bool xint = i >= CS && i < nx - CS;
  const int ccol = i < CS ? i : wcols + (i - e0);
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    const int y = y0 + r, j = j0 + y;
    if (j >= ny) break;
    const long long q = (long long)j * pitch + i;
    const long long* at = box + (y + R) * PW + lane + R;
    // derivative = factor * value per direction: a stencil sum in units of sigma, or a
    // closure or tap sum already scaled
    double dx, dy, fx = 1.0, fy = 1.0;
    if (xint && !taps) {
      dx = fx_d1<ORD>(at, 1);
      fx = prm.fx_sig[0];
    } else {
      dx = xint ? taps_by<double, ORD>([&](int p) { return in_at(j, p); }, i, prm.dx.taps) : s_cls[y][ccol];
    }
    if (j >= CS && j < ny - CS && !taps) {
      dy = fx_d1<ORD>(at, PW);
      fy = prm.fx_sig[1];
    } else if (j >= CS && j < ny - CS) {
      dy = taps_by<double, ORD>([&](int p) { return in_at(p, i); }, j, prm.dy.taps);
    } else {
      dy = closure_by<double, ORD>([&](int k) { return in_at(k, i); }, ny, j, prm.dy.cls);
    }
    double k;
    if constexpr (FIELDS) k = -fma(__ldg(prm.va + q), fx * dx, __ldg(prm.vb + q) * (fy * dy));
    else k = fma(fx, dx, fy * dy);
    if (i == 0 || j == 0 || i == nx - 1 || j == ny - 1) k = adv2d_sat<double>(prm, i, j, k, in_at(j, i));
    if constexpr (STAGE == ST_RHS) {
      prm.kout[q] = k;
    } else if constexpr (STAGE == ST_LAST) {
      prm.un[q] = fma(prm.c_acc, k, a0[r]);
    } else {
      prm.acc[q] = fma(prm.c_acc, k, STAGE == ST_FIRST ? u0[r] : a0[r]);
      prm.wout[q] = fma(prm.c_w, k, u0[r]);
    }
  }
}

}  // namespace sbp

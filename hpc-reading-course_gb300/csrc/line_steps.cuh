// line_steps.cuh -- many RK4 steps of a 1D problem (advection, reflection) in one launch.
//
// A stage of these grids is a few hundred to a few thousand points: launched one by one the
// stages cost 2.7 us each, nearly all of it launch and memory latency. Here one thread-block
// cluster holds the whole state in shared memory for all steps. Each CTA owns a run of points
// and keeps 4R halo points per side (R: the stencil's reach), so that it computes a whole step
// -- stage 1 on 3R halo points, stage 2 on 2R, ... -- with block barriers only; the new edge
// values then go to the neighbours' halos through distributed shared memory, and one cluster
// barrier ends the step. The state is double-buffered: a CTA may write its neighbour's next
// halo while the neighbour still reads the current one.
// Measured, us per step, stages launched one by one -> this: FP64 advection order 4, 201
// points 9.4 -> 3.0, 1601 9.0 -> 3.1, 6401 10.2 -> 6.5; reflection 201 13.6 -> 4.3; FP32
// advection 201 7.8 -> 2.1. What bounds it: a warp's FP64 instruction takes 64 clocks, and the
// cluster barrier ends each step. FP64 interior stencils are integer sums (with FP64 taps: 201
// points 3.3, 6401 8.7).
// FP32: the operations of line_point (line_kernels.cuh), in its order, the same bits.
#pragma once

#include <cooperative_groups.h>

#include "line_kernels.cuh"
#include "wave_cell.cuh"

namespace sbp {

// Points a CTA owns at least (several CTAs): its extended regions then hold no closure rows
// of a domain end that it does not own, and its halo lies within its neighbours' points.
constexpr int kLineMinChunk = 64;
constexpr int kLineMaxCtas = 8;

template <typename T, int ORD, int KIND> struct LineSteps {
  static constexpr int R = OpShape<ORD>::W / 2, H = 4 * R, NC = KIND == LK_REFL1D ? 2 : 1;
  static_assert(3 * R + OpShape<ORD>::CS <= kLineMinChunk && H <= kLineMinChunk, "halo within the neighbour");
  // planes of `len` values per component: u (two buffers), w (two), acc and the Kahan term
  static constexpr int planes = 6;
  static size_t smem(int chunk) { return sizeof(T) * NC * planes * (size_t)(chunk + 2 * H); }
};

// den times the interior stencil sum around c by integer arithmetic with the exponent of its
// own largest value (wave2d_fixed.cuh, fx_from<true>): some 100 integer instructions take half
// the time of four FP64 FMAs at 64 clocks each. False where the values leave the fixed-point
// range.
template <int ORD>
__device__ __forceinline__ bool fx_local(const double* c, double& out) {
  constexpr int R = OpShape<ORD>::W / 2;
  unsigned m = 0;
#pragma unroll
  for (int k = 1; k <= R; k++) {
    m = max(m, (unsigned)__double2hiint(c[k]) & 0x7FFFFFFFu);
    m = max(m, (unsigned)__double2hiint(c[-k]) & 0x7FFFFFFFu);
  }
  const int emax = (int)(m >> 20);
  long long d[R];  // v_k - v_-k
#pragma unroll
  for (int k = 1; k <= R; k++) {
    const double a = c[k], b = c[-k];
    d[k - 1] = fx_from<true>((unsigned)__double2loint(a), (unsigned)__double2hiint(a), emax) -
               fx_from<true>((unsigned)__double2loint(b), (unsigned)__double2hiint(b), emax);
  }
  long long s = d[0];
  if constexpr (ORD == 4) s = 8 * d[0] - d[1];
  if constexpr (ORD == 6) s = 45 * d[0] - 9 * d[1] + d[2];
  out = fx_to<true>(s, fx_base<true>(emax));
  if (m - (64u << 20) < (2031u - 64u) << 20) return true;
  if (m) return false;
  unsigned lo = 0;  // zeros, whose sum is 0, or subnormals
#pragma unroll
  for (int k = 1; k <= R; k++) lo |= (unsigned)__double2loint(c[k]) | (unsigned)__double2loint(c[-k]);
  return lo == 0;
}

template <typename T, int ORD, int KIND>
__global__ void __launch_bounds__(512) line_steps_kernel(const __grid_constant__ LineParams<T> prm, const int chunk,
                                                          const int steps, const T ca1, const T ca2, const T cw1,
                                                          const T cw3) {
  namespace cg = cooperative_groups;
  using L = LineSteps<T, ORD, KIND>;
  constexpr int R = L::R, H = L::H, NC = L::NC, CS = OpShape<ORD>::CS, CW = OpShape<ORD>::CW;
  extern __shared__ __align__(16) unsigned char line_smem[];
  const cg::cluster_group cluster = cg::this_cluster();
  const int nx = prm.nx, len = chunk + 2 * H, cta = (int)cluster.block_rank(), ctas = (int)cluster.num_blocks();
  const int a = cta * chunk, b = a + chunk < nx ? a + chunk : nx;  // this CTA's points
  const int base = a - H;                                          // grid index of local index 0
  T* const sm = reinterpret_cast<T*>(line_smem);
  const auto plane_of = [&](int p, int c) { return sm + (p * NC + c) * len; };  // u: 0, 1; w: 2, 3; acc 4; comp 5
  const int tid = threadIdx.x, nt = blockDim.x;
  const T sig = (T)prm.fx_sig[0], sa1 = ca1 * sig, sa2 = ca2 * sig, sw1 = cw1 * sig, sw3 = cw3 * sig;
  // the closure block: from the parameters, each row that a warp's lanes read is a
  // constant-bank access of its own (order 6: 4.5 us a step against 4.1)
  __shared__ T s_cls[6][9];
  for (int e = tid; e < CS * CW; e += nt) s_cls[e / CW][e % CW] = prm.dx.cls[e / CW][e % CW];
  for (int c = 0; c < NC; c++)
    for (int l = tid; l < len; l += nt) {
      const int i = base + l;
      const bool in = i >= 0 && i < nx;
      plane_of(0, c)[l] = in ? prm.un[c * prm.plane + i] : T(0);
      plane_of(5, c)[l] = in && prm.compensated && i >= a && i < b ? prm.comp[c * prm.plane + i] : T(0);
    }
  // Where thread slots are. FP64: the closure points of an end this CTA owns have a warp to themselves
  // (their rows of FP64 taps would hold up a warp of interior points), the other points follow.
  // FP32: point after point.
  const bool left = cta == 0, right = cta == ctas - 1;
  const int m0 = left ? CS : base, m1 = right ? nx - CS : base + len;  // the middle points
  const int s0 = left ? 32 : 0, s1 = s0 + ((m1 - m0 + 31) & ~31);
  const int slots = sizeof(T) == 8 ? s1 + (right ? 32 : 0) : len;
  const auto point_of = [&](int s) {  // the grid index of a slot, or -1
    if constexpr (sizeof(T) == 4) return base + s;
    if (s < s0) return s < CS ? s : -1;
    if (s < s1) return m0 + s - s0 < m1 ? m0 + s - s0 : -1;
    return s - s1 < CS ? nx - CS + s - s1 : -1;
  };
  cluster.sync();  // every CTA has read its halo from global memory and may be written to

  // stage rk of this CTA's points and (4 - rk) R halo points per side, from plane `in` to `out`
  const auto stage = [&](auto rk_, int u, int in, int out) {
    constexpr int rk = decltype(rk_)::value;
    const int lo = a - (4 - rk) * R > 0 ? a - (4 - rk) * R : 0, hi = b + (4 - rk) * R < nx ? b + (4 - rk) * R : nx;
    for (int s = tid; s < slots; s += nt) {  // a point keeps its thread through the stages
      const int i = point_of(s), l = i - base;
      if (i < lo || i >= hi) continue;
      T ca = (rk == 1 || rk == 4) ? ca1 : ca2, cw = rk == 3 ? cw3 : cw1;
      const auto d1 = [&](int c) {
        const T* line = plane_of(in, c) - base;
        const auto ld = [&](int q) { return line[q]; };
        return (i >= CS && i < nx - CS) ? taps_by<T, ORD>(ld, i, prm.dx.taps) : closure_by<T, ORD>(ld, nx, i, s_cls);
      };
      T k[NC];
      bool scaled = false;  // FP64 interior: k in units of fx_sig, folded into ca and cw
      if constexpr (sizeof(T) == 8) {
        if (i >= CS && i < nx - CS) {
          scaled = fx_local<ORD>(plane_of(in, 0) + l, k[NC - 1]);
          if constexpr (NC == 2) scaled = fx_local<ORD>(plane_of(in, 1) + l, k[0]) && scaled;
        }
      }
      if (scaled) {
        ca = (rk == 1 || rk == 4) ? sa1 : sa2, cw = rk == 3 ? sw3 : sw1;
        if constexpr (KIND == LK_ADV1D)
          if (prm.va) k[0] = -prm.va[i] * k[0];
      } else if constexpr (KIND == LK_ADV1D) {
        k[0] = d1(0);
        if (prm.va) k[0] = -prm.va[i] * k[0];
        k[0] = adv1d_sat<T>(prm, i, k[0], plane_of(in, 0)[l]);
      } else {
        k[NC - 1] = d1(0);
        k[0] = d1(NC - 1);
        if (prm.bc && (i == 0 || i == nx - 1)) k[0] = T(0);  // proj_dirichlet_bc_{l,r}
      }
#pragma unroll
      for (int c = 0; c < NC; c++) {
        T& acc = plane_of(4, c)[l];
        const T u0 = plane_of(u, c)[l];
        const bool own = i >= a && i < b;  // halo points need the stage input only
        if constexpr (rk == 1) {
          if (own) acc = prm.compensated ? ca * k[c] : fma(ca, k[c], u0);
          plane_of(out, c)[l] = fma(cw, k[c], u0);
        } else if constexpr (rk < 4) {
          if (own) acc = fma(ca, k[c], acc);
          plane_of(out, c)[l] = fma(cw, k[c], u0);
        } else {
          T d = fma(ca, k[c], acc);
          if (prm.compensated) {  // Kahan summation of the step increment into the FP32 state
            T& e = plane_of(5, c)[l];
            const T yv = d - e;
            const T tv = u0 + yv;
            e = (tv - u0) - yv;
            d = tv;
          }
          plane_of(out, c)[l] = d;
          // the neighbours' halos: point i is index i - (their base) there
          if (i < a + H && cta > 0) cluster.map_shared_rank(plane_of(out, c), cta - 1)[i - (base - chunk)] = d;
          if (i >= b - H && cta + 1 < ctas) cluster.map_shared_rank(plane_of(out, c), cta + 1)[i - (base + chunk)] = d;
        }
      }
    }
  };
  for (int s = 0; s < steps; s++) {
    const int u = s & 1;
    stage(std::integral_constant<int, 1>{}, u, u, 2);
    __syncthreads();
    stage(std::integral_constant<int, 2>{}, u, 2, 3);
    __syncthreads();
    stage(std::integral_constant<int, 3>{}, u, 3, 2);
    __syncthreads();
    stage(std::integral_constant<int, 4>{}, u, 2, u ^ 1);
    if (ctas > 1) cluster.sync();
    else __syncthreads();
  }
  for (int c = 0; c < NC; c++)
    for (int l = H + tid; l < H + b - a; l += nt) {
      prm.un[c * prm.plane + base + l] = plane_of(steps & 1, c)[l];
      if (prm.compensated) prm.comp[c * prm.plane + base + l] = plane_of(5, c)[l];
    }
}

}  // namespace sbp

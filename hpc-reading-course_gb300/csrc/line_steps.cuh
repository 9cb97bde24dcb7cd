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
// points 9.4 -> 3.3, 1601 9.0 -> 3.9, 6401 10.2 -> 8.7; reflection 201 13.6 -> 4.9; FP32
// advection 201 7.8 -> 2.1. What bounds it: a warp's FP64 instruction takes 64 clocks, so a
// stage's chain of about eight is 0.25 us, and the cluster barrier ends each step.
// The operations of a point are those of line_point (line_kernels.cuh), in its order, so FP32
// states get the same bits from both.
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
  cluster.sync();  // every CTA has read its halo from global memory and may be written to

  // stage rk of this CTA's points and (4 - rk) R halo points per side, from plane `in` to `out`
  const auto stage = [&](auto rk_, int u, int in, int out) {
    constexpr int rk = decltype(rk_)::value;
    const int lo = a - (4 - rk) * R > 0 ? a - (4 - rk) * R : 0, hi = b + (4 - rk) * R < nx ? b + (4 - rk) * R : nx;
    const T ca = (rk == 1 || rk == 4) ? ca1 : ca2, cw = rk == 3 ? cw3 : cw1;
    for (int l = tid; l < len; l += nt) {  // a point keeps its thread through the stages
      const int i = base + l;
      if (i < lo || i >= hi) continue;
      const auto d1 = [&](int c) {
        const T* line = plane_of(in, c) - base;
        const auto ld = [&](int q) { return line[q]; };
        return (i >= CS && i < nx - CS) ? taps_by<T, ORD>(ld, i, prm.dx.taps) : closure_by<T, ORD>(ld, nx, i, s_cls);
      };
      T k[NC];
      if constexpr (KIND == LK_ADV1D) {
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

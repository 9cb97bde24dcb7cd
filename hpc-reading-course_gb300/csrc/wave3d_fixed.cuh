// wave3d_fixed.cuh -- the FP64 stages of the 3D wave with integer stencils.
//
// The plane-ring kernel of wave3d.cu issued, in FP64, 24 tap FMAs of its 33 FP64 instructions
// per point-stage at order 4 and some 300 instructions per thread and plane for its 16-byte
// copies; at 12 warps per SM it took 700 clocks per warp and plane. Here a CTA of 256 threads
// owns a 32 x 8 column of points and marches along z: one thread issues the next planes' TMA
// boxes, all threads convert an arriving plane's p, w and the current plane's u, v boxes to
// words in place (wave2d_fixed.cuh), and the stencils are integer sums; the FP64 pipe keeps the
// update and, for p, the two spacing ratios: nine instructions.
// Measured, us per stage, plane ring -> this: order 4 49^3 50 -> 38, 97^3 138 -> 112,
// 201 x 193 x 161 552 -> 388, 256^3 1273 -> 831; order 2 256^3 838 -> 626; order 6 1764 -> 955.
// What bounds it now: the integer instructions and the FP64 pipe. Closure sums of the x columns
// shared out one per thread and x-face SAT on one warp, as in the 2D cells, measured slower here
// (two more barriers per plane).
//
// Rings, by plane: A holds p (x halo HX, y halo R) and w of planes k .. k + R and those in
// flight (a thread keeps its column's p and w along z in registers), B holds u (x halo), v (y
// halo) and the point boxes the stage update reads. Each group of boxes (plane m in A, plane m - R in B) completes one mbarrier; waits are bounded.
// Per plane one block barrier, "converted": past it every thread has left the previous plane, so
// that the slots that plane read may be refilled.
// Closure rows and planes with a value that has no word take FP64 taps from global memory; SAT
// in true units.
#pragma once

#include "line_kernels.cuh"
#include "wave2d.cuh"
#include "wave3d.cuh"

namespace sbp {

// Boundary terms on the faces the point lies on (FP64 arithmetic, as the 2D kernels):
// free surface (wave_eq_hom_rhs.h:389-441 per face): lower face F_ud -= bw_d p, upper F_ud += bw_d p;
// characteristic (Z = c = 1): lower face g = bw_d (p + u_d): F_ud -= g/2, F_p -= g/2;
// upper face g = bw_d (p - u_d): F_ud += g/2, F_p -= g/2.
template <typename T> struct Rhs4 { T u, v, w, p; };

template <typename T>
__device__ __noinline__ Rhs4<T> wave3d_sat(const Wave3Params<T>& prm, int i, int j, int k, T uc, T vc, T wc, T pc,
                                           Rhs4<T> kc) {
  // values and results by value: a noinline function taking arrays by reference
  // would keep the caller's arrays in local memory on every point. Only the
  // components a face changes go through FP64 (the others would round-trip
  // exactly), in the order of the faces, so that a point on one face costs about
  // ten FP64-pipe instructions.
  const T cen[3] = {uc, vc, wc};
  T f[3] = {kc.u, kc.v, kc.w};
  const int idx[3] = {i, j, k};
  const int n[3] = {prm.nx, prm.ny, prm.nz};
  const double p = (double)pc;
  double fp = (double)kc.p;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const bool lo = idx[d] == 0, hi = idx[d] == n[d] - 1;
    if (!lo && !hi) continue;
    const double ud = (double)cen[d];
    double fd = (double)f[d];
    if (prm.bc == BC_CHARACTERISTIC) {
      if (lo) {
        const double g = prm.bw[d] * (p + ud);
        fd -= 0.5 * g;
        fp -= 0.5 * g;
      }
      if (hi) {
        const double g = prm.bw[d] * (p - ud);
        fd += 0.5 * g;
        fp -= 0.5 * g;
      }
    } else {
      if (lo) fd -= prm.bw[d] * p;
      if (hi) fd += prm.bw[d] * p;
    }
    f[d] = (T)fd;
  }
  return Rhs4<T>{f[0], f[1], f[2], (T)fp};
}

struct Wave3Maps {
  CUtensorMap p, w, u, v;  // the stage input seen with the four boxes
  CUtensorMap n, a;        // u^n and acc as point boxes of all four components
};

constexpr int kF3X = 32, kF3Y = 8, kF3Threads = kF3X * kF3Y;

template <int ORD, int STAGE> struct Fixed3 {
  static constexpr int R = OpShape<ORD>::W / 2, W = OpShape<ORD>::W, TX = kF3X, TY = kF3Y;
  static constexpr int D = 1;                 // planes in flight beyond the one being converted
  static constexpr int HX = (R + 1) / 2 * 2;  // x halo: whole 16-byte units (TMA's rule on x)
  static constexpr int PX = TX + 2 * HX, PY = TY + 2 * R;
  static constexpr bool LOAD_N = STAGE == ST_MID || STAGE == ST_FIRST;  // first stage: u^n as doubles
  static constexpr bool LOAD_A = STAGE == ST_MID || STAGE == ST_LAST;
  static constexpr int al(int n) { return (n + 15) / 16 * 16; }  // TMA destinations: 128 bytes
  static constexpr int NP = PY * PX, NW = TY * TX, NU = TY * PX, NV = PY * TX, NPT = 4 * TY * TX;
  static constexpr int A_W = al(NP), A_SZ = A_W + al(NW);
  static constexpr int B_V = al(NU), B_N = B_V + al(NV), B_A = B_N + (LOAD_N ? NPT : 0);
  static constexpr int B_SZ = B_A + (LOAD_A ? NPT : 0);
  // Slots. When group g + D + 1 is issued, in iteration g after its first barrier, A's groups
  // g - R .. g + D hold planes still to be read (p of plane g - R; the z window is in
  // registers) and B's groups g .. g + D; the slot refilled is the one before them.
  static constexpr int SA = R + D + 2, SB = D + 2;
  static constexpr int SMEM = (SA * A_SZ + SB * B_SZ) * 8;
  static constexpr int PER_A = (NP + NW + kF3Threads - 1) / kF3Threads;
  static constexpr int PER_B = (NU + NV + kF3Threads - 1) / kF3Threads;
  static_assert(SMEM + 4096 <= 227 * 1024, "ring exceeds shared memory");
};

template <int ORD, int STAGE>
__global__ void __launch_bounds__(kF3Threads, 2)
    wave3d_fixed_kernel(const __grid_constant__ Wave3Maps maps, const __grid_constant__ Wave3Params<double> prm,
                        const int zchunk) {
  using G = Fixed3<ORD, STAGE>;
  constexpr int R = G::R, W = G::W, CS = OpShape<ORD>::CS, TX = G::TX, TY = G::TY, PX = G::PX, D = G::D;
  constexpr int SA = G::SA, SB = G::SB;
  extern __shared__ __align__(128) unsigned char f3_smem[];
  double* const sA = reinterpret_cast<double*>(f3_smem);
  double* const sB = sA + SA * G::A_SZ;
  __shared__ uint64_t full[SA];
  __shared__ int s_out[3][2];  // by group modulo 3: its p or w, its u or v boxes hold a value without a word
  if (prm.skip && *prm.skip) return;
  const int nx = prm.nx, ny = prm.ny, nz = prm.nz;
  const int pitch = (int)prm.pitch, slab = (int)prm.slab, plane = (int)prm.plane;  // 4 * plane < 2^31 (host)
  const double* __restrict__ U = prm.in;
  const double* __restrict__ V = U + plane;
  const double* __restrict__ Wc = V + plane;
  const double* __restrict__ P = Wc + plane;
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY, i = i0 + tx, j = j0 + ty;
  const bool live = i < nx && j < ny;
  const int k0 = blockIdx.z * zchunk, k1 = k0 + zchunk < nz ? k0 + zchunk : nz;
  if (tid == 0) {
    for (int s = 0; s < SA; s++) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  if (tid < 6) s_out[tid / 2][tid % 2] = 0;
  __syncthreads();

  // Group g (0, 1, ...): plane k0 - R + g of p and w into A's slot g % SA; from g = 2R on, while
  // it is this CTA's, plane k0 + g - 2R of u, v and the point boxes into B's slot. Planes outside
  // the grid are loaded as the maps' zero fill. Thread 0 only.
  const int groups = k1 - k0 + 2 * R;
  const auto issue = [&](int g) {
    if (g >= groups) return;
    if (g == 0 && prm.test_drop_tile == 1 + (int)(blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)))
      return;
    const int sa = g % SA, m = k0 - R + g, kb = m - R;
    double* a = sA + sa * G::A_SZ;
    const bool own = kb >= k0;
    mbar_arrive_expect_tx(&full[sa], 8u * (G::NP + G::NW + (own ? G::NU + G::NV + (G::LOAD_N ? G::NPT : 0) +
                                                                        (G::LOAD_A ? G::NPT : 0)
                                                                  : 0)));
    tma_load_4d(a, &maps.p, i0 - G::HX, j0 - R, m, 3, &full[sa]);
    tma_load_4d(a + G::A_W, &maps.w, i0, j0, m, 2, &full[sa]);
    if (own) {
      double* b = sB + (kb - k0) % SB * G::B_SZ;
      tma_load_4d(b, &maps.u, i0 - G::HX, j0, kb, 0, &full[sa]);
      tma_load_4d(b + G::B_V, &maps.v, i0, j0 - R, kb, 1, &full[sa]);
      if (G::LOAD_N) tma_load_4d(b + G::B_N, &maps.n, i0, j0, kb, 0, &full[sa]);
      if (G::LOAD_A) tma_load_4d(b + G::B_A, &maps.a, i0, j0, kb, 0, &full[sa]);
    }
  };
  int issued = 0;  // thread 0: groups issued
  if (tid == 0)
    for (; issued < D + 1; issued++) issue(issued);

  // register windows along z of this thread's column, planes k - R .. k + R
  long long zp[W], zw[W];
#pragma unroll
  for (int s = 0; s < W; s++) zp[s] = zw[s] = kFxNone;
  unsigned usable = ~0u;  // bit s: every value of the plane s before the latest has a word
  const int pc = (ty + R) * PX + tx + G::HX, wc = ty * TX + tx, uc = ty * PX + tx + G::HX, vc = (ty + R) * TX + tx;

#pragma unroll 1
  for (int g = 0; g < groups; g++) {
    const int sa = g % SA, kb = k0 - 2 * R + g;  // this group completes what plane kb needs
    const bool own = kb >= k0;
    double* a = sA + sa * G::A_SZ;
    double* b = sB + (own ? (kb - k0) % SB : 0) * G::B_SZ;
    long long* ia = reinterpret_cast<long long*>(a);
    long long* ib = reinterpret_cast<long long*>(b);
    const bool late = !mbar_wait_bounded(&full[sa], (g / SA) & 1, prm.wait_ns);  // the copy will not complete
    bool outa = false, outb = false;
#pragma unroll
    for (int c = 0; c < G::PER_A; c++) {
      const int e = tid + c * kF3Threads;
      if (e < G::NP) ia[e] = fx_pack(a[e], outa);
      else if (e < G::NP + G::NW) ia[G::A_W + e - G::NP] = fx_pack(a[G::A_W + e - G::NP], outa);
    }
    if (own) {
#pragma unroll
      for (int c = 0; c < G::PER_B; c++) {
        const int e = tid + c * kF3Threads;
        if (e < G::NU) ib[e] = fx_pack(b[e], outb);
        else if (e < G::NU + G::NV) ib[G::B_V + e - G::NU] = fx_pack(b[G::B_V + e - G::NU], outb);
      }
    }
    if (outa) s_out[g % 3][0] = 1;
    if (outb) s_out[g % 3][1] = 1;
    // order the generic writes before the TMA that refills these slots
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (__syncthreads_or(late)) {  // converted; every thread has left the previous plane
      if (tid == 0) {
        atomicOr(prm.err, ERR_TMA_TIMEOUT);
        // let the copies in flight land (bounded) before the CTA's shared memory goes
        for (int q = g; q < issued; q++) mbar_wait_bounded(&full[q % SA], (q / SA) & 1, prm.wait_ns);
      }
      return;
    }
    if (tid == 0 && issued < groups) issue(issued++);  // into slots the previous planes have left
    usable = usable << 1 | (s_out[g % 3][0] == 0);
    const bool uv_words = s_out[g % 3][1] == 0;
    if (tid < 2) s_out[(g + 2) % 3][tid] = 0;  // group g - 1's, read by all before the barrier
#pragma unroll
    for (int s = 0; s + 1 < W; s++) {
      zp[s] = zp[s + 1];
      zw[s] = zw[s + 1];
    }
    zp[W - 1] = ia[pc];
    zw[W - 1] = ia[G::A_W + wc];
    if (!own || !live) continue;

    const int k = kb, xo = k * slab + j * pitch, q = xo + i;
    const bool fx = uv_words && (usable & ((1u << W) - 1)) == (1u << W) - 1;
    const long long* ap = reinterpret_cast<const long long*>(sA + (g - R) % SA * G::A_SZ);  // plane k's p
    const bool xint = i >= CS && i < nx - CS, yint = j >= CS && j < ny - CS, zint = k >= CS && k < nz - CS;
    const auto far = [&](const double* line, int st, int n, int at, const DirTaps<double>& d, double isig) {
      return d1_line<double, ORD>(line, st, n, at, d) * isig;
    };
    double kf[4];  // the RHS in units of sigma
    kf[0] = xint && fx ? fx_d1<ORD>(ap + pc, 1)
                       : far(P + xo, 1, nx, i, prm.dx, prm.fx_isig[0]);
    kf[1] = yint && fx ? fx_d1<ORD>(ap + pc, PX)
                       : far(P + (k * slab + i), pitch, ny, j, prm.dy, prm.fx_isig[1]);
    kf[2] = zint && fx ? fx_d1<ORD>(zp + R, 1)
                       : far(P + (j * pitch + i), slab, nz, k, prm.dz, prm.fx_isig[2]);
    const double ux = xint && fx ? fx_d1<ORD>(ib + uc, 1)
                                 : far(U + xo, 1, nx, i, prm.dx, prm.fx_isig[0]);
    const double vy = yint && fx ? fx_d1<ORD>(ib + G::B_V + vc, TX)
                                 : far(V + (k * slab + i), pitch, ny, j, prm.dy, prm.fx_isig[1]);
    const double wz = zint && fx ? fx_d1<ORD>(zw + R, 1)
                                 : far(Wc + (j * pitch + i), slab, nz, k, prm.dz, prm.fx_isig[2]);
    kf[3] = fma(prm.fx_rho[1], wz, fma(prm.fx_rho[0], vy, ux));

    double ca[4], cw4[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      ca[c] = prm.fx_ca[c];
      cw4[c] = prm.fx_cw[c];
    }
    const bool face = prm.bc != BC_NONE && (i == 0 || j == 0 || k == 0 || i == nx - 1 || j == ny - 1 || k == nz - 1);
    if (STAGE == ST_RHS || face) {
#pragma unroll
      for (int c = 0; c < 4; c++) {  // true units
        kf[c] *= prm.fx_sig[c % 3];
        ca[c] = prm.c_acc;
        cw4[c] = prm.c_w;
      }
      if (face) {
        const Rhs4<double> r = wave3d_sat<double>(prm, i, j, k, U[q], V[q], Wc[q], P[q],
                                                  Rhs4<double>{kf[0], kf[1], kf[2], kf[3]});
        kf[0] = r.u;
        kf[1] = r.v;
        kf[2] = r.w;
        kf[3] = r.p;
      }
    }
    const double* un = b + G::B_N + wc;
    const double* ac = b + G::B_A + wc;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int o = c * plane + q;
      if constexpr (STAGE == ST_RHS) {
        prm.kout[o] = kf[c];
      } else if constexpr (STAGE == ST_FIRST) {
        st_stream(prm.acc + o, fma(ca[c], kf[c], un[c * TY * TX]));
        st_stream(prm.wout + o, fma(cw4[c], kf[c], un[c * TY * TX]));
      } else if constexpr (STAGE == ST_MID) {
        st_stream(prm.acc + o, fma(ca[c], kf[c], ac[c * TY * TX]));
        st_stream(prm.wout + o, fma(cw4[c], kf[c], un[c * TY * TX]));
      } else {  // ST_LAST
        prm.un[o] = fma(ca[c], kf[c], ac[c * TY * TX]);
      }
    }
  }
}

}  // namespace sbp

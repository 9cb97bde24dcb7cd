// wave2d_fixed.cuh -- the FP64 wave stages (constant and variable coefficients, the
// manufactured solution; RHS, RK4 and Fehlberg stages) with their interior stencils in
// exact integer arithmetic.
//
// GB300 issues FP64 FMAs at about 1/64 of its FP32 rate, and the FP64 tap
// chains of wave_tile_compute (4 derivatives x 4 taps at order 4, plus the
// stage update) keep that pipe busy long before HBM is. The interior stencils
// of the central SBP operators have rational weights with a small common
// denominator (code/include/sbpops/D1_central.h:245,254,266):
//     order 2: (1/2)  (v1 - v-1)
//     order 4: (1/12) (8 (v1 - v-1) - (v2 - v-2))
//     order 6: (1/60) (45 (v1 - v-1) - 9 (v2 - v-2) + (v3 - v-3))
// so den * sum is an integer combination of the point values, exact in int64.
//
// Constant coefficients, RHS and RK4 stages: each tile's stencil boxes are converted once, in
// place, to 64-bit integers in units of 2^(Emax - 1075), where Emax is the largest biased
// exponent among the box values of the group (p; u and v together): a double +-M 2^(E-1075)
// with its 53-bit mantissa M becomes +-trunc(M / 2^(Emax - E)), |V| < 2^53. The sums stay
// below 2^62 (|S| < 110 * 2^54 < 2^61 at order 6, and the u and v terms together), and one
// conversion back to a double carries the only other rounding: an error of a few 2^-52 of the
// box's largest magnitude, whatever the point's own.
//
// Every other stage (fx_fine) keeps each value whole: the boxes are converted to words that
// hold the signed mantissa above its exponent (fx_pack), and a stencil brings the words it
// reads to its own largest exponent. Its values are then in units of 2^-54 of the largest one
// it reads and its result is rounded to nearest: at every point the accuracy of FP64 taps,
// also for small values beside large ones. One value's conversion takes about 12 integer
// instructions and its use in a stencil seven, against about 20 and one in box units (variable
// coefficients at 2049^2, order 4: 139 us a stage, 123 in box units, 225 with FP64 taps).
// The integer work runs on the INT pipe; the
// FP64 pipe is left with the RK4 stage update, 1-2 FMAs per component, into
// which the scale sigma = -hi/den is folded (fx_ca, fx_cw).
//
// Closure rows (boundary strips) keep the FP64 taps read from global memory
// and are brought to the same units by 1/sigma; SAT terms are applied in FP64
// in true units as in wave_tile_compute. Boxes with values outside the fixed-point range:
// fx_tile_emax.
#pragma once

#include "sbp_device.cuh"

namespace sbp {

template <int ORD> struct FixDen;
template <> struct FixDen<2> { static constexpr int value = 2; };
template <> struct FixDen<4> { static constexpr int value = 12; };
template <> struct FixDen<6> { static constexpr int value = 60; };

// Which stages give each stencil its own exponent and round its sum to nearest. The RK4 and
// RHS stages of constant coefficients take their box's.
template <int KIND, int STAGE> constexpr bool fx_fine() {
  return is_rkf_stage(STAGE) || KIND == WK_VAR || KIND == WK_MMS;
}

// v (given as its two 32-bit words) as a signed integer in units of
// 2^(emax - 1075), FINE: 2^(emax - 1077), truncated towards zero; emax >= the exponent
// of v. Zero and subnormal values give 0, as does any shift of 64 or more.
template <bool FINE>
__device__ __forceinline__ long long fx_from(unsigned lo, unsigned hi, int emax) {
  const unsigned e = (hi >> 20) & 0x7FFu;
  unsigned mh = (hi & 0x000FFFFFu) | 0x00100000u, ml = lo;  // the 53-bit mantissa is mh:ml
  if constexpr (FINE) {
    mh = __funnelshift_l(ml, mh, 2);
    ml <<= 2;
  }
  const unsigned sh = e == 0 ? 64u : (unsigned)emax - e;
  const unsigned rlo = sh < 32 ? __funnelshift_rc(ml, mh, sh) : __funnelshift_rc(mh, 0u, sh - 32u);
  const unsigned rhi = __funnelshift_rc(mh, 0u, sh);
  const long long r = (long long)(((unsigned long long)rhi << 32) | rlo);
  const long long sg = (long long)((int)hi >> 31);  // 0 or -1
  return (r ^ sg) - sg;
}

// The exponent base fx_to takes for integers in fx_from's units.
template <bool FINE> __device__ __forceinline__ int fx_base(int emax) { return emax + (FINE ? 9 : 11); }

// s in fx_from's units as a double; eb = fx_base(emax), |s| < 2^63 (the tile guard keeps
// emax in [64, 2030], so the exponent stays normal). FINE: rounded to nearest (ties away
// from zero; a carry out of the mantissa moves into the exponent field), else truncated
// towards zero.
template <bool FINE>
__device__ __forceinline__ double fx_to(long long s, int eb) {
  constexpr int TOP = FINE ? 62 : 63;  // the bit the leading one is shifted to
  const long long sg = s >> 63;
  const unsigned long long a = (unsigned long long)((s ^ sg) - sg);
  const int lz = __clzll((long long)a);  // >= 1, without FINE >= 2
  unsigned long long n = a << ((lz - (63 - TOP)) & 63);
  if constexpr (FINE) n += 0x200ull;
  const unsigned mh = (unsigned)(n >> (TOP - 20));             // leading one + 20 fraction bits
  const unsigned ml = (unsigned)(n >> (TOP - 52));             // the other 32 fraction bits
  const unsigned hw = (((unsigned)(eb - lz - 1)) << 20) + mh;  // the leading one adds the last 1 to the exponent
  const double r = __hiloint2double((int)(hw | ((unsigned)sg & 0x80000000u)), (int)ml);
  return a == 0 ? 0.0 : r;
}

// den * (interior stencil sum) at the point c of an int64 line with stride st.
template <int ORD>
__device__ __forceinline__ long long fx_stencil(const long long* c, int st) {
  if constexpr (ORD == 2) {
    return c[st] - c[-st];
  } else if constexpr (ORD == 4) {
    return 8 * (c[st] - c[-st]) - (c[2 * st] - c[-2 * st]);
  } else {
    return 45 * (c[st] - c[-st]) - 9 * (c[2 * st] - c[-2 * st]) + (c[3 * st] - c[-3 * st]);
  }
}

// Whole values: a word is the signed mantissa, 53 bits and sign, above a 10-bit field r. The
// value's biased exponent is kFxTop - r; zero is a zero mantissa with r = kFxNone.
constexpr int kFxTop = 1087, kFxNone = 1023;

// The word of a double. Sets `out` if it has none: from 2^65 (3.7e19), Inf, NaN, or nonzero
// and below 2^-958.
__device__ __forceinline__ long long fx_pack(double v, bool& out) {
  const unsigned lo = (unsigned)__double2loint(v), hi = (unsigned)__double2hiint(v);
  const unsigned r = (unsigned)kFxTop - ((hi >> 20) & 0x7FFu);
  const bool zero = ((hi << 1) | lo) == 0;
  out |= !zero && r >= (unsigned)kFxNone;
  const unsigned mh = (hi & 0x000FFFFFu) | 0x00100000u;
  const long long m = (long long)(((unsigned long long)__funnelshift_l(lo, mh, 10) << 32) | (lo << 10));
  const long long sg = (long long)((int)hi >> 31);  // 0 or -1
  return zero ? (long long)kFxNone : (((m ^ sg) - sg) | (long long)(r & 1023u));
}

// The double of a word, exactly.
__device__ __forceinline__ double fx_unpack(long long w) {
  const unsigned r = (unsigned)w & 1023u;
  const long long m = w & ~1023ll, sg = w >> 63;
  const unsigned long long a = (unsigned long long)((m ^ sg) - sg);  // leading one at bit 62
  const unsigned hw = (((unsigned)kFxTop - r - 1) << 20) + (unsigned)(a >> 42);  // it adds the last 1 to the exponent
  const double v = __hiloint2double((int)(hw | ((unsigned)sg & 0x80000000u)), (int)(a >> 10));
  return a == 0 ? 0.0 : v;
}

// The largest exponent (smallest r) among the words that the stencil at c reads, and r.
template <int ORD>
__device__ __forceinline__ int fx_least(const long long* c, int st, int r = kFxNone) {
#pragma unroll
  for (int k = 1; k <= ORD / 2; k++) r = min(r, min((int)c[k * st] & 1023, (int)c[-k * st] & 1023));
  return r;
}

// den * (interior stencil sum) at c in units of 2^(kFxTop - r - 1077): a word is shifted down by
// 8 bits and its exponent's distance to r (shr.s64 takes any count: 64 and more give 0 or -1).
// 110 * 2 * 2^55 < 2^63: the sums at order 6, the u and v terms together, stay in range.
template <int ORD>
__device__ __forceinline__ long long fx_sum(const long long* c, int st, int r) {
  const auto at = [&](int k) {
    const long long w = c[k * st];
    long long t;
    asm("shr.s64 %0, %1, %2;" : "=l"(t) : "l"(w & ~1023ll), "r"(((int)w & 1023) - r + 8));
    return t;
  };
  if constexpr (ORD == 2) {
    return at(1) - at(-1);
  } else if constexpr (ORD == 4) {
    return 8 * (at(1) - at(-1)) - (at(2) - at(-2));
  } else {
    return 45 * (at(1) - at(-1)) - 9 * (at(2) - at(-2)) + (at(3) - at(-3));
  }
}

// den * (interior stencil sum) on words, as a double; and the sum of two such.
template <int ORD>
__device__ __forceinline__ double fx_d1(const long long* c, int st) {
  const int r = fx_least<ORD>(c, st);
  return fx_to<true>(fx_sum<ORD>(c, st, r), fx_base<true>(kFxTop - r));
}
template <int ORD>
__device__ __forceinline__ double fx_d1_sum(const long long* a, int sa, const long long* b, int sb) {
  const int r = fx_least<ORD>(b, sb, fx_least<ORD>(a, sa));
  return fx_to<true>(fx_sum<ORD>(a, sa, r) + fx_sum<ORD>(b, sb, r), fx_base<true>(kFxTop - r));
}

// The interior stencil at the point c of an FP64 line in global memory (scaled taps, the
// order of the FP64 tap kernels), for tiles whose values leave the fixed-point range.
template <int ORD>
__device__ __noinline__ double fx_taps_global(const double* c, long long st, const double (&taps)[7]) {
  constexpr int W = OpShape<ORD>::W, R = (W - 1) / 2;
  double s = taps[0] * c[-R * st];
#pragma unroll
  for (int k = 1; k < W; k++)
    if (k != R) s = fma(taps[k], c[(k - R) * st], s);
  return s;
}

// Where a tile's points live: the interior extent of the arrays holding them
// (the grid, or one subdomain of a decomposed grid), the global index of their
// first interior point, that point's array column and row (ghost lines before
// it), the row pitch, the component plane and the arrays' offset in the stage's
// buffers. The single grid: offsets zero, the arrays the whole buffers.
struct FxGeom {
  int nx, ny;
  int xoff, yoff;
  int col0, row0;
  long long pitch, plane, base;
};

// A subdomain of a decomposed grid: its interior points, the global index of its
// first interior point, and its arrays (row pitch, component plane, offset in the
// stage's buffers). Its first interior point sits at array column Tile::HX (the x
// ghost width, rounded up so every TMA x coordinate is 16-byte aligned) and row
// Tile::HY; the R ghost lines next to the interior hold the neighbours' values.
struct FxSub {
  int nx, ny, xoff, yoff;
  long long pitch, plane, base;
  int nbr[4];  // the neighbouring subdomain to the west, east, south, north, or -1
};
struct FxTile {
  int sub, i0, j0, pad;  // subdomain and tile origin in its interior indices
};

// A decomposed grid's tile as the producer hands it to the compute warps through
// shared memory (its geometry and origin), so they need no global loads per tile.
// A neighbour's arrays as a stage writes into its ghost lines: offset, row pitch,
// component plane and its interior extent across the shared edge (nx for a
// west/east neighbour, ny for a south/north one); n < 0 for none.
struct FxNbr {
  long long base, pitch, plane;
  int n, pad;
};
struct FxTileInfo {
  FxGeom g;
  int i0, j0;
  FxNbr nb[4];  // west, east, south, north
};
// Each tile's block in device memory (built by the host) and in a ring stage's slot:
// 192 bytes, a multiple of 16 for the bulk copy.
constexpr int kFxTileInfoBytes = 192;
static_assert(sizeof(FxTileInfo) <= kFxTileInfoBytes, "tile information slot");

// Decomposed grids: the halo exchange fused into the stages that produce the next
// stage input (the reference's VecScatter ghost update,
// code/src/scatter/scatter_ctx.cpp:149-211). Once a tile is done, each of its points
// within R of an edge shared with a neighbour copies its new value (w, or u^n in the
// last stage) into the neighbour's ghost line that mirrors it, so the next stage finds
// every ghost it reads without a separate exchange. Run by the 32 lanes of the
// exchange warp after the compute warps released the tile. The copies are enumerated
// side by side (each side's strip of the tile, component-major), and each lane issues
// U loads before its U stores, so one batch costs about two memory latencies.
template <typename Tile, int STAGE>
__device__ __forceinline__ void fx_exchange_tile(const WaveParams<double>& prm, const FxTileInfo& T, int lane) {
  constexpr int R = Tile::R, TY = Tile::TY, COL0 = Tile::HX, U = 4;
  const FxGeom& g = T.g;
  const int ie = min(T.i0 + kWaveTX, g.nx), je = min(T.j0 + TY, g.ny);
  // each side's strip of the tile, in the subdomain's interior indices: columns
  // [T.i0, iw) west, [ia, ie) east, rows [T.j0, js) south, [ja, je) north; the
  // strips of the sides without a neighbour are empty
  const int iw = min(ie, R), ia = max(T.i0, g.nx - R), js = min(je, R), ja = max(T.j0, g.ny - R);
  const int rows = je - T.j0, cols = ie - T.i0;
  const int c0 = T.nb[0].n >= 0 && iw > T.i0 ? 3 * (iw - T.i0) * rows : 0;
  const int c1 = T.nb[1].n >= 0 && ie > ia ? 3 * (ie - ia) * rows : 0;
  const int c2 = T.nb[2].n >= 0 && js > T.j0 ? 3 * cols * (js - T.j0) : 0;
  const int c3 = T.nb[3].n >= 0 && je > ja ? 3 * cols * (je - ja) : 0;
  const int total = c0 + c1 + c2 + c3;
  if (total == 0) return;
  double* obuf = STAGE == ST_LAST ? prm.un : prm.wout;
  for (int e0 = 0; e0 < total; e0 += 32 * U) {
    double v[U];
    long long dst[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      int e = e0 + lane + 32 * u;
      dst[u] = -1;
      if (e >= total) continue;
      int s, x0, w, y0, h;  // the side and its strip
      if (e < c0) {
        s = 0, x0 = T.i0, w = iw - T.i0, y0 = T.j0, h = rows;
      } else if ((e -= c0) < c1) {
        s = 1, x0 = ia, w = ie - ia, y0 = T.j0, h = rows;
      } else if ((e -= c1) < c2) {
        s = 2, x0 = T.i0, w = cols, y0 = T.j0, h = js - T.j0;
      } else {
        e -= c2;
        s = 3, x0 = T.i0, w = cols, y0 = ja, h = je - ja;
      }
      const int wh = w * h, c = e / wh, r = e - c * wh, j = y0 + r / w, i = x0 + r % w;
      v[u] = obuf[g.base + c * g.plane + (long long)(j + g.row0) * g.pitch + (i + g.col0)];
      const FxNbr& N = T.nb[s];
      const long long row = s == 0 || s == 1 ? j + g.row0 : (s == 2 ? N.n + j + g.row0 : j - g.ny + g.row0);
      const int col = s == 0 ? N.n + i + COL0 : (s == 1 ? i - g.nx + COL0 : i + COL0);
      dst[u] = N.base + c * N.plane + row * N.pitch + col;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (dst[u] >= 0) obuf[dst[u]] = v[u];
  }
}

// The threads of a fixed-point stage kernel: compute, converter and producer warps,
// and on a decomposed grid the exchange warp.
template <typename Tile, bool DEC>
constexpr int fx_kernel_threads() {
  return Tile::THREADS + (DEC ? 32 : 0);
}

// The exchange queue of a decomposed grid: the producer hands each released tile's
// geometry block to the exchange warp through the shared-memory slots after the NST
// ring stages' ones (Tile::OFF_TINFO), with a full/empty barrier pair per slot.
template <typename Tile>
struct FxExchangeQueue {
  static constexpr int SLOTS = 8 - Tile::NST;
  static_assert(SLOTS >= 2, "the tile geometry area leaves the exchange queue too few slots");
  unsigned char* slot0;
  uint64_t* full;
  uint64_t* empty;
  __device__ FxExchangeQueue(unsigned char* smem)
      : slot0(smem + Tile::OFF_TINFO + kFxTileInfoBytes * Tile::NST),
        full(reinterpret_cast<uint64_t*>(smem + Tile::OFF_XBAR)),
        empty(reinterpret_cast<uint64_t*>(smem + Tile::OFF_XBAR + 64)) {}
  __device__ FxTileInfo* slot(int s) const { return reinterpret_cast<FxTileInfo*>(slot0 + kFxTileInfoBytes * s); }
  // Push number q (all 32 lanes of the producer warp): the geometry block `from`, or
  // the end marker (i0 = -1) for nullptr. False if the wait for a free slot ran out.
  __device__ bool push(int q, const unsigned char* from, int lane, const WaveParams<double>& prm) const {
    const int s = q % SLOTS;
    if (q >= SLOTS && !mbar_wait_bounded(&empty[s], ((q / SLOTS) - 1) & 1, prm.wait_ns)) {
      if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
      return false;
    }
    int4* to = reinterpret_cast<int4*>(slot(s));
    if (from) {
      if (lane < kFxTileInfoBytes / 16) to[lane] = reinterpret_cast<const int4*>(from)[lane];
    } else if (lane == 0) {
      slot(s)->i0 = -1;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&full[s]);
    return true;
  }
};

// The exchange warp of a decomposed grid: takes the released tiles' geometry blocks
// from the exchange queue and runs their fused exchange, until the end marker. The
// compute warps' stores reach it through the ring stage's `empty` barrier and the
// queue's `full` barrier. Every wait is bounded.
template <typename Tile, int STAGE>
__device__ __forceinline__ void decomp_exchange(const WaveParams<double>& prm, const FxExchangeQueue<Tile>& xq,
                                                int lane) {
  constexpr int SLOTS = FxExchangeQueue<Tile>::SLOTS;
  for (int q = 0;; q++) {
    const int s = q % SLOTS;
    if (!mbar_wait_bounded(&xq.full[s], (q / SLOTS) & 1, prm.wait_ns)) {
      if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
      return;
    }
    const FxTileInfo& T = *xq.slot(s);
    if (T.i0 < 0) return;
    fx_exchange_tile<Tile, STAGE>(prm, T, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive(&xq.empty[s]);
  }
}

// The producer warp of a decomposed grid: lane 0 takes the tiles (dynamic queue or
// fixed stride) and issues each stage's loads -- TMA boxes with the maps of the tile's
// subdomain, and the tile's geometry block by a bulk copy on the stage's barrier --
// reading the next tile's descriptor one tile ahead. In the stages that produce the
// next stage input, each tile the compute warps release goes to the exchange queue
// (its geometry block copied by the 32 lanes) before its ring stage is refilled; the
// tiles still held at the end follow after their release, then the end marker.
// Every wait is bounded.
template <typename Tile, int STAGE>
__device__ __forceinline__ void decomp_produce(const WaveParams<double>& prm, unsigned char* smem, uint64_t* full,
                                               uint64_t* empty, int* tslot, const FxExchangeQueue<Tile>& xq,
                                               int lane) {
  constexpr int HY = Tile::HY, HX = Tile::HX, NST = Tile::NST;
  constexpr bool EXCH = STAGE == ST_FIRST || STAGE == ST_MID || STAGE == ST_LAST;
  const int ntiles = prm.dntiles;
  const bool dyn = prm.sched != nullptr;
  const unsigned char* tinfo = smem + Tile::OFF_TINFO;
  int k = 0, issued = 0, pushed = 0, sent = 0;  // sent: stage phases begun, the end marker's included
  int tile = 0;
  FxTile next{0, 0, 0, 0};
  if (lane == 0) {
    tile = dyn ? atomicAdd(prm.sched, 1) : (int)blockIdx.x;
    if (tile < ntiles) next = prm.dtiles[tile];
  }
  tile = __shfl_sync(0xffffffffu, tile, 0);
  bool ok = true;
  for (;; k++) {
    const int b = k % NST;
    if (k >= NST) {
      if (!mbar_wait_bounded(&empty[b], ((k / NST) - 1) & 1, prm.wait_ns)) {
        if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
        ok = false;
        break;
      }
      if constexpr (EXCH) {  // the tile this stage held is done: to the exchange warp
        if (!xq.push(pushed, tinfo + kFxTileInfoBytes * b, lane, prm)) {
          ok = false;
          break;
        }
        pushed++;
      }
    }
    if (tile >= ntiles) {
      if (lane == 0) {
        tslot[b] = -1;
        mbar_arrive(&full[b]);
      }
      sent = k + 1;
      break;
    }
    if (lane == 0) {
      tslot[b] = tile;
      const int cur = tile;
      const FxTile t = next;
      tile = dyn ? atomicAdd(prm.sched, 1) : tile + (int)gridDim.x;
      if (tile < ntiles) next = prm.dtiles[tile];  // in flight while this tile's loads are issued
      const CUtensorMap* in = prm.dmaps_in + 3 * t.sub;
      const CUtensorMap* na = prm.dmaps_na + 2 * t.sub;
      unsigned char* st = smem + b * Tile::STAGE_BYTES;
      // array coordinates: the interior starts at column HX, row HY
      const int x = t.i0, y = t.j0;
      mbar_arrive_expect_tx(&full[b], Tile::TX_BYTES + kFxTileInfoBytes);
      bulk_copy_g2s(smem + Tile::OFF_TINFO + kFxTileInfoBytes * b, prm.dtinfo + (long long)kFxTileInfoBytes * cur,
                    kFxTileInfoBytes, &full[b]);
      tma_load_3d(st, &in[0], x, y, 2, &full[b]);                     // p: origin (HX + i0 - HX, HY + j0 - HY)
      tma_load_3d(st + Tile::OFF_U, &in[1], x, y + HY, 0, &full[b]);  // u: x halo only
      tma_load_3d(st + Tile::OFF_V, &in[2], x + HX, y, 1, &full[b]);  // v: y halo only
      if (Tile::LOAD_UN) tma_load_3d(st + Tile::OFF_N, &na[0], x + HX, y + HY, 0, &full[b]);
      if (Tile::LOAD_ACC) tma_load_3d(st + Tile::OFF_A, &na[1], x + HX, y + HY, 0, &full[b]);
    }
    tile = __shfl_sync(0xffffffffu, tile, 0);
    issued = sent = k + 1;
  }
  if constexpr (EXCH) {
    // the tiles still held: to the exchange warp after their release; then the end marker
    for (int kk = pushed; ok && kk < issued; kk++) {
      if (!mbar_wait_bounded(&empty[kk % NST], (kk / NST) & 1, prm.wait_ns)) {
        if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
        ok = false;
        break;
      }
      ok = xq.push(pushed, tinfo + kFxTileInfoBytes * (kk % NST), lane, prm);
      pushed += ok;
    }
    if (ok) xq.push(pushed, nullptr, lane, prm);  // else the exchange warp's own wait runs out
  }
  if (lane == 0) {
    // the CTA must not exit with copies in flight
    for (int kk = (sent >= NST ? sent - NST : 0); kk < sent; kk++)
      if (!mbar_wait_bounded(&full[kk % NST], (kk / NST) & 1, prm.wait_ns)) atomicOr(prm.err, ERR_TMA_TIMEOUT);
    if (dyn) {
      __threadfence();
      if (atomicAdd(prm.sched + 1, 1) == (int)gridDim.x - 1) {
        atomicExch(prm.sched, 0);
        atomicExch(prm.sched + 1, 0);
      }
    }
  }
}

// One tile of a fixed-point FP64 stage for the compute warps: tile origin (i0, j0)
// in the arrays' interior indices. The stage's p, u, v boxes hold int64
// (converted by the converter warps); u^n, acc are FP64 point boxes. Closure rows
// and SAT faces follow the global indices I = xoff + i, J = yoff + j (prm.nx,
// prm.ny: the global grid); interior stencils read across subdomain edges from
// the ghost lines the boxes include. `in`, `wout` and the stage's RK4 coefficients
// (c_acc, c_w in true units, fx_ca / fx_cw scaled per component) come from the
// caller: the single grid passes prm's, a batch its instance's for the stage.
// KIND: WK_HOM (rho = K = 1); WK_CONST (rho = 1, constant K, folded into fx_sigp
// and the p coefficients; the SAT takes K); WK_VAR (1/rho and K from the tile's
// coefficient box multiply the scaled RHS; with prm.ysplit two blocks, each with its own
// y closures, and the interface SAT on the rows between them); WK_MMS (1/rho and the
// forcing, the latter in units of sigma and times `ct`, the stage's time factor).
// The variable kinds exist on a single grid only (no subdomain offsets).
// Fehlberg stages: u and k_1..k_{S-1} of the point are loaded ahead of the stencil
// arithmetic; stage 6 adds this thread's error terms to *errsq.
template <int ORD, int STAGE, typename Tile, int KIND = WK_HOM>
__device__ __forceinline__ void wave_tile_fixed(const WaveParams<double>& prm, const FxGeom& g, const double* in0,
                                                double* wout, const double c_acc, const double c_w,
                                                const double* fx_ca, const double* fx_cw, const unsigned char* st,
                                                const int i0, const int j0, const int warp, const int lane,
                                                const int ep, const int euv, const bool bad, uint64_t* dbar,
                                                uint32_t* dphase, const int b, const int k, const double ct = 0.0,
                                                double* errsq = nullptr) {
  constexpr int RKS = is_rkf_stage(STAGE) ? STAGE - ST_RKF1 + 1 : 1;
  constexpr bool FINE = fx_fine<KIND, STAGE>();
  constexpr int TY = Tile::TY, CS = OpShape<ORD>::CS;
  constexpr int HX = Tile::HX, HY = Tile::HY, PW = Tile::PW;
  constexpr int ROWS = TY / Tile::WARPS;
  constexpr int TPT = TY * kWaveTX;
  const int NX = prm.nx, NY = prm.ny;
  const long long pitch = g.pitch, plane = g.plane;
  const double* in = in0 + g.base;
  const long long* iP = reinterpret_cast<const long long*>(st);
  const long long* iU = reinterpret_cast<const long long*>(st + Tile::OFF_U);
  const long long* iV = reinterpret_cast<const long long*>(st + Tile::OFF_V);
  const double* sN = reinterpret_cast<const double*>(st + Tile::OFF_N);
  const double* sA = reinterpret_cast<const double*>(st + Tile::OFF_A);
  const double* sK = reinterpret_cast<const double*>(st + Tile::OFF_K);  // coefficient planes
  double* sD = reinterpret_cast<double*>(const_cast<unsigned char*>(st) + Tile::OFF_DEF);
  // x faces of the global grid inside this tile (their SAT goes to the deferred pass)
  const int iw = -g.xoff, ie = NX - 1 - g.xoff;  // local indices of global columns 0 and NX - 1
  const bool xfaces = dbar != nullptr && prm.bc != BC_NONE &&
                      ((iw >= i0 && iw < i0 + kWaveTX) || (ie >= i0 && ie < i0 + kWaveTX && ie < g.nx));
  const double sg[3] = {prm.fx_sig[0], prm.fx_sig[1], prm.fx_sigp};
  const int ebp = fx_base<false>(ep), ebuv = fx_base<false>(euv);
  const auto d1 = [&](const long long* c, int st, int eb) {
    if constexpr (FINE) return fx_d1<ORD>(c, st);
    else return fx_to<false>(fx_stencil<ORD>(c, st), eb);
  };
  (void)ebp;
  (void)ebuv;
  (void)sN;
  (void)sA;
  (void)sK;
  // rows that close a block from inside (two-block problems): the interface lines
  const int ys = KIND == WK_VAR ? prm.ysplit : 0;
  const auto interface_row = [&](int J) { return KIND == WK_VAR && ys > 0 && (J == ys - 1 || J == ys); };
#pragma unroll 1
  for (int rr = 0; rr < ROWS; rr++) {
    const int y = warp * ROWS + rr;
    const int j = j0 + y;
    if (j >= g.ny) continue;
    const int J = g.yoff + j;
    // the block's first row and height (one block unless ysplit is set)
    const int jb0 = (ys > 0 && J >= ys) ? ys : 0;
    const int nyb = ys > 0 ? (J >= ys ? NY - ys : ys) : NY;
    const bool yint = (J - jb0 >= CS) && (J - jb0 < nyb - CS);
    const long long rowq = (long long)(j + g.row0) * pitch;
#pragma unroll
    for (int cc = 0; cc < kWaveTX / 32; cc++) {
      const int x = lane + 32 * cc;
      const int i = i0 + x;
      if (i >= g.nx) continue;
      const int I = g.xoff + i;
      const bool xint = (I >= CS) && (I < NX - CS);
      const long long* cP = iP + (y + HY) * PW + (x + HX);
      const long long* cU = iU + y * PW + (x + HX);
      const long long* cV = iV + (y + HY) * kWaveTX + x;
      // closure lines start at the global first point of the line (inside the arrays
      // for a subdomain at the physical boundary, which holds a whole closure block)
      const double* xline = in + rowq + g.col0 - g.xoff;
      const double* yline = in + (long long)(g.row0 - g.yoff + jb0) * pitch + (i + g.col0);
      // Fehlberg stages: u and the earlier derivatives, in flight during the stencil arithmetic
      double pre[3][RKS];
      if constexpr (is_rkf_stage(STAGE)) {
#pragma unroll
        for (int c = 0; c < 3; c++) wave_rkf_preload<double, RKS>(prm, c * plane + rowq + i + g.col0, pre[c]);
      }
      (void)pre;
      // RHS in units of sigma per component: F_u = sx ku, F_v = sy kv, F_p = sx kp
      // (fx_fine, tiles with values that have no word: FP64 taps for the interior)
      const bool taps = FINE && bad, xfx = xint && !taps, yfx = yint && !taps;
      const auto other_x = [&](const double* line) {
        if (FINE && xint) return fx_taps_global<ORD>(line + I, 1, prm.dx.taps) * prm.fx_isig[0];
        return closure_line<double, ORD>(line, 1, NX, I, prm.dx.cls) * prm.fx_isig[0];
      };
      const auto other_y = [&](const double* line) {
        if (FINE && yint) return fx_taps_global<ORD>(line + (J - jb0) * pitch, pitch, prm.dy.taps) * prm.fx_isig[1];
        return closure_line<double, ORD>(line, pitch, nyb, J - jb0, prm.dy.cls) * prm.fx_isig[1];
      };
      double ku, kv, kp;
      if (xfx) {
        ku = d1(cP, 1, ebp);
      } else {
        ku = other_x(xline + 2 * plane);
      }
      if (yfx) {
        kv = d1(cP, PW, ebp);
      } else {
        kv = other_y(yline + 2 * plane);
      }
      if (xfx && yfx && prm.fx_square) {
        if constexpr (FINE) kp = fx_d1_sum<ORD>(cU, 1, cV, kWaveTX);
        else kp = fx_to<false>(fx_stencil<ORD>(cU, 1) + fx_stencil<ORD>(cV, kWaveTX), ebuv);
      } else {
        const double ax = xfx ? d1(cU, 1, ebuv) : other_x(xline);
        const double ay = yfx ? d1(cV, kWaveTX, ebuv) : other_y(yline + plane);
        kp = fma(prm.fx_rho, ay, ax);
      }
      if (!FINE && bad) ku = kv = kp = __longlong_as_double(0x7FF8000000000000ll);

      const long long q = rowq + i + g.col0;
      const int sp = y * kWaveTX + x;  // point within a 3-component smem box
      if constexpr (KIND == WK_VAR) {
        const double ri = sK[sp];
        ku *= ri;
        kv *= ri;
        kp *= sK[TPT + sp];
      } else if constexpr (KIND == WK_MMS) {
        const double ri = sK[sp];
        ku = fma(ct, sK[TPT + sp], ri * ku);
        kv = fma(ct, sK[2 * TPT + sp], ri * kv);
      }
      const bool edge = (I == 0) || (J == 0) || (I == NX - 1) || (J == NY - 1) || interface_row(J);
      if (prm.bc != BC_NONE && edge) {
        if (xfaces && J != 0 && J != NY - 1 && !interface_row(J)) {
          double* d = sD + ((I == 0 ? 0 : TY) + y) * 3;  // an x-face point only: deferred
          d[0] = ku;
          d[1] = kv;
          d[2] = kp;
          continue;
        }
        // SAT and the stage update in true units
        const double pc = in[2 * plane + q], uc = in[q], vc = in[plane + q];
        const Rhs3<double> r =
            apply_sat<double, KIND>(prm, in, I, J, pc, uc, vc, Rhs3<double>{sg[0] * ku, sg[1] * kv, sg[2] * kp});
        const double kt[3] = {r.u, r.v, r.p};
#pragma unroll
        for (int c = 0; c < 3; c++) {
          if constexpr (is_rkf_stage(STAGE)) {
            wave_point_rkf<double, STAGE, RKS>(prm, wout, c * plane + q, kt[c], pre[c], errsq);
          } else {
            const double cen = (STAGE == ST_FIRST) ? sN[c * TPT + sp] : 0.0;
            wave_point_store<double, STAGE, Tile>(prm, wout, c_acc, c_w, sA, sN, nullptr, sp, c,
                                                  g.base + c * plane + q, kt[c], cen);
          }
        }
        continue;
      }
      const double kf[3] = {ku, kv, kp};
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const long long o = g.base + c * plane + q;
        if constexpr (STAGE == ST_RHS) {
          prm.kout[o] = sg[c] * kf[c];
        } else if constexpr (is_rkf_stage(STAGE)) {
          wave_point_rkf<double, STAGE, RKS>(prm, wout, o, sg[c] * kf[c], pre[c], errsq);
        } else {
          const double cen = (STAGE == ST_FIRST) ? sN[c * TPT + sp] : 0.0;
          wave_point_store<double, STAGE, Tile>(prm, wout, fx_ca[c], fx_cw[c], sA, sN, nullptr, sp, c, o,
                                                kf[c], cen);
        }
      }
    }
  }
  if (xfaces) {
    __syncwarp();
    if (lane == 0) mbar_arrive(dbar);  // this warp's deferred entries are in shared memory
    const uint32_t par = (*dphase >> b) & 1u;
    *dphase ^= 1u << b;
    if (warp != k % Tile::WARPS) return;
    if (!mbar_wait_bounded(dbar, par, prm.wait_ns)) {
      if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
      return;
    }
    for (int e = lane; e < 2 * TY; e += 32) {
      const int side = e / TY, y = e - side * TY, j = j0 + y;
      const int I = side == 0 ? 0 : NX - 1, i = I - g.xoff, J = g.yoff + j;
      if (i < i0 || i >= i0 + kWaveTX || i >= g.nx || j >= g.ny || J == 0 || J == NY - 1 || interface_row(J)) continue;
      const int x = i - i0;
      const long long q = (long long)(j + g.row0) * pitch + i + g.col0;
      const double pc = in[2 * plane + q], uc = in[q], vc = in[plane + q];
      const double* d = sD + (side * TY + y) * 3;
      const Rhs3<double> r =
          apply_sat<double, KIND>(prm, in, I, J, pc, uc, vc, Rhs3<double>{sg[0] * d[0], sg[1] * d[1], sg[2] * d[2]});
      const double kt[3] = {r.u, r.v, r.p};
      const int sp = y * kWaveTX + x;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        if constexpr (is_rkf_stage(STAGE)) {
          double pre[RKS];
          wave_rkf_preload<double, RKS>(prm, c * plane + q, pre);
          wave_point_rkf<double, STAGE, RKS>(prm, wout, c * plane + q, kt[c], pre, errsq);
        } else {
          const double cen = (STAGE == ST_FIRST) ? sN[c * TPT + sp] : 0.0;
          wave_point_store<double, STAGE, Tile>(prm, wout, c_acc, c_w, sA, sN, nullptr, sp, c,
                                                g.base + c * plane + q, kt[c], cen);
        }
      }
    }
  }
}

// What the converter warps leave beside a converted stage, a pair per warp: the exponent maxima
// of p and of u and v, for stages that take their box's exponent. A box whose maximum is below
// 64 (values under 2^-959) converts to zeros, and one at 2031 or more (values from 2^1008, Inf,
// NaN) marks the tile bad: it is NaN throughout. Kernels that evaluate a bad tile with FP64 taps
// instead (TAPS) want one whose largest value is nonzero but below 2^-959 marked as well.
template <int CONV, bool TAPS>
__device__ __forceinline__ void fx_tile_emax(const int* wmax, int& ep, int& euv, bool& bad) {
  ep = 0;
  euv = 0;
#pragma unroll
  for (int c = 0; c < CONV; c++) {
    ep = max(ep, wmax[2 * c]);
    euv = max(euv, wmax[2 * c + 1]);
  }
  bad = ep >= 2031 || euv >= 2031;
  if (TAPS) bad = bad || (ep > 0 && ep < 64) || (euv > 0 && euv < 64);
  if (ep < 64) ep = 2111;  // every value converts to 0
  if (euv < 64) euv = 2111;
}

// Of stages on whole values: whether the warp met one without a word. FP64 taps from global
// memory then evaluate the tile.
template <int CONV>
__device__ __forceinline__ bool fx_tile_out(const int* wmax) {
  int o = 0;
#pragma unroll
  for (int c = 0; c < CONV; c++) o |= wmax[2 * c];
  return o != 0;
}

// Converter warps: the p, u and v boxes of one ring stage to words (FINE) or to int64 in units
// of the box's largest exponent, in place. t is the thread's index among the converter
// threads. Box units: the exponent maxima go through one barrier among the converters (fxa,
// bounded wait), each of which then takes the maximum over all, and so does every compute warp
// later, so nothing has to be reset between tiles. Returns false if the wait ran out.
template <typename Tile, bool FINE>
__device__ __forceinline__ bool fx_convert_stage(unsigned char* st, uint64_t* fxa, int* wmax, uint32_t parity,
                                                 unsigned long long wait_ns, int t) {
  constexpr int NT = 32 * Tile::CONV;
  constexpr int NP = Tile::PH * Tile::PW, NU = Tile::TY * Tile::PW, NV = Tile::PH * kWaveTX;
  const int lane = t & 31, cw = t >> 5;
  if constexpr (FINE) {
    bool out = false;
    const auto pack = [&](unsigned char* box, int n) {
      double* d = reinterpret_cast<double*>(box);
      long long* q = reinterpret_cast<long long*>(box);
#pragma unroll 4
      for (int e = t; e < n; e += NT) q[e] = fx_pack(d[e], out);
    };
    pack(st, NP);
    pack(st + Tile::OFF_U, NU);
    pack(st + Tile::OFF_V, NV);
    out = __any_sync(0xffffffffu, out);
    if (lane == 0) wmax[2 * cw] = out;
  } else {
    uint2* wP = reinterpret_cast<uint2*>(st);
    uint2* wU = reinterpret_cast<uint2*>(st + Tile::OFF_U);
    uint2* wV = reinterpret_cast<uint2*>(st + Tile::OFF_V);
    unsigned mp = 0, muv = 0;
    for (int e = t; e < NP; e += NT) mp = max(mp, wP[e].y & 0x7FF00000u);
    for (int e = t; e < NU; e += NT) muv = max(muv, wU[e].y & 0x7FF00000u);
    for (int e = t; e < NV; e += NT) muv = max(muv, wV[e].y & 0x7FF00000u);
    mp = __reduce_max_sync(0xffffffffu, mp);
    muv = __reduce_max_sync(0xffffffffu, muv);
    if (lane == 0) {
      wmax[2 * cw] = (int)(mp >> 20);
      wmax[2 * cw + 1] = (int)(muv >> 20);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(fxa);
    if (!mbar_wait_bounded(fxa, parity, wait_ns)) return false;
    int ep, euv;
    bool bad;
    fx_tile_emax<Tile::CONV, false>(wmax, ep, euv, bad);
    (void)bad;
    long long* iP = reinterpret_cast<long long*>(wP);
    long long* iU = reinterpret_cast<long long*>(wU);
    long long* iV = reinterpret_cast<long long*>(wV);
#pragma unroll 4
    for (int e = t; e < NP; e += NT) {
      const uint2 w = wP[e];
      iP[e] = fx_from<false>(w.x, w.y, ep);
    }
#pragma unroll 4
    for (int e = t; e < NU; e += NT) {
      const uint2 w = wU[e];
      iU[e] = fx_from<false>(w.x, w.y, euv);
    }
#pragma unroll 4
    for (int e = t; e < NV; e += NT) {
      const uint2 w = wV[e];
      iV[e] = fx_from<false>(w.x, w.y, euv);
    }
  }
  // the converted boxes were written through the generic proxy; order those writes
  // before the TMA (async proxy) refills the stage
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  return true;
}

// A fixed-point FP64 stage with warp roles: WARPS compute warps, CONV converter
// warps and one producer warp. Per ring stage: the producer's TMA loads complete
// `full` (1 arrival + bytes), the converters convert the stage's boxes and arrive on
// `conv` (CONV arrivals), the compute warps evaluate the tile and arrive on
// `empty` (WARPS arrivals), which lets the producer refill the stage. Conversion
// of the next tile thus overlaps the computation of the current one, and the
// compute warps meet no barrier but the deferred x-face pass. Every wait is
// bounded (prm.wait_ns); a wait that runs out sets the error word and the warp
// stops, so the others' waits run out in turn.
template <int ORD, int STAGE, bool DEC = false, int KIND = WK_HOM>
__global__ void __launch_bounds__(fx_kernel_threads<WaveStageTile<double, ORD, KIND, STAGE>, DEC>(), 1)
    wave_fixed_kernel(const __grid_constant__ CUtensorMap mapP, const __grid_constant__ CUtensorMap mapU,
                      const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapN,
                      const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapC,
                      const __grid_constant__ CUtensorMap mapK, const __grid_constant__ WaveParams<double> prm) {
  using Tile = WaveStageTile<double, ORD, KIND, STAGE>;
  static_assert(KIND == WK_HOM || !DEC, "decomposed grids: rho = K = 1");
  constexpr int TY = Tile::TY, NST = Tile::NST, WARPS = Tile::WARPS, CONV = Tile::CONV;
  static_assert(CONV >= 1, "the converter-warp kernel needs converter warps");
  extern __shared__ __align__(128) unsigned char smem[];
  if (prm.fx_sig[0] == 0.0 || prm.fx_sig[1] == 0.0) {  // the host did not set the fixed-point scales
    if (threadIdx.x == 0) atomicOr(prm.err, ERR_BAD_LAUNCH);
    return;
  }
  if (prm.skip && *prm.skip) return;  // uniform over the grid: set before this launch
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Tile::OFF_BAR);
  uint64_t* empty = full + NST;
  uint64_t* dbar = reinterpret_cast<uint64_t*>(smem + Tile::OFF_DBAR);
  int* tslot = reinterpret_cast<int*>(smem + Tile::OFF_BAR + 192);
  uint64_t* fxa = reinterpret_cast<uint64_t*>(smem + Tile::OFF_FX);  // [8]: exponent maxima known
  uint64_t* conv = fxa + 8;                                          // [8]: stage converted
  int* wmax = reinterpret_cast<int*>(smem + Tile::OFF_FX + 128);     // [8][8][2]
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], WARPS);
      mbar_init(&dbar[s], WARPS);
      mbar_init(&fxa[s], CONV);
      mbar_init(&conv[s], CONV);
    }
    if constexpr (DEC) {
      const FxExchangeQueue<Tile> xq(smem);
      for (int s = 0; s < FxExchangeQueue<Tile>::SLOTS; s++) {
        mbar_init(&xq.full[s], 1);
        mbar_init(&xq.empty[s], 1);
      }
    }
    fence_barrier_init();
  }
  __shared__ double s_ct;  // WK_MMS: the forcing's time factor, one cosine per CTA at most
  if constexpr (KIND == WK_MMS) {
    if (threadIdx.x == 32)
      s_ct = prm.tctl ? cos(5 * 3.14159265358979323846264 *
                            __dadd_rn(prm.tctl[0], __dmul_rn(prm.tc, prm.tctl[1])))
                      : (prm.ctp ? *prm.ctp : prm.ct);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntx = (prm.nx + kWaveTX - 1) / kWaveTX;

  if (warp == WARPS + CONV) {
    if constexpr (DEC)
      decomp_produce<Tile, STAGE>(prm, smem, full, empty, tslot, FxExchangeQueue<Tile>(smem), lane);
    else if (lane == 0)
      wave_produce<Tile>(mapP, mapU, mapV, mapN, mapA, mapC, mapK, prm, smem, full, empty, tslot,
                         prm.sched != nullptr);
    return;
  }
  if constexpr (DEC) {
    if (warp == WARPS + CONV + 1) {  // the exchange warp
      if constexpr (STAGE == ST_FIRST || STAGE == ST_MID || STAGE == ST_LAST)
        decomp_exchange<Tile, STAGE>(prm, FxExchangeQueue<Tile>(smem), lane);
      return;
    }
  }
  if (warp >= WARPS) {
    // ---------------- converters
    const int t = threadIdx.x - 32 * WARPS;
    for (int k = 0;; k++) {
      const int b = k % NST;
      if (!mbar_wait_bounded(&full[b], (k / NST) & 1, prm.wait_ns)) {
        if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
        break;
      }
      const int tile = tslot[b];
      if (tile >= 0 && !fx_convert_stage<Tile, fx_fine<KIND, STAGE>()>(smem + b * Tile::STAGE_BYTES, &fxa[b],
                                                                       wmax + 16 * b, (k / NST) & 1, prm.wait_ns, t)) {
        if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
        break;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&conv[b]);  // converted, or the end marker passed on
      if (tile < 0) break;
    }
    return;
  }
  // ---------------- compute warps
  uint32_t dphase = 0;  // parity of each stage's next deferred-pass barrier phase
  double errsq = 0.0;   // ST_RKF6: this thread's share of the weighted error sum
  const double ct = KIND == WK_MMS ? s_ct : 0.0;
  for (int k = 0;; k++) {
    const int b = k % NST;
    if (!mbar_wait_bounded(&conv[b], (k / NST) & 1, prm.wait_ns)) {
      if (lane == 0) atomicOr(prm.err, ERR_TMA_TIMEOUT);
      break;
    }
    const int tile = tslot[b];
    if (tile < 0) break;
    int i0, j0;
    FxGeom g;
    if constexpr (DEC) {
      const FxTileInfo* info = reinterpret_cast<const FxTileInfo*>(smem + Tile::OFF_TINFO + kFxTileInfoBytes * b);
      g = info->g;
      i0 = info->i0;
      j0 = info->j0;
    } else {
      i0 = (tile % ntx) * kWaveTX;
      j0 = (tile / ntx) * TY;
      g = FxGeom{prm.nx, prm.ny, 0, 0, 0, 0, prm.pitch, prm.plane, 0};
    }
    int ep = 0, euv = 0;
    bool bad;
    if constexpr (fx_fine<KIND, STAGE>()) bad = fx_tile_out<CONV>(wmax + 16 * b);
    else fx_tile_emax<CONV, false>(wmax + 16 * b, ep, euv, bad);
    wave_tile_fixed<ORD, STAGE, Tile, KIND>(prm, g, prm.in, prm.wout, prm.c_acc, prm.c_w, prm.fx_ca, prm.fx_cw,
                                            smem + b * Tile::STAGE_BYTES, i0, j0, warp, lane, ep, euv, bad, &dbar[b],
                                            &dphase, b, k, ct, &errsq);
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[b]);
  }
  if constexpr (STAGE == ST_RKF6) {
    // fixed-order sum over the compute threads -> one partial per CTA
    __shared__ double warp_sum[WARPS];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) errsq += __shfl_down_sync(0xffffffffu, errsq, off);
    if (lane == 0) warp_sum[warp] = errsq;
    asm volatile("bar.sync 1, %0;" ::"n"(32 * WARPS) : "memory");  // compute warps only
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int q = 0; q < WARPS; q++) s += warp_sum[q];
      prm.rkpart[blockIdx.x] = s;
    }
  }
}

}  // namespace sbp

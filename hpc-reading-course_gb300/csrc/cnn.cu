// cnn.cu -- the learned correction: a 4-layer 3x3 convolutional network
// (24 -> 32 -> 32 -> 32 -> 3 channels, ReLU between layers) trained and run on
// the GPU by the kernels in this file. No counterpart in the reference.
//
// Tensors are NHWC. Activations and weights are BF16; every product is
// accumulated in FP32 on the tensor cores; master weights, biases and Adam
// moments are FP32. Channel counts are padded to multiples of 16 (the MMA K
// step): input 24 -> 32, output 3 -> 16; the padding carries zeros.
//
//   conv3x3_tc_kernel     implicit GEMM on tcgen05 (TMA tiles, tensor-memory
//                         accumulator), M = 128 pixels, N = output channels,
//                         K = 9 taps x input channels; also computes the input
//                         gradient (dgrad) with the spatially flipped,
//                         transposed weights.
//   conv3x3_wgrad_tc_kernel  weight gradient on tcgen05, K = pixels: a column's three
//                         vertical taps stacked along M (MN-major operands),
//                         accumulated over all of a CTA's pixel tiles in tensor
//                         memory; weight_step_kernel adds the CTAs' sums up in
//                         CTA order (repeatable bits).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <random>
#include <string>
#include <vector>

#include "../../include/sbpgpu.h"
#include "launch.h"
#include "sbp_device.cuh"

namespace sbp {
namespace cnn {

typedef __nv_bfloat16 bf16;

constexpr int kLayers = 4;
constexpr int kCin[kLayers] = {32, 32, 32, 32};   // padded input channels
constexpr int kCout[kLayers] = {32, 32, 32, 16};  // padded output channels
constexpr int kInReal = 24, kOutReal = 3;

__device__ __forceinline__ uint32_t pack_pair(bf16 lo, bf16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// The widest pixel tiles: 32 x 4 pixels, and for images one or two pixels high 64 x 2.
constexpr int kConvMaxTw = 32, kConvStripTw = 64;
// A column box: 128 / tw + 2 rows of tw pixels, rounded up to whole 1024-byte units.
__host__ __device__ constexpr int conv_box_bytes(int tw, int rowb) {
  return ((128 / tw + 2) * tw * rowb + 1023) / 1024 * 1024;
}

// ---------------------------------------------------------------- tcgen05 convolution
// The forward and input-gradient 3x3 convolutions on the 5th-generation tensor cores:
// an implicit GEMM per 128-pixel tile (th x tw pixels of one image), M = 128 pixels,
// N = COUT, K = 9 taps x CIN. TMA loads the tile's three column boxes, one per horizontal
// tap offset and with a row above and below the tile (a 4D box {CIN, tw, th + 2, 1} of the
// NHWC activations: the image border comes back as zeros), and each tap's weight tile into
// shared memory, rows of CIN BF16 values swizzled by the TMA (64-byte swizzle for 32
// channels, 32-byte for 16) -- the K-major
// layout the MMA's shared-memory descriptors describe. One lane issues
// tcgen05.mma (kind::f16, BF16 inputs, FP32 accumulator in tensor memory) tap by
// tap once the boxes have landed, K = 16 per instruction; tcgen05.commit signals the
// epilogue, where each warp reads its 32 accumulator lanes (pixels) with
// tcgen05.ld, adds the bias, applies ReLU and stores. Every wait is bounded.

// Shared-memory descriptor of a K-major operand tile with rows of `rowb` bytes
// swizzled in 8-row atoms (stride between atoms: 8 rows), tcgen05 version.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr, uint32_t atom_bytes, uint32_t layout) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);  // start address
  d |= (uint64_t)1u << 16;                           // leading offset: unused by swizzled K-major tiles
  d |= (uint64_t)((atom_bytes >> 4) & 0x3FFFu) << 32;  // stride offset: one 8-row atom
  d |= (uint64_t)1u << 46;                           // descriptor version of tcgen05
  d |= (uint64_t)layout << 61;                       // swizzle mode
  return d;
}

// The same for an MN-major operand: rows along K of one swizzle span of M (or N)
// values; `lead` = byte stride between swizzle spans along M, `stride` = between
// 8-row groups along K.
__device__ __forceinline__ uint64_t umma_smem_desc_mn(uint32_t saddr, uint32_t lead, uint32_t stride,
                                                      uint32_t layout) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lead >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((stride >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)layout << 61;
  return d;
}

// Instruction descriptor of kind::f16: BF16 A and B (both K-major), FP32 D, M x N.
constexpr uint32_t umma_idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// One MMA, issued by the lanes with `leader` set: one lane of a converged warp. Predicated
// rather than branched around, so that the descriptors stay in uniform registers, which the
// instruction reads.
__device__ __forceinline__ void umma_bf16(uint32_t leader, uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accum), "r"(leader)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t leader, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n" ::"r"(smem_addr(bar)),
      "r"(leader)
      : "memory");
}

// A wait of a whole converged warp: true if it ended in time for every lane.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive accumulator columns of this thread's lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Eight mask values. Volatile: not before the kernel's wait for the ones that wrote them.
// Through L1, since a thread's four loads share two sectors.
__device__ __forceinline__ uint4 ld_mask(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

// Shared-memory layout of conv3x3_tc_kernel: a ring of NS column boxes (th + 2 rows of tw
// pixels of CIN BF16), the nine taps' weight tiles (COUT rows of CIN), barriers and the
// tensor-memory address; boxes and tiles 1024-byte aligned (whole swizzle atoms).
template <int CIN, int COUT>
struct TcConv {
  static_assert(CIN == 16 || CIN == 32, "input channels: one or two K steps of 16 per tap");
  static_assert(COUT == 16 || COUT == 32, "output channels: the MMA's N");
  static constexpr int ROWB = CIN * 2;  // bytes per row: the swizzle span
  static constexpr uint32_t LAYOUT = CIN == 32 ? 4u : 6u;  // 64-byte / 32-byte swizzle
  static constexpr uint32_t ATOM = 8 * ROWB;
  static constexpr int NS = 6;    // column boxes in flight: two pixel tiles per CTA
  static constexpr int slots(int tw) { return tw > kConvMaxTw ? 4 : NS; }
  static constexpr int CTAS = 2;  // resident CTAs per SM (forward pass at 8 x 258 x 257, launches not overlapped: 0.138 ms; three
                                  // CTAs with 4 boxes 0.138 ms, four with 3 boxes 0.146 ms)
  static constexpr int B_BYTES = COUT * ROWB;
  static constexpr int box_bytes(int tw) { return conv_box_bytes(tw, ROWB); }
  static constexpr int off_bar() { return ((9 * B_BYTES + 1023) / 1024) * 1024; }  // after the weights
  static constexpr int NACC = 2;  // accumulators of 32 columns (four: the same time)
  // full[NS], empty[NS], wbar, accfull[NACC], accempty[NACC], done; then the tensor-memory address
  static constexpr int NBAR = 2 * NS + 2 * NACC + 2;
  static constexpr int HEAD = (off_bar() + 8 * NBAR + 16 + 1023) / 1024 * 1024;  // weights, barriers
  static constexpr int smem(int tw) { return HEAD + slots(tw) * box_bytes(tw) + 1024; }  // + the dynamic base's slack
  static constexpr uint32_t IDESC = umma_idesc_bf16(128, COUT);
  static constexpr int THREADS = 192;  // producer, MMA issuer, four epilogue warps
  static_assert(B_BYTES % 256 == 0, "tiles start on swizzle atoms");
  static constexpr int SMEM_MAX = smem(kConvMaxTw) > smem(kConvStripTw) ? smem(kConvMaxTw) : smem(kConvStripTw);
  static_assert(CTAS * (SMEM_MAX + 1024) <= 228 * 1024, "shared memory");
};

// The two halves of grid_dependency_wait. A kernel whose CTAs take several tiles does not
// let the next kernel's CTAs in before it ends: they would take the places that free up
// first, two kernels' persistent CTAs sharing the SMs unevenly (training step at 8 x 258 x 257
// 366 us when let in at the start, 358 after the last loads, 344 at the end, 371 without
// overlap). With a tile per CTA (2 x 40 x 33) it does, after its loads: 75 us, 86 at the end,
// 112 without overlap.
__device__ __forceinline__ void grid_inputs_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_let_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Waits for the last loads of a ring of n slots, the next of which would go to slot s, after
// `round` times round: no copy may be in flight when a CTA exits.
__device__ __forceinline__ void drain_ring(uint64_t* full, int s, int round, int n) {
  int q = round > 0 ? s : 0, r = round > 0 ? round - 1 : 0;
  for (int left = round > 0 ? n : s; left > 0; left--) {
    mbar_wait_bounded(&full[q], r & 1);
    if (++q == n) {
      q = 0;
      r++;
    }
  }
}

// The pixel tiles of a persistent CTA: every gridDim.x-th, as tile column, tile row and
// image, stepped by carries instead of divided out of a tile number.
struct TileWalk {
  int w, h, b, dw, dh, db, ntw, nth;

  __device__ __forceinline__ TileWalk(int ntw_, int nth_) : ntw(ntw_), nth(nth_) {
    w = blockIdx.x % ntw;
    h = (blockIdx.x / ntw) % nth;
    b = blockIdx.x / (ntw * nth);
    dw = gridDim.x % ntw;
    dh = (gridDim.x / ntw) % nth;
    db = gridDim.x / (ntw * nth);
  }

  __device__ __forceinline__ void next() {
    w += dw;
    h += dh;
    b += db;
    if (w >= ntw) {
      w -= ntw;
      h++;
    }
    if (h >= nth) {
      h -= nth;
      b++;
    }
  }
};

// y[p][n] = act(bias[n] + sum_{tap,c} x[p + off(tap)][c] * w[n][tap][c]); x through xmap
// ({CIN, W, H, B}, box {CIN, tw, th + 2, 1}), w through wmap ({CIN, 9, COUT}). Persistent: a
// CTA takes every gridDim.x-th 128-pixel tile (th rows of tw pixels). Warp roles: warp 0 loads
// the weights once, then for each tile three boxes, one per horizontal tap offset, with a row
// above and below the tile, into a ring of NS slots; warp 1 (which owns the tensor memory)
// issues the nine taps' MMAs in tap order -- the vertical offsets are start addresses tw pixel
// rows apart in a box, whole 8-row swizzle atoms since tw is a multiple of 8 -- frees each box
// after its last tap with tcgen05.commit, and commits each pixel tile into one of two
// accumulators (32 columns each); warps 2-5 read an accumulator (warp w: lanes 32 (w % 4) ..),
// release it, and add bias, apply ReLU and store while the next tile accumulates in the other.
// Bounded waits.
// W, H here: the extents along and across a tile's rows. `turned`: those rows run down the image
// (xmap is then {CIN, image height, image width, B}); the taps change places with the weights'
// loads, and only the pixels' addresses differ.
//
// What bounded it was the MMA warp's instructions: with the loads, the stores and eight of
// nine MMAs left out the forward pass (8 x 258 x 257) still took 0.161 of its 0.197 ms.
// Issued from one lane's branch, each MMA builds its two descriptors in that lane and moves
// them to uniform registers; now the whole warp runs the loop, descriptors are a base plus
// constants, and only the MMAs and the commits are predicated on one lane: 0.138 ms (0.126
// with the kernels' launches overlapped). Three
// column boxes instead of nine shifted tiles (2.4 x fewer bytes through L2) made no
// difference before that.
//
// MASK (input gradients): the ReLU backward pass through `mask`, the post-activation
// values the output is the gradient of -- y is zero where the mask is not above zero.
// Each thread fetches its pixel's 64 mask bytes before it waits for the accumulator, so
// the fetch hides behind the MMAs; a separate pass reads and writes the gradient once
// more (8 x 258 x 257: 34 MB of mask instead of 102 MB).
template <int CIN, int COUT, bool RELU, bool OUT_F32, bool MASK>
__global__ void __launch_bounds__(TcConv<CIN, COUT>::THREADS, TcConv<CIN, COUT>::CTAS)
    conv3x3_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                      const float* __restrict__ bias, const bf16* __restrict__ mask, void* __restrict__ y, int B, int H,
                      int W, int tw, int th, bool turned, int* err) {
  static_assert(!MASK || (!RELU && !OUT_F32), "the mask is the input gradient's, in BF16");
  using L = TcConv<CIN, COUT>;
  constexpr int NS = L::NS;
  const int box = L::box_bytes(tw), box_tx = (th + 2) * tw * L::ROWB, ns = L::slots(tw);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  unsigned char* boxes = smem + L::HEAD;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::off_bar());
  uint64_t* empty = full + NS;
  uint64_t* wbar = empty + NS;
  uint64_t* accfull = wbar + 1;
  uint64_t* accempty = accfull + L::NACC;
  uint64_t* done = accempty + L::NACC;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntw = (W + tw - 1) / tw, nth = (H + th - 1) / th;
  const int ntiles = B * nth * ntw;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(wbar, 1);
    for (int s = 0; s < L::NACC; s++) {
      mbar_init(&accfull[s], 1);
      mbar_init(&accempty[s], 4);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tslot, 32 * L::NACC);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  grid_inputs_wait();  // nothing of the kernels before this one is read or overwritten above

  if (warp == 0) {  // ---- loads
    if (lane == 0) {
      mbar_arrive_expect_tx(wbar, 9 * L::B_BYTES);
      const int along = turned ? 3 : 1, over = turned ? 1 : 3;  // taps along and across the tile's rows
#pragma unroll
      for (int t = 0; t < 9; t++) tma_load_3d(smem + t * L::B_BYTES, &wmap, 0, t / 3 * over + t % 3 * along, 0, wbar);
      int s = 0, round = 0;  // the next slot, times round the ring
      bool ok = true;
      for (TileWalk t(ntw, nth); ok && t.b < B; t.next()) {
        const int w0 = t.w * tw, h0 = t.h * th, b = t.b;
        for (int dx = 0; dx < 3; dx++) {
          if (round > 0 && !mbar_wait_bounded(&empty[s], (round - 1) & 1)) {
            atomicOr(err, 1);
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&full[s], box_tx);
          tma_load_4d(boxes + s * box, &xmap, 0, w0 + dx - 1, h0 - 1, b, &full[s]);
          if (++s == ns) {
            s = 0;
            round++;
          }
        }
      }
      if (ntiles <= (int)gridDim.x) grid_let_next();
      mbar_wait_bounded(wbar, 0);
      drain_ring(full, s, round, ns);
    }
  } else if (warp == 1) {  // ---- MMAs
    const uint32_t leader = lane == 0;
    bool ok = mbar_wait_warp(wbar, 0);
    const uint64_t a0 = umma_smem_desc(smem_addr(boxes), L::ATOM, L::LAYOUT);
    const uint64_t b0 = umma_smem_desc(smem_addr(smem), L::ATOM, L::LAYOUT);
    const uint32_t box16 = (uint32_t)box >> 4, row16 = (uint32_t)(tw * L::ROWB) >> 4;  // as in descriptors
    int slot = 0, phase = 0, it = 0;
    for (int tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, it++) {
      const int buf = it % L::NACC;
      if (it >= L::NACC && !(ok = mbar_wait_warp(&accempty[buf], ((it / L::NACC) - 1) & 1))) break;
      tc_fence_after();
      const uint32_t d = tmem + (uint32_t)(32 * buf);
      int sl[3];
      uint64_t a[3];
#pragma unroll
      for (int dx = 0; dx < 3; dx++) {
        sl[dx] = slot;
        a[dx] = a0 + (uint64_t)(slot * box16);
        if (ok) ok = mbar_wait_warp(&full[slot], phase);
        if (++slot == ns) {
          slot = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int t = 0; t < 9; t++) {
        const int dy = t / 3, dx = t % 3;
#pragma unroll
        for (int kk = 0; kk < CIN / 16; kk++)  // 16 channels are 32 bytes
          umma_bf16(leader, d, a[dx] + dy * row16 + 2 * kk, b0 + (t * L::B_BYTES >> 4) + 2 * kk, L::IDESC,
                    (t | kk) != 0);
        if (dy == 2) umma_commit(leader, &empty[sl[dx]]);  // the box is free once the MMAs so far have read it
      }
      umma_commit(leader, &accfull[buf]);
    }
    if (!ok && leader) atomicOr(err, 1);
    umma_commit(leader, done);  // every MMA issued has completed once this arrives
    mbar_wait_warp(done, 0);
  } else {  // ---- epilogue: warps 2-5
    const int q = warp & 3;  // the lane quarter this warp may read
    float bv[COUT];
#pragma unroll
    for (int j = 0; j < COUT; j++) bv[j] = MASK ? 0.f : bias[j];  // input gradients have no bias
    int it = 0;
    const int m = 32 * q + lane;  // this thread's accumulator lane: pixel m of the tile
    const int hm = m / tw, wm = m % tw;
    for (TileWalk t(ntw, nth); t.b < B; t.next(), it++) {
      const int buf = it % L::NACC, b = t.b;
      const int hh = t.h * th + hm, ww = t.w * tw + wm;
      const bool inside = hh < H && ww < W;
      const long long p = turned ? ((long long)b * W + ww) * H + hh : ((long long)b * H + hh) * W + ww;
      uint4 mk[MASK ? COUT / 8 : 1];
      if (MASK && inside) {
#pragma unroll
        for (int j = 0; j < COUT / 8; j++) mk[j] = ld_mask(mask + p * COUT + 8 * j);
      }
      if (!mbar_wait_bounded(&accfull[buf], (it / L::NACC) & 1)) {
        if (lane == 0) atomicOr(err, 1);
        break;
      }
      tc_fence_after();
      uint32_t r[COUT];
      const uint32_t src = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * buf);
      tmem_ld16(src, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
      if (COUT == 32) tmem_ld16(src + 16, *reinterpret_cast<uint32_t(*)[16]>(&r[COUT == 32 ? 16 : 0]));
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&accempty[buf]);  // the accumulator may take a later tile
      if (!inside) continue;
      float v[COUT];
#pragma unroll
      for (int j = 0; j < COUT; j++) {
        v[j] = __uint_as_float(r[j]) + bv[j];
        if (RELU) v[j] = fmaxf(v[j], 0.f);
        if (MASK) {
          const uint4 u = mk[j / 8];
          const uint32_t w = (j / 2) % 4 == 0 ? u.x : (j / 2) % 4 == 1 ? u.y : (j / 2) % 4 == 2 ? u.z : u.w;
          // the BF16 value as FP32: its bits are the upper half
          if (!(__uint_as_float(j & 1 ? w & 0xffff0000u : w << 16) > 0.f)) v[j] = 0.f;
        }
      }
      if (OUT_F32) {
        float4* yp = reinterpret_cast<float4*>(static_cast<float*>(y) + p * COUT);
#pragma unroll
        for (int j = 0; j < COUT / 4; j++) yp[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      } else {
        uint4* yp = reinterpret_cast<uint4*>(static_cast<bf16*>(y) + p * COUT);
#pragma unroll
        for (int j = 0; j < COUT / 8; j++)
          yp[j] = make_uint4(pack_pair(__float2bfloat16(v[8 * j]), __float2bfloat16(v[8 * j + 1])),
                             pack_pair(__float2bfloat16(v[8 * j + 2]), __float2bfloat16(v[8 * j + 3])),
                             pack_pair(__float2bfloat16(v[8 * j + 4]), __float2bfloat16(v[8 * j + 5])),
                             pack_pair(__float2bfloat16(v[8 * j + 6]), __float2bfloat16(v[8 * j + 7])));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 32 * L::NACC);
  }
}

// ---------------------------------------------------------------- tcgen05 weight gradient
// dw[n][tap][c] += sum_p dy[p][n] * x[p + off(tap)][c] as tcgen05 MMAs with K = pixels:
// per 128-pixel tile, TMA loads the three column boxes of x (as in the forward pass) and
// the dy tile into one stage. Both operands are MN-major there (channels contiguous per
// pixel row). A column's three taps start one row of tw pixels apart in its box; with a
// fourth row offset, whose results are not used, they form one 128-row A operand (rows
// (dy, c): the spacing is the descriptor's leading offset), so three MMA groups -- one per
// column -- cover the nine taps with M = 128, N = COUT, eight K steps of 16 pixels each.
// The accumulators (3 x COUT tensor-memory columns) sum over every tile the CTA takes; at
// the end the four epilogue warps write them to the CTA's slice of the layer's part of
// dw_part, which weight_step_kernel adds up in CTA order (the same bits on every run).
template <int COUT>
struct TcWgrad {
  static_assert(COUT == 16 || COUT == 32, "output channels: the MMA's N");
  static constexpr int CIN = 32, A_ROWB = CIN * 2;
  static constexpr int B_ROWB = COUT * 2;
  static constexpr int B_BYTES = 128 * B_ROWB;   // the dy tile
  static constexpr uint32_t A_LAYOUT = 4u, B_LAYOUT = COUT == 32 ? 4u : 6u;  // 64-byte / 32-byte swizzle
  static constexpr uint32_t A_SBO = 8 * A_ROWB, B_SBO = 8 * B_ROWB;
  static constexpr int NST = 5;  // stages: the next tiles load while this one's MMAs run (8 x 258 x 257, with
                                 // the descriptors in uniform registers: 41 -> 32 us per layer)
  static constexpr int stages(int tw) { return tw > kConvMaxTw ? 3 : NST; }
  static constexpr int stage(int tw) { return 3 * conv_box_bytes(tw, A_ROWB) + B_BYTES; }
  static constexpr int HEAD = 1024;  // barriers, tensor-memory address
  static constexpr int smem(int tw) { return HEAD + stages(tw) * stage(tw) + 1024; }
  static constexpr uint32_t IDESC = umma_idesc_bf16(128, COUT) | (1u << 15) | (1u << 16);  // A, B MN-major
  static constexpr int THREADS = 192;
  static constexpr int SMEM_MAX = smem(kConvMaxTw) > smem(kConvStripTw) ? smem(kConvMaxTw) : smem(kConvStripTw);
  static_assert(SMEM_MAX <= 227 * 1024, "shared memory");
  // the fourth row offset of the last column reads one row of pixels past its box: the dy tile
  static_assert(B_BYTES >= kConvStripTw * A_ROWB, "operand reads stay in the stage");
};

template <int COUT>
__global__ void __launch_bounds__(TcWgrad<COUT>::THREADS, 1)
    conv3x3_wgrad_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap dymap,
                            float* __restrict__ dw_part, int B, int H, int W, int tw, int th, bool turned,
                            int* err) {
  using L = TcWgrad<COUT>;
  constexpr int NST = L::NST, CIN = L::CIN;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* head = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  unsigned char* smem = head + L::HEAD;
  const int box = conv_box_bytes(tw, L::A_ROWB), stage = L::stage(tw), nst = L::stages(tw);
  uint64_t* full = reinterpret_cast<uint64_t*>(head);
  uint64_t* empty = full + NST;
  uint64_t* accfull = empty + NST;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(accfull + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntw = (W + tw - 1) / tw, nth = (H + th - 1) / th;
  const int ntiles = B * nth * ntw;
  float* part = dw_part + (long long)blockIdx.x * COUT * 9 * CIN;  // this CTA's sums, every entry written
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accfull, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tslot, 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  grid_inputs_wait();  // nothing of the kernels before this one is read or overwritten above

  if (warp == 0) {  // ---- loads
    if (lane == 0) {
      int s = 0, round = 0;  // the next stage, times round the ring
      for (TileWalk t(ntw, nth); t.b < B; t.next()) {
        if (round > 0 && !mbar_wait_bounded(&empty[s], (round - 1) & 1)) {
          atomicOr(err, 1);
          break;
        }
        const int w0 = t.w * tw, h0 = t.h * th, b = t.b;
        unsigned char* st = smem + s * stage;
        mbar_arrive_expect_tx(&full[s], 3 * (th + 2) * tw * L::A_ROWB + L::B_BYTES);
        for (int dx = 0; dx < 3; dx++) tma_load_4d(st + dx * box, &xmap, 0, w0 + dx - 1, h0 - 1, b, &full[s]);
        tma_load_4d(st + 3 * box, &dymap, 0, w0, h0, b, &full[s]);
        if (++s == nst) {
          s = 0;
          round++;
        }
      }
      if (ntiles <= (int)gridDim.x) grid_let_next();
      drain_ring(full, s, round, nst);
    }
  } else if (warp == 1) {  // ---- MMAs
    const uint32_t leader = lane == 0;
    bool ok = true;
    const uint64_t a0 = umma_smem_desc_mn(smem_addr(smem), tw * L::A_ROWB, L::A_SBO, L::A_LAYOUT);
    const uint64_t b0 = umma_smem_desc_mn(smem_addr(smem) + 3 * box, L::B_SBO, L::B_SBO, L::B_LAYOUT);
    const uint32_t stage16 = (uint32_t)stage >> 4, box16 = (uint32_t)box >> 4;  // as in descriptors
    int s = 0, phase = 0, it = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
      if (!(ok = mbar_wait_warp(&full[s], phase))) break;
      tc_fence_after();
      const uint64_t a = a0 + (uint64_t)(s * stage16), b = b0 + (uint64_t)(s * stage16);
#pragma unroll
      for (int k = 0; k < 8; k++)  // 16 pixels = two 8-row groups per K step
#pragma unroll
        for (int g = 0; g < 3; g++)
          umma_bf16(leader, tmem + (uint32_t)(g * COUT), a + g * box16 + (2 * k * L::A_SBO >> 4),
                    b + (2 * k * L::B_SBO >> 4), L::IDESC, (it | k) != 0);
      umma_commit(leader, &empty[s]);
      if (++s == nst) {
        s = 0;
        phase ^= 1;
      }
    }
    if (!ok && leader) atomicOr(err, 1);
    umma_commit(leader, accfull);  // every MMA issued has completed once this arrives
  } else {  // ---- epilogue: warps 2-5, once per CTA
    const int q = warp & 3;  // lane quarter: row (vertical tap offset q, c = lane)
    if (mbar_wait_bounded(accfull, 0)) {
      tc_fence_after();
#pragma unroll
      for (int g = 0; g < 3; g++) {
        if (q == 3) continue;
        const int tap = turned ? 3 * g + q : 3 * q + g;
#pragma unroll
        for (int n0 = 0; n0 < COUT; n0 += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(g * COUT + n0), r);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; j++) part[((long long)(n0 + j) * 9 + tap) * CIN + lane] = __uint_as_float(r[j]);
        }
      }
    } else if (lane == 0) {
      atomicOr(err, 1);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
}

template <int COUT>
__global__ void bias_grad_kernel(const bf16* __restrict__ dy, float* __restrict__ db, long long P) {
  __shared__ float sh[COUT];
  for (int n = threadIdx.x; n < COUT; n += blockDim.x) sh[n] = 0.f;
  __syncthreads();
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < P * COUT; e += (long long)gridDim.x * blockDim.x)
    atomicAdd(&sh[e % COUT], __bfloat162float(dy[e]));
  __syncthreads();
  for (int n = threadIdx.x; n < COUT; n += blockDim.x) atomicAdd(&db[n], sh[n]);
}

// wT[c][tap][n] = w[n][8 - tap][c]: the weights of the input-gradient convolution.
__global__ void flip_weights_kernel(const bf16* __restrict__ w, bf16* __restrict__ wT, int cin, int cout) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= cin * 9 * cout) return;
  const int n = e % cout, tap = (e / cout) % 9, c = e / (cout * 9);
  wT[e] = w[((long long)n * 9 + (8 - tap)) * cin + c];
}

// x16[p][c] = c < 24 ? bf16(x[p][c]) : 0, c < 32. Bound by memory: a thread takes eight
// channels, one 16-byte store and, where x starts on a 16-byte boundary (VEC: rows are 96
// bytes, so every eight channels then do), two 16-byte loads; else eight single ones.
// (8 x 258 x 257, 85 MB: one channel per thread took 19.8 us.)
template <bool VEC>
__global__ void __launch_bounds__(256) pack_input_kernel(const float* __restrict__ x, bf16* __restrict__ x16, long long P) {
  static_assert(kCin[0] == 32 && kInReal == 24, "three groups of eight channels and one of zeros");
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < P * 4; e += (long long)gridDim.x * blockDim.x) {
    const int g = (int)(e & 3);
    float v[8] = {};
    if (g < 3) {
      const float* src = x + (e >> 2) * kInReal + 8 * g;
      if (VEC) {
        const float4 lo = __ldg(reinterpret_cast<const float4*>(src)), hi = __ldg(reinterpret_cast<const float4*>(src) + 1);
        v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w, v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
      } else {
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = __ldg(src + k);
      }
    }
    reinterpret_cast<uint4*>(x16)[e] = make_uint4(pack_pair(__float2bfloat16(v[0]), __float2bfloat16(v[1])),
                                                  pack_pair(__float2bfloat16(v[2]), __float2bfloat16(v[3])),
                                                  pack_pair(__float2bfloat16(v[4]), __float2bfloat16(v[5])),
                                                  pack_pair(__float2bfloat16(v[6]), __float2bfloat16(v[7])));
  }
}

// out3[p][c] = out16[p][c], c < 3
__global__ void unpack_output_kernel(const float* __restrict__ out16, float* __restrict__ out3, long long P) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < P * kOutReal;
       e += (long long)gridDim.x * blockDim.x)
    out3[e] = out16[(e / kOutReal) * 16 + e % kOutReal];
}

// Mean squared error over the 3 real channels; gradient (bf16, 16 channels) and the loss sum.
// Bound by memory: a thread takes a pixel, whose other 13 output channels it does not
// read (8 x 258 x 257: 40 MB moved instead of 57; one channel per thread took 17.0 us).
__global__ void mse_kernel(const float* __restrict__ out16, const float* __restrict__ target, bf16* __restrict__ d16,
                           float* __restrict__ loss, long long P) {
  static_assert(kOutReal == 3, "the first three channels");
  grid_dependency_wait();
  __shared__ float sh[256];
  float s = 0.f;
  const float scale = 2.f / (float)(P * kOutReal);
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const float4 o = __ldcg(reinterpret_cast<const float4*>(out16 + p * 16));
    const float r0 = o.x - target[3 * p], r1 = o.y - target[3 * p + 1], r2 = o.z - target[3 * p + 2];
    s += r0 * r0;
    s += r1 * r1;
    s += r2 * r2;
    uint4* d = reinterpret_cast<uint4*>(d16 + p * 16);
    d[0] = make_uint4(pack_pair(__float2bfloat16(scale * r0), __float2bfloat16(scale * r1)),
                      pack_pair(__float2bfloat16(scale * r2), __float2bfloat16(0.f)), 0u, 0u);
    d[1] = make_uint4(0u, 0u, 0u, 0u);
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, sh[0]);
}

// One layer's weights and what the training step keeps beside them.
struct LayerWeights {
  const float* part;  // the weight-gradient CTAs' partial sums [ctas][n]
  float *g, *p, *m, *v;
  bf16 *p16, *pT;     // the BF16 copy and the flipped, transposed one
  int n, cin, cout;
};

struct AllWeights {
  LayerWeights layer[kLayers];
};

// Volatile, so that a run of them stays ahead of the additions that use them.
__device__ __forceinline__ float ld_early(const float* p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// Every layer's weight gradient g[e] = sum over the weight-gradient CTAs of their partial
// sums, in CTA order (the same bits on every run), and with ADAM the step on the FP32
// master weights and their two BF16 copies, which the kernels read. With ADAM nothing is
// changed if a tensor-core kernel set *err.
// Bound by the latency of the loads: a thread's chain is `ctas` additions, so the loads
// are issued UN at a time ahead of them. One launch for the four layers: blockIdx.y.
// (One B x H x W = 8 x 258 x 257 step, 152 CTAs: a reduction per layer with one load per
// addition took 4 x 17.5 us, the Adam, copy and transpose launches 4 x 9.3 us.)
template <bool ADAM>
__global__ void __launch_bounds__(128) weight_step_kernel(const __grid_constant__ AllWeights a, int ctas, float lr,
                                                          float b1, float b2, float eps, float c1, float c2,
                                                          const int* __restrict__ err) {
  constexpr int UN = 38;
  grid_dependency_wait();
  const LayerWeights& w = a.layer[blockIdx.y];
  const int e = blockIdx.x * blockDim.x + threadIdx.x, n = w.n;
  if (e >= n || (ADAM && __ldcg(err))) return;
  float s = 0.f;
  const float* part = w.part + e;
  int c = 0;
  for (; c + UN <= ctas; c += UN) {
    float t[UN];
#pragma unroll
    for (int k = 0; k < UN; k++) t[k] = ld_early(part + (long long)(c + k) * n);
#pragma unroll
    for (int k = 0; k < UN; k++) s += t[k];
  }
  for (; c < ctas; c++) s += part[(long long)c * n];
  const float gg = 0.f + s;
  w.g[e] = gg;
  if (!ADAM) return;
  const float mm = b1 * w.m[e] + (1.f - b1) * gg;
  const float vv = b2 * w.v[e] + (1.f - b2) * gg * gg;
  w.m[e] = mm;
  w.v[e] = vv;
  const float upd = lr * (mm / c1) / (sqrtf(vv / c2) + eps);
  const float p = w.p[e] - upd;
  w.p[e] = p;
  const bf16 h = __float2bfloat16(p);
  w.p16[e] = h;
  const int ci = e % w.cin, tap = (e / w.cin) % 9, co = e / (9 * w.cin);
  w.pT[((long long)ci * 9 + (8 - tap)) * w.cout + co] = h;
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ a, bf16* __restrict__ b, int n) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) b[e] = __float2bfloat16(a[e]);
}

// Features of a layered wave state (AoS FP64 u, v, p on ny = blocks x block_rows
// rows of nx points) for the network. In the impedance-scaled variables
// q = (Z u, Z v, p), Z = sqrt(rho K), the coarse solve's error does not depend
// on the layer away from the interface (equal wave speeds). Per point, divided
// by the feature scale s (inv_scale = 1/s):
//   x[0..2]   = d2x q    undivided second differences along x,
//   x[3..5]   = d2y q    along y, within the point's block (no differencing
//                        across the interface line, which both blocks hold),
//   x[6..8]   = d4x q    undivided fourth differences along x,
//   x[9..11]  = d4y q    along y, within the block,
//   x[12..23] = t x[0..11]   t = +1 in block 0, -1 above (the layer tag),
// with each centre clamped one (two, for d4) point(s) in from an edge, so the
// difference is one-sided there. The differences are taken in FP64 before the
// network's BF16 rounding. The features are high-pass and linear in the state;
// the network's ReLU layers without biases are positively homogeneous, so a
// smooth or zero state gets a proportionally small or zero correction.
__device__ __forceinline__ void zq(const double* __restrict__ state, const double* __restrict__ rho,
                                   const double* __restrict__ K, long long p, double (&q)[3]) {
  const double z = sqrt(rho[p] * K[p]);
  q[0] = z * state[3 * p + 0];
  q[1] = z * state[3 * p + 1];
  q[2] = state[3 * p + 2];
}

// Second (D4 = false) or fourth (D4 = true) undivided difference of q at point p0 with stride st.
template <bool D4>
__device__ __forceinline__ void diff_q(const double* __restrict__ state, const double* __restrict__ rho,
                                       const double* __restrict__ K, long long p0, long long st, double (&d)[3]) {
  double a[3], b[3], m[3];
  zq(state, rho, K, p0, m);
  if (!D4) {
    zq(state, rho, K, p0 - st, a);
    zq(state, rho, K, p0 + st, b);
    for (int c = 0; c < 3; c++) d[c] = a[c] - 2.0 * m[c] + b[c];
  } else {
    double a2[3], b2[3];
    zq(state, rho, K, p0 - 2 * st, a2);
    zq(state, rho, K, p0 - st, a);
    zq(state, rho, K, p0 + st, b);
    zq(state, rho, K, p0 + 2 * st, b2);
    for (int c = 0; c < 3; c++) d[c] = a2[c] - 4.0 * a[c] + 6.0 * m[c] - 4.0 * b[c] + b2[c];
  }
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__global__ void features_kernel(const double* __restrict__ state, const double* __restrict__ rho,
                                const double* __restrict__ K, float* __restrict__ x, int nx, int ny, int block_rows,
                                double inv_scale) {
  const long long P = (long long)nx * ny;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(p / nx), i = (int)(p % nx);
    const int b = j / block_rows, r = j % block_rows;
    const long long row0 = (long long)b * block_rows;
    double f[12], d[3];
    diff_q<false>(state, rho, K, (long long)j * nx + clampi(i, 1, nx - 2), 1, d);
    for (int c = 0; c < 3; c++) f[c] = d[c];
    diff_q<false>(state, rho, K, (row0 + clampi(r, 1, block_rows - 2)) * nx + i, nx, d);
    for (int c = 0; c < 3; c++) f[3 + c] = d[c];
    diff_q<true>(state, rho, K, (long long)j * nx + clampi(i, 2, nx - 3), 1, d);
    for (int c = 0; c < 3; c++) f[6 + c] = d[c];
    diff_q<true>(state, rho, K, (row0 + clampi(r, 2, block_rows - 3)) * nx + i, nx, d);
    for (int c = 0; c < 3; c++) f[9 + c] = d[c];
    const double t = b == 0 ? 1.0 : -1.0;
    for (int c = 0; c < 12; c++) {
      x[(long long)kInReal * p + c] = (float)(f[c] * inv_scale);
      x[(long long)kInReal * p + 12 + c] = (float)(t * f[c] * inv_scale);
    }
  }
}

// The network's output is a correction of q = (Z u, Z v, p) in units of `scale`:
// state[p] += scale * (delta[p][0] / Z, delta[p][1] / Z, delta[p][2]).
__global__ void correct_kernel(double* __restrict__ state, const float* __restrict__ delta,
                               const double* __restrict__ rho, const double* __restrict__ K, long long P,
                               double scale) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const double zi = scale / sqrt(rho[p] * K[p]);
    state[3 * p + 0] += zi * (double)delta[3 * p + 0];
    state[3 * p + 1] += zi * (double)delta[3 * p + 1];
    state[3 * p + 2] += scale * (double)delta[3 * p + 2];
  }
}

inline int blocks_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  return (int)(b > 4096 ? 4096 : (b < 1 ? 1 : b));
}

}  // namespace cnn
}  // namespace sbp

using namespace sbp::cnn;

struct sbp_cnn {
  int H = 0, W = 0, maxB = 0, device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  long long step = 0;
  float* wm[kLayers] = {};   // FP32 master weights [cout][9][cin]
  bf16* wb[kLayers] = {};    // BF16 copies
  bf16* wT[kLayers] = {};    // flipped, transposed (input-gradient) weights
  float* bias[kLayers] = {};
  float *mw[kLayers] = {}, *vw[kLayers] = {}, *mbias[kLayers] = {}, *vbias[kLayers] = {};
  float *gw[kLayers] = {}, *gb[kLayers] = {};
  bf16* act[kLayers] = {};   // layer inputs: act[0] = packed input, act[l] = output of layer l-1
  bf16* dact = nullptr;      // gradient buffers (two, ping-pong)
  bf16* dact2 = nullptr;
  float* out16 = nullptr;    // last layer output (FP32, 16 channels)
  float* loss = nullptr;
  int* err = nullptr;        // the tensor-core convolutions' error word (a bounded wait ran out)
  int tw = 0, th = 0;        // the tensor-core kernels' pixel tile: th rows of tw pixels, th * tw = 128
  bool turned = false;       // whether those rows run down the image instead of along it
  int across() const { return turned ? W : H; }  // the image's extent across a tile's rows, and along them
  int along() const { return turned ? H : W; }
  // pixel tiles of a batch
  long long tiles(int batch) const {
    return (long long)batch * ((across() + th - 1) / th) * ((along() + tw - 1) / tw);
  }
  int nsm = 1;               // SMs: the persistent convolutions' grid
  float* dw_part[kLayers] = {};  // the weight gradients' per-CTA sums ([nsm][wcount(l)] each, one block)
  long long launches = 0;
  std::string msg;
};

namespace {

thread_local std::string g_cnn_error;

int cfail(sbp_cnn* c, int code, const std::string& m) {
  if (c) c->msg = m;
  else g_cnn_error = m;
  return code;
}

#define CCK(call)                                                                        \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      return cfail(c, SBP_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

long long wcount(int l) { return (long long)kCout[l] * 9 * kCin[l]; }

void cnn_release(sbp_cnn* c) {
  for (int l = 0; l < kLayers; l++) {
    void* ps[] = {c->wm[l], c->wb[l], c->wT[l], c->bias[l], c->mw[l], c->vw[l], c->mbias[l], c->vbias[l],
                  c->gw[l], c->gb[l], c->act[l]};
    for (void* p : ps)
      if (p) cudaFree(p);
  }
  void* ps[] = {c->dact, c->dact2, c->out16, c->loss, c->err, c->dw_part[0]};
  for (void* p : ps)
    if (p) cudaFree(p);
  if (c->own_stream && c->stream) cudaStreamDestroy(c->stream);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// The tensor maps of one convolution: the NHWC BF16 input ({ch, W, H, B}, turned {ch, H, W, B},
// box {ch, bw, bh, 1}) and the weights ([cout][9][ch]: {ch, 9, cout}, box {ch, 1, cout}), rows
// swizzled over their ch * 2 bytes. Out-of-range boxes read zeros (the image border).
cudaError_t encode_conv_maps(const sbp_cnn* c, const bf16* x, const bf16* w, int ch, int cout, int batch, int bw,
                             int bh, CUtensorMap* xm, CUtensorMap* wm) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  const CUtensorMapSwizzle sw = ch == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
  const cuuint64_t xd[4] = {(cuuint64_t)ch, (cuuint64_t)c->along(), (cuuint64_t)c->across(), (cuuint64_t)batch};
  const cuuint64_t px = (cuuint64_t)ch * 2, row = (cuuint64_t)c->W * ch * 2;
  const cuuint64_t xs[3] = {c->turned ? row : px, c->turned ? px : row, (cuuint64_t)c->H * row};
  const cuuint32_t xb[4] = {(cuuint32_t)ch, (cuuint32_t)bw, (cuuint32_t)bh, 1};
  const cuuint32_t e[4] = {1, 1, 1, 1};
  if (enc(xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(x), xd, xs, xb, e, CU_TENSOR_MAP_INTERLEAVE_NONE,
          sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  const cuuint64_t wd[3] = {(cuuint64_t)ch, 9, (cuuint64_t)cout};
  const cuuint64_t ws[2] = {(cuuint64_t)ch * 2, (cuuint64_t)9 * ch * 2};
  const cuuint32_t wbx[3] = {(cuuint32_t)ch, 1, (cuuint32_t)cout};
  if (enc(wm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(w), wd, ws, wbx, e, CU_TENSOR_MAP_INTERLEAVE_NONE,
          sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  return cudaSuccess;
}

template <int CIN, int COUT, bool RELU, bool OUT_F32, bool MASK>
cudaError_t configure_tc() {
  return cudaFuncSetAttribute(conv3x3_tc_kernel<CIN, COUT, RELU, OUT_F32, MASK>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, TcConv<CIN, COUT>::SMEM_MAX);
}

template <int CIN, int COUT, bool RELU, bool OUT_F32, bool MASK>
cudaError_t launch_tc(const bf16* x, const bf16* w, const float* bias, const bf16* mask, void* y, const sbp_cnn* c,
                      int batch, cudaStream_t s) {
  CUtensorMap xm, wm;
  cudaError_t e = encode_conv_maps(c, x, w, CIN, COUT, batch, c->tw, c->th + 2, &xm, &wm);
  if (e != cudaSuccess) return e;
  const long long tiles = c->tiles(batch);
  const long long slots = (long long)TcConv<CIN, COUT>::CTAS * c->nsm;  // persistent: every CTA resident
  const unsigned grid = (unsigned)(tiles < slots ? tiles : slots);
  return sbp::launch_overlapped(conv3x3_tc_kernel<CIN, COUT, RELU, OUT_F32, MASK>, dim3(grid),
                           dim3(TcConv<CIN, COUT>::THREADS), TcConv<CIN, COUT>::smem(c->tw), s, xm, wm, bias, mask, y,
                           batch, c->across(), c->along(), c->tw, c->th, c->turned, c->err);
}

template <int COUT>
cudaError_t configure_wgrad_tc() {
  return cudaFuncSetAttribute(conv3x3_wgrad_tc_kernel<COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              TcWgrad<COUT>::SMEM_MAX);
}

// Shared-memory opt-in of the tensor-core convolutions (outside stream capture).
cudaError_t configure_convs() {
  cudaError_t e;
  if ((e = configure_tc<32, 32, true, false, false>()) != cudaSuccess) return e;
  if ((e = configure_tc<32, 16, false, true, false>()) != cudaSuccess) return e;
  if ((e = configure_tc<32, 32, false, false, true>()) != cudaSuccess) return e;
  if ((e = configure_tc<16, 32, false, false, true>()) != cudaSuccess) return e;
  if ((e = configure_wgrad_tc<32>()) != cudaSuccess) return e;
  return configure_wgrad_tc<16>();
}

// Launch one conv of layer l (forward), or its input-gradient conv with the ReLU
// backward pass through the layer's input.
cudaError_t conv_fwd(int l, const bf16* x, void* y, const sbp_cnn* c, int batch, cudaStream_t s) {
  if (l < kLayers - 1) return launch_tc<32, 32, true, false, false>(x, c->wb[l], c->bias[l], nullptr, y, c, batch, s);
  return launch_tc<32, 16, false, true, false>(x, c->wb[l], c->bias[l], nullptr, y, c, batch, s);
}

cudaError_t conv_dgrad(int l, const bf16* dy, bf16* dx, const sbp_cnn* c, int batch, cudaStream_t s) {
  if (l == kLayers - 1) return launch_tc<16, 32, false, false, true>(dy, c->wT[l], nullptr, c->act[l], dx, c, batch, s);
  return launch_tc<32, 32, false, false, true>(dy, c->wT[l], nullptr, c->act[l], dx, c, batch, s);
}

// CTAs of the weight gradients: each leaves one partial sum.
unsigned wgrad_ctas(const sbp_cnn* c, int batch) {
  const long long tiles = c->tiles(batch);
  return (unsigned)(tiles < c->nsm ? tiles : c->nsm);
}

// Partial sums of the weight gradient of layer l (x: its input, 32 channels; dy: its output gradient).
cudaError_t conv_wgrad(int l, const bf16* x, const bf16* dy, const sbp_cnn* c, int batch, cudaStream_t s) {
  CUtensorMap xm, dym, unused;
  const int cout = kCout[l];
  // x: 32-channel tap tiles; dy: one unshifted tile of cout channels (its map from the same
  // encoder, with dy as the "input" and the weights map unused)
  cudaError_t e = encode_conv_maps(c, x, c->wb[l], 32, cout, batch, c->tw, c->th + 2, &xm, &unused);
  if (e == cudaSuccess) e = encode_conv_maps(c, dy, c->wb[l], cout, cout, batch, c->tw, c->th, &dym, &unused);
  if (e != cudaSuccess) return e;
  const unsigned grid = wgrad_ctas(c, batch);
  if (cout == 32)
    return sbp::launch_overlapped(conv3x3_wgrad_tc_kernel<32>, dim3(grid), dim3(TcWgrad<32>::THREADS),
                             TcWgrad<32>::smem(c->tw), s, xm, dym, c->dw_part[l], batch, c->across(), c->along(), c->tw,
                             c->th, c->turned, c->err);
  return sbp::launch_overlapped(conv3x3_wgrad_tc_kernel<16>, dim3(grid), dim3(TcWgrad<16>::THREADS),
                           TcWgrad<16>::smem(c->tw), s, xm, dym, c->dw_part[l], batch, c->across(), c->along(), c->tw,
                           c->th, c->turned, c->err);
}

AllWeights all_weights(const sbp_cnn* c) {
  AllWeights a;
  for (int l = 0; l < kLayers; l++)
    a.layer[l] = LayerWeights{c->dw_part[l], c->gw[l], c->wm[l], c->mw[l], c->vw[l], c->wb[l], c->wT[l],
                              (int)wcount(l), kCin[l], kCout[l]};
  return a;
}

inline dim3 weight_step_grid() {
  long long n = 0;
  for (int l = 0; l < kLayers; l++) n = std::max(n, wcount(l));
  return dim3((unsigned)((n + 127) / 128), kLayers);
}

cudaError_t bias_grad(int l, const bf16* dy, float* db, int batch, const sbp_cnn* c, cudaStream_t s) {
  const long long P = (long long)batch * c->H * c->W;
  if (kCout[l] == 32)
    bias_grad_kernel<32><<<blocks_for(P * 32, 256), 256, 0, s>>>(dy, db, P);
  else
    bias_grad_kernel<16><<<blocks_for(P * 16, 256), 256, 0, s>>>(dy, db, P);
  return cudaGetLastError();
}

int refresh_weights(sbp_cnn* c) {
  for (int l = 0; l < kLayers; l++) {
    const int n = (int)wcount(l);
    f32_to_bf16_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(c->wm[l], c->wb[l], n);
    flip_weights_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(c->wb[l], c->wT[l], kCin[l], kCout[l]);
    c->launches += 2;
  }
  CCK(cudaGetLastError());
  return SBP_OK;
}

int run_forward(sbp_cnn* c, const float* x, int batch) {
  const long long P = (long long)batch * c->H * c->W;
  if (reinterpret_cast<uintptr_t>(x) % 16 == 0)
    pack_input_kernel<true><<<blocks_for(P * 4, 256), 256, 0, c->stream>>>(x, c->act[0], P);
  else
    pack_input_kernel<false><<<blocks_for(P * 4, 256), 256, 0, c->stream>>>(x, c->act[0], P);
  c->launches++;
  for (int l = 0; l < kLayers; l++) {
    void* y = (l == kLayers - 1) ? (void*)c->out16 : (void*)c->act[l + 1];
    CCK(conv_fwd(l, c->act[l], y, c, batch, c->stream));
    c->launches++;
  }
  return SBP_OK;
}

// Masks that keep padded channels of parameters at zero (never trained).
bool weight_is_real(int l, long long e) {
  const int cin = kCin[l];
  const int ci = (int)(e % cin);
  const int n = (int)(e / (9LL * cin));
  if (l == 0 && ci >= kInReal) return false;
  if (l == kLayers - 1 && n >= kOutReal) return false;
  return true;
}

}  // namespace

extern "C" {

int sbp_cnn_create(int height, int width, int max_batch, int device, void* stream, sbp_cnn** out) {
  if (!out || height < 1 || width < 1 || max_batch < 1) return cfail(nullptr, SBP_ERR_INVALID, "bad network size");
  *out = nullptr;
  sbp_cnn* c = new (std::nothrow) sbp_cnn();
  if (!c) return cfail(nullptr, SBP_ERR_INVALID, "out of host memory");
  c->H = height;
  c->W = width;
  c->maxB = max_batch;
  c->device = device;
  auto bad = [&](const std::string& m) {
    g_cnn_error = m;
    cnn_release(c);
    delete c;
    return SBP_ERR_CUDA;
  };
  if (cudaSetDevice(device) != cudaSuccess) return bad("cudaSetDevice failed");
  if (stream) {
    c->stream = (cudaStream_t)stream;
  } else {
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) return bad("stream");
    c->own_stream = true;
  }
  const long long P = (long long)max_batch * height * width;
  for (int l = 0; l < kLayers; l++) {
    const size_t nw = (size_t)wcount(l), nb = (size_t)kCout[l];
    if (cudaMalloc(&c->wm[l], nw * 4) || cudaMalloc(&c->wb[l], nw * 2) || cudaMalloc(&c->wT[l], nw * 2) ||
        cudaMalloc(&c->bias[l], nb * 4) || cudaMalloc(&c->mw[l], nw * 4) || cudaMalloc(&c->vw[l], nw * 4) ||
        cudaMalloc(&c->mbias[l], nb * 4) || cudaMalloc(&c->vbias[l], nb * 4) || cudaMalloc(&c->gw[l], nw * 4) ||
        cudaMalloc(&c->gb[l], nb * 4) || cudaMalloc(&c->act[l], (size_t)P * kCin[l] * 2))
      return bad("cudaMalloc(network)");
    cudaMemset(c->mw[l], 0, nw * 4);
    cudaMemset(c->vw[l], 0, nw * 4);
    cudaMemset(c->mbias[l], 0, nb * 4);
    cudaMemset(c->vbias[l], 0, nb * 4);
  }
  if (cudaMalloc(&c->dact, (size_t)P * 32 * 2) || cudaMalloc(&c->dact2, (size_t)P * 32 * 2) ||
      cudaMalloc(&c->out16, (size_t)P * 16 * 4) || cudaMalloc(&c->loss, 4) || cudaMalloc(&c->err, 4))
    return bad("cudaMalloc(activations)");
  cudaMemset(c->err, 0, 4);
  // the tensor-core kernels' tile: 128 pixels, th rows of tw, the shape whose tiles cover the
  // image with the fewest padding pixels (ties: the first tried). tw >= 8: a row of pixels is
  // whole swizzle atoms, so that the vertical taps can start at any row of a box; tw <= 32: wider
  // tiles' boxes are mostly halo (64: 4 rows for 2) and five of them overfill shared memory.
  // Images up to four pixels wide turn the tile, one or two pixels high or wide take 64 x 2:
  // forward pass at 8 x 32768 x 1 122 us (with upright tiles of 8 x 16 pixels 282), 8 x 1 x 32768
  // 122 (32 x 4 pixels: 160), 8 x 20000 x 3 135 (201).
  long long best = -1;
  for (int t = 0; t < (width <= 4 ? 2 : 1); t++) {
    const int along = t ? height : width, across = t ? width : height;
    for (int tw : {32, 16, 8, kConvStripTw}) {
      if (tw > kConvMaxTw && across > 2) continue;
      const int th = 128 / tw;
      const long long area = (long long)((along + tw - 1) / tw) * tw * ((across + th - 1) / th) * th;
      if (best < 0 || area < best) {
        best = area;
        c->tw = tw;
        c->th = th;
        c->turned = t != 0;
      }
    }
  }
  if (configure_convs() != cudaSuccess) return bad("cudaFuncSetAttribute(convolutions)");
  if (cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || c->nsm < 1)
    return bad("cudaDeviceGetAttribute(SMs)");
  long long sums = 0;
  for (int l = 0; l < kLayers; l++) sums += wcount(l);
  if (cudaMalloc(&c->dw_part[0], (size_t)(c->nsm * sums) * sizeof(float)) != cudaSuccess)
    return bad("cudaMalloc(weight-gradient partial sums)");
  for (int l = 1; l < kLayers; l++) c->dw_part[l] = c->dw_part[l - 1] + c->nsm * wcount(l - 1);
  if (!encode_fn()) return bad("cuTensorMapEncodeTiled is not available from the driver");
  // a network that failed its initialisation is released, not handed out
  const int rc = sbp_cnn_init(c, 1234);
  if (rc) {
    g_cnn_error = c->msg;
    cnn_release(c);
    delete c;
    return rc;
  }
  *out = c;
  return SBP_OK;
}

int sbp_cnn_destroy(sbp_cnn* c) {
  if (!c) return SBP_ERR_INVALID;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  cnn_release(c);
  delete c;
  return SBP_OK;
}

const char* sbp_cnn_last_error(const sbp_cnn* c) { return c ? c->msg.c_str() : g_cnn_error.c_str(); }

long long sbp_cnn_param_count(void) {
  long long n = 0;
  for (int l = 0; l < kLayers; l++) n += wcount(l) + kCout[l];
  return n;
}

int sbp_cnn_init(sbp_cnn* c, unsigned long long seed) {
  if (!c) return SBP_ERR_INVALID;
  CCK(cudaSetDevice(c->device));
  std::mt19937_64 rng(seed);
  for (int l = 0; l < kLayers; l++) {
    const long long n = wcount(l);
    const int fan_in = 9 * (l == 0 ? kInReal : kCin[l]);
    // He-normal hidden layers; the output layer starts at zero, so the untrained network is the
    // zero correction and training moves away from it only where that lowers the error.
    std::normal_distribution<double> nd(0.0, std::sqrt(2.0 / fan_in) * (l == kLayers - 1 ? 0.0 : 1.0));
    std::vector<float> w(n);
    for (long long e = 0; e < n; e++) w[e] = weight_is_real(l, e) ? (float)nd(rng) : 0.f;
    std::vector<float> b(kCout[l], 0.f);
    CCK(cudaMemcpyAsync(c->wm[l], w.data(), n * 4, cudaMemcpyHostToDevice, c->stream));
    CCK(cudaMemcpyAsync(c->bias[l], b.data(), b.size() * 4, cudaMemcpyHostToDevice, c->stream));
    CCK(cudaMemsetAsync(c->mw[l], 0, n * 4, c->stream));
    CCK(cudaMemsetAsync(c->vw[l], 0, n * 4, c->stream));
    CCK(cudaMemsetAsync(c->mbias[l], 0, kCout[l] * 4, c->stream));
    CCK(cudaMemsetAsync(c->vbias[l], 0, kCout[l] * 4, c->stream));
  }
  c->step = 0;
  int rc = refresh_weights(c);
  if (rc) return rc;
  CCK(cudaStreamSynchronize(c->stream));
  return SBP_OK;
}

// Parameters as one FP32 vector: per layer, weights [cout][9][cin] then bias [cout].
int sbp_cnn_get_params(sbp_cnn* c, float* host, long long n) {
  if (!c || !host || n != sbp_cnn_param_count()) return SBP_ERR_INVALID;
  CCK(cudaSetDevice(c->device));
  long long o = 0;
  for (int l = 0; l < kLayers; l++) {
    CCK(cudaMemcpyAsync(host + o, c->wm[l], wcount(l) * 4, cudaMemcpyDeviceToHost, c->stream));
    o += wcount(l);
    CCK(cudaMemcpyAsync(host + o, c->bias[l], kCout[l] * 4, cudaMemcpyDeviceToHost, c->stream));
    o += kCout[l];
  }
  CCK(cudaStreamSynchronize(c->stream));
  return SBP_OK;
}

int sbp_cnn_set_params(sbp_cnn* c, const float* host, long long n) {
  if (!c || !host || n != sbp_cnn_param_count()) return SBP_ERR_INVALID;
  CCK(cudaSetDevice(c->device));
  long long o = 0;
  for (int l = 0; l < kLayers; l++) {
    CCK(cudaMemcpyAsync(c->wm[l], host + o, wcount(l) * 4, cudaMemcpyHostToDevice, c->stream));
    o += wcount(l);
    CCK(cudaMemcpyAsync(c->bias[l], host + o, kCout[l] * 4, cudaMemcpyHostToDevice, c->stream));
    o += kCout[l];
  }
  int rc = refresh_weights(c);
  if (rc) return rc;
  CCK(cudaStreamSynchronize(c->stream));
  return SBP_OK;
}

// out = network(x): x, out device arrays, NHWC FP32, 4 and 3 channels.
int sbp_cnn_forward(sbp_cnn* c, const float* x, int batch, float* out) {
  if (!c || !x || !out || batch < 1 || batch > c->maxB) return SBP_ERR_INVALID;
  CCK(cudaSetDevice(c->device));
  int rc = run_forward(c, x, batch);
  if (rc) return rc;
  const long long P = (long long)batch * c->H * c->W;
  unpack_output_kernel<<<blocks_for(P * 3, 256), 256, 0, c->stream>>>(c->out16, out, P);
  c->launches++;
  int e = 0;
  CCK(cudaMemcpyAsync(&e, c->err, 4, cudaMemcpyDeviceToHost, c->stream));
  CCK(cudaStreamSynchronize(c->stream));
  if (e) {
    CCK(cudaMemsetAsync(c->err, 0, 4, c->stream));
    return cfail(c, SBP_ERR_DEVICE, "a tensor-core convolution's wait for its tiles ran out");
  }
  return SBP_OK;
}

// Gradients of the mean squared error of network(x) against target (both device, NHWC FP32,
// 4 and 3 channels), without updating the parameters; written as one FP32 vector in the
// layout of sbp_cnn_get_params (host `grad`, may be NULL). Returns the loss in *loss.
// lr > 0: the training step, which updates the weights (biases stay untrained, their gradients are skipped).
static int backward(sbp_cnn* c, const float* x, const float* target, int batch, float* loss, float lr) {
  const bool train = lr > 0;
  const long long P = (long long)batch * c->H * c->W;
  CCK(cudaMemsetAsync(c->loss, 0, 4, c->stream));
  int rc = run_forward(c, x, batch);
  if (rc) return rc;
  CCK(sbp::launch_overlapped(mse_kernel, dim3(blocks_for(P, 256)), dim3(256), 0, c->stream, c->out16, target, c->dact,
                        c->loss, P));
  c->launches++;
  if (!train)
    for (int l = 0; l < kLayers; l++) CCK(cudaMemsetAsync(c->gb[l], 0, kCout[l] * 4, c->stream));
  bf16* dcur = c->dact;   // gradient w.r.t. the output of layer l (pre-activation once masked)
  bf16* dnext = c->dact2;
  for (int l = kLayers - 1; l >= 0; l--) {
    CCK(conv_wgrad(l, c->act[l], dcur, c, batch, c->stream));
    c->launches++;
    if (!train) {
      CCK(bias_grad(l, dcur, c->gb[l], batch, c, c->stream));
      c->launches++;
    }
    if (l == 0) break;
    CCK(conv_dgrad(l, dcur, dnext, c, batch, c->stream));
    c->launches++;
    bf16* tmp = dcur;
    dcur = dnext;
    dnext = tmp;
  }
  const AllWeights a = all_weights(c);
  const int ctas = (int)wgrad_ctas(c, batch);
  if (train) {
    const float b1 = 0.9f, b2 = 0.999f, t = (float)(c->step + 1);
    const float c1 = 1.f - std::pow(b1, t), c2 = 1.f - std::pow(b2, t);
    // padded channels stay zero: their gradients are zero (zero inputs / zero targets) and
    // Adam leaves zero-gradient entries unchanged.
    CCK(sbp::launch_overlapped(weight_step_kernel<true>, weight_step_grid(), dim3(128), 0, c->stream, a, ctas, lr, b1, b2,
                          1e-8f, c1, c2, c->err));
  } else {
    CCK(sbp::launch_overlapped(weight_step_kernel<false>, weight_step_grid(), dim3(128), 0, c->stream, a, ctas, 0.f, 0.f,
                          0.f, 0.f, 1.f, 1.f, c->err));
  }
  c->launches++;
  float h = 0;
  int e = 0;
  CCK(cudaMemcpyAsync(&h, c->loss, 4, cudaMemcpyDeviceToHost, c->stream));
  CCK(cudaMemcpyAsync(&e, c->err, 4, cudaMemcpyDeviceToHost, c->stream));
  CCK(cudaStreamSynchronize(c->stream));
  if (e) {
    CCK(cudaMemsetAsync(c->err, 0, 4, c->stream));
    return cfail(c, SBP_ERR_DEVICE, "a tensor-core convolution's wait for its tiles ran out");
  }
  if (train) c->step++;
  if (loss) *loss = h / (float)(P * kOutReal);
  return SBP_OK;
}

int sbp_cnn_gradients(sbp_cnn* c, const float* x, const float* target, int batch, float* grad, long long n,
                      float* loss) {
  if (!c || !x || !target || batch < 1 || batch > c->maxB) return SBP_ERR_INVALID;
  if (grad && n != sbp_cnn_param_count()) return SBP_ERR_INVALID;
  CCK(cudaSetDevice(c->device));
  int rc = backward(c, x, target, batch, loss, 0.f);
  if (rc || !grad) return rc;
  long long o = 0;
  for (int l = 0; l < kLayers; l++) {
    CCK(cudaMemcpyAsync(grad + o, c->gw[l], wcount(l) * 4, cudaMemcpyDeviceToHost, c->stream));
    o += wcount(l);
    CCK(cudaMemcpyAsync(grad + o, c->gb[l], kCout[l] * 4, cudaMemcpyDeviceToHost, c->stream));
    o += kCout[l];
  }
  CCK(cudaStreamSynchronize(c->stream));
  return SBP_OK;
}

// One Adam step (beta1 0.9, beta2 0.999, eps 1e-8) on the mean squared error.
// Weights are trained; biases keep their values (zero from sbp_cnn_init), so
// the trained network maps zero features to zero outputs.
int sbp_cnn_train_step(sbp_cnn* c, const float* x, const float* target, int batch, float lr, float* loss) {
  if (!c || !x || !target || batch < 1 || batch > c->maxB || !(lr > 0)) return SBP_ERR_INVALID;
  CCK(cudaSetDevice(c->device));
  return backward(c, x, target, batch, loss, lr);
}

int sbp_cnn_features(const double* state, const double* rho, const double* K, int nx, int ny, int block_rows,
                     double inv_scale, float* x, void* stream) {
  if (!state || !rho || !K || !x || nx < 5 || block_rows < 5 || ny < block_rows || ny % block_rows)
    return SBP_ERR_INVALID;
  const long long P = (long long)nx * ny;
  features_kernel<<<blocks_for(P, 256), 256, 0, (cudaStream_t)stream>>>(state, rho, K, x, nx, ny, block_rows,
                                                                        inv_scale);
  return cudaGetLastError() == cudaSuccess ? SBP_OK : SBP_ERR_CUDA;
}

int sbp_cnn_correct(double* state, const float* delta, const double* rho, const double* K, long long npts,
                    double scale, void* stream) {
  if (!state || !delta || !rho || !K || npts < 1) return SBP_ERR_INVALID;
  correct_kernel<<<blocks_for(npts, 256), 256, 0, (cudaStream_t)stream>>>(state, delta, rho, K, npts, scale);
  return cudaGetLastError() == cudaSuccess ? SBP_OK : SBP_ERR_CUDA;
}

long long sbp_cnn_launch_count(const sbp_cnn* c) { return c ? c->launches : SBP_ERR_INVALID; }

}  // extern "C"

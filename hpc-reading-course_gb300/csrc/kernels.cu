// kernels.cu -- launchers for the scalar/1D stage kernels, the AoS <-> SoA
// layout kernels at the reference boundary, the FP64 norm reductions and the
// FP64 throughput probe.
#include "adv_cell.cuh"
#include "launch.h"
#include "line_steps.cuh"

namespace sbp {

int wave_smem_bytes(int order, bool fp32) {
  switch (order) {
    case 2: return fp32 ? WaveStageTile<float, 2, WK_HOM, ST_MID>::SMEM : WaveStageTile<double, 2, WK_HOM, ST_MID>::SMEM;
    case 4: return fp32 ? WaveStageTile<float, 4, WK_HOM, ST_MID>::SMEM : WaveStageTile<double, 4, WK_HOM, ST_MID>::SMEM;
    case 6: return fp32 ? WaveStageTile<float, 6, WK_HOM, ST_MID>::SMEM : WaveStageTile<double, 6, WK_HOM, ST_MID>::SMEM;
    default: return -1;
  }
}

int device_sm_count() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 148;
  if (dev < 64 && cache[dev]) return cache[dev];
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  if (dev < 64) cache[dev] = n;
  return n;
}

// ---------------------------------------------------------------- line kernels
namespace {
template <int ORD, bool FIELDS, int ROWS>
cudaError_t adv_cell_stage(int stage, const LineParams<double>& prm, cudaStream_t s) {
  constexpr int TY = kCellThreads / 32 * ROWS;
  const dim3 grid((prm.nx + kCellTX - 1) / kCellTX, (prm.ny + TY - 1) / TY);
  switch (stage) {
    case ST_RHS: return launch_overlapped(adv_cell_kernel<ORD, ST_RHS, FIELDS, ROWS>, grid, kCellThreads, 0, s, prm);
    case ST_FIRST: return launch_overlapped(adv_cell_kernel<ORD, ST_FIRST, FIELDS, ROWS>, grid, kCellThreads, 0, s, prm);
    case ST_MID: return launch_overlapped(adv_cell_kernel<ORD, ST_MID, FIELDS, ROWS>, grid, kCellThreads, 0, s, prm);
    case ST_LAST: return launch_overlapped(adv_cell_kernel<ORD, ST_LAST, FIELDS, ROWS>, grid, kCellThreads, 0, s, prm);
    default: return cudaErrorInvalidValue;
  }
}

template <typename T, int ORD, int KIND>
cudaError_t line_stage(int stage, const LineParams<T>& prm, cudaStream_t s) {
  if constexpr (KIND == LK_ADV2D && sizeof(T) == 8) {
    // us per stage, line form / cells of one row per thread: order 2 201^2 3.8 / 3.8, 257^2 4.0 /
    // 4.3, 801x101 4.1 / 3.8, 361^2 5.4 / 4.6, 513^2 8.5 / 5.3; order 4 161^2 3.5 / 3.7, 201^2 4.9 /
    // 3.5, 513^2 12.0 / 6.1; order 6 161^2 4.1 / 4.5, 201^2 5.9 / 4.5. With velocity fields: order 2
    // 257^2 5.9 / 7.8, 361^2 7.5 / 8.1, 401^2 8.2 / 8.1, 513^2 13.5 / 9.3; order 4 161^2 4.6 / 6.0,
    // 201^2 6.7 / 5.9, 257^2 6.8 / 7.0, 361^2 9.0 / 7.7; order 6 161^2 5.3 / 7.2, 201^2 7.7 / 6.7.
    // Cells of one / two rows: 513^2 5.3 / 6.0, 6.1 / 6.4, 7.3 / 7.3 at orders 2, 4 and 6, 801^2 9.1 /
    // 9.0, 10.7 / 10.4, 12.9 / 12.2, 2049^2 48 / 44, 57 / 50, 69 / 59; with fields 801^2 14.7 / 16.0,
    // 15.4 / 16.5, 16.7 / 17.5, 1001^2 19.7 / 20.7, 20.6 / 21.4, 22.6 / 22.7, 2049^2 71 / 68, 79 / 73,
    // 89 / 77.
    const long long points = (long long)prm.nx * prm.ny;
    if (points > (ORD == 2 ? (prm.va ? 160000 : 80000) : 40000)) {
      if (points <= (prm.va ? 1100000 : 450000))
        return prm.va ? adv_cell_stage<ORD, true, 1>(stage, prm, s) : adv_cell_stage<ORD, false, 1>(stage, prm, s);
      return prm.va ? adv_cell_stage<ORD, true, 2>(stage, prm, s) : adv_cell_stage<ORD, false, 2>(stage, prm, s);
    }
  }
  const dim3 block(KIND == LK_ADV2D ? 32 : 128, KIND == LK_ADV2D ? 8 : 1);
  const dim3 grid((prm.nx + block.x - 1) / block.x, (prm.ny + block.y - 1) / block.y);
  switch (stage) {
    case ST_RHS: line_stage_kernel<T, ORD, KIND, ST_RHS><<<grid, block, 0, s>>>(prm); break;
    case ST_FIRST: line_stage_kernel<T, ORD, KIND, ST_FIRST><<<grid, block, 0, s>>>(prm); break;
    case ST_MID: line_stage_kernel<T, ORD, KIND, ST_MID><<<grid, block, 0, s>>>(prm); break;
    case ST_LAST: line_stage_kernel<T, ORD, KIND, ST_LAST><<<grid, block, 0, s>>>(prm); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <typename T, int ORD>
cudaError_t line_order(int kind, int stage, const LineParams<T>& prm, cudaStream_t s) {
  switch (kind) {
    case LK_ADV1D: return line_stage<T, ORD, LK_ADV1D>(stage, prm, s);
    case LK_REFL1D: return line_stage<T, ORD, LK_REFL1D>(stage, prm, s);
    case LK_ADV2D: return line_stage<T, ORD, LK_ADV2D>(stage, prm, s);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace

template <typename T>
cudaError_t launch_line(int order, int kind, int stage, const LineParams<T>& prm, cudaStream_t s) {
  switch (order) {
    case 2: return line_order<T, 2>(kind, stage, prm, s);
    case 4: return line_order<T, 4>(kind, stage, prm, s);
    case 6: return line_order<T, 6>(kind, stage, prm, s);
    default: return cudaErrorInvalidValue;
  }
}
template cudaError_t launch_line<double>(int, int, int, const LineParams<double>&, cudaStream_t);
template cudaError_t launch_line<float>(int, int, int, const LineParams<float>&, cudaStream_t);

// ---------------------------------------------------------------- 1D step loops
namespace {
// CTAs of the cluster: 128 points each, up to the eight CTAs that every device can place
// (32 to 128 points per CTA measured the same, 256 or more slower: 201 points 3.4 us a step
// at 128, 3.8 at 256; 1601 points 4.0 at 8 CTAs, 5.5 at 512 points each).
inline int line_ctas(long long nx) {
  long long c = (nx + 127) / 128;
  if (c > kLineMaxCtas) c = kLineMaxCtas;
  while (c > 1 && nx / c < kLineMinChunk) c--;
  return (int)(c < 1 ? 1 : c);
}
inline int line_chunk(long long nx) {
  const int c = line_ctas(nx);
  return (int)((nx + c - 1) / c);
}
constexpr size_t kLineSmemMax = 200 * 1024;

template <typename T, int ORD, int KIND>
cudaError_t steps_one(const LineParams<T>& prm, double dt, int steps, cudaStream_t s) {
  const int chunk = line_chunk(prm.nx), ctas = (prm.nx + chunk - 1) / chunk;
  int threads = (chunk + 8 * (OpShape<ORD>::W / 2) + 31) / 32 * 32;
  if (sizeof(T) == 8) threads += ctas == 1 ? 64 : 32;  // the closure points' warps
  if (threads > 512) threads = 512;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = LineSteps<T, ORD, KIND>::smem(chunk);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, line_steps_kernel<T, ORD, KIND>, prm, chunk, steps, (T)(dt / 6), (T)(dt / 3),
                            (T)(0.5 * dt), (T)dt);
}
template <typename T, int ORD, int KIND> cudaError_t steps_configure() {
  return cudaFuncSetAttribute(line_steps_kernel<T, ORD, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kLineSmemMax);
}
}  // namespace

// Above about 6000 points eight CTAs' FP64 pipes take as long as the launches they replace
// (reflection at 6401 points: 13.9 us a step against 12.8).
bool line_steps_takes(long long nx, int kind, int elem_bytes) {
  return nx <= (elem_bytes == 4 ? 8192 : (kind == LK_REFL1D ? 5000 : 6500));
}

template <typename T>
cudaError_t launch_line_steps(int order, int kind, const LineParams<T>& prm, double dt, int steps, cudaStream_t s) {
  const bool adv = kind == LK_ADV1D;
  switch (order) {
    case 2: return adv ? steps_one<T, 2, LK_ADV1D>(prm, dt, steps, s) : steps_one<T, 2, LK_REFL1D>(prm, dt, steps, s);
    case 4: return adv ? steps_one<T, 4, LK_ADV1D>(prm, dt, steps, s) : steps_one<T, 4, LK_REFL1D>(prm, dt, steps, s);
    case 6: return adv ? steps_one<T, 6, LK_ADV1D>(prm, dt, steps, s) : steps_one<T, 6, LK_REFL1D>(prm, dt, steps, s);
    default: return cudaErrorInvalidValue;
  }
}
template <typename T> cudaError_t configure_line_steps(int order, int kind) {
  const bool adv = kind == LK_ADV1D;
  switch (order) {
    case 2: return adv ? steps_configure<T, 2, LK_ADV1D>() : steps_configure<T, 2, LK_REFL1D>();
    case 4: return adv ? steps_configure<T, 4, LK_ADV1D>() : steps_configure<T, 4, LK_REFL1D>();
    case 6: return adv ? steps_configure<T, 6, LK_ADV1D>() : steps_configure<T, 6, LK_REFL1D>();
    default: return cudaErrorInvalidValue;
  }
}
template cudaError_t launch_line_steps<double>(int, int, const LineParams<double>&, double, int, cudaStream_t);
template cudaError_t launch_line_steps<float>(int, int, const LineParams<float>&, double, int, cudaStream_t);
template cudaError_t configure_line_steps<double>(int, int);
template cudaError_t configure_line_steps<float>(int, int);

// ---------------------------------------------------------------- manufactured solution
// code/demo/wave/wave_eq_rhs.h:42-64 with the time factor cos(5 pi t) left out. Run once
// when a context is created: evaluated per point and stage, the four trigonometric
// functions and three divisions held a 161 x 161 stage at 55 us on the FP64 pipe.
__global__ void __launch_bounds__(256)
    mms_coefficients_kernel(double* __restrict__ out, int nx, int ny, long long pitch, long long plane, double xl0,
                            double xl1, double hix, double hiy, double isx, double isy) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nx) return;
  const double PI = 3.14159265358979323846264;
  const double x = xl0 + (double)i / hix;
  const double s3x = sin(3 * PI * x), c3x = cos(3 * PI * x);
  for (int j = blockIdx.y; j < ny; j += gridDim.y) {
    const double y = xl1 + (double)j / hiy;
    const long long q = (long long)j * pitch + i;
    out[q] = 1. / (2 + x * y);
    out[plane + q] = isx * (-(3 * PI * c3x * sin(4 * PI * y) * (x * y + 1)) / (x * y + 2));
    out[2 * plane + q] = isy * (-(4 * PI * cos(4 * PI * y) * s3x * (x * y + 1)) / (x * y + 2));
  }
}

cudaError_t launch_mms_coefficients(double* out, int nx, int ny, long long pitch, long long plane, double xl0,
                                    double xl1, double hix, double hiy, int order, cudaStream_t s) {
  const double den = fixed_denominator(order);
  const dim3 grid((nx + 255) / 256, ny < 1024 ? ny : 1024);
  mms_coefficients_kernel<<<grid, 256, 0, s>>>(out, nx, ny, pitch, plane, xl0, xl1, hix, hiy, -den / hix, -den / hiy);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- layout
// One thread per (point, component) of the AoS array: reads are contiguous,
// writes go to `dofs` planes (contiguous per component within a warp).
template <typename T>
__global__ void pack_kernel(const double* __restrict__ aos, T* __restrict__ soa, int nx, int ny, int dofs,
                            long long pitch, long long plane) {
  const long long n = (long long)nx * ny * dofs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const long long pt = e / dofs;
    const int c = (int)(e - pt * dofs);
    const long long j = pt / nx, i = pt - j * nx;
    soa[c * plane + j * pitch + i] = (T)aos[e];
  }
}

template <typename T>
__global__ void unpack_kernel(const T* __restrict__ soa, double* __restrict__ aos, int nx, int ny, int dofs,
                              long long pitch, long long plane) {
  const long long n = (long long)nx * ny * dofs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const long long pt = e / dofs;
    const int c = (int)(e - pt * dofs);
    const long long j = pt / nx, i = pt - j * nx;
    aos[e] = (double)soa[c * plane + j * pitch + i];
  }
}

static int grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b > 152LL * 16) b = 152LL * 16;
  return (int)(b < 1 ? 1 : b);
}

template <typename T>
cudaError_t launch_pack(const double* aos, T* soa, int nx, int ny, int dofs, long long pitch, long long plane,
                        cudaStream_t s) {
  const long long n = (long long)nx * ny * dofs;
  pack_kernel<T><<<grid_for(n, 256), 256, 0, s>>>(aos, soa, nx, ny, dofs, pitch, plane);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_unpack(const T* soa, double* aos, int nx, int ny, int dofs, long long pitch, long long plane,
                          cudaStream_t s) {
  const long long n = (long long)nx * ny * dofs;
  unpack_kernel<T><<<grid_for(n, 256), 256, 0, s>>>(soa, aos, nx, ny, dofs, pitch, plane);
  return cudaGetLastError();
}
template cudaError_t launch_pack<double>(const double*, double*, int, int, int, long long, long long, cudaStream_t);
template cudaError_t launch_pack<float>(const double*, float*, int, int, int, long long, long long, cudaStream_t);
template cudaError_t launch_unpack<double>(const double*, double*, int, int, int, long long, long long, cudaStream_t);
template cudaError_t launch_unpack<float>(const float*, double*, int, int, int, long long, long long, cudaStream_t);

// ---------------------------------------------------------------- reductions
// Two passes with a fixed block count, so the summation order (and the FP64
// result) does not depend on timing.
constexpr int kReduceThreads = 256;

__device__ __forceinline__ void block_reduce2(double& sum, double& mx, double* sh) {
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_down_sync(0xffffffffu, sum, o);
    mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sh[warp] = sum;
    sh[32 + warp] = mx;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    sum = lane < nw ? sh[lane] : 0.0;
    mx = lane < nw ? sh[32 + lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_down_sync(0xffffffffu, sum, o);
      mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kReduceThreads)
    error_partial_kernel(const T* __restrict__ soa, const double* __restrict__ aos, int nx, int ny, int dofs,
                         long long pitch, long long plane, double* __restrict__ partial) {
  __shared__ double sh[64];
  double sum = 0.0, mx = 0.0;
  const long long n = (long long)nx * ny * dofs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const long long pt = e / dofs;
    const int c = (int)(e - pt * dofs);
    const long long j = pt / nx, i = pt - j * nx;
    const double d = fabs(aos[e] - (double)soa[c * plane + j * pitch + i]);
    sum += d * d;
    mx = fmax(mx, d);
  }
  block_reduce2(sum, mx, sh);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = sum;
    partial[2 * blockIdx.x + 1] = mx;
  }
}

__global__ void __launch_bounds__(kReduceThreads) final_reduce_kernel(const double* __restrict__ partial, int nblocks,
                                                                      double* __restrict__ out) {
  __shared__ double sh[64];
  double sum = 0.0, mx = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
    sum += partial[2 * b];
    mx = fmax(mx, partial[2 * b + 1]);
  }
  block_reduce2(sum, mx, sh);
  if (threadIdx.x == 0) {
    out[0] = sum;
    out[1] = mx;
  }
}

template <typename T>
cudaError_t launch_error_norms(const T* soa, const double* aos, int nx, int ny, int dofs, long long pitch,
                               long long plane, double* partial, double* out, cudaStream_t s) {
  error_partial_kernel<T><<<kReduceBlocks, kReduceThreads, 0, s>>>(soa, aos, nx, ny, dofs, pitch, plane, partial);
  final_reduce_kernel<<<1, kReduceThreads, 0, s>>>(partial, kReduceBlocks, out);
  return cudaGetLastError();
}
template cudaError_t launch_error_norms<double>(const double*, const double*, int, int, int, long long, long long,
                                                double*, double*, cudaStream_t);
template cudaError_t launch_error_norms<float>(const float*, const double*, int, int, int, long long, long long,
                                               double*, double*, cudaStream_t);

// Quadrature weights of the closures (code/include/sbpops/H_central.h:193-212).
__constant__ double c_hquad[3][6] = {
    {1. / 2, 0, 0, 0, 0, 0},
    {17. / 48, 59. / 48, 43. / 48, 49. / 48, 0, 0},
    {13649. / 43200, 12013. / 8640, 2711. / 4320, 5359. / 4320, 7877. / 8640, 43801. / 43200}};

__device__ __forceinline__ double hweight(int n, int i, int cs, int oi) {
  if (i < cs) return c_hquad[oi][i];
  if (i >= n - cs) return c_hquad[oi][n - 1 - i];
  return 1.0;
}

template <typename T>
__global__ void __launch_bounds__(kReduceThreads)
    hnorm_partial_kernel(const T* __restrict__ soa, int nx, int ny, int dofs, long long pitch, long long plane,
                         int order, double hx, double hy, int ysplit, double* __restrict__ partial, int nz,
                         double hz) {
  __shared__ double sh[64];
  const int oi = order / 2 - 1, cs = (order == 2) ? 1 : (order == 4 ? 4 : 6);
  double sum = 0.0, mx = 0.0;
  const long long n = (long long)nx * ny * nz;
  for (long long pt = blockIdx.x * (long long)blockDim.x + threadIdx.x; pt < n; pt += (long long)gridDim.x * blockDim.x) {
    const long long r = pt / nx, i = pt - r * nx;  // row r = j + ny * k
    const long long kz = r / ny, j = r - kz * ny;
    // two-block grids: each block has its own quadrature in y
    const int jb0 = (ysplit > 0 && j >= ysplit) ? ysplit : 0;
    const int nyb = (ysplit > 0) ? (j >= ysplit ? ny - ysplit : ysplit) : ny;
    double w = hx * hweight(nx, (int)i, cs, oi) * (ny > 1 ? hy * hweight(nyb, (int)j - jb0, cs, oi) : 1.0);
    if (nz > 1) w *= hz * hweight(nz, (int)kz, cs, oi);
    double s = 0.0;
    for (int c = 0; c < dofs; c++) {
      const double x = (double)soa[c * plane + r * pitch + i];
      s += x * x;
    }
    sum += w * s;
  }
  block_reduce2(sum, mx, sh);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = sum;
    partial[2 * blockIdx.x + 1] = 0.0;
  }
}

template <typename T>
cudaError_t launch_hnorm(const T* soa, int nx, int ny, int dofs, long long pitch, long long plane, int order,
                         double hx, double hy, int ysplit, double* partial, double* out, cudaStream_t s, int nz,
                         double hz) {
  hnorm_partial_kernel<T><<<kReduceBlocks, kReduceThreads, 0, s>>>(soa, nx, ny, dofs, pitch, plane, order, hx, hy,
                                                                   ysplit, partial, nz, hz);
  final_reduce_kernel<<<1, kReduceThreads, 0, s>>>(partial, kReduceBlocks, out);
  return cudaGetLastError();
}
template cudaError_t launch_hnorm<double>(const double*, int, int, int, long long, long long, int, double, double,
                                          int, double*, double*, cudaStream_t, int, double);
template cudaError_t launch_hnorm<float>(const float*, int, int, int, long long, long long, int, double, double, int,
                                         double*, double*, cudaStream_t, int, double);

// ---------------------------------------------------------------- FP64 probe
__global__ void dfma_probe_kernel(double* out, int iters) {
  double a[8];
#pragma unroll
  for (int k = 0; k < 8; k++) a[k] = 1.0 + 1e-9 * (threadIdx.x + k);
  const double m = 0.9999999, c = 1e-7;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = fma(a[k], m, c);
  }
  double s = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) s += a[k];
  if (s == 12345.678) out[0] = s;  // keeps the chains live; never true in practice
  if (threadIdx.x == 0 && blockIdx.x == 0) out[1] = s;
}

cudaError_t launch_dfma_probe(double* out, int blocks, int threads, int iters, cudaStream_t s) {
  dfma_probe_kernel<<<blocks, threads, 0, s>>>(out, iters);
  return cudaGetLastError();
}

}  // namespace sbp

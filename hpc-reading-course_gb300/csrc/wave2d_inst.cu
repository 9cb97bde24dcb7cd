// wave2d_inst.cu -- instantiations and launcher of the fused wave stage kernel
// for one SBP order. The build compiles this file once per order with
// -DSBP_ORDER=2, 4 or 6 so the three orders compile in parallel.
#include "launch.h"

#ifndef SBP_ORDER
#error "compile with -DSBP_ORDER=2, 4 or 6"
#endif

#define CAT_(a, b) a##b
#define CAT(a, b) CAT_(a, b)
#define LAUNCH_WAVE CAT(launch_wave_o, SBP_ORDER)
#define CONFIGURE_WAVE CAT(configure_wave_o, SBP_ORDER)
#define LAUNCH_CELL CAT(launch_cell_o, SBP_ORDER)
#define LAUNCH_STEP CAT(launch_step_o, SBP_ORDER)
#define CONFIGURE_STEP CAT(configure_step_o, SBP_ORDER)

namespace sbp {

namespace {

// FP64 stages run the fixed-point kernel with converter warps (wave_fixed_kernel), FP32
// ones wave_stage_kernel.
template <typename T, int KIND, int STAGE>
cudaError_t configure_one() {
  if constexpr (wave_fixed<T, KIND, STAGE>())
    return cudaFuncSetAttribute(wave_fixed_kernel<SBP_ORDER, STAGE, false, KIND>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                WaveStageTile<T, SBP_ORDER, KIND, STAGE>::SMEM);
  else
    return cudaFuncSetAttribute(wave_stage_kernel<T, SBP_ORDER, KIND, STAGE>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                WaveStageTile<T, SBP_ORDER, KIND, STAGE>::SMEM);
}

template <typename T, int KIND>
cudaError_t configure_kind() {
  cudaError_t e;
  if ((e = configure_one<T, KIND, ST_RHS>()) != cudaSuccess) return e;
  if ((e = configure_one<T, KIND, ST_FIRST>()) != cudaSuccess) return e;
  if ((e = configure_one<T, KIND, ST_MID>()) != cudaSuccess) return e;
  if ((e = configure_one<T, KIND, ST_LAST>()) != cudaSuccess) return e;
  if constexpr (sizeof(T) == 8) {  // the Fehlberg stages (FP64 only)
    if ((e = configure_one<T, KIND, ST_RKF1>()) != cudaSuccess) return e;
    if ((e = configure_one<T, KIND, ST_RKF1 + 1>()) != cudaSuccess) return e;
    if ((e = configure_one<T, KIND, ST_RKF1 + 2>()) != cudaSuccess) return e;
    if ((e = configure_one<T, KIND, ST_RKF1 + 3>()) != cudaSuccess) return e;
    if ((e = configure_one<T, KIND, ST_RKF1 + 4>()) != cudaSuccess) return e;
    if ((e = configure_one<T, KIND, ST_RKF6>()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <typename T, int KIND, int STAGE>
cudaError_t launch_one(const WaveMaps& m, const WaveParams<T>& prm, dim3 grid, cudaStream_t s) {
  using Tile = WaveStageTile<T, SBP_ORDER, KIND, STAGE>;
  if constexpr (wave_fixed<T, KIND, STAGE>())
    wave_fixed_kernel<SBP_ORDER, STAGE, false, KIND><<<grid, Tile::THREADS, Tile::SMEM, s>>>(m.p, m.u, m.v, m.n, m.a,
                                                                                            m.c, m.k, prm);
  else
    wave_stage_kernel<T, SBP_ORDER, KIND, STAGE>
        <<<grid, Tile::THREADS, Tile::SMEM, s>>>(m.p, m.u, m.v, m.n, m.a, m.c, m.k, prm);
  return cudaGetLastError();
}

template <typename T, int KIND>
cudaError_t launch_kind(int stage, const WaveMaps& m, const WaveParams<T>& prm, dim3 grid, cudaStream_t s) {
  switch (stage) {
    case ST_RHS: return launch_one<T, KIND, ST_RHS>(m, prm, grid, s);
    case ST_FIRST: return launch_one<T, KIND, ST_FIRST>(m, prm, grid, s);
    case ST_MID: return launch_one<T, KIND, ST_MID>(m, prm, grid, s);
    case ST_LAST: return launch_one<T, KIND, ST_LAST>(m, prm, grid, s);
    default: break;
  }
  if constexpr (sizeof(T) == 8) {
    switch (stage) {
      case ST_RKF1: return launch_one<T, KIND, ST_RKF1>(m, prm, grid, s);
      case ST_RKF1 + 1: return launch_one<T, KIND, ST_RKF1 + 1>(m, prm, grid, s);
      case ST_RKF1 + 2: return launch_one<T, KIND, ST_RKF1 + 2>(m, prm, grid, s);
      case ST_RKF1 + 3: return launch_one<T, KIND, ST_RKF1 + 3>(m, prm, grid, s);
      case ST_RKF1 + 4: return launch_one<T, KIND, ST_RKF1 + 4>(m, prm, grid, s);
      case ST_RKF6: return launch_one<T, KIND, ST_RKF6>(m, prm, grid, s);
      default: break;
    }
  }
  return cudaErrorInvalidValue;
}

template <typename T, int KIND, int STAGE, bool AOS = false>
cudaError_t cell_one(const WaveParams<T>& prm, cudaStream_t s) {
  return launch_overlapped(wave_cell_kernel<T, SBP_ORDER, KIND, STAGE, AOS>,
                           cell_grid(prm.nx, prm.ny), kCellThreads, 0, s, prm);
}

template <typename T, int KIND>
cudaError_t cell_kind(int stage, bool aos, const WaveParams<T>& prm, cudaStream_t s) {
  if (aos) return stage == ST_RHS ? cell_one<T, KIND, ST_RHS, true>(prm, s) : cudaErrorInvalidValue;
  switch (stage) {
    case ST_RHS: return cell_one<T, KIND, ST_RHS>(prm, s);
    case ST_FIRST: return cell_one<T, KIND, ST_FIRST>(prm, s);
    case ST_MID: return cell_one<T, KIND, ST_MID>(prm, s);
    case ST_LAST: return cell_one<T, KIND, ST_LAST>(prm, s);
    default: break;
  }
  if constexpr (sizeof(T) == 8) {
    switch (stage) {
      case ST_RKF1: return cell_one<T, KIND, ST_RKF1>(prm, s);
      case ST_RKF1 + 1: return cell_one<T, KIND, ST_RKF1 + 1>(prm, s);
      case ST_RKF1 + 2: return cell_one<T, KIND, ST_RKF1 + 2>(prm, s);
      case ST_RKF1 + 3: return cell_one<T, KIND, ST_RKF1 + 3>(prm, s);
      case ST_RKF1 + 4: return cell_one<T, KIND, ST_RKF1 + 4>(prm, s);
      case ST_RKF6: return cell_one<T, KIND, ST_RKF6>(prm, s);
      default: break;
    }
  }
  return cudaErrorInvalidValue;
}

template <int KIND, int TC>
constexpr int step_smem() {
  return WaveStep<SBP_ORDER, TC>::smem(KIND == WK_VAR ? 2 : (KIND == WK_MMS ? 3 : 0));
}

template <int KIND, int TC>
cudaError_t step_one(const WaveParams<double>& prm, const WaveStepCoef& cf, cudaStream_t s) {
  const dim3 grid((prm.nx + TC - 1) / TC, (prm.ny + TC - 1) / TC);
  return launch_overlapped(wave_step_kernel<SBP_ORDER, KIND, TC>, grid, kStepThreads, step_smem<KIND, TC>(), s, prm, cf);
}

// The smaller cell where its CTAs fit the SMs at once, else the larger.
template <int KIND>
cudaError_t step_kind(const WaveParams<double>& prm, const WaveStepCoef& cf, cudaStream_t s) {
  const long long small = (long long)((prm.nx + kStepSmall - 1) / kStepSmall) * ((prm.ny + kStepSmall - 1) / kStepSmall);
  if (small <= device_sm_count()) return step_one<KIND, kStepSmall>(prm, cf, s);
  return step_one<KIND, step_large(SBP_ORDER)>(prm, cf, s);
}

template <int KIND, int TC> cudaError_t step_configure_one() {
  return cudaFuncSetAttribute(wave_step_kernel<SBP_ORDER, KIND, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              step_smem<KIND, TC>());
}
template <int KIND> cudaError_t step_configure() {
  const cudaError_t e = step_configure_one<KIND, kStepSmall>();
  return e != cudaSuccess ? e : step_configure_one<KIND, step_large(SBP_ORDER)>();
}

}  // namespace

cudaError_t LAUNCH_STEP(int kind, const WaveParams<double>& prm, const WaveStepCoef& cf, cudaStream_t s) {
  switch (kind) {
    case WK_HOM: return step_kind<WK_HOM>(prm, cf, s);
    case WK_VAR: return step_kind<WK_VAR>(prm, cf, s);
    case WK_MMS: return step_kind<WK_MMS>(prm, cf, s);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t CONFIGURE_STEP(int kind) {
  switch (kind) {
    case WK_HOM: return step_configure<WK_HOM>();
    case WK_VAR: return step_configure<WK_VAR>();
    case WK_MMS: return step_configure<WK_MMS>();
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t LAUNCH_CELL<double>(int kind, int stage, bool aos, const WaveParams<double>& prm, cudaStream_t s) {
  switch (kind) {
    case WK_HOM: return cell_kind<double, WK_HOM>(stage, aos, prm, s);
    case WK_VAR: return cell_kind<double, WK_VAR>(stage, aos, prm, s);
    case WK_MMS: return cell_kind<double, WK_MMS>(stage, aos, prm, s);
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t LAUNCH_CELL<float>(int kind, int stage, bool aos, const WaveParams<float>& prm, cudaStream_t s) {
  switch (kind) {
    case WK_HOM: return cell_kind<float, WK_HOM>(stage, aos, prm, s);
    case WK_VAR: return cell_kind<float, WK_VAR>(stage, aos, prm, s);
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t CONFIGURE_WAVE<double>(int kind) {
  switch (kind) {
    case WK_HOM: return configure_kind<double, WK_HOM>();
    case WK_VAR: return configure_kind<double, WK_VAR>();
    case WK_MMS: return configure_kind<double, WK_MMS>();
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t CONFIGURE_WAVE<float>(int kind) {
  switch (kind) {
    case WK_HOM: return configure_kind<float, WK_HOM>();
    case WK_VAR: return configure_kind<float, WK_VAR>();
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t LAUNCH_WAVE<double>(int kind, int stage, const WaveMaps& m, const WaveParams<double>& prm, dim3 grid,
                                cudaStream_t s) {
  switch (kind) {
    case WK_HOM: return launch_kind<double, WK_HOM>(stage, m, prm, grid, s);
    case WK_VAR: return launch_kind<double, WK_VAR>(stage, m, prm, grid, s);
    case WK_MMS: return launch_kind<double, WK_MMS>(stage, m, prm, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t LAUNCH_WAVE<float>(int kind, int stage, const WaveMaps& m, const WaveParams<float>& prm, dim3 grid,
                               cudaStream_t s) {
  switch (kind) {
    case WK_HOM: return launch_kind<float, WK_HOM>(stage, m, prm, grid, s);
    case WK_VAR: return launch_kind<float, WK_VAR>(stage, m, prm, grid, s);
    default: return cudaErrorInvalidValue;  // the manufactured-solution problem is FP64 only
  }
}

}  // namespace sbp

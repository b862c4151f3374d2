// Operand staging kernels shared by the tensor-core forward and backward.
#pragma once

#include <cuda_fp16.h>

#include "d2c_common.cuh"
#include "sm100_ptx.cuh"

namespace d2c {
namespace {

// round-to-nearest fp32 -> fp16 with saturation to the largest finite half (|x| > 65504 is clamped)
__device__ __forceinline__ uint32_t pack_f16x2_sat(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// x [B][C][Vin] fp32 -> x_cl [B][Vin][C] channels-last: fp16 (saturating), or fp32 for the fp32-parity mode.  fp32: infinities are
// replaced by the largest finite float (as the fp16 staging saturates).
// `zero` is cleared on the side (the output that partial tiles are added to); nan_flag (nullable) is set to 1 where x holds a NaN:
// the kernel before, which this one may run beside, clears it, so it is set after the wait.
// Bound by HBM.  Block: 64 channels x kVox voxels; all of a thread's loads are requested before the first is stored, and it
// writes 16 bytes.  (8 loads and 4- or 8-byte writes a thread: fp32, 512 channels on 2 x 8 x 30 x 54 with the output cleared, 46 us,
// now 26; fp16, 1024 channels on 8 x 30 x 54, 35 us, now 17.)
template <typename T, int kVox>
static __global__ void __launch_bounds__(256)
stage_input_cl_kernel(int C, long long Vin, const float* __restrict__ x, T* __restrict__ x_cl, ZeroFill zero,
                      int* __restrict__ nan_flag) {
  next_kernel_may_start();
  constexpr int kPer = 16 / sizeof(T);             // channels a thread writes
  constexpr int kLanes = 64 / kPer;                // threads per voxel
  __shared__ float tile[64][kVox + 1];
  const int b = blockIdx.z, c0 = blockIdx.y * 64;
  const long long v0 = (long long)blockIdx.x * kVox;
  bool nan = false;
  {
    constexpr int kRowsPass = 256 / kVox, kLoads = 64 / kRowsPass;
    const int tx = threadIdx.x % kVox, ty = threadIdx.x / kVox;
    const long long v = v0 + tx;
    const float* src = x + ((long long)b * C + c0) * Vin + v;
    float f[kLoads];
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int cc = ty + kRowsPass * i;
      f[i] = (v < Vin && c0 + cc < C) ? __ldg(src + (long long)cc * Vin) : 0.f;
    }
    zero_fill(zero, blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z),
              (long long)gridDim.x * gridDim.y * gridDim.z);
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      nan |= isnan(f[i]);
      if (sizeof(T) == 4 && isinf(f[i])) f[i] = copysignf(3.402823466e+38f, f[i]);
      tile[ty + kRowsPass * i][tx] = f[i];
    }
  }
  nan = __syncthreads_or(nan);
  const int q = threadIdx.x % kLanes, c = q * kPer;
#pragma unroll
  for (int vv = threadIdx.x / kLanes; vv < kVox; vv += 256 / kLanes) {
    const long long v = v0 + vv;
    if (v >= Vin || c0 + c >= C) continue;         // C is a multiple of 32
    T* dst = x_cl + ((long long)b * Vin + v) * C + c0 + c;
    if constexpr (sizeof(T) == 2) {
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = pack_f16x2_sat(tile[c + 2 * e][vv], tile[c + 2 * e + 1][vv]);
      *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
      *reinterpret_cast<float4*>(dst) = make_float4(tile[c][vv], tile[c + 1][vv], tile[c + 2][vv], tile[c + 3][vv]);
    }
  }
  if (threadIdx.x == 0) {
    wait_for_kernels_before();
    if (nan && nan_flag) *nan_flag = 1;
  }
}

// Blocks of 64 voxels, of 32 where that leaves multiprocessors without one.  beside: may run at the same time as the kernel before.
template <typename T>
static int launch_stage_input(const Geom& g, const float* x, T* x_cl, const ZeroFill& zero, int* nan_flag, int sm_count,
                              cudaStream_t st, bool beside = false) {
  dim3 grid((unsigned)((g.Vin + 63) / 64), (unsigned)((g.Cin + 63) / 64), (unsigned)g.B);
  auto kernel = stage_input_cl_kernel<T, 64>;
  if ((long long)grid.x * grid.y * grid.z < 2LL * sm_count) {
    grid.x = (unsigned)((g.Vin + 31) / 32);
    kernel = stage_input_cl_kernel<T, 32>;
  }
  if (beside)
    D2C_CUDA_TRY(launch_beside(kernel, grid, 256, 0, st, g.Cin, g.Vin, x, x_cl, zero, nan_flag));
  else
    kernel<<<grid, 256, 0, st>>>(g.Cin, g.Vin, x, x_cl, zero, nan_flag);
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

}  // namespace
}  // namespace d2c

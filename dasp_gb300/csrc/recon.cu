// Consumer of the centroids: the reconstructor matrix-vector step of DASP's
// tomoRecon (science/tomoRecon.py:1077-1107 decay, :1196-1223 MVM):
//   act[i] = decay_i * act[i] - gain_i * sum_j R[i, j] x[j]
// with R (nacts x ncents, row-major float32) resident in HBM.  The step is
// bound by reading R once: one warp per actuator row, eight 16-byte loads (or
// sixteen 4-byte ones where rows are not 16-byte aligned) in flight per lane,
// x read through L1 (every row reads it), float32 accumulation as the
// reference's float32 dot, decay and gain fused into the same pass.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "../../include/shwfs.h"
#include "engine_internal.h"

namespace shwfs {

namespace {

constexpr int kMvmThreads = 256, kMvmWarps = kMvmThreads / 32;
constexpr int kMvmUnroll = 8;    // 16-byte loads of R in flight per lane
constexpr int kMvmUnroll1 = 16;  // 4-byte loads, rows of other alignments

// WPR warps share a row (interleaved blocks of 32 loads): few long rows would
// otherwise leave the SMs short of loads in flight.  Launched programmatically:
// the CTAs take their places as those of the kernel before end, and read
// nothing until it has completed.  5316 x 7944 (169 MB, 25.2 us at the measured
// copy rate) 28.9 -> 26.9 us a step, 3001 x 4002 17.0 -> 11.2, 1000 x 1001 6.2
// -> 4.0; rows that are not 16-byte aligned (5316 x 7943) 32.9 -> 31.8, in
// 4-byte loads: 16-byte ones from each row's first boundary, with x then in
// 4-byte loads, took 37.
template <bool VEC, int WPR>
__global__ void __launch_bounds__(kMvmThreads) mvm_update_kernel(const float* __restrict__ R, int nacts, int ncents,
                                                                 const float* __restrict__ x,
                                                                 const float* __restrict__ gains, float gain,
                                                                 const float* __restrict__ decay, float decay_s,
                                                                 float* __restrict__ act) {
  __shared__ float s_part[kMvmWarps];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int rows = kMvmWarps / WPR, step = 32 * WPR;
  const int seg = warp % WPR;  // this warp's share of its row
  const int first = seg * 32 + lane;
  for (int row0 = blockIdx.x * rows; row0 < nacts; row0 += gridDim.x * rows) {
    const int row = row0 + warp / WPR;
    float acc = 0.f;
    if (row < nacts) {
      const float* r = R + (long long)row * ncents;
      if (VEC) {
        // 16-byte chunks, kMvmUnroll per lane per pass
        const int nq = ncents >> 2;
        const float4* r4 = reinterpret_cast<const float4*>(r);
        const float4* x4 = reinterpret_cast<const float4*>(x);
        int q = first;
        for (; q + step * (kMvmUnroll - 1) < nq; q += step * kMvmUnroll) {
          float4 a[kMvmUnroll];
#pragma unroll
          for (int u = 0; u < kMvmUnroll; u++) a[u] = __ldcs(r4 + q + step * u);
#pragma unroll
          for (int u = 0; u < kMvmUnroll; u++) {
            const float4 b = x4[q + step * u];
            acc += a[u].x * b.x + a[u].y * b.y + a[u].z * b.z + a[u].w * b.w;
          }
        }
        for (; q < nq; q += step) {
          const float4 a0 = __ldcs(r4 + q), b0 = x4[q];
          acc += a0.x * b0.x + a0.y * b0.y + a0.z * b0.z + a0.w * b0.w;
        }
      } else {
        // coalesced 4-byte loads: a 128-byte line per warp and load
        int j = first;
        for (; j + step * (kMvmUnroll1 - 1) < ncents; j += step * kMvmUnroll1) {
          float a[kMvmUnroll1];
#pragma unroll
          for (int u = 0; u < kMvmUnroll1; u++) a[u] = __ldcs(r + j + step * u);
#pragma unroll
          for (int u = 0; u < kMvmUnroll1; u++) acc += a[u] * x[j + step * u];
        }
        for (; j < ncents; j += step) acc += __ldcs(r + j) * x[j];
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    if constexpr (WPR > 1) {
      if (lane == 0) s_part[warp] = acc;
      __syncthreads();
      if (seg == 0)
        for (int k = 1; k < WPR; k++) acc += s_part[warp + k];
      __syncthreads();
    }
    if (row0 + gridDim.x * rows >= nacts) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (lane == 0 && seg == 0 && row < nacts) {
      const float d = decay ? decay[row] : decay_s;
      const float g = gains ? gains[row] : gain;
      act[row] = d * act[row] - g * acc;
    }
  }
}

// warps per row: about 32 warps per SM, each with at least two loads per lane
int mvm_wpr(int nacts, int ncents, int sms, bool vec) {
  int w = 1;
  while (w < kMvmWarps && (long long)nacts * w < 32LL * sms && ncents >= 2 * w * 64 * (vec ? 4 : 1)) w *= 2;
  return w;
}

}  // namespace

}  // namespace shwfs

extern "C" shwfs_status shwfs_mvm_update(int nacts, int ncents, const float* R, const float* x, const float* gains,
                                         float gain, const float* decay, float decay_scalar, float* act,
                                         void* stream) {
  if (nacts < 1 || ncents < 1 || !R || !x || !act)
    return shwfs::engine_fail(SHWFS_ERR_INVALID, "mvm_update: bad arguments");
  const bool vec = (ncents & 3) == 0 && ((uintptr_t)R & 15) == 0 && ((uintptr_t)x & 15) == 0;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int wpr = shwfs::mvm_wpr(nacts, ncents, sms, vec), rows = shwfs::kMvmWarps / wpr;
  cudaStream_t st = (cudaStream_t)stream;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::max(1, std::min((nacts + rows - 1) / rows, sms * 8)));
  cfg.blockDim = dim3(shwfs::kMvmThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  using Kern = void (*)(const float*, int, int, const float*, const float*, float, const float*, float, float*);
  static const Kern kerns[2][4] = {{shwfs::mvm_update_kernel<false, 1>, shwfs::mvm_update_kernel<false, 2>,
                                    shwfs::mvm_update_kernel<false, 4>, shwfs::mvm_update_kernel<false, 8>},
                                   {shwfs::mvm_update_kernel<true, 1>, shwfs::mvm_update_kernel<true, 2>,
                                    shwfs::mvm_update_kernel<true, 4>, shwfs::mvm_update_kernel<true, 8>}};
  const Kern kern = kerns[vec ? 1 : 0][wpr == 1 ? 0 : (wpr == 2 ? 1 : (wpr == 4 ? 2 : 3))];
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, R, nacts, ncents, x, gains, gain, decay, decay_scalar, act);
  if (e == cudaSuccess && !stream) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess)
    return shwfs::engine_fail(SHWFS_ERR_CUDA, (std::string("mvm_update: ") + cudaGetErrorString(e)).c_str());
  return SHWFS_OK;
}

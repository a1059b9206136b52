// Image-input path of the WFS step (runSlope): centroids from a detector
// image instead of phase (cmod/src/centmodule.c:1987-2127).
//
// Per lit subaperture: the subaperture window is cut from the 2-D detector
// image (default tiling by nimg, or the caller's subapLocation rows/cols) or
// taken from a 4-D (nsubx,nsubx,nimg,nimg) image; as in the reference the
// window lands in the top-left of the nimg x nimg image and pixels outside it
// keep their previous bimg values.  Then, for a science source, readCCD with
// no noise (threshold only) over the first nexposed pixels in storage order,
// and the shared post stages (brightest pixels, power, bimg, centroids).
#include <algorithm>

#include "wfs_plain.cuh"

namespace shwfs {

__device__ __forceinline__ void subap_window(const WfsArgs& a, const int* loc, int i, int& r0, int& r1, int& c0,
                                             int& c1) {
  if (loc) {
    r0 = loc[i * 4];
    r1 = loc[i * 4 + 1];
    c0 = loc[i * 4 + 2];
    c1 = loc[i * 4 + 3];
  } else {
    r0 = (i / a.nsubx) * a.m;
    r1 = r0 + a.m;
    c0 = (i % a.nsubx) * a.m;
    c1 = c0 + a.m;
  }
}

constexpr int kImageThreads = 256;
constexpr int kImageUnroll = 4;  // detector pixels in flight per thread
constexpr int kImageTilesPerSM = 4;

// Bound by the link the detector frame and the outputs travel on (a host
// frame's 1.6 MB each way at about 150 GB/s: 11 us for the 74x74 sensor) and by
// its latency, so every thread has kImageUnroll loads in flight and the tiles
// are small enough that two or more CTAs per SM share the frame: 40
// subapertures per 128-thread CTA with one load in flight per thread took 58 us
// of kernel time.  One call on the 74x74 sensor's 740 x 740 host frame: 71 ->
// 34 us; one to eight tiles per SM measured alike (32.5 to 35 us).  Unlit subapertures' centroids are zeroed here too
// (a.zeroUnlit) instead of in a launch of their own.
__global__ void __launch_bounds__(kImageThreads)
    wfs_image_kernel(const WfsArgs a, const float* __restrict__ img, int dims, int npxlx, const int* loc) {
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const int tid = threadIdx.x;
  const int m = a.m, mm = m * m;
  const bool cw2d = a.centWeightDim == 2;
  float* s_cw = smem;
  float* s_sub0 = smem + (((cw2d ? mm : 0) + 3) & ~3);
  const int persub = (mm + 3) & ~3;
  __shared__ int s_subap[64];
  __shared__ int s_frame[64];
  __shared__ int s_nexp[64];
  __shared__ int2 s_size[64];        // rows and columns of the window
  __shared__ long long s_src[64];  // its first pixel in the image
  if (a.zeroUnlit)
    // unlit subapertures: centroids 0 (within centroidsFromImage)
    for (int u = blockIdx.x * blockDim.x + tid; u < a.nunlit; u += gridDim.x * blockDim.x) {
      float* c = a.cents + 2LL * a.unlit[u];
      c[0] = 0.f;
      c[1] = 0.f;
    }
  if (cw2d)
    for (int k = tid; k < mm; k += blockDim.x) s_cw[k] = a.centWeight[k];
  const int TS = a.TS;
  const int ntiles = (a.nlit + TS - 1) / TS;
  const int pitch = dims == 4 ? m : npxlx;
  const float inv_mm = 1.0f / (float)mm, inv_m = 1.0f / (float)m;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int w0 = tile * TS;
    const int ns = min(TS, a.nlit - w0);
    __syncthreads();
    for (int s = tid; s < ns; s += blockDim.x) {
      const int i = a.lit[w0 + s];
      int r0 = 0, r1 = m, c0 = 0, c1 = m;
      if (dims != 4) subap_window(a, loc, i, r0, r1, c0, c1);
      s_subap[s] = i;
      s_frame[s] = 0;
      s_src[s] = dims == 4 ? (long long)i * mm : (long long)r0 * npxlx + c0;
      s_size[s] = make_int2(r1 - r0, c1 - c0);
      s_nexp[s] = (r1 - r0) * (c1 - c0);
    }
    __syncthreads();
    for (int wb = tid; wb < ns * mm; wb += kImageUnroll * kImageThreads) {
      float v[kImageUnroll];
#pragma unroll
      for (int u = 0; u < kImageUnroll; u++) {
        const int w = wb + u * kImageThreads;
        v[u] = 0.f;
        if (w >= ns * mm) continue;
        const int s = div_small(w, mm, inv_mm), pix = w - s * mm;
        const int j = div_small(pix, m, inv_m), k = pix - j * m;
        v[u] = (j < s_size[s].x && k < s_size[s].y) ? img[s_src[s] + (long long)j * pitch + k]
                                                    : a.bimg[(long long)s_subap[s] * mm + pix];
      }
#pragma unroll
      for (int u = 0; u < kImageUnroll; u++) {
        const int w = wb + u * kImageThreads;
        if (w >= ns * mm) continue;
        const int s = div_small(w, mm, inv_mm), pix = w - s * mm;
        float x = v[u];
        if (a.calsource == 0 && pix < s_nexp[s]) x = threshold_px(x + 0.f, a.floorv, a.threshType);
        s_sub0[s * persub + pix] = x;
      }
    }
    __syncthreads();
    post_tile(a, ns, s_subap, s_frame, s_cw, [&](int s) { return s_sub0 + s * persub; },
              [&](int s) { return s_nexp[s]; });
  }
}

cudaError_t launch_image(const WfsArgs& a0, const float* img, int dims, int npxlx, const int* loc, int numSMs,
                         cudaStream_t stream, bool* didUnlit) {
  WfsArgs a = a0;
  const int mm = a.m * a.m;
  // subapertures per CTA: at most 4096 pixels, and few enough that every SM
  // gets kImageTilesPerSM tiles
  a.TS = std::max(1, std::min({64, 4096 / mm, (a.nlit + kImageTilesPerSM * numSMs - 1) / (kImageTilesPerSM * numSMs)}));
  a.zeroUnlit = didUnlit && !a.imageOnly && a.unlit && a.nunlit > 0;
  if (didUnlit) *didUnlit = !a.imageOnly;
  const int smem = ((((a.centWeightDim == 2 ? mm : 0) + 3) & ~3) + a.TS * ((mm + 3) & ~3)) * 4;
  cudaError_t e = kernel_smem_setup((const void*)wfs_image_kernel, smem, kImageThreads, nullptr);
  if (e != cudaSuccess) return e;
  const int ntiles = (a.nlit + a.TS - 1) / a.TS;
  const int grid = ntiles < numSMs * 8 ? (ntiles > 0 ? ntiles : 1) : numSMs * 8;
  wfs_image_kernel<<<grid, kImageThreads, smem, stream>>>(a, img, dims, npxlx, loc);
  return cudaGetLastError();
}

}  // namespace shwfs

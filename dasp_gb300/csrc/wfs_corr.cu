// Correlation centroiding (cmod/src/centmodule.c:1898-1925 and 2044-2066):
// from each lit subaperture's final image in bimg, the correlation image with
// the subaperture's pattern (corrsize x corrsize), its threshold, the
// correlation image written to corrimg, then the centroid stage on it.
//
//   mode 1  calcCorrelation (:1403-1486): r2hc(zero-padded image) times the
//           half-complex pattern, hc2r -- computed as the circular
//           convolution of the padded image with hc2r(pattern), which the
//           host builds once per pattern (the half-complex product is the
//           product of the complex spectra)
//   mode 2  diffCorrelation mode 1: mean squared difference over the overlap
//   mode 3  diffCorrelation mode 2: the reference's abs-difference branch,
//           with its own indexing
//   mode 4  diffCorrelation mode 3: squared difference / (flux of image *
//           flux of pattern) over the overlap
//   mode 5  bruteCorrelation (:1339-1398): overlap sums of the product
// then thresholdCorrelation (:1488-1505) over corrsize^2 pixels and
// computeCoG/computeFit with corrsize (centre on brightest for modes 1 and 5,
// faintest otherwise).
#include <algorithm>

#include "wfs_plain.cuh"

namespace shwfs {

namespace {

constexpr int kCorrThreads = 128;
constexpr int kCorrMaxTS = 32;

// Mode 1's layout: per subaperture the image with rows padded to a multiple
// of four floats, and its pattern with every row extended so that a strip's
// taps are consecutive: entry mp + t of row r is K[r][(t - (cs - m) / 2) mod
// cs], t = -mp .. strips * strip - 1 (t = 0 is 16-byte aligned)
struct CorrStrips {
  int strip;   // outputs per thread: 8 (0: the general code of the other modes)
  int strips;  // per output row
  int row;     // floats per extended row
  int mp;      // floats per image row, and taps ahead of t = 0
};
inline CorrStrips corr_strips(int mode, int m, int cs) {
  CorrStrips g{0, 0, cs, m};
  if (mode != 1) return g;
  g.strip = 8;
  g.strips = (cs + g.strip - 1) / g.strip;
  g.mp = (m + 3) & ~3;
  g.row = g.mp + g.strips * g.strip;
  // consecutive lanes take consecutive strips, then rows: a row length of
  // strips (mod 8) strip widths keeps the 16-byte loads of a strip width of
  // four on consecutive addresses (mod 128 bytes)
  while ((g.row / 4) % 8 != (g.strips * g.strip / 4) % 8) g.row += 4;
  return g;
}

// overlap of pattern and image for output offset i (diffCorrelation
// :1228-1240): start in the pattern, start in the image, extent
__device__ __forceinline__ void overlap(int i, int nimg, int cs, int ncen, int& sref, int& sin_, int& len) {
  const int off = i - ncen / 2;
  len = cs < nimg ? cs : nimg;
  sref = -off - (nimg - cs) / 2;
  if (sref < 0) sref = 0;
  sin_ = (nimg - cs) / 2 + off;
  if (sin_ < 0) sin_ = 0;
  if (sin_ + len > nimg) len = nimg - sin_;
  if (sref + len > cs) len = cs - sref;
}

// One correlation row's strip of STRIP outputs for mode 1, each accumulated
// over the M x M image pixels in row-major order.  A pattern row's taps of the
// whole strip and the image row (the same for neighbouring lanes) come in
// 16-byte loads, then STRIP x M multiply-adds in registers.
template <int STRIP, int M>
__device__ __forceinline__ void corr_strip(const float* img, const float* E, int erow, int y, int x0, int cs, int off,
                                           float (&acc)[STRIP]) {
  constexpr int MP = (M + 3) & ~3;
#pragma unroll
  for (int e = 0; e < STRIP; e++) acc[e] = 0.f;
  int ky = y - off;
  if (ky < 0) ky += cs;
#pragma unroll 1
  for (int p = 0; p < M; p++) {
    const float* er = E + ky * erow + x0;
    float w[MP + STRIP], im[MP];  // w[MP + t]: tap t = x - q of the strip
#pragma unroll
    for (int e = 0; e < MP + STRIP; e += 4) {
      const float4 t = *reinterpret_cast<const float4*>(er + e);
      w[e] = t.x, w[e + 1] = t.y, w[e + 2] = t.z, w[e + 3] = t.w;
    }
#pragma unroll
    for (int q = 0; q < MP; q += 4) {
      const float4 t = *reinterpret_cast<const float4*>(img + p * MP + q);
      im[q] = t.x, im[q + 1] = t.y, im[q + 2] = t.z, im[q + 3] = t.w;
    }
#pragma unroll
    for (int q = 0; q < M; q++)
#pragma unroll
      for (int e = 0; e < STRIP; e++) acc[e] += im[q] * w[MP + e - q];
    if (--ky < 0) ky += cs;
  }
}

// the same for any m, four taps and pixels at a time
template <int STRIP>
__device__ __forceinline__ void corr_strip_any(const float* img, int m, int mp, const float* E, int erow, int y, int x0,
                                               int cs, int off, float (&acc)[STRIP]) {
#pragma unroll
  for (int e = 0; e < STRIP; e++) acc[e] = 0.f;
  int ky = y - off;
  if (ky < 0) ky += cs;
  for (int p = 0; p < m; p++) {
    const float* er = E + ky * erow + mp + x0;
    const float* ir = img + p * mp;
    float w[STRIP + 4];  // w[e + 4 - j]: tap of output e at pixel q + j
#pragma unroll
    for (int e = 0; e < STRIP; e++) w[e + 4] = er[e];
    for (int q = 0; q < m; q += 4) {
      const float4 im = *reinterpret_cast<const float4*>(ir + q);
      const float4 t = *reinterpret_cast<const float4*>(er - q - 4);
      const float px[4] = {im.x, im.y, im.z, im.w};
      w[0] = t.x, w[1] = t.y, w[2] = t.z, w[3] = t.w;
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (q + j < m) {
#pragma unroll
          for (int e = 0; e < STRIP; e++) acc[e] += px[j] * w[e + 4 - j];
        }
#pragma unroll
      for (int e = STRIP + 3; e >= 4; e--) w[e] = w[e - 4];  // slide by four
    }
    if (--ky < 0) ky += cs;
  }
}

// Bound by shared-memory bandwidth (mode 1): corrsize^2 m^2 multiply-adds per
// subaperture, 159 M for the 74x74 sensor with 20x20 patterns of 10x10 images.
// One output per thread with two loads and a conditional wrap per
// multiply-add took 121 us; strips of eight outputs along a row, with a row's
// taps and pixels loaded 16 bytes at a time, take 30 us (38 % of the
// instructions are the multiply-adds).  Small CTAs of as many subapertures as
// give every thread about two strips keep all of one frame resident.  One
// runSlope call with the correlation: 154 -> 46 us.
template <int STRIP, int M>
__global__ void __launch_bounds__(kCorrThreads)
    wfs_corr_kernel(const WfsArgs a, const CorrArgs c, const CorrStrips g) {
  extern __shared__ __align__(16) float smem_corr[];
  __shared__ int s_subap[kCorrMaxTS];
  __shared__ int s_frame[kCorrMaxTS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int m = a.m, mm = m * m, cs = c.cs, cc = cs * cs, ncen = a.ncen;
  const bool cw2d = a.centWeightDim == 2;
  // per subaperture: the image, the pattern (or hc2r(pattern) for mode 1),
  // then the correlation image; the first two 16-byte aligned
  const int imgF = m * g.mp, patF = cs * g.row;
  float* imgs = smem_corr;
  float* Ks = imgs + ((c.TS * imgF + 3) & ~3);
  float* corr = Ks + c.TS * patF;
  float* s_cw = corr + c.TS * cc;
  if (cw2d)
    for (int k = tid; k < cc; k += blockDim.x) s_cw[k] = a.centWeight[k];
  WfsArgs ac = a;  // the centroid stage sees corrsize x corrsize images
  ac.m = cs;
  const long long nwork = (long long)a.nlit * a.nframes;
  const long long ntiles = (nwork + c.TS - 1) / c.TS;
  const int shift = cs - (g.mp + (cs - m) / 2) % cs;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long w0 = tile * c.TS;
    const int ns = (int)min((long long)c.TS, nwork - w0);
    __syncthreads();
    for (int s = tid; s < ns; s += blockDim.x) {
      const long long w = w0 + s;
      s_frame[s] = (int)(w / a.nlit);
      s_subap[s] = a.lit[w % a.nlit];
    }
    __syncthreads();
    // images and patterns a subaperture at a time: a warp per row, the lanes
    // along it, eight rows' loads in flight (flattened indices with a division
    // and a wrap per element took twice the multiply-adds' instructions)
    for (int s = 0; s < ns; s++) {
      const float* src = a.bimg + (long long)s_frame[s] * a.bimgFrameStride + (long long)s_subap[s] * mm;
      for (int q = lane; q < g.mp; q += 32)
#pragma unroll 4
        for (int p = warp; p < m; p += kCorrThreads / 32)
          imgs[s * imgF + p * g.mp + q] = q < m ? src[p * m + q] : 0.f;
      src = c.K + (long long)s_subap[s] * cc;
      if constexpr (STRIP > 0) {
        for (int e = lane; e < g.mp + g.strips * STRIP; e += 32) {
          int x = e + shift;  // circular index of extended entry e
          while (x >= cs) x -= cs;
#pragma unroll 8
          for (int y = warp; y < cs; y += kCorrThreads / 32) Ks[s * patF + y * g.row + e] = src[y * cs + x];
        }
      } else {
#pragma unroll 4
        for (int e = tid; e < cc; e += kCorrThreads) Ks[s * cc + e] = src[e];
      }
    }
    __syncthreads();
    // ---- correlation images ----
    if constexpr (STRIP > 0) {
      const int per = cs * g.strips, off = (cs - m) / 2;
      const float inv_per = 1.0f / (float)per, inv_strips = 1.0f / (float)g.strips;
      for (int w = tid; w < ns * per; w += blockDim.x) {
        const int s = div_small(w, per, inv_per), o = w - s * per;
        const int y = div_small(o, g.strips, inv_strips), x0 = (o - y * g.strips) * STRIP;
        float acc[STRIP];
        if constexpr (M > 0)
          corr_strip<STRIP, M>(imgs + s * imgF, Ks + s * patF, g.row, y, x0, cs, off, acc);
        else
          corr_strip_any<STRIP>(imgs + s * imgF, m, g.mp, Ks + s * patF, g.row, y, x0, cs, off, acc);
        float* out = corr + s * cc + y * cs + x0;
        if (x0 + STRIP <= cs && (cs & 3) == 0) {
#pragma unroll
          for (int e = 0; e < STRIP; e += 4)
            *reinterpret_cast<float4*>(out + e) = make_float4(acc[e], acc[e + 1], acc[e + 2], acc[e + 3]);
        } else {
#pragma unroll
          for (int e = 0; e < STRIP; e++)
            if (x0 + e < cs) out[e] = acc[e];
        }
      }
    } else
    for (int w = tid; w < ns * cc; w += blockDim.x) {
      const int s = w / cc, o = w - s * cc, y = o / cs, x = o - y * cs;
      const float* img = imgs + s * imgF;
      const float* K = Ks + s * patF;
      float v = 0.f;
      if (c.mode == 3) {
        // the abs-difference branch writes output (i + (nimg-ncen)/2,
        // j + (nimg-ncen)/2) of a corrsize-wide array
        const int i = y - (m - ncen) / 2, j = x - (m - ncen) / 2;
        if (i >= 0 && i < ncen && j >= 0 && j < ncen) {
          const int my = cs - abs(ncen / 2 - i), mx = cs - abs(ncen / 2 - j);
          float sacc = 0.f;
          for (int yy = 0; yy < my; yy++)
            for (int xx = 0; xx < mx; xx++) {
              float d;
              if (i < ncen / 2) {
                if (j < ncen / 2)
                  d = K[yy * cs + xx] - img[(ncen / 2 - i + yy) * m + ncen / 2 - j + xx];
                else
                  d = K[yy * cs + j - ncen / 2 + xx] - img[(ncen / 2 - i + yy) * m + xx];
              } else {
                if (j < ncen / 2)
                  d = K[(i - ncen / 2 + yy) * cs + xx] - img[yy * m + ncen / 2 - j + xx];
                else
                  d = K[(i - ncen / 2 + yy) * cs + j - ncen / 2 + xx] - img[yy * m + xx];
              }
              sacc += fabsf(d);
            }
          v = sacc * sacc / (float)(my * mx);
        }
      } else {
        const int i = y - (cs - ncen) / 2, j = x - (cs - ncen) / 2;
        if (i >= 0 && i < ncen && j >= 0 && j < ncen) {
          int srefy, siny, my, srefx, sinx, mx;
          overlap(i, m, cs, ncen, srefy, siny, my);
          overlap(j, m, cs, ncen, srefx, sinx, mx);
          float sacc = 0.f, tot = 0.f, tot2 = 0.f;
          for (int yy = 0; yy < my; yy++)
            for (int xx = 0; xx < mx; xx++) {
              const float b = img[(siny + yy) * m + sinx + xx];
              const float p = K[(srefy + yy) * cs + srefx + xx];
              if (c.mode == 5) {
                sacc += p * b;
              } else {
                const float d = p - b;
                sacc += d * d;
                tot += b;
                tot2 += p;
              }
            }
          if (c.mode == 2) {
            if (mx != 0 && my != 0) v = sacc / (float)(mx * my);
          } else if (c.mode == 4) {
            if (tot != 0.f && tot2 != 0.f) v = sacc / (tot * tot2);
          } else if (mx != 0 && my != 0) {
            v = sacc;
          }
        }
      }
      corr[w] = v;
    }
    __syncthreads();
    // ---- threshold (a fraction of the maximum when 0 < thresh <= 1), and
    // the thresholded image to corrimg: one warp per subaperture ----
    for (int s = warp; s < ns; s += nwarps) {
      float* im = corr + s * cc;
      float t = c.thresh;
      if (t <= 1.f && t > 0.f) {
        float mx = 0.f;
        for (int k = lane; k < cc; k += 32) mx = fmaxf(mx, im[k]);
#pragma unroll
        for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        t = mx * t;
      }
      __syncwarp();
      float* out = c.corrimg + (long long)s_frame[s] * c.corrimgFrameStride + (long long)s_subap[s] * cc;
      for (int k = lane; k < cc; k += 32) {
        const float v = im[k] < t ? 0.f : im[k] - t;
        im[k] = v;
        out[k] = v;
      }
    }
    __syncthreads();
    centroid_tile(ac, ns, s_subap, s_frame, s_cw, [&](int s) { return corr + s * cc; });
    if (ac.gaussianFit > 0 && ac.opticalBinning != 1) {
      // the Gaussian fit logs its input in place (cmod/src/centmodule.c:
      // 1087-1096); with correlation that input is the corrimg output
      __syncthreads();
      for (int s = warp; s < ns; s += nwarps) {
        float* out = c.corrimg + (long long)s_frame[s] * c.corrimgFrameStride + (long long)s_subap[s] * cc;
        for (int k = lane; k < cc; k += 32) out[k] = corr[s * cc + k];
      }
    }
  }
}

// testcorrelation: the correlation of one n x n image with a pattern whose
// inverse transform is K (mode 1 with corrsize = nimg = n: a circular
// convolution, summed in the correlation kernel's order)
__global__ void test_corr_kernel(int n, const float* __restrict__ img, const float* __restrict__ K,
                                 float* __restrict__ out) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n * n) return;
  const int y = o / n, x = o - y * n;
  float v = 0.f;
  for (int p = 0; p < n; p++) {
    int ky = y - p;
    if (ky < 0) ky += n;
    int kx = x;
    for (int q = 0; q < n; q++) {
      v += img[p * n + q] * K[ky * n + kx];
      kx = kx == 0 ? n - 1 : kx - 1;
    }
  }
  out[o] = v;
}

}  // namespace

cudaError_t launch_test_corr(int n, const float* img, const float* K, float* out, cudaStream_t stream) {
  const int nn = n * n;
  test_corr_kernel<<<(nn + 255) / 256, 256, 0, stream>>>(n, img, K, out);
  return cudaGetLastError();
}

cudaError_t launch_corr(const WfsArgs& a, CorrArgs c, int numSMs, cudaStream_t stream) {
  const long long nwork = (long long)a.nlit * a.nframes;
  if (nwork == 0) return cudaSuccess;
  const int cc = c.cs * c.cs;
  const CorrStrips g = corr_strips(c.mode, a.m, c.cs);
  const int per = a.m * g.mp + c.cs * g.row + cc;  // floats per subaperture
  // up to about two strips (or eight outputs of the other modes) per thread,
  // within 48 KB, and no more than an even share of the SMs; of these the tile
  // whose last round of threads is fullest
  const int items = g.strip ? c.cs * g.strips : std::max(1, cc / 4);
  long long most = (2 * kCorrThreads + items - 1) / items;
  most = std::min<long long>(most, 12288 / per);
  most = std::min<long long>(most, (nwork + numSMs - 1) / numSMs);
  most = std::max<long long>(1, std::min<long long>(most, kCorrMaxTS));
  double best = 0.0;
  for (int t = (int)most; t >= 1; t--) {
    const double use = (double)t * items / ((t * items + kCorrThreads - 1) / kCorrThreads * kCorrThreads);
    if (use > best + 0.01) {
      best = use;
      c.TS = t;
    }
  }
  const int smem = (c.TS * per + 4 + (a.centWeightDim == 2 ? cc : 0)) * (int)sizeof(float);
  // image widths of 4 to 16 pixels have their row loop unrolled (16 covers the
  // sensors in use; a wider image amortises the general loop over more pixels)
  using Kern = void (*)(const WfsArgs, const CorrArgs, const CorrStrips);
  static const Kern sized[13] = {wfs_corr_kernel<8, 4>,  wfs_corr_kernel<8, 5>,  wfs_corr_kernel<8, 6>,
                                 wfs_corr_kernel<8, 7>,  wfs_corr_kernel<8, 8>,  wfs_corr_kernel<8, 9>,
                                 wfs_corr_kernel<8, 10>, wfs_corr_kernel<8, 11>, wfs_corr_kernel<8, 12>,
                                 wfs_corr_kernel<8, 13>, wfs_corr_kernel<8, 14>, wfs_corr_kernel<8, 15>,
                                 wfs_corr_kernel<8, 16>};
  const Kern kern = g.strip == 0               ? wfs_corr_kernel<0, 0>
                    : a.m >= 4 && a.m <= 16 ? sized[a.m - 4]
                                            : wfs_corr_kernel<8, 0>;
  cudaError_t e = kernel_smem_setup((const void*)kern, smem, kCorrThreads, nullptr);
  if (e != cudaSuccess) return e;
  const long long ntiles = (nwork + c.TS - 1) / c.TS;
  const long long cap = (long long)numSMs * 16;
  const int grid = (int)(ntiles < cap ? ntiles : cap);
  kern<<<grid, kCorrThreads, smem, stream>>>(a, c, g);
  return cudaGetLastError();
}

}  // namespace shwfs

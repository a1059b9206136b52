// FP32 image formation, one warp per group of subaperture-frames: the stages
//
//   1 field             conj(pup*exp(i(phs-tilt))), lanes over the pixels  (centmodule.c:473-497)
//   2 row FFTs          the p non-zero rows, an N-point FFT per lane; inputs
//                       from N/2 on are zero and left out of the transform
//   3 column FFTs, |F|^2  two neighbouring rows per complex value            (:498-504, :430-471)
//   4 spot-PSF convolution (r2c rows two per complex FFT, column FFT *
//     PSF spectrum * inverse column FFT in registers, c2r rows)             (:524-564)
//   5 binning, normalisation, sky                                           (:609-651, 1829-1872)
//   6 threshold, pixel power, window CoG, calibration, references of frames
//     without noise (:1893-1961); other frames leave the pre-noise images in
//     bimg for the noise/centroid kernel (wfs_post.cu)
//
// run within a warp, on one complex buffer per subaperture of N/2 rows that
// every stage transforms in place: a lane reads its row (column) into
// registers, transforms it and writes it back, so the only synchronisation is
// __syncwarp and 8 to 20 independent warps per SM hide each other's latency.
// Bound by instruction issue (the transforms' additions and multiplications
// and their shared-memory accesses; 2.4 GFLOP and 51 MB for 16 frames of the
// 74x74 sensor, 30 us at the nominal FP32 rate and 8 us of memory time).  The
// block form (wfs_plain.cuh), which keeps 128 threads in step over uneven
// stages and transforms the zero inputs and the unbinned image too, took 341
// us there, this one 121 (130 with scalar butterflies and five CTAs per SM at
// 20 points); one frame of the 74x74 LGS sensor (fftsize 32, a PSF per
// subaperture) 114 and 27 us, one 8x8 frame through host arrays 32 and 17.
//
// The field is conjugated because |DFT(conj E)|^2 at u is |DFT(E)|^2 at N - u:
// the 180-degree rotation of the power spectrum (addPowerSpecCentral) is then
// a shift by one, which the next stage applies by reading its constant
// indices rotated.  The DC and Nyquist columns of a row-transformed real
// image are real and share one complex column (PACK below), which makes N/2
// columns of N/2 + 1 and N/2 slots per lane group in every stage.  When the
// image bins F by F pixels, F = 2 or 4, the product with the PSF spectrum is
// multiplied by the response of the sum of F pixels and folded to N/F
// frequencies per axis, so that the inverse transforms are of that size and
// give the binned image.
//
// Even N, with no PSF or an N x N PSF, no pre-binning, phase-only input, no
// optical binning (form_covers); everything else takes the block form.
#pragma once
#include <array>
#include <map>
#include <type_traits>

#include "wfs_plain.cuh"

namespace shwfs {

// ---- transforms whose inputs from NZ on are zero ----
template <int R, int S, int NZ>
__device__ __forceinline__ void butterfly_nz(float2 (&a)[R]) {
  if constexpr (NZ >= R) {
    butterfly<R, S>(a);
  } else if constexpr (NZ == 1) {
#pragma unroll
    for (int k = 1; k < R; k++) a[k] = a[0];
  } else if constexpr (R == 3) {  // NZ == 2
    constexpr float h = 0.866025403784438647f;  // sin(2 pi / 3)
    const float2 b = make_float2(a[0].x - 0.5f * a[1].x, a[0].y - 0.5f * a[1].y);
    const float2 d = cscale(cmuli(a[1]), S * h);
    a[0] = cadd(a[0], a[1]);
    a[1] = cadd(b, d);
    a[2] = csub(b, d);
  } else if constexpr (R == 4) {  // NZ == 2 or 3
    float2 i1 = cmuli(a[1]);
    if (S < 0) i1 = make_float2(-i1.x, -i1.y);
    const float2 s = NZ == 3 ? padd(a[0], a[2]) : a[0], d = NZ == 3 ? psub(a[0], a[2]) : a[0], b = a[1];
    a[0] = padd(s, b);
    a[2] = psub(s, b);
    a[1] = cadd(d, i1);
    a[3] = csub(d, i1);
  } else {  // R == 5, NZ == 2, 3 or 4
    constexpr float c1 = 0.309016994374947424f, c2 = -0.809016994374947424f;  // cos(2 pi / 5), cos(4 pi / 5)
    constexpr float s1 = 0.951056516295153572f, s2 = 0.587785252292473129f;   // sin(2 pi / 5), sin(4 pi / 5)
    const float2 x0 = a[0], x1 = a[1], x2 = a[2], x3 = a[3];
    float2 b1 = pfma(c1, x1, x0), b2 = pfma(c2, x1, x0), e1 = pmul(s1, x1), e2 = pmul(s2, x1);
    a[0] = padd(x0, x1);
    if constexpr (NZ > 2) {
      const float2 t2 = NZ > 3 ? padd(x2, x3) : x2, t4 = NZ > 3 ? psub(x2, x3) : x2;
      b1 = pfma(c2, t2, b1);
      b2 = pfma(c1, t2, b2);
      e1 = pfma(s2, t4, e1);
      e2 = pfma(-s1, t4, e2);
      a[0] = padd(a[0], t2);
    }
    const float2 d1 = cscale(cmuli(e1), (float)S), d2 = cscale(cmuli(e2), (float)S);
    a[1] = cadd(b1, d1);
    a[4] = csub(b1, d1);
    a[2] = cadd(b2, d2);
    a[3] = csub(b2, d2);
  }
}

// fft<N, S, NT> of x with x[j] = 0 for j >= NZ (those entries are not read)
template <int N, int S, int NT, int NZ>
__device__ __forceinline__ void fft_nz(float2 (&x)[N]) {
  if constexpr (NZ >= N) {
    fft<N, S, NT>(x);
  } else if constexpr (N == 2 || N == 3 || N == 4 || N == 5) {
    butterfly_nz<N, S, NZ>(x);
  } else {
    constexpr int R = first_radix(N);
    constexpr int M = N / R;
    constexpr int RZ = NZ < R ? NZ : R;  // sub-sequences with a non-zero input
    float2 sub[RZ][M];
    auto one = [&](auto rc) {
      constexpr int r = decltype(rc)::value;
      if constexpr (r < RZ) {
        constexpr int nz = (NZ - r + R - 1) / R;
#pragma unroll
        for (int q = 0; q < nz; q++) sub[r][q] = x[R * q + r];
        fft_nz<M, S, NT, nz>(sub[r]);
      }
    };
    one(std::integral_constant<int, 0>{});
    one(std::integral_constant<int, 1>{});
    one(std::integral_constant<int, 2>{});
    one(std::integral_constant<int, 3>{});
    one(std::integral_constant<int, 4>{});
#pragma unroll
    for (int k1 = 0; k1 < M; k1++) {
      float2 t[R];
      t[0] = sub[0][k1];
#pragma unroll
      for (int r = 1; r < RZ; r++) t[r] = k1 == 0 ? sub[r][0] : cmul(sub[r][k1], twiddle<NT, S>(r * k1 * (NT / N)));
      butterfly_nz<R, S, RZ>(t);
#pragma unroll
      for (int k2 = 0; k2 < R; k2++) x[k1 + M * k2] = t[k2];
    }
  }
}

// ---- geometry ----
template <int N>
struct FormGeom {
  static constexpr int H = N / 2;                 // rows of the complex buffer, lanes of a subaperture
  static constexpr int ZS = N + 1;                // its row stride (complex): odd, conflict-free down a column
  static constexpr int S = 32 / H < 1 ? 1 : 32 / H;  // most subaperture-frames per warp
};
// one warp's shared memory in floats: the complex buffers, the final images
// and the centroid row sums of S subaperture-frames
__host__ __device__ inline int form_warp_floats(int N, int S, int m, int ncen) {
  return ((2 * (N / 2) * (N + 1) * S + m * m * S + 3) & ~3) + 2 * S * ncen;
}
// per-CTA constants in floats: the pixel table, the PSF spectrum (2-D PSF),
// the bin tables and the centroid weights (2-D)
__host__ __device__ inline int form_const_floats(int N, int P, int p, int C, int m, bool psf2d, bool cw2d) {
  return ((4 * p * p + (psf2d ? 2 * P * (P / 2 + 1) : 0) + 3 * C + 2 * m + (cw2d ? m * m : 0)) + 3) & ~3;
}
constexpr int kFormWarps = 4;

// sum of exp(2 pi i j k / N) over j < F: the response of the sum of F pixels
template <int N, int F>
struct BinTable {
  float2 v[N];
};
template <int N, int F>
__host__ __device__ constexpr BinTable<N, F> make_bin_table() {
  BinTable<N, F> t{};
  for (int k = 0; k < N; k++) {
    double c = 0.0, s = 0.0;
    for (int j = 0; j < F; j++) {
      const CS e = cos_sin_frac(j * k % N, N);
      c += e.c;
      s += e.s;
    }
    t.v[k] = float2{(float)c, (float)s};
  }
  return t;
}

template <int N, int P, int F>
__device__ __forceinline__ void form_body(const WfsArgs& a, long long warp0, long long nwarps) {
  using G = FormGeom<N>;
  constexpr int H = G::H, ZS = G::ZS;
  constexpr int M = N / F;  // size of the inverse transforms
  constexpr BinTable<N, F> kBin = make_bin_table<N, F>();
  static_assert(P == 0 || P == N, "the PSF has the FFT's size");
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int p = a.p, pp = p * p, C = a.C, m = a.m, mm = m * m, ncen = a.ncen;
  const bool cw2d = a.centWeightDim == 2;
  const bool psf2d = P > 0 && a.psfDim == 2;
  constexpr int HS = N / 2 + 1;
  const int S = a.TS;  // subaperture-frames per warp (at most G::S)

  // --- per-CTA constants ---
  int4* s_pix = reinterpret_cast<int4*>(smem);  // {phase offset, buffer slot, tilt, -} of each pixel
  float2* s_psf = reinterpret_cast<float2*>(smem + 4 * pp);
  float* s_binT = smem + 4 * pp + (psf2d ? 2 * N * HS : 0);
  float* s_binN = s_binT + C;
  int* s_binII = reinterpret_cast<int*>(s_binN + C);
  int* s_binLo = s_binII + C;
  int* s_binHi = s_binLo + m;
  float* s_cw = reinterpret_cast<float*>(s_binHi + m);
  float* mine = smem + form_const_floats(N, P, p, C, m, psf2d, cw2d) + warp * form_warp_floats(N, S, m, ncen);
  float2* zb = reinterpret_cast<float2*>(mine);
  float* img = mine + 2 * H * ZS * S;
  float* rows = mine + ((2 * H * ZS * S + mm * S + 3) & ~3);
  __shared__ long long s_src[kFormWarps][8], s_dst[kFormWarps][8];  // phase and image offsets of the group's items
  __shared__ int s_sub[kFormWarps][8], s_frm[kFormWarps][8];
  __shared__ float2 s_norm[kFormWarps][8];  // scale, sky

  for (int k = tid; k < pp; k += blockDim.x) {
    const int r = k / p, j = k - r * p;
    s_pix[k] = make_int4(r * a.W + j, r * ZS + j, __float_as_int(a.tilt[k]), 0);
  }
  if (psf2d)
    // column 0 takes the DC and the Nyquist column at once: y' = A y + B
    // conj(y(-k)) with A, B the mean and half the difference of the two
    for (int k = tid; k < N * HS; k += blockDim.x) {
      const int c = k % HS;
      float2 v = a.psfSpec[k];
      if (c == 0) {
        const float2 n = a.psfSpec[k + N / 2];
        v = make_float2(0.5f * (v.x + n.x), 0.5f * (v.y + n.y));
      } else if (c == N / 2) {
        const float2 d = a.psfSpec[k - N / 2];
        v = make_float2(0.5f * (d.x - v.x), 0.5f * (d.y - v.y));
      }
      s_psf[k] = v;
    }
  if (F == 1) {
    for (int k = tid; k < C; k += blockDim.x) {
      s_binT[k] = a.binT[k];
      s_binN[k] = a.binN[k];
      s_binII[k] = a.binII[k];
    }
    for (int k = tid; k < m; k += blockDim.x) {
      s_binLo[k] = a.binLo[k];
      s_binHi[k] = a.binHi[k];
    }
  }
  if (cw2d)
    for (int k = tid; k < mm; k += blockDim.x) s_cw[k] = a.centWeight[k];
  __syncthreads();
  // the noise/centroid kernel launched programmatically behind this one may
  // become resident; it waits for the whole grid before it reads bimg
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (a.zeroUnlit) {
    // unlit subapertures: centroids 0 (cmod/src/centmodule.c:1964-1981)
    const long long nu = (long long)a.nunlit * a.nframes;
    for (long long u = warp0 * 32 + lane; u < nu; u += nwarps * 32) {
      const int f = (int)(u / a.nunlit), i = a.unlit[u - (long long)f * a.nunlit];
      float* c = a.cents + (long long)f * a.centsFrameStride + 2LL * i;
      c[0] = 0.f;
      c[1] = 0.f;
    }
  }

  const bool storePre = a.mode & kStorePreNoise;
  const int rofs = P > 0 ? 1 : (N - (N - C) / 2 - C + 1) % N;  // image row i is |F|^2 row (i + rofs) mod N
  const int whole = C % m == 0 ? C / m : 0;  // pixels binned per axis, 0 when fractional
  const float inv_m = 1.0f / (float)m, inv_nc = 1.0f / (float)ncen;
  const long long nwork = (long long)a.nlit * a.nframes;
  const long long ngroups = (nwork + S - 1) / S;
  for (long long g = warp0; g < ngroups; g += nwarps) {
    const int ns = (int)min((long long)S, nwork - g * S);
    if (lane < ns) {
      const long long w = g * S + lane;
      const int f = nwork < 0x7fffffffLL ? (int)((unsigned)w / (unsigned)a.nlit) : (int)(w / a.nlit);
      const int i = a.lit[w - (long long)f * a.nlit];
      const int sy = i / a.nsubx, sx = i - sy * a.nsubx;
      s_src[warp][lane] = (long long)f * a.phsFrameStride + (long long)(sy * p) * a.W + sx * p;
      s_dst[warp][lane] = (long long)f * a.bimgFrameStride + (long long)i * mm;
      s_sub[warp][lane] = i;
      s_frm[warp][lane] = f;
      const float totsig = a.totsig[i], fr = a.frac[i];
      float scale = 1.f;
      if (totsig > 0.f) scale = a.sigArr ? a.sigArr[i] / totsig : a.sig * fr / totsig;
      const float skyv = a.sky * fr;
      // the row transforms of the convolution leave out their factor 1/2
      s_norm[warp][lane] = make_float2(P > 0 ? 0.5f * scale : scale, skyv);
      if (storePre && a.poisFlag) a.poisFlag[i] = (totsig > 0.f || skyv > 0.f || a.skyArr) ? 1 : 0;
    }
    if (p < H)
      for (int k = lane; k < ns * H * ZS; k += 32) zb[k] = make_float2(0.f, 0.f);
    __syncwarp();

    // ---- 1: field ----
    {
      int s = 0, pix = lane;
      while (pix >= pp) {
        pix -= pp;
        s++;
      }
      while (s < ns) {
        const int4 e = s_pix[pix];
        const float t = a.phs[s_src[warp][s] + e.x] - __int_as_float(e.z);
        const float amp = a.pup[(long long)s_sub[warp][s] * pp + pix];
        float sn, cs;
        sincosf(t, &sn, &cs);
        zb[s * (H * ZS) + e.y] = make_float2(amp * cs, -(amp * sn));
        pix += 32;
        while (pix >= pp) {
          pix -= pp;
          s++;
        }
      }
    }
    __syncwarp();

    // lane -> (subaperture, row or column) of the stages with H per subaperture
    const int ls = lane / H, lq = lane - ls * H;
    const bool on = ls < ns;
    // ---- 2: row FFTs ----
    if (on && lq < p) {
      float2* r = zb + ls * (H * ZS) + lq * ZS;
      float2 x[N];
#pragma unroll
      for (int j = 0; j < H; j++) x[j] = r[j];
      fft_nz<N, -1, N, H>(x);
#pragma unroll
      for (int k = 0; k < N; k++) r[k] = x[k];
    }
    __syncwarp();
    // ---- 3: column FFTs, |F|^2 of rows 2q and 2q + 1 as one complex value ----
#pragma unroll 1
    for (int w = lane; w < ns * N; w += 32) {
      const int s = w / N;
      float2* c = zb + s * (H * ZS) + (w - s * N);
      float2 x[N];
#pragma unroll
      for (int r = 0; r < H; r++) x[r] = c[r * ZS];
      fft_nz<N, -1, N, H>(x);
#pragma unroll
      for (int q = 0; q < H; q++)
        c[q * ZS] = make_float2(x[2 * q].x * x[2 * q].x + x[2 * q].y * x[2 * q].y,
                                x[2 * q + 1].x * x[2 * q + 1].x + x[2 * q + 1].y * x[2 * q + 1].y);
    }
    __syncwarp();

    if constexpr (P > 0) {
      // ---- 4a: r2c of row pairs (X, Y the spectra of rows 2q and 2q + 1,
      // doubled); entry 0 of each holds its real DC and Nyquist values ----
      if (on) {
        float2* r = zb + ls * (H * ZS) + lq * ZS;
        float2 z[N];
#pragma unroll
        for (int n = 0; n < N; n++) z[n] = r[(n + 1) % N];
        fft<N, -1>(z);
        r[0] = make_float2(2.f * z[0].x, 2.f * z[H].x);
        r[H] = make_float2(2.f * z[0].y, 2.f * z[H].y);
#pragma unroll
        for (int k = 1; k < H; k++) {
          const float2 u = z[k], v = z[N - k];
          r[k] = make_float2(u.x + v.x, u.y - v.y);
          r[H + k] = make_float2(u.y + v.y, v.x - u.x);
        }
      }
      __syncwarp();
      // ---- 4b: column FFT, * PSF spectrum, [fold], inverse column FFT ----
      if (on) {
        float2* c = zb + ls * (H * ZS) + lq;
        const float2* psf = psf2d ? s_psf : a.psfSpec + (long long)s_sub[warp][ls] * N * HS;
        float2 y[N];
#pragma unroll
        for (int r = 0; r < N; r++) y[r] = c[(((r + 1) % N) >> 1) * ZS + (((r + 1) % N) & 1) * H];
        fft<N, -1>(y);
#pragma unroll
        for (int k = 0; k <= H; k++) {
          const int n = (N - k) % N;
          float2 ak = psf[k * HS + lq], an = psf[n * HS + lq], bk, bn;
          const float2 yk = y[k], yn = y[n];
          if (lq == 0) {
            bk = psf[k * HS + H];
            bn = psf[n * HS + H];
            if (!psf2d) {
              const float2 dk = ak, dn = an;
              ak = make_float2(0.5f * (dk.x + bk.x), 0.5f * (dk.y + bk.y));
              bk = make_float2(0.5f * (dk.x - bk.x), 0.5f * (dk.y - bk.y));
              an = make_float2(0.5f * (dn.x + bn.x), 0.5f * (dn.y + bn.y));
              bn = make_float2(0.5f * (dn.x - bn.x), 0.5f * (dn.y - bn.y));
            }
          }
          y[k] = cmul(ak, yk);
          if (n != k) y[n] = cmul(an, yn);
          if (lq == 0) {
            y[k] = cadd(y[k], cmul(bk, cconj(yn)));
            if (n != k) y[n] = cadd(y[n], cmul(bn, cconj(yk)));
          }
        }
        float2 v[M];
#pragma unroll
        for (int k = 0; k < M; k++) {
          v[k] = F == 1 ? y[k] : cmul(y[k], kBin.v[k]);
#pragma unroll
          for (int f = 1; f < F; f++) v[k] = cadd(v[k], cmul(y[k + f * M], kBin.v[k + f * M]));
        }
        fft<M, 1, N>(v);
#pragma unroll
        for (int r = 0; r < M; r++) c[(r >> 1) * ZS + (r & 1) * H] = v[r];
      }
      __syncwarp();
      // ---- 4c: c2r of row pairs [folded]: pixel x of rows 2q and 2q + 1 as
      // one complex value ----
      if (on && lq < (M + 1) / 2) {
        float2* r = zb + ls * (H * ZS) + lq * ZS;
        const bool two = 2 * lq + 1 < M;
        float2 z[M];
        const float2 x0 = r[0], y0 = two ? r[H] : make_float2(0.f, 0.f);
        if constexpr (F > 1) {
          // frequency i of the real row whose entries start at o
          auto at = [&](int o, int i) {
            return i == H ? make_float2(o ? y0.y : x0.y, 0.f) : (i < H ? r[o + i] : cconj(r[o + N - i]));
          };
          z[0] = make_float2(F * x0.x, F * y0.x);
#pragma unroll
          for (int l = 1; l <= M / 2; l++) {
            float2 X = make_float2(0.f, 0.f), Y = X;
#pragma unroll
            for (int f = 0; f < F; f++) {
              const float2 bf = kBin.v[l + f * M];
              X = f == 0 ? cmul(at(0, l), bf) : cadd(X, cmul(at(0, l + f * M), bf));
              if (two) Y = f == 0 ? cmul(at(H, l), bf) : cadd(Y, cmul(at(H, l + f * M), bf));
            }
            if (2 * l == M) {
              z[l] = make_float2(X.x, Y.x);
            } else {
              z[l] = make_float2(X.x - Y.y, X.y + Y.x);
              z[M - l] = make_float2(X.x + Y.y, Y.x - X.y);
            }
          }
        } else {
          z[0] = make_float2(x0.x, y0.x);
          z[H] = make_float2(x0.y, y0.y);
#pragma unroll
          for (int l = 1; l < H; l++) {
            const float2 X = r[l], Y = r[H + l];
            z[l] = make_float2(X.x - Y.y, X.y + Y.x);
            z[N - l] = make_float2(X.x + Y.y, Y.x - X.y);
          }
        }
        fft<M, 1, N>(z);
#pragma unroll
        for (int x = 0; x < M; x++) r[x] = z[x];
      }
      __syncwarp();
    }

    // ---- 5: bin, normalise, sky [threshold, power] -> bimg ----
    const float* zf = reinterpret_cast<const float*>(zb);
    int s5 = 0, pix5 = lane;
    while (pix5 >= mm) {
      pix5 -= mm;
      s5++;
    }
    for (int w = lane; w < ns * mm; w += 32) {
      const int s = s5, pix = pix5;
      pix5 += 32;
      while (pix5 >= mm) {
        pix5 -= mm;
        s5++;
      }
      int I, J;
      if constexpr (F > 1) {
        I = pix / M;
        J = pix - I * M;
      } else {
        I = div_small(pix, m, inv_m);
        J = pix - I * m;
      }
      const float* z = zf + s * (2 * H * ZS);
      auto at = [&](int i, int j) {  // pixel (i, j) of the C x C image
        if (P == 0) {
          i += rofs;
          j += rofs;
          if (i >= N) i -= N;
          if (j >= N) j -= N;
        }
        return z[2 * ((i >> 1) * ZS + j) + (i & 1)];
      };
      float v;
      if (F > 1 || C == m) {
        v = at(I, J);
      } else if (whole == 2) {
        v = at(2 * I, 2 * J) + at(2 * I, 2 * J + 1) + at(2 * I + 1, 2 * J) + at(2 * I + 1, 2 * J + 1);
      } else if (whole) {
        v = 0.f;
        for (int i = whole * I; i < whole * (I + 1); i++)
          for (int j = whole * J; j < whole * (J + 1); j++) v += at(i, j);
      } else {
        v = 0.f;
        const int ilo = s_binLo[I], ihi = s_binHi[I], jlo = s_binLo[J], jhi = s_binHi[J];
        for (int ii = ilo; ii <= ihi; ii++) {
          const int iiv = s_binII[ii];
          const bool lastI = ii == C - 1;
          for (int jj = jlo; jj <= jhi; jj++) {
            const int jjv = s_binII[jj];
            const bool lastJ = jj == C - 1;
            if (iiv == I) {
              if (jjv == J)
                v += s_binT[ii] * s_binT[jj] * at(ii, jj);
              else if (jjv + 1 == J && !lastJ)
                v += s_binT[ii] * s_binN[jj] * at(ii, jj + 1);
            } else if (iiv + 1 == I && !lastI) {
              if (jjv == J)
                v += s_binN[ii] * s_binT[jj] * at(ii + 1, jj);
              else if (jjv + 1 == J && !lastJ)
                v += s_binN[ii] * s_binN[jj] * at(ii + 1, jj + 1);
            }
          }
        }
      }
      const float2 nv = s_norm[warp][s];
      v *= nv.x;
      if (nv.y > 0.f) v += nv.y;
      if (a.skyArr) v += a.skyArr[(long long)s_sub[warp][s] * mm + pix];
      if (!storePre) {
        v = threshold_px(v + a.readBg, a.floorv, a.threshType);
        if (a.pxlPower == 2.f)
          v = v * v;
        else if (a.pxlPower != 1.f && a.pxlPower != 0.f)
          v = powf(v, a.pxlPower);
        img[w] = v;
      }
      a.bimg[s_dst[warp][s] + pix] = v;
    }
    if (!storePre && !a.imageOnly && !a.skipCents) {
      __syncwarp();
      // ---- 6: centred-window CoG: sums of each window row, then of the rows,
      // with coordinates from the image centre (taking it off afterwards
      // cancels most of the digits) ----
      const int sx0 = (m - ncen) / 2;
      const float mid = 0.5f * (float)(m - 1);
      for (int t = lane; t < ns * ncen; t += 32) {
        const int s = div_small(t, ncen, inv_nc), r = sx0 + (t - s * ncen);
        const float* row = img + s * mm + r * m + sx0;
        const float* wrow = cw2d ? s_cw + r * m + sx0
                                 : (a.centWeightDim == 4 ? a.centWeight + (long long)s_sub[warp][s] * mm + r * m + sx0
                                                         : nullptr);
        float ps = 0.f, px = 0.f;
        for (int c = 0; c < ncen; c++) {
          const float v = wrow ? row[c] * wrow[c] : row[c];
          ps += v;
          px += v * ((float)(sx0 + c) - mid);
        }
        rows[2 * t] = ps;
        rows[2 * t + 1] = px;
      }
      __syncwarp();
      if (lane < ns) {
        float sum = 0.f, sxv = 0.f, syv = 0.f;
        for (int rr = 0; rr < ncen; rr++) {
          const float ps = rows[2 * (lane * ncen + rr)];
          sum += ps;
          sxv += rows[2 * (lane * ncen + rr) + 1];
          syv += ps * ((float)(sx0 + rr) - mid);
        }
        float cx = 0.f, cy = 0.f;
        if (sum > 0.f) {
          cx = sxv / sum;
          cy = syv / sum;
        }
        calibrate_and_store(a, s_sub[warp][lane], s_frm[warp][lane], cx, cy);
      }
    }
    __syncwarp();  // the group's buffers and tables are consumed
  }
}

// CTAs per SM that the registers are cut for: the most that do not spill in the
// form's main variants (20 points: six at 80 registers 122 us, five 125).
template <int N>
constexpr int form_min_blocks() {
  return N <= 20 ? 6 : (N <= 24 ? 5 : (N <= 32 ? 4 : 2));
}
template <int N, int P, int F>
__global__ void __launch_bounds__(32 * kFormWarps, form_min_blocks<N>()) wfs_form_kernel(const __grid_constant__ WfsArgs a) {
  const int warps = blockDim.x >> 5;
  form_body<N, P, F>(a, (long long)blockIdx.x * warps + (threadIdx.x >> 5), (long long)gridDim.x * warps);
}

// Several handles of one instantiation in one launch (the multi-sensor
// batches): handle h owns CTAs [ctaStart[h], ctaStart[h+1]) and each of them
// loops over that handle's groups, as in a launch of its own.
constexpr int kFormMulti = 8;
struct FormMulti {
  WfsArgs a[kFormMulti];
  int ctaStart[kFormMulti + 1];
  int n;
};
template <int N, int P, int F>
__global__ void __launch_bounds__(32 * kFormWarps, form_min_blocks<N>())
    wfs_form_multi_kernel(const __grid_constant__ FormMulti m) {
  int h = 0;
  while (h + 1 < m.n && (int)blockIdx.x >= m.ctaStart[h + 1]) h++;
  const int warps = blockDim.x >> 5;
  form_body<N, P, F>(m.a[h], (long long)((int)blockIdx.x - m.ctaStart[h]) * warps + (threadIdx.x >> 5),
                     (long long)(m.ctaStart[h + 1] - m.ctaStart[h]) * warps);
}

// ---- registry of the compiled instantiations ----
struct FormEntry {
  int maxS;  // most subaperture-frames per warp
  cudaError_t (*launch)(const WfsArgs&, int grid, int threads, int smem, cudaStream_t);
  cudaError_t (*occupancy)(int* ctas_per_sm, int threads, int smem);
  cudaError_t (*launch_multi)(const FormMulti& m, int threads, int smem, cudaStream_t);
  cudaError_t (*occupancy_multi)(int* ctas_per_sm, int threads, int smem);
};
// (fftsize, 0 without a spot PSF else fftsize, pixels binned per axis in the
// transforms: 1, 2 or 4)
using FormKey = std::array<int, 3>;
inline std::map<FormKey, FormEntry>& form_registry() {
  static std::map<FormKey, FormEntry> r;
  return r;
}

template <int N, int P, int F>
struct FormRegistrar {
  static cudaError_t launch(const WfsArgs& a, int grid, int threads, int smem, cudaStream_t stream) {
    cudaError_t e = kernel_smem_setup((const void*)wfs_form_kernel<N, P, F>, smem, threads, nullptr);
    if (e != cudaSuccess) return e;
    wfs_form_kernel<N, P, F><<<grid, threads, smem, stream>>>(a);
    return cudaGetLastError();
  }
  static cudaError_t occupancy(int* ctas, int threads, int smem) {
    return kernel_smem_setup((const void*)wfs_form_kernel<N, P, F>, smem, threads, ctas);
  }
  static cudaError_t launch_multi(const FormMulti& m, int threads, int smem, cudaStream_t stream) {
    cudaError_t e = kernel_smem_setup((const void*)wfs_form_multi_kernel<N, P, F>, smem, threads, nullptr);
    if (e != cudaSuccess) return e;
    wfs_form_multi_kernel<N, P, F><<<m.ctaStart[m.n], threads, smem, stream>>>(m);
    return cudaGetLastError();
  }
  static cudaError_t occupancy_multi(int* ctas, int threads, int smem) {
    return kernel_smem_setup((const void*)wfs_form_multi_kernel<N, P, F>, smem, threads, ctas);
  }
  FormRegistrar() {
    form_registry()[FormKey{N, P, F}] =
        FormEntry{FormGeom<N>::S, &launch, &occupancy, &launch_multi, &occupancy_multi};
  }
};

// fftsize N without a PSF, with an N x N PSF, and with one and images of N / 2
// pixels; SHWFS_REGISTER_FORM4 (N a multiple of 4): of N / 4 pixels too
#define SHWFS_REGISTER_FORM(N)                               \
  static ::shwfs::FormRegistrar<N, 0, 1> shwfs_form_##N##_0; \
  static ::shwfs::FormRegistrar<N, N, 1> shwfs_form_##N##_1; \
  static ::shwfs::FormRegistrar<N, N, 2> shwfs_form_##N##_2;
#define SHWFS_REGISTER_FORM4(N) \
  SHWFS_REGISTER_FORM(N)        \
  static ::shwfs::FormRegistrar<N, N, 4> shwfs_form_##N##_4;

}  // namespace shwfs

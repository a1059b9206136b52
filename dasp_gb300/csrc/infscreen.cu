// Infinite phase screen resident on the device (science/infScrn.py
// addNewColumnOnEnd :747-791, addNewRowOnEnd :825-855, addNewColumnOnStart
// :793-823, addNewRowOnStart :857-887): each new column (row) is
// A Z + coeff B n + step, Z the last two columns (rows) stacked oldest first,
// n standard normals; A and B come from the host in float64.  At the start
// of the screen the reference uses AStart, A with its two column blocks in
// reverse order (:722-731), on the first two lines stacked first line first:
// that is A applied with the second line in A's first block and the edge
// line in its second, which is how the kernel pairs them.
// The screen is a circular buffer in both axes: logical (y, x) lives at
// ((rs + y) % ny, (cs + x) % nx), so appending overwrites the oldest column
// (row) in place instead of shifting the screen as the reference does.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/shwfs.h"
#include "engine_internal.h"
#include "shwfs_dev.cuh"

struct shwfs_screen {
  int ny = 0, nx = 0;
  int rs = 0, cs = 0;             // circular starts (rows, columns)
  float* scr = nullptr;           // ny x nx, physical order
  double* a[2] = {nullptr, nullptr};  // [0] columns: ny x 2ny; [1] rows: nx x 2nx
  double* b[2] = {nullptr, nullptr};  // [0] ny x ny; [1] nx x nx
  double* noise = nullptr;        // max(ny, nx): injected normals of one line
  int numSMs = 1;
  int device = 0;
  cudaMemPool_t pool = nullptr;   // the device's scratch pool, shared by its screens
  shwfs::PhiloxKeys keys{};
  unsigned long long added = 0;   // extrusions so far (the noise stream's frame index)
  cudaStream_t stream = nullptr;
};

namespace shwfs {

namespace {

// (double)x by integer operations for zeros and normal values: the
// conversion instruction runs on the FP64 pipe, which the kernels below are
// bound by
__device__ __forceinline__ double to_double(float x) {
  const uint32_t u = __float_as_uint(x), m = u & 0x7fffffffu;
  if (m - 1u < 0x007fffffu || m >= 0x7f800000u) return (double)x;  // subnormal, infinite or NaN
  const uint32_t hi = (u & 0x80000000u) | (m ? (m >> 3) + 0x38000000u : 0u);
  return __hiloint2double((int)hi, (int)(u << 29));
}

// One new line (axis 0 a column, 1 a row): kLineThreads threads per output
// element, rowsPerCta elements per CTA, so that about one CTA per SM covers
// the line.  Bound by reading A and B once (24 len^2 bytes, L2-resident
// between lines) and by the FP64 rate (3 len^2 multiply-adds at about two a
// cycle and SM: 2.6 us for 741 elements); a warp per element with its z
// gathered by modulo from the circular buffer took 35 us for 741.  Here a
// thread has all its 36 matrix elements of a chunk in flight before the
// vectors are staged in shared memory, and the line's normals, B n and the
// matrix loads, which do not depend on the line before, run ahead of
// griddepcontrol.wait: successive lines are launched programmatically and
// overlap in that part.
constexpr int kLineThreads = 64;  // per output element
constexpr int kLineUnroll = 12;     // elements of each of A's two blocks and of B per thread and chunk
constexpr int kLineChunk = kLineThreads * kLineUnroll;
constexpr int kLineMaxRows = 8;

__global__ void __launch_bounds__(kLineThreads* kLineMaxRows)
    screen_line_kernel(float* __restrict__ scr, int ny, int nx, int rs, int cs, int axis, int start,
                       const double* __restrict__ A, const double* __restrict__ B, const PhiloxKeys keys,
                       unsigned long long ext, const double* __restrict__ noise, double coeff, double step) {
  __shared__ double s_n[kLineChunk], s_z[2][kLineChunk];
  __shared__ double s_red[kLineThreads * kLineMaxRows];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int len = axis == 0 ? ny : nx;  // output length; Z has 2 len entries
  const int tid = threadIdx.x, t = tid & (kLineThreads - 1), g = tid / kLineThreads;
  const int rows = blockDim.x / kLineThreads;
  const int i = blockIdx.x * rows + g;
  const bool live = i < len;
  const double* ar = A + (long long)(live ? i : 0) * 2 * len;
  const double* br = B + (long long)(live ? i : 0) * len;
  // physical position of line l of A's block l: at the end, 0 the older of
  // the last two lines and 1 the last; at the start, 0 the second line and 1
  // the first (the edge)
  int line[2];
  const int lines = axis == 0 ? nx : ny, origin = axis == 0 ? cs : rs, along = axis == 0 ? rs : cs;
#pragma unroll
  for (int l = 0; l < 2; l++) {
    line[l] = origin + (start ? 1 - l : lines - 2 + l);
    if (line[l] >= lines) line[l] -= lines;
  }
  double az = 0.0, bn = 0.0;
  for (int j0 = 0; j0 < len; j0 += kLineChunk) {
    const int cnt = min(kLineChunk, len - j0);
    double a0[kLineUnroll], a1[kLineUnroll], b[kLineUnroll];
#pragma unroll
    for (int u = 0; u < kLineUnroll; u++) {
      const int j = t + u * kLineThreads;
      const bool in = live && j < cnt;
      b[u] = in ? br[j0 + j] : 0.0;
      a0[u] = in ? ar[j0 + j] : 0.0;
      a1[u] = in ? ar[len + j0 + j] : 0.0;
    }
    if (j0) __syncthreads();  // the previous chunk's vectors are consumed
    // standard normals of this extrusion: element j from the stream of
    // (seed, extrusion, j, purpose 3)
    for (int j = tid; j < cnt; j += blockDim.x) {
      if (noise) {
        s_n[j] = noise[j0 + j];
      } else {
        KeyedStream st(keys, ext, j0 + j, 0, 3);
        s_n[j] = to_double(normal_counter(st));
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kLineUnroll; u++) {
      const int j = t + u * kLineThreads;
      if (j < cnt) bn = fma(b[u], s_n[j], bn);
    }
    // the lines before this one are complete and visible from here on
    if (j0 == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int j = tid; j < cnt; j += blockDim.x) {
      int k = along + j0 + j;
      if (k >= len) k -= len;
#pragma unroll
      for (int l = 0; l < 2; l++)
        s_z[l][j] = to_double(axis == 0 ? scr[(long long)k * nx + line[l]] : scr[(long long)line[l] * nx + k]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kLineUnroll; u++) {
      const int j = t + u * kLineThreads;
      if (j < cnt) {
        az = fma(a0[u], s_z[0][j], az);
        az = fma(a1[u], s_z[1][j], az);
      }
    }
  }
  s_red[tid] = fma(bn, coeff, az);
  __syncthreads();
  // one warp per element sums its threads' parts
  const int w = tid >> 5, lane = tid & 31, io = blockIdx.x * rows + w;
  if (w < rows && io < len) {
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < kLineThreads / 32; k++) v += s_red[w * kLineThreads + k * 32 + lane];
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) {
      // the new line replaces the one dropped: at the end the first line
      // (physical column cs, row rs), at the start the last
      int pl = start ? origin - 1 : origin, k = along + io;
      if (pl < 0) pl += lines;
      if (k >= len) k -= len;
      scr[axis == 0 ? (long long)k * nx + pl : (long long)pl * nx + k] = (float)(v + step);
    }
  }
}

// an h x w window, a block per row, with the circular wraps by comparison (a
// 64-bit division and two modulo operations per pixel took 6 us for
// 740 x 740 against 1 us of copy time); launched programmatically behind the
// line kernels
constexpr int kWinThreads = 256;
__global__ void __launch_bounds__(kWinThreads)
    screen_window_kernel(const float* scr, int ny, int nx, int rs, int cs, int y0, int x0, int h, int w,
                         float* __restrict__ out, long long stride) {
  int px0 = cs + x0;  // physical column of the window's first
  if (px0 >= nx) px0 -= nx;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int y = blockIdx.x; y < h; y += gridDim.x) {
    int py = rs + y0 + y;
    if (py >= ny) py -= ny;
    const float* src = scr + (long long)py * nx;
    float* dst = out + y * stride;
#pragma unroll 4
    for (int x = threadIdx.x; x < w; x += kWinThreads) {
      int px = px0 + x;
      if (px >= nx) px -= nx;
      dst[x] = src[px];
    }
  }
}

// one pupil-phase layer: the window of a screen and its sub-pixel shift
struct LayerWin {
  const float* scr;
  int ny, nx, rs, cs;  // the screen's size and circular starts
  int y0, x0;          // logical top-left of the (npup+1) square window
  float s1, s2, s3, s4;  // bilinear weights (1-x)(1-y), (1-x)y, x(1-y), xy
};
constexpr int kMaxLayers = 16;
// threads per block of both pupil-phase kernels (their reductions assume it)
constexpr int kPupilThreads = 256;
// a block's tile: 64 columns, four groups of kPupilRun rows
constexpr int kPupilCols = 64, kPupilRun = 4, kPupilRows = kPupilThreads / kPupilCols * kPupilRun;
constexpr int kPupilMaxBlocks = 1024;
struct LayerSet {
  LayerWin l[kMaxLayers];
  int n;
};

// sum over the block of one double per thread, in warp 0; kept to one warp's
// additions, the FP64 pipe taking about 20 cycles for each
__device__ __forceinline__ double block_sum(double v, double* red) {
  red[threadIdx.x] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 0; k < kPupilThreads / 32; k++) s += red[k * 32 + threadIdx.x];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;
}

// createPupilPhs (util/atmos.py:678-733) for sources at infinity: each
// layer's window shifted by linearshift (cmod/src/interpmodule.c:1234-1300,
// float products and sums in its order, no contraction) and the layers
// added in order; then (second kernel) the piston over the pupil removed
// and the result multiplied by the pupil and scaled (:818-833).
// Bound by reading each layer's window once and writing the phase (13 MB
// for 740 x 740 and four layers, 2 us); one pixel per thread with a 64-bit
// division and eight modulo operations per layer took 19 us.  A thread walks
// kPupilRun rows down a column, so that a window row it read as the lower
// neighbour serves as the next row's upper one, and the circular wraps are
// comparisons.  Both kernels, 740 x 740 and four layers: 31.6 -> 14.7 us a
// call, of which the host's part is now the longer one.
__global__ void __launch_bounds__(kPupilThreads)
    pupil_layers_kernel(const __grid_constant__ LayerSet L, int npup, float* __restrict__ out,
                        const float* __restrict__ pfn, double* __restrict__ partial) {
  __shared__ double red[kPupilThreads];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tx = (npup + kPupilCols - 1) / kPupilCols, ty = (npup + kPupilRows - 1) / kPupilRows;
  double acc = 0.0;
  for (int tile = blockIdx.x; tile < tx * ty; tile += gridDim.x) {
    const int by = tile / tx, bx = tile - by * tx;
    const int x = bx * kPupilCols + (int)(threadIdx.x & (kPupilCols - 1));
    const int y = by * kPupilRows + (int)(threadIdx.x / kPupilCols) * kPupilRun;
    const int ny = min(kPupilRun, npup - y);
    if (x >= npup || ny <= 0) continue;
    float pf[kPupilRun], o[kPupilRun];
#pragma unroll
    for (int r = 0; r < kPupilRun; r++) {
      pf[r] = r < ny ? pfn[(long long)(y + r) * npup + x] : 0.f;
      o[r] = 0.f;
    }
    for (int q = 0; q < L.n; q++) {
      const LayerWin& w = L.l[q];
      int c0 = w.cs + w.x0 + x, row = w.rs + w.y0 + y;
      while (c0 >= w.nx) c0 -= w.nx;
      while (row >= w.ny) row -= w.ny;
      const int c1 = c0 + 1 == w.nx ? 0 : c0 + 1;
      float v0[kPupilRun + 1], v1[kPupilRun + 1];
#pragma unroll
      for (int r = 0; r <= kPupilRun; r++) {
        // rows past the pupil's last one are not read
        const float* src = w.scr + (long long)row * w.nx;
        v0[r] = r <= ny ? src[c0] : 0.f;
        v1[r] = r <= ny ? src[c1] : 0.f;
        if (++row == w.ny) row = 0;
      }
#pragma unroll
      for (int r = 0; r < kPupilRun; r++) {
        float f = __fmul_rn(v0[r], w.s1);
        f = __fadd_rn(f, __fmul_rn(v0[r + 1], w.s2));
        f = __fadd_rn(f, __fmul_rn(v1[r], w.s3));
        f = __fadd_rn(f, __fmul_rn(v1[r + 1], w.s4));
        o[r] = __fadd_rn(o[r], f);
      }
    }
#pragma unroll
    for (int r = 0; r < kPupilRun; r++)
      if (r < ny) {
        out[(long long)(y + r) * npup + x] = o[r];
        acc = fma(to_double(o[r]), to_double(pf[r]), acc);  // the product is exact
      }
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

// The finish: one block per SM, its first warp sums the layer blocks' parts
// (all blocks in the same order, so all subtract the same piston) while the
// others' pixels are on their way; 256-thread blocks that each summed them
// with all warps and divided in every thread spent 12 us on FP64.
constexpr int kFinishThreads = 1024;
__global__ void __launch_bounds__(kFinishThreads)
    pupil_finish_kernel(float* __restrict__ out, const float* __restrict__ pfn, long long n,
                        const double* __restrict__ partial, int nparts, double area, int removePiston, float scale,
                        int vec) {
  __shared__ float s_pist;
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  // launched programmatically: the layers' phase and its partial sums are
  // complete and visible from here on
  asm volatile("griddepcontrol.wait;" ::: "memory");
  float pist = 0.f;
  auto one = [&](float v, float p) { return __fmul_rn(__fmul_rn(__fsub_rn(v, pist), p), scale); };
  float4* o4 = reinterpret_cast<float4*>(out);
  const float4* p4 = reinterpret_cast<const float4*>(pfn);
  const long long nq = vec ? n >> 2 : 0;  // 16-byte loads and stores
  float4 v, p;
  if (first < nq) {
    v = o4[first];
    p = p4[first];
  }
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int b = threadIdx.x; b < nparts; b += 32) s += partial[b];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) s_pist = removePiston ? (float)(s / area) : 0.f;
  }
  __syncthreads();
  pist = s_pist;
  if (first < nq) o4[first] = make_float4(one(v.x, p.x), one(v.y, p.y), one(v.z, p.z), one(v.w, p.w));
  for (long long k = first + stride; k < nq; k += stride) {
    v = o4[k];
    p = p4[k];
    o4[k] = make_float4(one(v.x, p.x), one(v.y, p.y), one(v.z, p.z), one(v.w, p.w));
  }
  for (long long k = (nq << 2) + first; k < n; k += stride) out[k] = one(out[k], pfn[k]);
}

// Stream-ordered scratch of the pupil phase (its partial sums): one pool per
// device, made with the first screen on it and destroyed with the last, that
// keeps up to kScratchKeep bytes across synchronisations.  The device's
// default pool gives its memory back at every synchronisation, and a call
// after one then waited about 200 us for it to be mapped again.
constexpr uint64_t kScratchKeep = 64u << 20;
struct ScratchPool {
  cudaMemPool_t pool = nullptr;
  int users = 0;
};
std::mutex scratchMutex;
std::map<int, ScratchPool>& scratchPools = *new std::map<int, ScratchPool>;  // outlives every screen

cudaError_t scratch_acquire(int dev, cudaStream_t st, cudaMemPool_t* out) {
  std::lock_guard<std::mutex> lock(scratchMutex);
  ScratchPool& p = scratchPools[dev];
  if (!p.pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaError_t e = cudaMemPoolCreate(&p.pool, &props);
    if (e != cudaSuccess) {
      p.pool = nullptr;
      return e;
    }
    uint64_t keep = kScratchKeep;
    e = cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    // the first block of memory is mapped here
    void* first = nullptr;
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&first, 1024, p.pool, st);
    if (e == cudaSuccess) e = cudaFreeAsync(first, st);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(p.pool);
      p.pool = nullptr;
      return e;
    }
  }
  p.users++;
  *out = p.pool;
  return cudaSuccess;
}

void scratch_release(int dev) {
  std::lock_guard<std::mutex> lock(scratchMutex);
  ScratchPool& p = scratchPools[dev];
  if (p.users > 0 && --p.users == 0) {
    cudaMemPoolDestroy(p.pool);  // pending frees complete first
    p.pool = nullptr;
  }
}

}  // namespace

}  // namespace shwfs

using shwfs::engine_fail;

namespace {

shwfs_status cuda_fail(cudaError_t e, const char* what) {
  return engine_fail(SHWFS_ERR_CUDA, (std::string(what) + ": " + cudaGetErrorString(e)).c_str());
}

#define SCK(call, what)                          \
  do {                                           \
    cudaError_t e_ = (call);                     \
    if (e_ != cudaSuccess) return cuda_fail(e_, what); \
  } while (0)

template <typename T>
cudaError_t upload(T** dst, const T* src, size_t n) {
  cudaError_t e = cudaMalloc((void**)dst, n * sizeof(T));
  if (e != cudaSuccess) return e;
  return cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice);
}

void release(shwfs_screen* s) {
  cudaFree(s->scr);
  for (int k = 0; k < 2; k++) {
    cudaFree(s->a[k]);
    cudaFree(s->b[k]);
  }
  cudaFree(s->noise);
  if (s->stream) cudaStreamDestroy(s->stream);
  if (s->pool) shwfs::scratch_release(s->device);
  delete s;
}

}  // namespace

extern "C" {

shwfs_status shwfs_screen_create(int ny, int nx, const float* init, const double* ay, const double* by,
                                 const double* ax, const double* bx, uint64_t seed, shwfs_screen** out) {
  if (!out || !init || ny < 3 || nx < 3 || (int64_t)ny * nx > ((int64_t)1 << 30))
    return engine_fail(SHWFS_ERR_INVALID, "screen_create: bad size or null argument");
  if (!ay && !ax) return engine_fail(SHWFS_ERR_INVALID, "screen_create: give the column and/or row matrices");
  if ((ay && !by) || (ax && !bx)) return engine_fail(SHWFS_ERR_INVALID, "screen_create: A without B");
  shwfs_screen* s = new shwfs_screen;
  s->ny = ny;
  s->nx = nx;
  s->keys = shwfs::PhiloxKeys{};
  {
    shwfs::WfsArgs tmp;
    memset(&tmp, 0, sizeof(tmp));
    tmp.seed = seed;
    shwfs::set_philox_keys(tmp);
    s->keys = tmp.philoxKeys;
  }
  cudaError_t e = cudaGetDevice(&s->device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&s->numSMs, cudaDevAttrMultiProcessorCount, s->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = shwfs::scratch_acquire(s->device, s->stream, &s->pool);
  if (e == cudaSuccess) e = upload(&s->scr, init, (size_t)ny * nx);
  if (e == cudaSuccess && ay) e = upload(&s->a[0], ay, (size_t)ny * 2 * ny);
  if (e == cudaSuccess && by) e = upload(&s->b[0], by, (size_t)ny * ny);
  if (e == cudaSuccess && ax) e = upload(&s->a[1], ax, (size_t)nx * 2 * nx);
  if (e == cudaSuccess && bx) e = upload(&s->b[1], bx, (size_t)nx * nx);
  if (e == cudaSuccess) e = cudaMalloc((void**)&s->noise, (size_t)std::max(ny, nx) * sizeof(double));
  if (e != cudaSuccess) {
    release(s);
    return cuda_fail(e, "screen_create");
  }
  *out = s;
  return SHWFS_OK;
}

shwfs_status shwfs_screen_add(shwfs_screen* s, int axis, int n, double coeff_turb, double step, const double* noise,
                              void* stream) {
  if (!s || axis < 0 || axis > 3 || n < 0) return engine_fail(SHWFS_ERR_INVALID, "screen_add: bad arguments");
  const int start = axis >= 2 ? 1 : 0;
  axis &= 1;
  if (!s->a[axis]) return engine_fail(SHWFS_ERR_INVALID, "screen_add: no matrices for this axis");
  cudaStream_t st = stream ? (cudaStream_t)stream : s->stream;
  const int len = axis == 0 ? s->ny : s->nx;
  // elements per CTA: about one CTA per SM (more for lines of over eight
  // elements per SM)
  const int rows = std::max(1, std::min(shwfs::kLineMaxRows, (len + s->numSMs - 1) / s->numSMs));
  for (int k = 0; k < n; k++) {
    if (noise)
      SCK(cudaMemcpyAsync(s->noise, noise + (size_t)k * len, len * sizeof(double), cudaMemcpyHostToDevice, st),
          "screen_add noise");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((len + rows - 1) / rows));
    cfg.blockDim = dim3((unsigned)(rows * shwfs::kLineThreads));
    cfg.stream = st;
    // programmatic launch: injected normals are read ahead of the kernel's
    // wait, so a line that takes them is launched in plain stream order
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = noise ? 0 : 1;
    const double* injected = noise ? s->noise : nullptr;
    SCK(cudaLaunchKernelEx(&cfg, shwfs::screen_line_kernel, s->scr, s->ny, s->nx, s->rs, s->cs, axis, start,
                           (const double*)s->a[axis], (const double*)s->b[axis], s->keys, s->added, injected,
                           coeff_turb, k == 0 ? step : 0.0),
        "screen_line_kernel");
    if (axis == 0)
      s->cs = start ? (s->cs + s->nx - 1) % s->nx : (s->cs + 1) % s->nx;
    else
      s->rs = start ? (s->rs + s->ny - 1) % s->ny : (s->rs + 1) % s->ny;
    s->added++;  // the next extrusion's injected noise overwrites s->noise in stream order
  }
  if (!stream) SCK(cudaStreamSynchronize(st), "screen_add sync");
  return SHWFS_OK;
}

shwfs_status shwfs_screen_window(shwfs_screen* s, int y0, int x0, int h, int w, float* out, int64_t out_stride,
                                 void* stream) {
  if (!s || !out || y0 < 0 || x0 < 0 || h < 1 || w < 1 || y0 + h > s->ny || x0 + w > s->nx || out_stride < w)
    return engine_fail(SHWFS_ERR_INVALID, "screen_window: window outside the screen");
  cudaStream_t st = stream ? (cudaStream_t)stream : s->stream;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min(h, s->numSMs * 8));
  cfg.blockDim = dim3(shwfs::kWinThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SCK(cudaLaunchKernelEx(&cfg, shwfs::screen_window_kernel, (const float*)s->scr, s->ny, s->nx, s->rs, s->cs, y0, x0, h, w,
                         out, (long long)out_stride),
      "screen_window_kernel");
  if (!stream) SCK(cudaStreamSynchronize(st), "screen_window sync");
  return SHWFS_OK;
}

shwfs_status shwfs_screens_pupil_phase(shwfs_screen* const* screens, int nlayers, const int* y0, const int* x0,
                                       const float* yshift, const float* xshift, int npup, const float* pupil,
                                       double pupil_area, int remove_piston, float scale, float* out, void* stream) {
  if (!screens || nlayers < 1 || nlayers > shwfs::kMaxLayers || !y0 || !x0 || !yshift || !xshift || npup < 1 ||
      !pupil || !out || !(pupil_area > 0.0))
    return engine_fail(SHWFS_ERR_INVALID, "screens_pupil_phase: bad arguments (1..16 layers, npup >= 1, area > 0)");
  shwfs::LayerSet L{};
  L.n = nlayers;
  for (int q = 0; q < nlayers; q++) {
    const shwfs_screen* s = screens[q];
    if (!s) return engine_fail(SHWFS_ERR_INVALID, "screens_pupil_phase: null screen");
    if (y0[q] < 0 || x0[q] < 0 || y0[q] + npup + 1 > s->ny || x0[q] + npup + 1 > s->nx)
      return engine_fail(SHWFS_ERR_INVALID, "screens_pupil_phase: window (npup+1 square) outside a screen");
    const float xs = xshift[q], ys = yshift[q];
    if (!(xs >= 0.f && xs <= 1.f && ys >= 0.f && ys <= 1.f))
      return engine_fail(SHWFS_ERR_INVALID, "screens_pupil_phase: shifts must be in [0, 1]");
    shwfs::LayerWin& w = L.l[q];
    w.scr = s->scr;
    w.ny = s->ny;
    w.nx = s->nx;
    w.rs = s->rs;
    w.cs = s->cs;
    w.y0 = y0[q];
    w.x0 = x0[q];
    // linearshift's weights in float (cmod/src/interpmodule.c:1277-1280)
    w.s1 = (float)((1.0 - (double)xs) * (1.0 - (double)ys));
    w.s2 = (float)((1.0 - (double)xs) * (double)ys);
    w.s3 = (float)((double)xs * (1.0 - (double)ys));
    w.s4 = xs * ys;
  }
  cudaStream_t st = stream ? (cudaStream_t)stream : screens[0]->stream;
  const long long n = (long long)npup * npup;
  const int tiles = ((npup + shwfs::kPupilCols - 1) / shwfs::kPupilCols) * ((npup + shwfs::kPupilRows - 1) / shwfs::kPupilRows);
  const int blocks = std::min(tiles, shwfs::kPupilMaxBlocks);
  int dev = 0;
  SCK(cudaGetDevice(&dev), "screens_pupil_phase");
  double* partial = nullptr;
  // the screens' scratch pool belongs to their device
  SCK(dev == screens[0]->device
          ? cudaMallocFromPoolAsync((void**)&partial, (size_t)blocks * sizeof(double), screens[0]->pool, st)
          : cudaMallocAsync((void**)&partial, (size_t)blocks * sizeof(double), st),
      "screens_pupil_phase");
  shwfs::pupil_layers_kernel<<<blocks, shwfs::kPupilThreads, 0, st>>>(L, npup, out, pupil, partial);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min<long long>((n + shwfs::kFinishThreads - 1) / shwfs::kFinishThreads,
                                                     (long long)screens[0]->numSMs));
    cfg.blockDim = dim3(shwfs::kFinishThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int vec = (((uintptr_t)out | (uintptr_t)pupil) & 15) == 0 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, shwfs::pupil_finish_kernel, out, pupil, n, (const double*)partial, blocks, pupil_area,
                           remove_piston, scale, vec);
  }
  cudaFreeAsync(partial, st);
  if (e != cudaSuccess) return cuda_fail(e, "pupil phase kernels");
  if (!stream) SCK(cudaStreamSynchronize(st), "screens_pupil_phase sync");
  return SHWFS_OK;
}

shwfs_status shwfs_screen_read(shwfs_screen* s, float* host_out) {
  if (!s || !host_out) return engine_fail(SHWFS_ERR_INVALID, "screen_read: null argument");
  float* d = nullptr;
  SCK(cudaMalloc((void**)&d, (size_t)s->ny * s->nx * sizeof(float)), "screen_read");
  shwfs_status r = shwfs_screen_window(s, 0, 0, s->ny, s->nx, d, s->nx, s->stream);
  if (r == SHWFS_OK) {
    cudaError_t e = cudaStreamSynchronize(s->stream);
    if (e == cudaSuccess) e = cudaMemcpy(host_out, d, (size_t)s->ny * s->nx * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) r = cuda_fail(e, "screen_read");
  }
  cudaFree(d);
  return r;
}

shwfs_status shwfs_screen_free(shwfs_screen* s) {
  if (s) {
    cudaStreamSynchronize(s->stream);
    release(s);
  }
  return SHWFS_OK;
}

}  // extern "C"

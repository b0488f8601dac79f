// api.cu -- status handling, macrocell build and frame-buffer read.
#include <cstdio>
#include <cstring>
#include <string>
#include <algorithm>
#include <cuda_runtime.h>
#include "gbv_volume.cuh"
#include "gbv_internal.h"
#include "../../include/gbvol_diag.h"

namespace gbv {

static thread_local std::string g_last_error;

gbv_status set_error(gbv_status st, const char *msg) {
  g_last_error = msg ? msg : "";
  return st;
}

gbv_status check_cuda(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return GBV_OK;
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  g_last_error = m;
  return e == cudaErrorMemoryAllocation ? GBV_ERROR_OUT_OF_MEMORY : GBV_ERROR_CUDA;
}

gbv_status check_launch(const char *what) { return check_cuda(cudaGetLastError(), what); }

// -------------------------------------------------------------------------
// Macrocell ranges over the (cpm+1)^3 footprint (StructuredData.cu:45-57,
// inclusive upper corner, clipped to the volume).  min/max are exact, so the
// result is independent of the reduction order.
//
// A block takes a strip of K macrocells along x, K cpm <= 128: a thread per
// column runs over half of the footprint's (y, z) rows, so that a warp reads
// 128 consecutive bytes of a row, then a warp per macrocell reduces its
// cpm + 1 columns.  The strip's last column, which belongs to its last
// macrocell alone, is shared out by rows.  Macrocells of more than 64 cells
// are strips of one (K = 1): their columns are one range, whatever their
// number.
//
// What bounds it: the volume's read.  One warp per macrocell read rows of
// cpm + 1 values with two divisions a value: 256^3 at 16^3 cells 79 us (0.85
// TB/s); a strip per block: 24 us (2.8).
// -------------------------------------------------------------------------
constexpr int kStripCols = 128;
__global__ void __launch_bounds__(2 * kStripCols) mc_ranges_kernel(const float *__restrict__ scalars, int nx, int ny,
                                                                   int nz, int cpm, int mx_, int my_, int mz_, int K,
                                                                   float2 *__restrict__ ranges) {
  __shared__ float s_lo[2][kStripCols], s_hi[2][kStripCols], s_wlo[8], s_whi[8];
  const int strips = (mx_ + K - 1) / K;
  const long long blk = blockIdx.x;
  const int sx = (int)(blk % strips), cy = (int)((blk / strips) % my_), cz = (int)(blk / ((long long)strips * my_));
  const int tx = threadIdx.x & (kStripCols - 1), half = threadIdx.x / kStripCols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = sx * K * cpm, y0 = cy * cpm, z0 = cz * cpm;
  const int cols = min(K * cpm + 1, nx - x0), ey = min(cpm + 1, ny - y0), ez = min(cpm + 1, nz - z0);
  const float INF = __int_as_float(0x7f800000);
  const float *base = scalars + (size_t)x0 + (size_t)nx * ((size_t)y0 + (size_t)ny * z0);
  const size_t plane = (size_t)nx * ny;
  float lo = INF, hi = -INF;  // interval::extend: NaN never replaces the bound
  const int own = K > 1 ? min(cols, kStripCols) : cols;  // columns the threads take whole
  for (int x = tx; x < own; x += kStripCols)
    for (int z = half; z < ez; z += 2) {
      const float *row = base + x + plane * z;
#pragma unroll 8
      for (int y = 0; y < ey; y++) {
        const float v = __ldg(row + (size_t)nx * y);
        lo = mn(lo, v);
        hi = mx(hi, v);
      }
    }
  float elo = INF, ehi = -INF;  // the strip's last column, by rows
  if (own < cols)
    for (int r = threadIdx.x; r < ey * ez; r += 2 * kStripCols) {
      const float v = __ldg(base + (cols - 1) + (size_t)nx * (r % ey) + plane * (r / ey));
      elo = mn(elo, v);
      ehi = mx(ehi, v);
    }
  if (K == 1) {
    elo = mn(elo, lo);
    ehi = mx(ehi, hi);
  } else {
    s_lo[half][tx] = lo;
    s_hi[half][tx] = hi;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    elo = mn(elo, __shfl_xor_sync(0xffffffffu, elo, o));
    ehi = mx(ehi, __shfl_xor_sync(0xffffffffu, ehi, o));
  }
  if (lane == 0) {
    s_wlo[warp] = elo;
    s_whi[warp] = ehi;
  }
  __syncthreads();
  for (int k = warp; k < K && sx * K + k < mx_; k += 8) {
    lo = INF;
    hi = -INF;
    if (K > 1)
      for (int i = lane; i < 2 * (cpm + 1); i += 32) {
        const int c = k * cpm + (i >> 1);
        if (c < own) {
          lo = mn(lo, s_lo[i & 1][c]);
          hi = mx(hi, s_hi[i & 1][c]);
        }
      }
    // the shared-out column (or, for K = 1, all columns)
    if (lane < 8 && (K == 1 || (own < cols && k * cpm + cpm == cols - 1))) {
      lo = mn(lo, s_wlo[lane]);
      hi = mx(hi, s_whi[lane]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = mn(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = mx(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) ranges[(size_t)sx * K + k + (size_t)mx_ * ((size_t)cy + (size_t)my_ * cz)] = make_float2(lo, hi);
  }
}

// The same for fields of few voxels along x, whose strips would leave most of a
// block's columns empty.  A block takes rows of macrocells along x; per row
// 2^wl threads stand for its columns and 2^sl slices share its (y, z) rows,
// 256 threads in all.  Then 2^pl threads reduce the partial ranges of a
// macrocell's columns.
// What bounds it: for macrocells of a few cells the reduction, else the read.
// 8 x 700 x 600 at 6^3 cells: a warp per macrocell 21 us, a strip per block 59
// us, this 12 us.
// Taken where it was the faster one, in fields of nx x 700 x 600: 16 at 24^3
// cells 15 us (strips 18), but 17 at 24^3 23 us (18); 24 at 8^3 28 us (30), 32
// at 12^3 25 us (31); 33 at 6^3 47 us (64), but at 12^3 44 us (33).
inline bool mc_ranges_thin(int nx, int cpm) {
  return nx <= 16 || (nx <= 32 && cpm <= 12) || (nx <= 64 && cpm <= 6);
}
constexpr int kThinThreads = 256;
constexpr long long kFillBlocks = 8 * 152;  // resident blocks of the GPU's SMs
__global__ void __launch_bounds__(kThinThreads) mc_ranges_thin_kernel(const float *__restrict__ scalars, int nx, int ny,
                                                                      int nz, int cpm, int mx_, int my_, int mz_,
                                                                      int wl, int sl, int pl,
                                                                      float2 *__restrict__ ranges) {
  __shared__ float s_lo[kThinThreads], s_hi[kThinThreads];
  const int t = threadIdx.x, x = t & ((1 << wl) - 1), slice = (t >> wl) & ((1 << sl) - 1);
  const int G = kThinThreads >> (wl + sl);
  const int rows = my_ * mz_, first = blockIdx.x * G;
  const float INF = __int_as_float(0x7f800000);
  float lo = INF, hi = -INF;  // interval::extend: NaN never replaces the bound
  const int row = first + (t >> (wl + sl));
  if (row < rows && x < nx) {
    const int y0 = row % my_ * cpm, z0 = row / my_ * cpm;
    const int ey = min(cpm + 1, ny - y0), ez = min(cpm + 1, nz - z0);
    const float *base = scalars + (size_t)x + (size_t)nx * ((size_t)y0 + (size_t)ny * z0);
    const int dy = (1 << sl) % ey, dz = (1 << sl) / ey;
    int y = slice % ey, z = slice / ey;
#pragma unroll 4
    while (z < ez) {
      const float v = __ldg(base + (size_t)nx * ((size_t)y + (size_t)ny * z));
      lo = mn(lo, v);
      hi = mx(hi, v);
      y += dy;
      z += dz;
      if (y >= ey) {
        y -= ey;
        z++;
      }
    }
  }
  s_lo[t] = lo;
  s_hi[t] = hi;
  __syncthreads();
  const int parts = min(cpm + 1, nx) << sl;
  for (int m0 = 0; m0 < G * mx_; m0 += kThinThreads >> pl) {
    const int m = m0 + (t >> pl), g = m / mx_, k = m % mx_;
    const bool valid = m < G * mx_ && first + g < rows;
    lo = INF;
    hi = -INF;
    for (int i = t & ((1 << pl) - 1); valid && i < parts; i += 1 << pl) {
      const int c = k * cpm + (i >> sl);
      if (c >= nx) break;
      const int at = (((g << sl) + (i & ((1 << sl) - 1))) << wl) + c;
      lo = mn(lo, s_lo[at]);
      hi = mx(hi, s_hi[at]);
    }
    for (int o = 1 << pl >> 1; o > 0; o >>= 1) {
      lo = mn(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = mx(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (valid && (t & ((1 << pl) - 1)) == 0) ranges[(size_t)(first + g) * mx_ + k] = make_float2(lo, hi);
  }
}

gbv_status launch_mc_ranges(const float *d_scalars, const int dims[3], int cpm, const int M[3], float2 *ranges,
                            cudaStream_t stream) {
  if (mc_ranges_thin(dims[0], cpm)) {
    int wl = 1, sl = 0;
    while (1 << wl < dims[0]) wl++;
    // more slices while the blocks do not fill the GPU, at least four rows each
    const long long rows = (long long)std::min(cpm + 1, dims[1]) * std::min(cpm + 1, dims[2]);
    while (wl + sl < 8 && 8ll << sl <= rows && ((long long)M[1] * M[2] << (wl + sl)) < kThinThreads * kFillBlocks) sl++;
    const long long parts = (long long)std::min(cpm + 1, dims[0]) << sl;
    const int pl = parts <= 16 ? 0 : parts <= 128 ? 3 : 5;
    const int G = kThinThreads >> (wl + sl);
    const long long blocks = ((long long)M[1] * M[2] + G - 1) / G;
    mc_ranges_thin_kernel<<<(unsigned)blocks, kThinThreads, 0, stream>>>(d_scalars, dims[0], dims[1], dims[2], cpm,
                                                                         M[0], M[1], M[2], wl, sl, pl, ranges);
    return check_launch("mc_ranges_thin_kernel");
  }
  const int K = cpm <= kStripCols / 2 ? kStripCols / cpm : 1;
  const long long blocks = (((long long)M[0] + K - 1) / K) * M[1] * M[2];
  mc_ranges_kernel<<<(unsigned)blocks, 2 * kStripCols, 0, stream>>>(d_scalars, dims[0], dims[1], dims[2], cpm, M[0],
                                                                    M[1], M[2], K, ranges);
  return check_launch("mc_ranges_kernel");
}

// mapMCs (MCGrid.cu:94-116): one thread per macrocell
__global__ void majorants_kernel(const float2 *__restrict__ ranges, long long numMC, const float4 *__restrict__ tf,
                                 int n, float lo, float span, float bd, float *__restrict__ out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= numMC) return;
  float2 r = ranges[i];
  out[i] = xf_majorant(tf, n, lo, span, bd, r.x, r.y);
}

// linearizeColorAndNormalKernel (TiledFB.cu:13-50); make_8bit and
// linear_to_srgb (math.h:52-116) are in gbv_math.cuh
__global__ void tonemap_kernel(const float4 *__restrict__ accum, long long n, float accumScale, int format,
                               void *out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 a = accum[i];
  float4 c = make_float4(a.x * accumScale, a.y * accumScale, a.z * accumScale, a.w * accumScale);
  if (format == GBV_FB_FLOAT4) {
    reinterpret_cast<float4 *>(out)[i] = c;
    return;
  }
  if (format == GBV_FB_RGBA8_SRGB) {
    c.x = linear_to_srgb(c.x);
    c.y = linear_to_srgb(c.y);
    c.z = linear_to_srgb(c.z);
  }
  reinterpret_cast<uint32_t *>(out)[i] =
      (make_8bit(c.x) << 0) + (make_8bit(c.y) << 8) + (make_8bit(c.z) << 16) + (make_8bit(c.w) << 24);
}

// Normalised integer texels (cudaReadModeNormalizedFloat of the reference's
// CUDA texture objects, rtcore/cudaCommon/TextureData.cu:34-39; the CPU
// backend's getTexel<unsigned char>, rtcore/embree/Texture.cpp:216-225):
// v / 255 or v / 65535, one IEEE division per texel.
// What bounds it: memory.  One texel a thread took 46 us for 16.8 M 8-bit texels
// (1.8 TB/s); 16 bytes of them a thread takes 21 us (4.0).
template <typename T>
__global__ void __launch_bounds__(256) normalize_texels_kernel(const T *__restrict__ in, long long n, float scale_max,
                                                               float *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)in[i] / scale_max;
}
// Arrays that are both 16-byte aligned: `vectors` threads take 16 bytes of
// texels each, the others the remainder one by one.
template <typename T>
__global__ void __launch_bounds__(256) normalize_vectors_kernel(const T *__restrict__ in, long long n, long long vectors,
                                                                float scale_max, float *__restrict__ out) {
  constexpr int kPer = 16 / sizeof(T);
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < vectors) {
    union { uint4 q; T t[kPer]; } v;
    v.q = __ldg(reinterpret_cast<const uint4 *>(in) + i);
    float4 *o = reinterpret_cast<float4 *>(out) + i * (kPer / 4);
#pragma unroll
    for (int k = 0; k < kPer / 4; k++)
      o[k] = make_float4((float)v.t[4 * k] / scale_max, (float)v.t[4 * k + 1] / scale_max,
                         (float)v.t[4 * k + 2] / scale_max, (float)v.t[4 * k + 3] / scale_max);
    return;
  }
  const long long r = vectors * kPer + (i - vectors);
  if (r < n) out[r] = (float)in[r] / scale_max;
}
template <typename T>
static gbv_status launch_normalize(const void *in, long long n, float scale_max, float *out, cudaStream_t stream) {
  const T *t = reinterpret_cast<const T *>(in);
  if ((((uintptr_t)in | (uintptr_t)out) & 15) != 0) {
    normalize_texels_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(t, n, scale_max, out);
    return check_launch("normalize_texels_kernel");
  }
  const long long per = 16 / sizeof(T), vectors = n / per, threads = vectors + (n - vectors * per);
  normalize_vectors_kernel<T><<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(t, n, vectors, scale_max, out);
  return check_launch("normalize_vectors_kernel");
}

__global__ void sincos_angle_kernel(const float *__restrict__ x, long long n, float *__restrict__ sn,
                                    float *__restrict__ cs) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s, c;
  sincos_angle(x[i], s, c);
  sn[i] = s;
  cs[i] = c;
}

}  // namespace gbv

using namespace gbv;

extern "C" {

const char *gbv_last_error(void) { return g_last_error.c_str(); }
int gbv_version(void) { return 1; }

gbv_status gbv_release_scratch(void) {
  int dev = 0;
  const gbv_status st = check_cuda(cudaGetDevice(&dev), "gbv_release_scratch");
  return st != GBV_OK ? st : check_cuda(release_scratch(dev), "gbv_release_scratch");
}

gbv_status gbv_mc_dims(const int dims[3], int cells_per_mc, int mc_dims[3]) {
  if (!dims || !mc_dims || cells_per_mc <= 0) return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_mc_dims: bad argument");
  for (int i = 0; i < 3; i++) {
    if (dims[i] < 0) return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_mc_dims: negative dims");
    int cells = dims[i] - 1;
    mc_dims[i] = cells <= 0 ? 0 : (cells + cells_per_mc - 1) / cells_per_mc;
  }
  long long n = (long long)mc_dims[0] * mc_dims[1] * mc_dims[2];
  if (n != (long long)(int)n)
    return set_error(GBV_ERROR_INVALID_ARGUMENT, "number of macrocells cannot be expressed in a 32-bit value");
  return GBV_OK;
}

gbv_status gbv_build_mc_ranges(const float *d_scalars, const int dims[3], int cells_per_mc, float *d_ranges,
                               void *stream) {
  int M[3];
  gbv_status st = gbv_mc_dims(dims, cells_per_mc, M);
  if (st != GBV_OK) return st;
  if (!d_scalars || !d_ranges) return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_build_mc_ranges: null pointer");
  long long n = (long long)M[0] * M[1] * M[2];
  if (n == 0) return GBV_OK;
  return launch_mc_ranges(d_scalars, dims, cells_per_mc, M, reinterpret_cast<float2 *>(d_ranges),
                          (cudaStream_t)stream);
}

gbv_status gbv_map_majorants(const float *d_ranges, int num_mc, const float *d_tf, int tf_n, float domain_lo,
                             float domain_hi, float base_density, float *d_majorants, void *stream) {
  if (!d_ranges || !d_tf || !d_majorants || num_mc < 0 || tf_n < 2)
    return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_map_majorants: bad argument");
  if (num_mc == 0) return GBV_OK;
  int bs = 256;
  majorants_kernel<<<(num_mc + bs - 1) / bs, bs, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const float2 *>(d_ranges), num_mc, reinterpret_cast<const float4 *>(d_tf), tf_n, domain_lo,
      domain_hi - domain_lo, base_density, d_majorants);
  return check_launch("majorants_kernel");
}

gbv_status gbv_tonemap(const float *d_accum, int width, int height, int accum_id, int format, void *d_out,
                       void *stream) {
  if (!d_accum || !d_out || width <= 0 || height <= 0 || accum_id <= 0)
    return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_tonemap: bad argument (accum_id must be >= 1)");
  if (format < GBV_FB_FLOAT4 || format > GBV_FB_RGBA8_SRGB)
    return set_error(GBV_ERROR_UNSUPPORTED, "gbv_tonemap: unsupported format");
  long long n = (long long)width * height;
  float accumScale = 1.f / (float)accum_id;
  tonemap_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const float4 *>(d_accum), n, accumScale, format, d_out);
  return check_launch("tonemap_kernel");
}

gbv_status gbv_selftest_sincos(const float *x, long long n, float *sn, float *cs, int on_device, void *stream) {
  if (!x || !sn || !cs || n < 0) return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_selftest_sincos: bad argument");
  if (n == 0) return GBV_OK;
  if (!on_device) {
    for (long long i = 0; i < n; i++) sincos_angle(x[i], sn[i], cs[i]);
    return GBV_OK;
  }
  sincos_angle_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(x, n, sn, cs);
  return check_launch("sincos_angle_kernel");
}

__global__ void angles_kernel(const float *__restrict__ y, const float *__restrict__ x, long long n,
                              float *__restrict__ acos_x, float *__restrict__ atan2_yx) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  acos_x[i] = acos_angle(x[i]);
  atan2_yx[i] = atan2_angle(y[i], x[i]);
}

gbv_status gbv_selftest_angles(const float *y, const float *x, long long n, float *acos_x, float *atan2_yx,
                               int on_device, void *stream) {
  if (!y || !x || !acos_x || !atan2_yx || n < 0)
    return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_selftest_angles: bad argument");
  if (n == 0) return GBV_OK;
  if (!on_device) {
    for (long long i = 0; i < n; i++) {
      acos_x[i] = acos_angle(x[i]);
      atan2_yx[i] = atan2_angle(y[i], x[i]);
    }
    return GBV_OK;
  }
  angles_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(y, x, n, acos_x, atan2_yx);
  return check_launch("angles_kernel");
}

gbv_status gbv_normalize_texels(const void *d_texels, int bits, long long n, float *d_scalars, void *stream) {
  if (!d_texels || !d_scalars || n < 0 || (bits != 8 && bits != 16))
    return set_error(GBV_ERROR_INVALID_ARGUMENT, "gbv_normalize_texels: bad argument (bits must be 8 or 16)");
  if (n == 0) return GBV_OK;
  return bits == 8 ? launch_normalize<uint8_t>(d_texels, n, 255.f, d_scalars, (cudaStream_t)stream)
                   : launch_normalize<uint16_t>(d_texels, n, 65535.f, d_scalars, (cudaStream_t)stream);
}

}  // extern "C"

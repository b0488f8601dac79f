// render_kernel.cuh -- the structured-volume frame render on sm_103a: device
// code, the persistent kernel and its launch templates (instantiated once per
// voxel store in render_store_*.cu).
//
// Every pixel accumulates its fragments in the reference's order (pass-major,
// then generation; within a generation the shadow ray before the bounce ray)
// with plain adds: a path sums its pixel's passes one after the other, or
// logs one pass's fragments, which a second kernel adds up in that order.  A
// pass follows Context::renderTiles (barney/Context.cpp:142-185):
// _generateRays, then per generation the trace (MCVolumeAccel::isProg) and
// _shadeRays/bounce (barney/kernels/shadeRays.cu:477-1041) of the pixel's
// queued rays.
#pragma once
#include <cstring>
#include <type_traits>
#include <vector>
#include <cuda_runtime.h>
#include "gbv_volume.cuh"
#include "gbv_internal.h"

namespace gbv {

struct DirLightDev { vec3 direction; float radiance; vec3 color; };
struct M3 { vec3 vx, vy, vz; };
__device__ __forceinline__ vec3 xfm_vector(const M3 &m, vec3 v) { return m.vx * v.x + m.vy * v.y + m.vz * v.z; }

struct EnvDev {
  const float4 *tex;
  const float *cdf_y, *cdf_x;
  int W, H;
  int addr[2];
  M3 toWorld, toLocal;
  float scale;
};

struct RenderParams {
  FieldGeom F;
  XF xf;
  MCGridDev G;
  // camera (PerspectiveCamera::commit)
  vec3 lens00, dir00, du, dv;
  int W, H;
  float aspect;  // W / H
  int numDir;
  DirLightDev dir[4];
  int hasEnv;
  EnvDev env;
  float4 bg;
  float ambient;
  int multi, volMS, maxVB;
  float aniso, scatAlb;
  float4 *accum;
  int accumIdStart, spp;
  unsigned long long *counters;
  int *capFlag;   // if set, a loop-cap event stores 1 here (no counting needed)
  int skip;       // seek rounds per traversal iteration
  int threshold;  // keep tracing while at least this % of the lanes does
  int idlePolls;  // a warp that finds no work this many times in a row gives up (a loop-cap event)
  // shared-memory staging (offsets in 32-bit words of the dynamic smem)
  int maskWords;  // >0: bitmask of non-zero majorants staged at offset 0 (a multiple of 4 words)
  const uint32_t *maskSrc;  // the bitmask in HBM (16-byte aligned), staged by one bulk copy; null: by ballots
  int cdfYOff;    // >=0: env cdf_y staged here
  int pivOff;     // >=0: per-row pivots of cdf_x staged here
  int pivPerRow;
  int rowOff;     // >=0: per env-map row (pdf_y, pdf denominator) staged here
  int profile;    // accumulate per-phase cycle counts
  int poolOff;    // the block's path pool starts here
  int slots;      // path slots a block uses (a multiple of 32)
  // The warp tiles that may see the field (its projection's rectangle, in
  // tiles), numbered row by row; the other tiles are the outer ones
  int rx, ry, rw, rh;
  // What the launch hands out: `whole` inner tiles with all their passes, then
  // each pass of `split` inner tiles by itself (its fragments logged and added
  // up in order by finish_kernel, which also renders the outer tiles)
  long long whole, split, outer;
  uint32_t *log;  // null: split == 0
  int logHits;    // fragments a record has room for
  int maskMode;   // 0: the staged bitmask arrives by one bulk copy of a precomputed mask; 1: by ballots
  // voxel store of this scene (see make_store)
  const void *vox;
  const float2 *so;
  BrickGeom brick;
  NvdbGrid nvdb;  // GBV_LAYOUT_NANOVDB: the grid (vox is its buffer)
  vec3 rcpMc;     // 1 / macrocell spacing
  // frame partition across ranks (TiledFB.cu:226-255): with numRanks > 1
  // this launch renders only the 32x32-pixel tiles rank, rank + numRanks, ...
  int rank, numRanks;
  // the world's instances: the volume's stream hash, and an iso-surface
  // (gbv_iso_surface) with its matte material, intersected before the
  // volume when its instance index is the lower one
  uint64_t volHash;
  int hasVolume;
  int isoOn, isoFirst;
  float isoValue, isoDelta, isoAlpha;
  const float2 *isoRanges;
  vec3 isoAlbedo;
  uint64_t isoHash;
  // auxiliary channels (gbv_scene.d_depth, ...; null: not written) and the
  // hit IDs they take
  float *depth;
  int *primId, *instId, *objId;
  int volInst, isoInst, volUser, isoUser;
};

// The reference frame buffer's tiles (TiledFB tileSize) and their
// round-robin assignment to ranks: rank r owns tiles r, r + R, r + 2R, ...
// of the row-major tile grid (TiledFB::resize numActiveTilesThisGPU and
// setTileCoordsKernel, barney/fb/TiledFB.cu:226-255).
constexpr int kRefTile = 32;
__host__ __device__ inline long long owned_ref_tiles(int W, int H, int rank, int numRanks) {
  const long long total = (((long long)W + kRefTile - 1) / kRefTile) * (((long long)H + kRefTile - 1) / kRefTile);
  return total > rank ? (total - rank + numRanks - 1) / numRanks : 0;
}
// 8x4-pixel warp tiles one (non-batched) launch hands out
__host__ __device__ inline long long warp_tile_count(const RenderParams &p) {
  if (p.numRanks > 1) return owned_ref_tiles(p.W, p.H, p.rank, p.numRanks) * 32;
  return (((long long)p.W + 7) >> 3) * (((long long)p.H + 3) >> 2);
}

// what one launch hands out (see RenderParams::whole)
__host__ __device__ inline long long launch_tiles(const RenderParams &L) { return L.whole + L.split * L.spp; }
// the i-th tile inside (outside) the field's rectangle, row-major
__device__ __forceinline__ int inner_tile(const RenderParams &p, int i) {
  const int tilesX = (int)(((long long)p.W + 7) >> 3);
  return p.rw == 0 ? i : (p.ry + i / p.rw) * tilesX + p.rx + i % p.rw;
}
__device__ __forceinline__ int outer_tile(const RenderParams &p, int i) {
  const int tilesX = (int)(((long long)p.W + 7) >> 3), side = tilesX - p.rw;
  if (i < p.ry * tilesX) return i;  // the rows before the rectangle
  i -= p.ry * tilesX;
  if (i >= p.rh * side) return (p.ry + p.rh) * tilesX + i - p.rh * side;  // the rows after it
  const int col = i % side;
  return (p.ry + i / side) * tilesX + (col < p.rx ? col : col + p.rw);
}
// the last item whose first tile is at or before t, searched by the whole
// warp: a load per 32-fold of items
__device__ __forceinline__ int tile_item_warp(const long long *__restrict__ start, int numItems, long long t) {
  const int lane = threadIdx.x & 31;
  int lo = 0, n = numItems;  // it is one of lo .. lo + n - 1
  while (n > 1) {
    const int step = (n + 31) / 32, i = lo + lane * step;
    const int at = __popc(__ballot_sync(0xffffffffu, lane * step < n && start[i] <= t)) - 1;
    n = min(step, n - at * step);
    lo += at * step;
  }
  return lo;
}
// a warp tile's upper-left pixel
template <bool Batch>
__device__ __forceinline__ void tile_corner(const RenderParams &L, const RenderParams &tp, int tile, int &tx, int &ty) {
  if (!Batch && L.numRanks > 1) {  // the k-th 32x32 tile this rank owns, 4x8 warp tiles in it
    const long long big = (long long)L.rank + (long long)(tile >> 5) * L.numRanks;
    const int bigX = (int)(((long long)tp.W + kRefTile - 1) / kRefTile);
    tx = (int)(big % bigX) * kRefTile + (tile & 3) * 8;
    ty = (int)(big / bigX) * kRefTile + ((tile >> 2) & 7) * 4;
  } else {
    const int tilesX = (int)(((long long)tp.W + 7) >> 3);
    tx = (tile % tilesX) * 8;
    ty = (tile / tilesX) * 4;
  }
}

template <class Store> __device__ __forceinline__ Store make_store(const RenderParams &p);
template <> __device__ __forceinline__ StoreLinearF32 make_store<StoreLinearF32>(const RenderParams &p) {
  return StoreLinearF32{reinterpret_cast<const float *>(p.vox), p.F.N[0], p.F.N[1]};
}
template <> __device__ __forceinline__ StoreNanoVDB make_store<StoreNanoVDB>(const RenderParams &p) {
  return StoreNanoVDB{p.nvdb};
}
#define GBV_BRICK_STORE(FMT)                                                                         \
  template <> __device__ __forceinline__ StoreBrickCorners<FMT> make_store<StoreBrickCorners<FMT>>(  \
      const RenderParams &p) {                                                                       \
    return StoreBrickCorners<FMT>{p.vox, p.so, p.brick};                                             \
  }
GBV_BRICK_STORE(GBV_VOXEL_F32)
GBV_BRICK_STORE(GBV_VOXEL_F16)
GBV_BRICK_STORE(GBV_VOXEL_BF16)
GBV_BRICK_STORE(GBV_VOXEL_U8_SCALED)
#undef GBV_BRICK_STORE

// Dynamic shared memory of the render kernel (layout in RenderParams).
extern __shared__ uint32_t g_smem[];

// One warp per 32 macrocells: bit k of word w is set when macrocell
// 32 w + k has a non-zero majorant (words up to `words`, zero-padded).
static __global__ void __launch_bounds__(256) majorant_mask_kernel(const float *__restrict__ maj, int nmc, int words,
                                                            uint32_t *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  for (int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w < words;
       w += (int)((gridDim.x * blockDim.x) >> 5)) {
    const int i = w * 32 + lane;
    const float m = i < nmc ? __ldg(maj + i) : 0.f;
    const unsigned b = __ballot_sync(0xffffffffu, m != 0.f);
    if (lane == 0) out[w] = b;
  }
}

// Stages the bitmask of non-zero majorants in shared-memory words
// [0, p.maskWords).  With the precomputed mask in HBM (p.maskSrc) one thread
// issues one bulk copy (cp.async.bulk global -> shared, completion counted
// in bytes on an mbarrier) and every thread waits on the barrier; the wait
// is bounded, and a copy that has not completed in time (which no working
// GPU produces) sets *capFlag and the block builds the mask from the
// majorants with warp ballots instead (the same bits).  Without a
// precomputed mask the warps build it that way directly.  Every thread of
// the block calls this.
__device__ __forceinline__ void stage_majorant_mask(const RenderParams &p) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  bool staged = false;
  if (p.maskSrc) {
    __shared__ __align__(8) unsigned long long mbar;
    const unsigned mb = (unsigned)__cvta_generic_to_shared(&mbar);
    const unsigned bytes = (unsigned)p.maskWords * 4u;
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              (unsigned)__cvta_generic_to_shared(g_smem)),
          "l"(p.maskSrc), "r"(bytes), "r"(mb)
          : "memory");
    }
    __syncthreads();  // the barrier is initialised before anyone waits on it
    unsigned done = 0;
    for (int it = 0; it < (1 << 20) && !done; it++)
      asm volatile(
          "{\n .reg .pred P;\n mbarrier.try_wait.parity.shared::cta.b64 P, [%1], 0;\n selp.u32 %0, 1, 0, P;\n}"
          : "=r"(done)
          : "r"(mb)
          : "memory");
    staged = __syncthreads_and(done != 0) != 0;
    if (!staged && threadIdx.x == 0 && p.capFlag) *p.capFlag = 1;
  }
  if (!staged) {
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int nmc = p.G.M[0] * p.G.M[1] * p.G.M[2];
    for (int w = warp; w < p.maskWords; w += nwarps) {
      const int i = w * 32 + lane;
      const float m = i < nmc ? __ldg(p.G.maj + i) : 0.f;
      const unsigned b = __ballot_sync(FULL, m != 0.f);
      if (lane == 0) g_smem[w] = b;
    }
  }
}

struct LightSample {
  vec3 radiance, direction;
  float distance, pdf;
};

// fmod(x, y), whose result is exact by definition (x - n y for the integer n
// that truncates x / y, carrying the sign of x).  The wrap addressing of an
// env-map lookup only meets |x| < 2|y|: there the result is x itself, or
// |x| - |y| with the sign of x, a subtraction that is exact because
// |y| <= |x| < 2|y| (Sterbenz's lemma).  Other arguments (and NaN, inf, zero
// y) go to fmodf.  Identical results, a few instructions instead of a
// general remainder.
static __device__ __noinline__ float fmod_general(float x, float y) { return fmodf(x, y); }
__device__ __forceinline__ float fmod_wrap(float x, float y) {
  const float ax = fabsf(x), ay = fabsf(y);
  if (ax < ay) return x;
  if (ax < 2.f * ay) return copysignf(ax - ay, x);
  return fmod_general(x, y);
}

// rtcore/embree/Texture.cpp:25-93, mirror mode (out of line: env maps here
// wrap or clamp)
static __device__ __noinline__ void compute_address_mirror(float tc, int N, int &i0, int &i1, float &f) {
  tc = tc * (float)N + .5f;
  float fc = floorf(tc);
  int ic = (int)fc;
  f = tc - (float)ic;
  int a = ic - 1, b = ic;
  if (a < 0) a = -a;
  if (b < 0) b = -b;
  a = a % (2 * N);
  b = b % (2 * N);
  if (a >= N) a = 2 * N - 1 - a;
  if (b >= N) b = 2 * N - 1 - b;
  i0 = a;
  i1 = b;
}
// rtcore/embree/Texture.cpp:25-93 (normalized coordinates)
__device__ __forceinline__ void compute_address(int mode, float tc, int N, int &i0, int &i1, float &f) {
  i0 = 0; i1 = 0; f = 0.f;
  if (mode == GBV_ADDR_WRAP) {
    tc = tc * (float)N - .5f;
    tc = fmod_wrap(tc, (float)N);
    if (tc < 0.f) tc += (float)N;
    float fc = floorf(tc);
    int ic = (int)fc;
    f = tc - (float)ic;
    i0 = ic;
    i1 = (int)fmod_wrap(tc + 1.f, (float)N);
  } else if (mode == GBV_ADDR_MIRROR) {
    compute_address_mirror(tc, N, i0, i1, f);
  } else if (mode == GBV_ADDR_CLAMP) {
    tc = tc * (float)N;
    if (tc - .5f <= 0.f) { i0 = i1 = 0; f = 0.f; }
    else if (tc - .5f >= (float)(N - 1)) { i0 = i1 = N - 1; f = 0.f; }
    else {
      f = (tc - .5f) - (float)(int)(tc - .5f);
      i0 = (int)(tc - .5f);
      i1 = i0 + 1;
    }
  }
}
__device__ __forceinline__ float4 lerp4(float f, float4 a, float4 b) {
  return make_float4((1.f - f) * a.x + f * b.x, (1.f - f) * a.y + f * b.y, (1.f - f) * a.z + f * b.z,
                     (1.f - f) * a.w + f * b.w);
}
// rtcore/embree/Texture.cpp:295-321 (one call site: the shading phase
// fetches the texels of the env-map samples and the miss lookups together)
__device__ __forceinline__ float4 tex2D(const EnvDev &e, float u, float v) {
  int x0, x1, y0, y1;
  float fx, fy;
  compute_address(e.addr[0], u, e.W, x0, x1, fx);
  compute_address(e.addr[1], v, e.H, y0, y1, fy);
  float4 v00 = __ldg(e.tex + (size_t)x0 + (size_t)y0 * e.W), v01 = __ldg(e.tex + (size_t)x1 + (size_t)y0 * e.W);
  float4 v10 = __ldg(e.tex + (size_t)x0 + (size_t)y1 * e.W), v11 = __ldg(e.tex + (size_t)x1 + (size_t)y1 * e.W);
  return lerp4(fy, lerp4(fx, v00, v01), lerp4(fx, v10, v11));
}

// DG.h:97-106 (acos and atan2 by this library's series, gbv_math.cuh)
__device__ __forceinline__ float spherical_theta(vec3 v) { return acos_angle(clampv(v.z, -1.f, 1.f)); }
__device__ __forceinline__ float spherical_phi(vec3 v) {
  float p = atan2_angle(v.y, v.x);
  return (p < 0.f) ? (p + float(2.f * 3.14159265358979323846)) : p;
}
// (theta, phi) of a direction in the env map's frame, for the env-map pdf
// and the env lookup
__device__ __forceinline__ float2 spherical_theta_phi(vec3 v) {
  return make_float2(spherical_theta(v), spherical_phi(v));
}
// EnvMap.h:98-134
__device__ __forceinline__ float cdf_get_pdf(int position, const float *cdf, int N) {
  float at = __ldg(cdf + position);
  float before = position ? __ldg(cdf + position - 1) : 0.f;
  return (float)N * (at - before);
}
__device__ __forceinline__ int sample_cdf(const float *cdf, int N, float v, float &pdf) {
  int begin = 0, end = N;
  while ((end - begin) > 1) {
    int mid = (begin + end) / 2;
    float f_mid = __ldg(cdf + mid - 1);
    if (v < f_mid) end = mid;
    else begin = mid;
  }
  float at = __ldg(cdf + begin);
  float before = begin ? __ldg(cdf + begin - 1) : 0.f;
  pdf = (float)N * (at - before);
  return begin;
}
// cdfGetPDF / sampleCDF on the staged cdf_y (binary search in shared memory)
__device__ __forceinline__ float cdf_y_at(const RenderParams &p, int i) {
  return p.cdfYOff >= 0 ? __int_as_float(g_smem[p.cdfYOff + i]) : __ldg(p.env.cdf_y + i);
}
__device__ __forceinline__ int sample_cdf_y(const RenderParams &p, float v, float &pdf) {
  const int N = p.env.H;
  int begin = 0, end = N;
  while ((end - begin) > 1) {
    int mid = (begin + end) / 2;
    if (v < cdf_y_at(p, mid - 1)) end = mid;
    else begin = mid;
  }
  const float at = cdf_y_at(p, begin);
  const float before = begin ? cdf_y_at(p, begin - 1) : 0.f;
  pdf = (float)N * (at - before);
  return begin;
}
// sampleCDF over one row of cdf_x.  The binary search returns the number of
// entries cdf[0..N-2] that are <= v (the CDF is non-decreasing); with staged
// pivots (the last counted entry of every 32-entry segment) the same count is
// the number of segments whose pivot is <= v, times 32, plus a count inside
// the next segment, whose 32 entries are fetched with independent loads.
static __device__ __noinline__ int sample_cdf_x_pivots(const RenderParams &p, int row, float v, float &pdf) {
  const int N = p.env.W;
  const float *cdf = p.env.cdf_x + (size_t)row * N;
  const float *piv = reinterpret_cast<const float *>(g_smem + p.pivOff) + (size_t)row * p.pivPerRow;
  const int nseg = p.pivPerRow;
  int lo = 0, hi = nseg;  // first segment whose pivot is > v
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (piv[mid] <= v) lo = mid + 1;
    else hi = mid;
  }
  int begin;
  if (lo == nseg) {
    begin = N - 1;
  } else {
    const int s0 = lo * 32;
    const int last = min(s0 + 31, N - 2);
    float seg[32];
#pragma unroll
    for (int k = 0; k < 32; k++) seg[k] = (s0 + k <= last) ? __ldg(cdf + s0 + k) : 0.f;
    int c = 0;
#pragma unroll
    for (int k = 0; k < 32; k++) c += (s0 + k <= last && seg[k] <= v) ? 1 : 0;
    begin = s0 + c;
  }
  const float at = __ldg(cdf + begin);
  const float before = begin ? __ldg(cdf + begin - 1) : 0.f;
  pdf = (float)N * (at - before);
  return begin;
}
__device__ __forceinline__ int sample_cdf_x(const RenderParams &p, int row, float v, float &pdf) {
  if (p.pivOff >= 0) return sample_cdf_x_pivots(p, row, v, pdf);
  return sample_cdf(p.env.cdf_x + (size_t)row * p.env.W, p.env.W, v, pdf);
}

// Code layout.  The render kernel is limited as much by instruction fetch
// as by memory: warps of one SM sit in different phases (start, traverse,
// shade) at once, so the whole loop body is the instruction working set
// (ncu: about 40% of the stall samples of a 1080p launch are "no
// instruction").  The shading helpers are inlined: the trace set-up, the
// texel fetch, the env coordinates and the bounce have one call site each,
// only the env pdf (one call per MIS weight) is duplicated, and no registers
// are saved around calls (measured on the 512^3 frame: +9% against
// out-of-line helpers).  Rarely taken branches (general fmod, mirror addressing, the
// pivot search, subnormal half rounding) stay out of line.
// The two factors of the env-map pdf that depend on the pixel row only
// (EnvMap.h:160-179): the row's marginal pdf and the solid-angle
// denominator 2 pi^2 sin(theta) at the row centre.
__device__ __forceinline__ float2 env_row_terms(const EnvDev &e, int py) {
  const float pdf_y = (float)e.H * (__ldg(e.cdf_y + py) - (py ? __ldg(e.cdf_y + py - 1) : 0.f));
  const float rel_y = ((float)py + .5f) / (float)e.H;
  const float theta2 = kPi * rel_y;
  float sinTheta2, cosTheta2;
  sincos_angle(theta2, sinTheta2, cosTheta2);
  return make_float2(pdf_y, kTwoPi * kPi * sinTheta2);
}
// EnvMap.h:136-180.  With the row terms staged in shared memory (rowOff >= 0,
// computed by the same expressions at kernel start) the pdf is one shared
// and two global loads.
__device__ __forceinline__ float env_pdf(const RenderParams &p, vec3 dir) {
  if (!p.hasEnv) return kOneOverFourPi;
  const EnvDev &e = p.env;
  const float2 tp = spherical_theta_phi(xfm_vector(e.toLocal, dir));
  float theta = tp.x;
  float phi = tp.y;
  float u = phi * kOneOverTwoPi, v = theta * kOneOverPi;
  int px = (int)clampv(u * (float)e.W, 0.f, (float)e.W - 1.f);
  int py = (int)clampv(v * (float)e.H, 0.f, (float)e.H - 1.f);
  const float2 row = p.rowOff >= 0 ? reinterpret_cast<const float2 *>(g_smem + p.rowOff)[py] : env_row_terms(e, py);
  float pdf_x = cdf_get_pdf(px, e.cdf_x + (size_t)py * e.W, e.W);
  return pdf_x * row.x * 1.f / row.y;
}
// EnvMap.h:198-250, in two parts.  The light selection of sampleLights
// needs only the sample's radiance, so the direction and pdf (two
// sine/cosine pairs, a transform and a division) are formed only when the
// env light is the one selected; they use no random numbers, so the random
// stream is consumed exactly as in one piece.
struct EnvPick {
  vec3 radiance; // scale * texel(sx, sy)
  float sx, sy;  // sampled texture coordinates
  float pdfxy;   // pdf_x * pdf_y
};
// The random draws and CDF searches of the sample; the texel at (sx, sy)
// is fetched by the caller (see the shading phase of render_kernel).
__device__ __forceinline__ EnvPick env_pick_coords(const RenderParams &p, Random &r) {
  const EnvDev &e = p.env;
  EnvPick k;
  float r_y = r();
  float r_x = r();
  float pdf_y, pdf_x;
  int iy = sample_cdf_y(p, r_y, pdf_y);
  int ix = sample_cdf_x(p, iy, r_x, pdf_x);
  k.sx = ((float)ix + r()) / (float)e.W;
  k.sy = ((float)iy + r()) / (float)e.H;
  k.pdfxy = pdf_x * pdf_y;
  return k;
}
__device__ __forceinline__ void env_pick_direction(const RenderParams &p, const EnvPick &k, LightSample &s) {
  const EnvDev &e = p.env;
  const float phi = kTwoPi * k.sx;
  const float theta = kPi * k.sy;
  float sinTheta, cosTheta, sinPhi, cosPhi;
  sincos_angle(theta, sinTheta, cosTheta);  // theta in [0, pi]
  sincos_angle(phi, sinPhi, cosPhi);        // phi in [0, 2 pi]
  vec3 d;
  d.z = cosTheta;
  d.x = cosPhi * sinTheta;
  d.y = sinPhi * sinTheta;
  s.direction = xfm_vector(e.toWorld, d);
  s.pdf = k.pdfxy * 1.f / (kTwoPi * kPi * sinTheta);
}

// DG.h:183-193
__device__ __forceinline__ vec3 random_direction(Random &rng) {
#pragma unroll 1
  for (int k = 0; k < 64; k++) {
    vec3 v;
    v.x = 1.f - 2.f * rng();
    v.y = 1.f - 2.f * rng();
    v.z = 1.f - 2.f * rng();
    if (dot(v, v) <= 1.f) return normalize(v);
  }
  return vec3(0.f, 0.f, 1.f);
}

// shadeRays.cu:141-191.  Surf = false: a volume hit, whose normal is zero
// (weight 1); Surf = true: the light's weight is dot(lightDir, N) for the
// front-facing surface normal N.
template <bool Surf = false>
__device__ __forceinline__ bool sample_dir_lights(const RenderParams &p, Random &random, LightSample &ls,
                                                  vec3 N = vec3()) {
  if (p.numDir == 0) return false;
  int lID[2];
  float weights[2];
  float sumWeights = 0.f;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    lID[i] = mn((int)(random() * (float)p.numDir), p.numDir - 1);
    weights[i] = 0.f;
    const DirLightDev &light = p.dir[lID[i]];
    vec3 lr = light.color * light.radiance;
    float weight = 1.f;  // N == 0
    if (Surf) {
      weight = is_zero(N) ? 1.f : dot(-light.direction, N);
      if (weight <= 1e-3f) continue;
    }
    weight *= reduce_max(lr);
    if (weight <= 1e-3f) continue;
    weights[i] = weight;
    sumWeights += weight;
  }
  if (sumWeights == 0.f) return false;
  float r = random() * sumWeights;
  int i = 0;
  while (i < 2 && r >= weights[i]) { r -= weights[i]; ++i; }
  if (i == 2) return false;
  const DirLightDev &light = p.dir[lID[i]];
  ls.direction = -light.direction;
  ls.distance = __int_as_float(0x7f800000);
  ls.radiance = light.color * light.radiance * 1.f / (weights[i] / sumWeights * (2.f / (float)p.numDir));
  ls.pdf = __int_as_float(0x7f800000);
  return weights[i] != 0.f;
}

// shadeRays.cu:268-404 (no area or point lights in this world).  Surf:
// sampling at a surface of front-facing normal N, where the ambient light's
// direction turns into N's hemisphere (radiance 2 pi ambient, pdf 1/(2 pi)).
template <bool Surf = false>
__device__ __forceinline__ bool sample_lights(const RenderParams &p, Random &random, const EnvPick &pick,
                                              LightSample &ls, bool &needsMIS, bool &isDir, vec3 N = vec3()) {
  needsMIS = false;
  LightSample els;
  if (p.hasEnv) {
    els.radiance = pick.radiance;
    els.distance = __int_as_float(0x7f800000);
  } else {
    els.direction = random_direction(random);
    els.distance = __int_as_float(0x7f800000);
    if (Surf && !is_zero(N)) {
      els.radiance = vec3(kTwoPi * p.ambient);
      if (dot(els.direction, N) < 0.f) els.direction = -els.direction;
      els.pdf = kOneOverTwoPi;
    } else {
      els.radiance = vec3(kFourPi * p.ambient);
      els.pdf = kOneOverFourPi;
    }
  }
  float elsWeight = reduce_max(els.radiance);
  LightSample dls;
  dls.pdf = 0.f;
  float dlsWeight = sample_dir_lights<Surf>(p, random, dls, N) ? reduce_max(dls.radiance) : 0.f;
  float alsWeight = 0.f, plsWeight = 0.f;
  float sumWeights = alsWeight + dlsWeight + elsWeight + plsWeight;
  if (sumWeights == 0.f) return false;
  elsWeight *= 1.f / sumWeights;
  alsWeight *= 1.f / sumWeights;
  dlsWeight *= 1.f / sumWeights;
  float r = random();
  if (r <= alsWeight) {
    return false;  // empty area-light sample (pdf 0)
  } else if (r <= alsWeight + elsWeight) {
    if (p.hasEnv) env_pick_direction(p, pick, els);
    ls = els;
    ls.radiance = ls.radiance * (1.f / elsWeight);
    needsMIS = true;
  } else if (r <= alsWeight + elsWeight + plsWeight) {
    return false;
  } else {
    ls = dls;
    ls.radiance = ls.radiance * (1.f / dlsWeight);
    isDir = true;
  }
  if (isnan(ls.pdf) || (ls.pdf <= 0.f)) return false;
  return true;
}

// radianceFromEnv (shadeRays.cu:437-456) up to the texture read: the
// env-map coordinates of a ray direction
__device__ __forceinline__ float2 env_miss_coords(const RenderParams &p, vec3 rayDir) {
  vec3 d = xfm_vector(p.env.toLocal, normalize(rayDir));
  const float2 tp = spherical_theta_phi(d);
  float theta = tp.x;
  float phi = tp.y;
  const float invPi = 1.f / (float)3.14159265358979323846;
  const float inv2Pi = 1.f / (2.f * (float)3.14159265358979323846);
  return make_float2(phi * inv2Pi, theta * invPi);
}

// Phase.h:49-57
__device__ __forceinline__ float hg_phase(float g, float cosTheta) {
  if (fabsf(g) < 1e-3f) return kOneOverFourPi;
  float g2 = g * g;
  float denom = 1.f + g2 - 2.f * g * cosTheta;
  return kOneOverFourPi * (1.f - g2) / (denom * sqrtf(denom));
}
__device__ __forceinline__ float phase_pdf(const RenderParams &p, float g, vec3 wo, vec3 wi) {
  if (!p.multi) return kOneOverFourPi;
  if (fabsf(g) < 1e-3f) return kOneOverFourPi;  // isotropic: no directions needed
  vec3 wi_in = normalize(-wo);
  return hg_phase(g, dot(wi_in, normalize(wi)));
}
// Phase.h:74-99
__device__ __forceinline__ vec3 sample_hg_direction(vec3 wi_in, float g, Random &random) {
  float u0 = random();
  float u1 = random();
  float cosTheta;
  if (fabsf(g) < 1e-3f) cosTheta = 1.f - 2.f * u0;
  else {
    float sqrTerm = (1.f - g * g) / (1.f + g - 2.f * g * u0);
    cosTheta = (1.f + g * g - sqrTerm * sqrTerm) / (2.f * g);
  }
  float sinTheta = sqrtf(mx(0.f, 1.f - cosTheta * cosTheta));
  float phi = kTwoPi * u1;
  float sinPhi, cosPhi;
  sincos_angle(phi, sinPhi, cosPhi);  // phi in [0, 2 pi)
  vec3 local(cosPhi * sinTheta, sinPhi * sinTheta, cosTheta);
  vec3 w = normalize(wi_in);
  vec3 u, v;
  if (fabsf(w.x) > 0.1f) u = normalize(cross(vec3(0.f, 1.f, 0.f), w));
  else u = normalize(cross(vec3(1.f, 0.f, 0.f), w));
  v = cross(w, u);
  return normalize(local.x * u + local.y * v + local.z * w);
}

// Per-ray state of the pixel's path (Ray + PathState, render/Ray.h:18-99)
struct PathRay {
  vec3 org, dir;
  float tMax;
  RNGSeed seed;
  vec3h tp;
  float misWeight;
  int numVolumeBounces;
  int numDiffuseBounces;  // surface bounces (iso-surface worlds only)
};

struct ShadeOut {
  vec3 fragment;
  bool shadowValid;
  PathRay shadow;
};

// bounce() for a volume hit (shadeRays.cu:605-878).  Updates `ray`; a dead
// ray has tMax = -1.
// `random` is the hit's stream, Random2(ray.rngSeed, tHit), already derived
// (it advanced ray.seed); with an env map `pick` holds the light sample's
// texel coordinates and radiance.
__device__ __forceinline__ void bounce_volume_hit(const RenderParams &p, PathRay &ray, const Hit &h, vec3 P,
                                                  int pathDepth, Random &random, const EnvPick &pick,
                                                  ShadeOut &out) {
  out.shadowValid = false;
  const float tHit = h.t;
  const vec3 albedo = p.multi ? p.scatAlb * h.rgb : .7f * h.rgb;
  const float g = p.multi ? p.aniso : 0.f;
  const vec3 incomingThroughput = from_half(ray.tp);
  const vec3 wo = -normalize(ray.dir);
  const float offsetEpsilon = mx(1e-4f, 1e-6f * reduce_max(vabs(P)));
  LightSample ls;
  bool needsMIS = false, isDir = false;
  if (sample_lights(p, random, pick, ls, needsMIS, isDir)) {
    float density = p.multi ? phase_pdf(p, g, wo, ls.direction) : kOneOverFourPi;
    vec3 fr = density * albedo;
    if (!(density > 0.f) || reduce_max(fr) < 1e-4f) {
      out.shadowValid = false;
    } else {
      fr = vmin(fr, vec3(13.f));
      vec3 tp_sr = incomingThroughput * (isinf(ls.pdf) ? 1.f : 1.f / ls.pdf) * fr * ls.radiance * 1.f;
      out.shadow.dir = ls.direction;
      out.shadow.org = P + offsetEpsilon * wo;
      out.shadow.tMax = ls.distance * (1.f - 2.f * offsetEpsilon);
      out.shadow.tp = to_half(tp_sr);
      out.shadow.seed = ray.seed;
      ray.seed.next_h((uint64_t)hit_hash(tHit));
      out.shadow.misWeight = 1.f;
      out.shadowValid = true;
      if (!isDir && needsMIS) {
        float pdf_l = env_pdf(p, ls.direction);
        float pdf_s = p.multi ? phase_pdf(p, g, wo, ls.direction) : kOneOverFourPi;
        out.shadow.misWeight = pdf_l / (pdf_l + pdf_s + 1e-10f);
        if (out.shadow.misWeight < 1e-5f) out.shadowValid = false;
      }
    }
  }
  if (pathDepth >= 10) {  // MAX_PATH_DEPTH
    ray.tMax = -1.f;
    return;
  }
  ray.tMax = __int_as_float(0x7f800000);
  if (!p.multi) {
    // SCI_VIS_MODE: a volume scatter ends the path after its shadow ray
    // (the scatter direction is drawn but never used).
    ray.tMax = -1.f;
    return;
  }
  vec3 wi_in = normalize(-wo);
  vec3 sdir = sample_hg_direction(wi_in, g, random);
  float spdf = hg_phase(g, dot(wi_in, sdir));
  vec3 sf_r = albedo * spdf;
  if (!(spdf > 0.f) || spdf <= 1e-6f) return;
  if (!p.volMS || ray.numVolumeBounces >= p.maxVB) {
    ray.tMax = -1.f;
    return;
  }
  ray.numVolumeBounces = ray.numVolumeBounces + 1;
  ray.org = P + (1.f * offsetEpsilon) * wo;
  ray.dir = normalize(sdir);
  vec3 scatterFactor = sf_r * 1.f / (isinf(spdf) ? 1.f : (spdf + 1e-10f));
  scatterFactor = vmin(scatterFactor, vec3(2.5f));
  ray.tp = to_half(from_half(ray.tp) * scatterFactor);
  if (needsMIS && !isinf(spdf)) {
    float pdf_s = phase_pdf(p, g, wo, ray.dir);
    float pdf_l = env_pdf(p, ray.dir);
    ray.misWeight = pdf_s / (pdf_s + pdf_l);
  } else {
    ray.misWeight = 1.f;
  }
}

// owl::common::frame: the orthonormal frame about a unit normal N that
// xfmVector(frame(N), v) uses -- dx the longer of (1,0,0) x N and
// (0,1,0) x N, normalized, dy = normalize(N x dx)
__device__ __forceinline__ void frame_of(vec3 N, vec3 &dx, vec3 &dy) {
  const vec3 dx0 = cross(vec3(1.f, 0.f, 0.f), N), dx1 = cross(vec3(0.f, 1.f, 0.f), N);
  dx = normalize(dot(dx0, dx0) > dot(dx1, dx1) ? dx0 : dx1);
  dy = normalize(cross(N, dx));
}
// Lambertian::pdf (packedBSDF/Lambertian.h:46-55): the cosine-hemisphere
// pdf about the normal turned toward wi
__device__ __forceinline__ float lambert_pdf(vec3 Ng, vec3 wi) {
  const vec3 N = dot(wi, Ng) < 0.f ? -Ng : Ng;
  return mx(dot(wi, N), 0.f) * kOneOverPi;
}

// bounce() for an iso-surface hit (shadeRays.cu:541-878 with isVolumeHit
// false), the matte material's Lambertian (AnariMatte.h:50-62,
// packedBSDF/Lambertian.h:57-90): Ng = normalize(ray.N), offsets and light
// sampling along the front-facing normal, the cosine factors of the surface
// branches and a diffuse scatter, at most MAX_DIFFUSE_BOUNCES = 1 per path
// (shadeRays.cu:18, 795-808).  Updates `ray` like bounce_volume_hit.
static __device__ __noinline__ void bounce_surface_hit(const RenderParams &p, PathRay &ray, vec3h Nh, float tHit,
                                                      vec3 P, int pathDepth, Random &random, const EnvPick &pick,
                                                      ShadeOut &out) {
  out.shadowValid = false;
  const vec3 Ng = normalize(from_half(Nh));
  const vec3 Ngff = dot(ray.dir, Ng) < 0.f ? Ng : -Ng;
  const vec3 incomingThroughput = from_half(ray.tp);
  const vec3 wo = -normalize(ray.dir);
  const float offsetEpsilon = mx(1e-4f, 1e-6f * reduce_max(vabs(P)));
  LightSample ls;
  bool needsMIS = false, isDir = false;
  if (sample_lights<true>(p, random, pick, ls, needsMIS, isDir, Ngff)) {
    // Lambertian::eval: the cosine against the unflipped normal
    const float cosThetaI = mx(dot(ls.direction, Ng), 0.f);
    vec3 fr = p.isoAlbedo * kOneOverPi * cosThetaI;
    if (!(cosThetaI * kOneOverPi > 0.f) || reduce_max(fr) < 1e-4f) {
      out.shadowValid = false;
    } else {
      fr = vmin(fr, vec3(13.f));
      vec3 tp_sr = incomingThroughput * (isinf(ls.pdf) ? 1.f : 1.f / ls.pdf) * fr * ls.radiance *
                   (kOneOverPi * fabsf(dot(Ng, ls.direction)));
      out.shadow.dir = ls.direction;
      out.shadow.org = P + offsetEpsilon * Ngff;
      out.shadow.tMax = ls.distance * (1.f - 2.f * offsetEpsilon);
      out.shadow.tp = to_half(tp_sr);
      out.shadow.seed = ray.seed;
      ray.seed.next_h((uint64_t)hit_hash(tHit));
      out.shadow.misWeight = 1.f;
      out.shadowValid = true;
      if (!isDir && needsMIS) {
        const float pdf_l = env_pdf(p, ls.direction);
        const float pdf_s = lambert_pdf(Ng, ls.direction);
        out.shadow.misWeight = pdf_l / (pdf_l + pdf_s + 1e-10f);
        if (out.shadow.misWeight < 1e-5f) out.shadowValid = false;
      }
    }
  }
  if (pathDepth >= 10) {  // MAX_PATH_DEPTH
    ray.tMax = -1.f;
    return;
  }
  ray.tMax = __int_as_float(0x7f800000);
  // Lambertian::scatter: cosineSampleHemisphere (DG.h:135-168) about the
  // normal turned toward wo.  Its vec2f s(random(), random()) takes the
  // second argument's draw first, as the reference's CPU backend (built
  // with gcc, which evaluates arguments right to left) does.
  const vec3 N = dot(wo, Ng) < 0.f ? -Ng : Ng;
  const float r0 = random();
  const float r1 = random();
  const float phi = kTwoPi * r1;
  const float cosTheta = sqrtf(r0);
  const float sinTheta = sqrtf(1.0f - r0);
  float sinPhi, cosPhi;
  sincos_angle(phi, sinPhi, cosPhi);  // phi in [0, 2 pi)
  vec3 dx, dy;
  frame_of(N, dx, dy);
  const vec3 sdir = dx * (cosPhi * sinTheta) + dy * (sinPhi * sinTheta) + N * cosTheta;
  const float spdf = cosTheta * kOneOverPi;
  if (!(spdf > 0.f) || spdf <= 1e-6f) return;  // the ray stays alive unchanged
  if (ray.numDiffuseBounces >= 1) {
    ray.tMax = -1.f;
    return;
  }
  ray.numDiffuseBounces = ray.numDiffuseBounces + 1;
  ray.org = P + (1.f * offsetEpsilon) * Ngff;
  ray.dir = normalize(sdir);
  vec3 scatterFactor = p.isoAlbedo * fabsf(dot(Ng, normalize(ray.dir))) / (isinf(spdf) ? 1.f : (spdf + 1e-10f));
  scatterFactor = vmin(scatterFactor, vec3(2.5f));
  ray.tp = to_half(from_half(ray.tp) * scatterFactor);
  if (needsMIS && !isinf(spdf)) {
    const float pdf_s = lambert_pdf(Ng, ray.dir);
    const float pdf_l = env_pdf(p, ray.dir);
    ray.misWeight = pdf_s / (pdf_s + pdf_l);
  } else {
    ray.misWeight = 1.f;
  }
}

__device__ __forceinline__ void accum_add(float4 &acc, vec3 frag) {
  if (frag.x > 0.f) acc.x += frag.x;
  if (frag.y > 0.f) acc.y += frag.y;
  if (frag.z > 0.f) acc.z += frag.z;
}

// -------------------------------------------------------------------------
// Traversal of one ray through the macrocell grid: dda::dda3 (DDA.h:65-206)
// with Woodcock::sampleRange (Volume.h:188-223) inside each cell of non-zero
// majorant, as set up by MCVolumeAccel::isProg (MCAccelerator.h:569-708).
// The state advances by bounded units so that a warp's lanes stay in one
// loop: per warp iteration a lane makes at most `skip` (default
// kSkipDefault) cell tests and distance draws to reach its next sample
// position, then the warp's ready lanes take their density samples together.
// -------------------------------------------------------------------------
// Defaults of the launch shape and the scheduling limits of the frame kernel
// (512^3 1080p 16-pass frame / 256^3 720p 1 pass, ms; results never depend on
// them):
// * rounds a seek makes before the warp samples: 2: 6.59 / 0.508, 3: 6.28 /
//   0.485, 4: 6.16 / 0.491, 6: 6.16 / 0.505;
// * a warp leaves tracing for a waiting stage below this share of its lanes:
//   10%: 6.24 / 0.491, 25%: 6.15 / 0.496, 30%: 6.22 / 0.507, 50%: 7.53 / 0.540,
//   65%: 11.2 / 0.618;
// * kRefillMin, the rays a refill waits for: 4: 6.21 / 0.503, 8: 6.11 / 0.493,
//   12: 6.16 / 0.490;
// * kFull, the paths that make a stage worth leaving another for: 16: 6.24 /
//   0.513, 24: 6.18 / 0.496, 28: 6.16 / 0.490, 30: 6.15 / 0.495.
constexpr int kSkipDefault = 4;
// A batch's lanes read their scene's record from memory at every seek: one
// that goes on to its next position reads it less often (64 uneven scenes, 8
// passes, when this was chosen: 4 rounds 6.25 ms, 16: 5.83, 64: 5.53).
constexpr int kBatchSkipDefault = 64;
constexpr int kThresholdDefault = 25;
constexpr int kRefillMin = 12, kFull = 28;
constexpr int kRepeatMin = 24;     // lanes for which starting passes goes on
constexpr int kIdlePolls = 1 << 24;  // polls (1 us) a warp without work makes at most

// Per-lane event counts; with On == false the counting and its registers
// compile away (timed launches pass no counter buffer).
template <bool On> struct Ctr {
  static constexpr bool kOn = On;
  unsigned samples = 0, mcs = 0, rays = 0, caps = 0, cells = 0;
};
#define GBV_COUNT(cnt, field) \
  do {                       \
    if (cnt.kOn) cnt.field++; \
  } while (0)
constexpr int kWoodcockCap = 1 << 20;
enum { TR_CONTINUE = 0, TR_HIT = 1, TR_MISS = 2 };

struct Traversal {
  vec3 org, dir;   // trace direction: zero components replaced by 1e-6
  float rayTMax;   // ray.tMax of the ray record
  vec3 t_next, t_step;
  int cx, cy, cz;
  int stopx, stopy, stopz;
  float ray_t0, tMax, ncb;
  float t, segHi, maj; // delta tracking in the current cell
  Random rng;
  int inCell;
  int steps;           // Woodcock steps in the current cell
  int cells;           // cells visited
};

__device__ __forceinline__ float majorant_at(const MCGridDev &G, int cx, int cy, int cz) {
  return __ldg(G.maj + (cx + G.M[0] * (cy + G.M[1] * cz)));
}

// Box test, RNG stream and DDA set-up.  Returns false when the ray reaches
// no cell.  `seed` advances exactly when the reference advances ray.rngSeed
// (once the box test passes); the stream is Random2(seed, streamHash), the
// hash of the geometry's instance (hash(0, 0, 0) for a lone volume).
template <class Cnt>
__device__ __forceinline__ bool trace_begin(const FieldGeom &F, const MCGridDev &G, const vec3 &rcpMc, vec3 org,
                                            vec3 rayDir, float rayTMax, RNGSeed &seed, Traversal &T, Cnt &cnt,
                                            uint64_t streamHash = kVolumeStreamHash) {
  GBV_COUNT(cnt, rays);
  vec3 dir = rayDir;
  if (dir.x == 0.f) dir.x = 1e-6f;
  if (dir.y == 0.f) dir.y = 1e-6f;
  if (dir.z == 0.f) dir.z = 1e-6f;
  if (G.M[0] <= 0 || G.M[1] <= 0 || G.M[2] <= 0) return false;
  float tLo = 0.f, tHi = rayTMax;
  if (!box_test(org, dir, tLo, tHi, F.boundsLo, F.boundsHi)) return false;
  const vec3 dda_org = (org - G.origin) * rcpMc;
  const vec3 dda_dir = dir * rcpMc;
  T.rng = Random::derive(seed, streamHash);
  const float tMax = tHi;
  const vec3 f_size((float)G.M[0], (float)G.M[1], (float)G.M[2]);
  const vec3 rcp_dir = rcp(dda_dir);
  vec3 t_lo = (vec3(0.f) - dda_org) * rcp_dir;
  vec3 t_hi = (f_size - dda_org) * rcp_dir;
  vec3 t_nr = vmin(t_lo, t_hi), t_fr = vmax(t_lo, t_hi);
  const float INF = __int_as_float(0x7f800000);
  if (dda_dir.x == 0.f) {
    if (dda_org.x < 0.f || dda_org.x > f_size.x) return false;
    t_nr.x = -INF; t_fr.x = INF;
  }
  if (dda_dir.y == 0.f) {
    if (dda_org.y < 0.f || dda_org.y > f_size.y) return false;
    t_nr.y = -INF; t_fr.y = INF;
  }
  if (dda_dir.z == 0.f) {
    if (dda_org.z < 0.f || dda_org.z > f_size.z) return false;
    t_nr.z = -INF; t_fr.z = INF;
  }
  const float ray_t0 = mx(0.f, reduce_max(t_nr));
  const float ray_t1 = mn(tMax, reduce_min(t_fr));
  if (ray_t0 > ray_t1) return false;
  const vec3 oiv = dda_org + ray_t0 * dda_dir;
  const vec3 f_cell = vmax(vec3(0.f), vmin(f_size - vec3(1.f), vfloor(oiv)));
  const vec3 f_end(dda_dir.x > 0.f ? f_cell.x + 1.f : f_cell.x, dda_dir.y > 0.f ? f_cell.y + 1.f : f_cell.y,
                   dda_dir.z > 0.f ? f_cell.z + 1.f : f_cell.z);
  T.t_step = vabs(rcp_dir);
  T.t_next = vec3((dda_dir.x == 0.f) ? INF : (fabsf(f_end.x - oiv.x) * T.t_step.x),
                  (dda_dir.y == 0.f) ? INF : (fabsf(f_end.y - oiv.y) * T.t_step.y),
                  (dda_dir.z == 0.f) ? INF : (fabsf(f_end.z - oiv.z) * T.t_step.z));
  T.stopx = dda_dir.x > 0.f ? G.M[0] : -1;
  T.stopy = dda_dir.y > 0.f ? G.M[1] : -1;
  T.stopz = dda_dir.z > 0.f ? G.M[2] : -1;
  T.cx = (int)f_cell.x;
  T.cy = (int)f_cell.y;
  T.cz = (int)f_cell.z;
  T.ray_t0 = ray_t0;
  T.tMax = tMax;
  T.ncb = 0.f;
  T.org = org;
  T.dir = dir;
  T.rayTMax = rayTMax;
  T.inCell = 0;
  T.cells = 0;
  return true;
}

// next_cell_begin = t_closest, then step every axis whose t_next equals it;
// false when the ray leaves the grid (its state is then not used again).
// Selects instead of branches: every lane that steps runs the same code.
__device__ __forceinline__ bool trace_advance(Traversal &T, float tc) {
  const bool ax = T.t_next.x == tc, ay = T.t_next.y == tc, az = T.t_next.z == tc;
  T.ncb = tc;
  T.t_next.x = ax ? T.t_next.x + T.t_step.x : T.t_next.x;
  T.t_next.y = ay ? T.t_next.y + T.t_step.y : T.t_next.y;
  T.t_next.z = az ? T.t_next.z + T.t_step.z : T.t_next.z;
  T.cx += ax ? (T.stopx >> 31) | 1 : 0;
  T.cy += ay ? (T.stopy >> 31) | 1 : 0;
  T.cz += az ? (T.stopz >> 31) | 1 : 0;
  return !((T.cx == T.stopx) | (T.cy == T.stopy) | (T.cz == T.stopz));
}

// The traversal is split so that the expensive part, the density sample,
// runs for all of a warp's tracing lanes at once.  trace_seek advances a lane
// toward its next sample position (T.inCell = 2: a position is ready) by at
// most `rounds` rounds of: test the macrocell it stands before (T.inCell 0;
// 1: inside one of non-zero majorant), draw a Woodcock distance inside it,
// and, from an empty cell or past the cell's end, step to the next cell.
// trace_sample then samples there and makes the accept test.  Every lane
// performs exactly the operations, in exactly the order, of the
// one-step-at-a-time loop (dda::dda3 with Woodcock::sampleRange inside each
// cell); only the grouping of a lane's steps into warp iterations differs.
// A round has one copy of each step and the lanes meet again after each, so
// that lanes crossing empty cells and lanes leaving a cell step together.
template <class Cnt>
__device__ __forceinline__ int trace_seek(const MCGridDev &G, Traversal &T, Cnt &cnt, int rounds, bool staged,
                                          int *capFlag) {
  const int maxCells = G.M[0] + G.M[1] + G.M[2] + 8;
  int state = TR_CONTINUE;
#pragma unroll 1
  for (int round = 0; round < rounds && T.inCell != 2 && state == TR_CONTINUE; round++) {
    const float tc = reduce_min(T.t_next);
    bool step = false;
    if (T.inCell == 0) {
      GBV_COUNT(cnt, cells);
      const int ci = T.cx + G.M[0] * (T.cy + G.M[1] * T.cz);
      const bool nonzero = staged ? ((g_smem[ci >> 5] >> (ci & 31)) & 1u) != 0u : __ldg(G.maj + ci) != 0.f;
      if (++T.cells > maxCells) {
        GBV_COUNT(cnt, caps);
        if (capFlag) *capFlag = 1;
        state = TR_MISS;
      } else if (nonzero) {
        T.maj = __ldg(G.maj + ci);
        T.inCell = 1;
        T.t = T.ray_t0 + T.ncb;
        T.segHi = mn(T.ray_t0 + mn(tc, T.tMax), T.rayTMax);
        T.steps = 0;
        GBV_COUNT(cnt, mcs);
      } else {
        step = true;
      }
    }
    if (T.inCell == 1) {
      const float r = T.rng();
      const float dt = -fastLog(1.f - r) / T.maj;
      T.t += dt;
      T.inCell = 2;
      if (T.t >= T.segHi || ++T.steps > kWoodcockCap) {
        if (T.steps > kWoodcockCap) {
          GBV_COUNT(cnt, caps);
          if (capFlag) *capFlag = 1;
        }
        T.inCell = 0;
        step = true;
      }
    }
    if (step && !trace_advance(T, tc)) state = TR_MISS;
  }
  return state;
}

template <class Store, class Cnt>
__device__ __forceinline__ int trace_sample(const FieldGeom &F, const Store &store, const XF &xf, Traversal &T,
                                            Hit &h, Cnt &cnt) {
  T.inCell = 1;
  const vec3 P = T.org + T.t * T.dir;
  // Volume::DD::sampleAndMap (Volume.h:66-80): NaN maps to zeros
  const float f = sample_field(F, store, P);
  GBV_COUNT(cnt, samples);
  float w = 0.f;
  XFSegment seg;
  if (!isnan(f)) {
    seg = xf_segment(xf, f);
    w = seg.opacity() * xf.baseDensity;
  }
  if (w >= T.rng() * T.maj) {
    h.hit = true;
    h.t = T.t;
    h.rgb = isnan(f) ? vec3(0.f) : seg.color();
    return TR_HIT;
  }
  return TR_CONTINUE;
}

// i / 10 as a float
static __constant__ float kTenths[11] = {0.f / 10.f, 1.f / 10.f, 2.f / 10.f, 3.f / 10.f, 4.f / 10.f, 5.f / 10.f,
                                         6.f / 10.f, 7.f / 10.f, 8.f / 10.f, 9.f / 10.f, 10.f / 10.f};
// The hit search and normal of MCIsoSurfaceAccel::isProg
// (MCAccelerator.h:393-503) along a DDA that trace_begin set up: per
// macrocell whose scalar range holds the iso value, the cell's t range is
// cut into 10 sub-steps; the first sub-step whose end values bracket the
// value gives the hit t by linear interpolation.  The normal is the central
// difference of the field at +-delta per axis, one-sided where a sample
// falls outside the field, normalized.  Returns whether t < tmax.
// `stop`: the search may end before a macrocell that begins beyond it (a
// crossing found there would lie beyond `stop`: an interpolated t is never
// more than a few ulps below its cell's start, far inside the 1e-5 margin);
// +inf searches the whole ray.
template <class Store>
__device__ __forceinline__ bool iso_search(const FieldGeom &F, const Store &renderStore, const MCGridDev &G,
                                           const float2 *__restrict__ ranges, float iso, float delta, Traversal &T,
                                           float tmax, float &tOut, vec3 &N,
                                           float stop = __int_as_float_hd(0x7f800000), bool normal = true) {
  // the sub-steps' samples lie close together along the ray: read through L1
  const auto &store = via_l1(renderStore);
  const int maxCells = G.M[0] + G.M[1] + G.M[2] + 8;
  float tHit = tmax;
  bool stopped = false;
  auto crosses = [&](float tt0, float ff0, float tt1, float ff1) {
    if (isnan(ff0) || isnan(ff1) || !(iso >= mn(ff0, ff1) && iso <= mx(ff0, ff1))) return false;
    float t = (iso - ff0) / (ff1 - ff0);
    t = lerp_l(t, tt0, tt1);
    tHit = mn(tHit, t);
    return tHit < tmax;
  };
  // Each lane walks to its next macrocell that holds the value, then all of
  // them sample theirs: a cell's 11 samples are most of the search, and a lane
  // that sampled where it stood left those that had only to walk on waiting
  // (256^3, 960x540, 8 passes through isotropic fog: 5.78 -> 5.22 ms; two samples at a time 6.4,
  // at most 8 cells a walk the same; a shadow ray needs no normal: -> 5.15).
  // Half of its stalls were instruction fetch (8.5 of 17 cycles per issued
  // instruction): one copy of the sample in a cell and one at the normal,
  // instead of 9, -> 4.46.
  bool more = true;
#pragma unroll 1
  for (int it = 0; more;) {
    float tc = 0.f, t0 = 0.f, t1 = 0.f;
    bool holds = false;
#pragma unroll 1
    while (more && !holds) {
      more = it++ < maxCells;
      tc = reduce_min(T.t_next);
      t0 = T.ray_t0 + T.ncb;
      t1 = T.ray_t0 + mn(tc, T.tMax);
      more = more && !(t0 > stop + fabsf(stop) * 1e-5f);
      if (!more) break;
      // the iso lambda (MCAccelerator.h:405-471)
      if (!(t0 >= mn(t1, tmax))) {
        const float2 vr = __ldg(ranges + (T.cx + G.M[0] * (T.cy + G.M[1] * T.cz)));
        holds = iso >= vr.x && iso <= vr.y;
      }
      if (!holds) more = trace_advance(T, tc);
    }
    if (!holds) break;
    float tt1 = t0, ff1 = __int_as_float(0x7fffffff);  // no sample before the first
#pragma unroll 1
    for (int i = 0; i <= 10 && !stopped; i++) {
      const float tt0 = tt1;
      const float ff0 = ff1;
      if (i > 0) tt1 = lerp_l(kTenths[i], t0, t1);
      ff1 = sample_field(F, store, T.org + tt1 * T.dir);
      stopped = crosses(tt0, ff0, tt1, ff1);
    }
    more = !stopped && trace_advance(T, tc);
  }
  if (!(tHit < tmax)) return false;
  tOut = tHit;
  if (!normal) return true;
  const vec3 P = T.org + tHit * T.dir;
  const float d = delta;
  // the hit, then the two neighbours along each axis: one copy of the sample
  float fP = 0.f, f0 = 0.f;
  N = vec3(0.f);
#pragma unroll 1
  for (int k = 0; k < 7; k++) {
    const int axis = (k - 1) >> 1;
    const float o = k & 1 ? -d : d;
    const vec3 off(axis == 0 ? o : 0.f, axis == 1 ? o : 0.f, axis == 2 ? o : 0.f);
    float f1 = sample_field(F, store, k == 0 ? P : P + off);
    if (k == 0) {
      fP = f1;
    } else if (k & 1) {
      f0 = f1;
    } else {
      float n = 2.f;
      if (isnan(f0)) { n -= 1.f; f0 = fP; }
      if (isnan(f1)) { n -= 1.f; f1 = fP; }
      const float c = n == 0.f ? 0.f : (f1 - f0) / n;
      if (axis == 0) N.x = c;
      if (axis == 1) N.y = c;
      if (axis == 2) N.z = c;
    }
  }
  if (is_zero(N)) N = -normalize(T.dir);
  N = normalize(N);
  return true;
}

// The iso-surface's intersection program for a render ray (org, rayDir,
// [0, tmax]): the box test and the geometry's random stream
// Random2(seed, hash(instance, 0, 0)), which advances `seed`; the hit
// search; the material's opacity test (opacity < 1: the ray passes when
// rng() > opacity, MCAccelerator.h:533-539); and Ray::setHit's record (the
// hit point and the normal in half precision).  Returns whether the surface
// records a hit.
// The iso-surface's box test and random stream alone -- what its
// intersection program does to the ray's seed -- when it runs before the
// volume's: the search itself waits until the volume's first collision is
// known (iso_trace_after).  Returns whether the box test passed; the stream's
// state goes to *rng.
__device__ __forceinline__ bool iso_begin(const RenderParams &p, vec3 org, vec3 rayDir, float tmax, RNGSeed &seed,
                                          uint64_t &rng) {
  vec3 dir = rayDir;
  if (dir.x == 0.f) dir.x = 1e-6f;
  if (dir.y == 0.f) dir.y = 1e-6f;
  if (dir.z == 0.f) dir.z = 1e-6f;
  if (p.G.M[0] <= 0 || p.G.M[1] <= 0 || p.G.M[2] <= 0) return false;
  float tLo = 0.f, tHi = tmax;
  if (!box_test(org, dir, tLo, tHi, p.F.boundsLo, p.F.boundsHi)) return false;
  rng = Random::derive(seed, p.isoHash).s.state;
  return true;
}

// The rest of that program, after the volume traced without the surface's
// bound and found its first collision at `stop` (+inf: none): the search on
// the ray's own [0, tmax], as the program makes it, ends at `stop`; the
// surface's hit counts when its t is at most `stop` (the volume's tracking,
// bounded by the surface's hit, would have stopped there: the surface wins a
// tie), after the material's opacity test on the stream iso_begin made.
// The final hit, point, normal and every random stream equal those of
// running the surface's program first.
template <class Store>
static __device__ __noinline__ bool iso_trace_after(const RenderParams &p, vec3 org, vec3 rayDir, float tmax,
                                                    float stop, uint64_t rng, bool normal, float &tOut, vec3h &Nh) {
  Traversal T;
  Ctr<false> none;
  RNGSeed scratch;  // the stream was derived by iso_begin
  scratch.state = 0;
  if (!trace_begin(p.F, p.G, p.rcpMc, org, rayDir, tmax, scratch, T, none, p.isoHash)) return false;
  float t;
  vec3 N;
  if (!iso_search(p.F, make_store<Store>(p), p.G, p.isoRanges, p.isoValue, p.isoDelta, T, tmax, t, N, stop, normal))
    return false;
  if (!(t <= stop)) return false;
  Random r;
  r.s.state = rng;
  if (p.isoAlpha < 1.f && r() > p.isoAlpha) return false;
  tOut = t;
  if (normal) Nh = to_half(N);
  return true;
}

template <class Store>
static __device__ __noinline__ bool iso_trace(const RenderParams &p, vec3 org, vec3 rayDir, float tmax, RNGSeed &seed,
                                              bool normal, float &tOut, vec3h &Nh) {
  Traversal T;
  Ctr<false> none;
  if (!trace_begin(p.F, p.G, p.rcpMc, org, rayDir, tmax, seed, T, none, p.isoHash)) return false;
  float t;
  vec3 N;
  if (!iso_search(p.F, make_store<Store>(p), p.G, p.isoRanges, p.isoValue, p.isoDelta, T, tmax, t, N,
                  __int_as_float(0x7f800000), normal))
    return false;
  if (p.isoAlpha < 1.f && T.rng() > p.isoAlpha) return false;
  tOut = t;
  if (normal) Nh = to_half(N);
  return true;
}

// The auxiliary channels of pixel px from its primary ray (shadeRays.cu:
// 1003-1023): pass 0 writes the depth (the ray's tMax: the closest hit's t,
// or the generated 1e30 on a miss) and the closest hit's IDs (primitive 0 of
// the user geometry, its instance index and userID; -1 on a miss); later
// passes keep the smaller depth.  The lane owns the pixel: no atomics.
static __device__ __noinline__ void write_aux(const RenderParams &p, size_t px, int accumID, float z, int hitKind) {
  if (accumID == 0) {
    if (p.depth) p.depth[px] = z;
    if (p.primId) p.primId[px] = hitKind ? 0 : -1;
    if (p.instId) p.instId[px] = hitKind == 1 ? p.volInst : hitKind == 2 ? p.isoInst : -1;
    if (p.objId) p.objId[px] = hitKind == 1 ? p.volUser : hitKind == 2 ? p.isoUser : -1;
  } else if (p.depth && z < p.depth[px]) {
    p.depth[px] = z;
  }
}

// -------------------------------------------------------------------------
// The persistent frame kernel.  A path lives in a slot of its block's pool in
// shared memory; a block (one per SM) has more paths than lanes.  A warp takes
// up to 32 paths that wait for the same stage and runs that stage for them:
// starting passes and shading misses, tracing, the iso-surface search, shading
// hits.
//
// What bounds it: instruction issue.  A ray is a few cells, draws and samples
// of very different number, a hit's shading a few thousand instructions; a
// lane that owns its pixel from generation to shading leaves the others of
// its warp waiting in every phase (8.6 of 32 lanes active per instruction),
// and warps in different phases evict one another's code (41% of the stall
// cycles were instruction fetch).  Taking paths by stage gives 15 to 20 active
// lanes; letting the block's warps leave tracing for shading together
// (PathPool::shading) keeps them in the same code: 16.2 -> 14.5 ms from the
// pool, -> 12.4 ms from the common phase, -> 11.7 ms from refilling lanes in
// batches (512^3, 1080p, 16 passes, as each was made; with passes logged, see
// below, and later changes such a frame takes 6.2 ms).  The register budget
// matters little to its middle (128 registers a thread 6.27 ms, 96 6.16, 80
// 6.14) and much to its end, see default_budget.
//
// A path that sums all of its pixel's passes runs them one after the other,
// so the last pixels' passes hold a small frame's end: 50 to 80% of its time.
// The tiles that see the field come first and, as far as the log has room,
// pass by pass (F_SPLIT), each pass's fragments logged: 256^2 x 16 passes of a
// 64^3 volume 0.65 -> 0.18 ms, 853x479 x 8 passes 1.27 -> 0.38 ms, 1280x720 x
// 4 passes multi-scatter 2.83 -> 1.24 ms.
// -------------------------------------------------------------------------
// Path slots of a block
constexpr int kSlots = 1024;
// Threads of a block, by the register budget gbv_render_config.blocks_per_sm
// asks for (4: 128 registers a thread, 5: 96, 6: 80)
__host__ __device__ constexpr int block_threads(int budget) { return budget * 128; }

__device__ __forceinline__ float4 miss_color(const RenderParams &p, int iy) {
  float4 m = p.bg;
  if (!(p.bg.w >= 0.f)) {
    const float t = ((float)iy + .5f) / (float)p.H;
    m.x = (1.0f - t) * 0.9f + t * 0.15f;
    m.y = (1.0f - t) * 0.9f + t * 0.25f;
    m.z = (1.0f - t) * 0.9f + t * .8f;
    m.w = (1.0f - t) * 1.f + t * 1.f;
  }
  return m;
}

// _generateRays (generateRays.cu:72-243), perspective camera, no aperture
__device__ __forceinline__ void generate_primary(const RenderParams &p, int ix, int iy, int accumID, PathRay &ray) {
  Random rand = Random::from_pair((unsigned)(ix + p.W * accumID), (unsigned)(iy + p.H * accumID));
  ray.seed = seeded((uint32_t)(ix + accumID * p.W), (uint32_t)iy);
  const float pixel_u = (accumID == 0) ? .5f : rand();
  const float pixel_v = (accumID == 0) ? .5f : rand();
  const float image_u = ((float)ix + pixel_u) / (float)p.W;
  const float image_v = ((float)iy + pixel_v) / (float)p.H;
  const vec3 d = p.dir00 + (1.f * p.aspect * (image_u - .5f)) * p.du + (1.f * (image_v - .5f)) * p.dv;
  ray.org = p.lens00;
  ray.dir = normalize(d);
  ray.tMax = 1e30f;
  ray.tp = vec3h{0x3c00, 0x3c00, 0x3c00};  // 1.0 in half
  ray.misWeight = 0.f;
  ray.numVolumeBounces = 0;
  ray.numDiffuseBounces = 0;
}

// A primary ray that leaves the world: its fragment, and its alpha in w
__device__ __forceinline__ float4 primary_miss(const RenderParams &p, int iy, vec3 dir, int accumID) {
  const float4 miss = miss_color(p, iy);
  vec3 frag(miss.x, miss.y, miss.z);
  if (p.hasEnv) {
    const float2 uv = env_miss_coords(p, dir);
    const float4 t = tex2D(p.env, uv.x, uv.y);
    frag = p.env.scale * vec3(t.x, t.y, t.z);
  }
  frag = vmin(frag, vec3(10.f * (float)(1 + accumID)));
  return make_float4(frag.x, frag.y, frag.z, miss.w);
}
__device__ __forceinline__ void add_miss(float4 &acc, float4 miss, int accumID) {
  if (accumID == 0) {
    acc = miss;
  } else {
    if (miss.w > 0.f) acc.w += miss.w;
    accum_add(acc, vec3(miss.x, miss.y, miss.z));
  }
}
// What a path waits for; each is a bitmask over the block's slots in shared
// memory.  Publishing a path sets its bit (after a fence), taking it clears
// the bit: whoever clears it owns the path.
enum {
  Q_FREE = 0,   // no pixel
  Q_START = 1,  // F_FRESH: its next pass is to be generated; else its main ray left the world
  Q_READY = 2,  // a ray (F_SHADOW: the shadow ray) is to be traced
  Q_HIT = 3,    // its main ray has a hit to shade
  Q_ISO = 4,    // the volume is traced, the iso-surface search is to run
  Q_COUNT = 5
};
// Control word of a path: flags, generation in bits 8..15
constexpr uint32_t F_FRESH = 1u, F_SHADOW = 2u, F_ALIVE = 4u, F_ISOBOX = 8u, F_SPLIT = 16u,
                   F_LONE = 32u /* a shadow ray of a path that goes on elsewhere */,
                   F_VOLHIT = 1u << 16, F_SURFHIT = 2u << 16,
                   kHitMask = 3u << 16;
// Words of a path's record.  The main ray's hit (t, rgb, the surface's
// normal) shares the shadow ray's words: a main ray's hit is shaded before
// its shadow ray exists.
// A split path (one pass of a pixel, F_SPLIT) keeps no sum: W_ACC holds its
// record's index in the log and the fragments it has logged.
enum {
  W_REC = 23, W_MASK = 24,
  W_ORG = 0, W_DIR = 3, W_SEED = 6, W_TP = 8 /* 3 halves, bounce counts */, W_MIS = 10,
  W_SORG = 11, W_SDIR = 14, W_STMAX = 17, W_SSEED = 18, W_STP = 20, W_SMIS = 22,
  W_HT = 11, W_HRGB = 12, W_HN = 15,
  W_ACC = 23, W_IX = 27, W_IY = 28, W_PASS = 29, W_CTL = 30, W_ITEM = 31, W_ISORNG = 32
};

// Record of a split path in the log: the fragments it logged (a bit per
// generation; kLogMissed: the primary ray itself missed), the pass's alpha,
// then 3 floats per generation -- the shadow ray's fragment of a hit, or the
// miss that ends the path.  Each generation adds at most one fragment to a
// pixel that is not zero, so adding a pixel's records pass by pass and
// generation by generation is the order in which a lane that owned the pixel
// would add them.
constexpr uint32_t kLogMissed = 1u << 31;
__host__ __device__ constexpr int log_words(int hits) { return 2 + 3 * hits; }
__device__ __forceinline__ void log_fragment(const RenderParams &L, uint32_t rec, int gen, vec3 f) {
  if (gen >= L.logHits) return;  // path_hits bounds the generations
  float *r = reinterpret_cast<float *>(L.log) + (size_t)rec * log_words(L.logHits) + 2 + 3 * gen;
  r[0] = f.x;
  r[1] = f.y;
  r[2] = f.z;
}
__device__ __forceinline__ void log_end(const RenderParams &L, uint32_t rec, uint32_t mask, float alpha) {
  uint32_t *r = L.log + (size_t)rec * log_words(L.logHits);
  r[0] = mask;
  r[1] = __float_as_uint(alpha);
}

// Position of the r-th set bit (r < popc(bits)).
__device__ __forceinline__ int nth_bit(uint32_t bits, int r) {
  int p = 0;
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) {
    const int t = __popc(bits & ((1u << h) - 1u));
    const bool up = r >= t;
    r -= up ? t : 0;
    p += up ? h : 0;
    bits = up ? bits >> h : bits;
  }
  return p;
}
__device__ __forceinline__ int warp_scan(int v) {  // inclusive sum over the warp's lanes
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, v, o);
    if ((int)(threadIdx.x & 31) >= o) v += x;
  }
  return v;
}

// The paths of one block, field-major: lane k of a stage reads word f of
// slot j at bank j mod 32.
template <bool Iso> struct PathPool {
  static constexpr int kWords = Iso ? 34 : 32;
  static constexpr int kStride = kWords * kSlots + Q_COUNT * (kSlots / 32) + 1 + 6 * 24;
  uint32_t *w;
  __device__ __forceinline__ uint32_t u(int f, int k) const { return w[f * kSlots + k]; }
  __device__ __forceinline__ void setu(int f, int k, uint32_t v) const { w[f * kSlots + k] = v; }
  __device__ __forceinline__ float f(int i, int k) const { return __uint_as_float(w[i * kSlots + k]); }
  __device__ __forceinline__ void setf(int i, int k, float v) const { w[i * kSlots + k] = __float_as_uint(v); }
  __device__ __forceinline__ vec3 v3(int i, int k) const { return vec3(f(i, k), f(i + 1, k), f(i + 2, k)); }
  __device__ __forceinline__ void setv3(int i, int k, vec3 v) const {
    setf(i, k, v.x);
    setf(i + 1, k, v.y);
    setf(i + 2, k, v.z);
  }
  __device__ __forceinline__ uint64_t u64(int i, int k) const {
    return (uint64_t)u(i, k) | ((uint64_t)u(i + 1, k) << 32);
  }
  __device__ __forceinline__ void setu64(int i, int k, uint64_t v) const {
    setu(i, k, (uint32_t)v);
    setu(i + 1, k, (uint32_t)(v >> 32));
  }
  __device__ __forceinline__ float4 acc(int k) const {
    return make_float4(f(W_ACC, k), f(W_ACC + 1, k), f(W_ACC + 2, k), f(W_ACC + 3, k));
  }
  __device__ __forceinline__ void setacc(int k, float4 a) const {
    setf(W_ACC, k, a.x);
    setf(W_ACC + 1, k, a.y);
    setf(W_ACC + 2, k, a.z);
    setf(W_ACC + 3, k, a.w);
  }
  __device__ __forceinline__ vec3h half3(int i, int k) const {
    const uint32_t a = u(i, k), b = u(i + 1, k);
    return vec3h{(uint16_t)(a & 0xffffu), (uint16_t)(a >> 16), (uint16_t)(b & 0xffffu)};
  }
  __device__ __forceinline__ void sethalf3(int i, int k, vec3h h, uint32_t upper = 0) const {
    setu(i, k, (uint32_t)h.x | ((uint32_t)h.y << 16));
    setu(i + 1, k, (uint32_t)h.z | (upper << 16));
  }
  __device__ __forceinline__ uint32_t *queue(int q) const { return w + kWords * kSlots + q * (kSlots / 32); }
  // Hands path k to whoever takes it from queue q.
  __device__ __forceinline__ void publish(int q, int k) const {
    __threadfence_block();
    atomicOr(queue(q) + (k >> 5), 1u << (k & 31));
  }
  // The block's phase: whether warps leave tracing for the shading stages
  // (whole warp; one lane's read, so that the warp agrees).
  __device__ __forceinline__ bool shading() const {
    const volatile uint32_t *m = queue(Q_COUNT);
    return __shfl_sync(0xffffffffu, *m, 0) != 0u;
  }
  __device__ __forceinline__ void set_shading(uint32_t on) const {
    volatile uint32_t *m = queue(Q_COUNT);
    if ((threadIdx.x & 31) == 0) *m = on;
    __syncwarp();
  }
  // Paths waiting in queue q (whole warp).
  __device__ __forceinline__ int waiting(int q) const {
    const volatile uint32_t *m = queue(q);
    return (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(m[threadIdx.x & 31]));
  }
  // Takes up to `want` (<= 32) paths from queue q (whole warp): lane i gets
  // the i-th of the n taken, other lanes -1.  rot spreads the warps over the
  // queue's words.
  __device__ __forceinline__ int take(int q, int want, int rot, int &n) const {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    volatile uint32_t *m = queue(q);
    const int at = (lane + rot) & 31;
    const uint32_t bits = m[at];
    const int c = __popc(bits);
    const int before = warp_scan(c) - c;
    const int mine = min(max(want - before, 0), c);
    const uint32_t sel = mine == c ? bits : bits & ((1u << nth_bit(bits, mine)) - 1u);
    const uint32_t got = sel ? atomicAnd(const_cast<uint32_t *>(m) + at, ~sel) & sel : 0u;
    // the lane that took a path is seldom the one that reads its record: the
    // barrier orders their accesses (the shuffles below order no memory)
    __threadfence_block();
    __syncwarp();
    const int g = __popc(got), upTo = warp_scan(g);
    n = __shfl_sync(FULL, upTo, 31);
    const int first = upTo - g;
    int l = 0;  // the word lane i's path is in: the last one that starts at or before i
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
      const int x = __shfl_sync(FULL, first, l + h);
      l += x <= lane ? h : 0;
    }
    const uint32_t word = __shfl_sync(FULL, got, l);
    const int r = lane - __shfl_sync(FULL, first, l);
    return lane < n ? ((l + rot) & 31) * 32 + nth_bit(word, r) : -1;
  }
};

// Batch: the launch renders `numItems` scenes (items[]), whose 8x4-pixel
// tiles are numbered consecutively (tileStart[] holds the prefix sums); a
// lane reads the scene of the path it works on.  Otherwise the launch renders
// the one scene `p0`.  Launch-wide settings (passes, thresholds, counters)
// always come from p0.  Count: whether to count events (see Ctr) and, with
// a profile requested in the launch config (gbv_render_config.profile),
// cycles and lanes per phase (the timed kernel, Count =
// false, carries no profiling code).
// p0 is __grid_constant__ so that helpers can take it by reference without a
// copy to local memory.
// Iso: the world holds an iso-surface (p0.isoOn; never batched): each trace
// also runs its intersection program, before the volume's when its instance
// index is the lower one (p0.isoFirst) and otherwise after it, each bounded
// by the other's hit, and shading takes the surface branch on its hits.
template <class Store, int Budget, bool Batch, bool Count, bool Iso = false>
__global__ void __launch_bounds__(block_threads(Budget), 1)
    render_kernel(const __grid_constant__ RenderParams p0, const RenderParams *__restrict__ items,
                  const long long *__restrict__ tileStart, int numItems, int *__restrict__ pool) {
  static_assert(!(Iso && Batch), "batched launches render volume-only worlds");
  using Pool = PathPool<Iso>;
  const unsigned FULL = 0xffffffffu;
  const float INF = __int_as_float(0x7f800000);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int rot = 2 * warp;
  const RenderParams &L = p0;  // launch-wide settings
  asm volatile("griddepcontrol.launch_dependents;");  // finish_kernel may start where a block has ended
  // ---- stage the majorant bitmask and env-map tables in shared memory ----
  if (!Batch) {
    const RenderParams &p = p0;
    if (p.maskWords > 0) stage_majorant_mask(p);
    if (p.cdfYOff >= 0)
      for (int i = threadIdx.x; i < p.env.H; i += blockDim.x) g_smem[p.cdfYOff + i] = __float_as_uint(__ldg(p.env.cdf_y + i));
    if (p.pivOff >= 0) {
      const int total = p.env.H * p.pivPerRow;
      for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int row = i / p.pivPerRow, k = i - row * p.pivPerRow;
        const int last = min(k * 32 + 31, p.env.W - 2);
        g_smem[p.pivOff + i] = __float_as_uint(__ldg(p.env.cdf_x + (size_t)row * p.env.W + last));
      }
    }
    if (p.rowOff >= 0)
      for (int i = threadIdx.x; i < p.env.H; i += blockDim.x)
        reinterpret_cast<float2 *>(g_smem + p.rowOff)[i] = env_row_terms(p.env, i);
  }
  const Pool P{g_smem + L.poolOff};
  for (int i = threadIdx.x; i <= Q_COUNT * (kSlots / 32); i += blockDim.x)
    P.queue(0)[i] = i < L.slots / 32 ? 0xffffffffu : 0u;  // slots [0, L.slots) are free
  __syncthreads();
  if (lane == 0) P.queue(Q_COUNT)[1 + 6 * warp + 1] = 32u;  // the warp has no tile yet
  __syncwarp();
  Ctr<Count> cnt;
  bool poolDone = false;
  // the lane's trace
  int cur = -1;  // slot of the ray it traces
  Traversal T;
  unsigned long long cyc[3] = {0ull, 0ull, 0ull};
  // profile: traversal iterations and tracing lanes summed over them, shading
  // passes and shaded lanes summed over them (lane 0 of each warp counts)
  unsigned long long simt[4] = {0ull, 0ull, 0ull, 0ull};

  // The pass of path k is complete: the next one, or the pixel is finished.
  auto end_pass = [&](const RenderParams &p, int k, uint32_t ctl) -> int {
    if (ctl & F_SPLIT) {
      if (!(ctl & F_LONE)) log_end(L, P.u(W_REC, k), P.u(W_MASK, k), 1.f);
      return Q_FREE;
    }
    const int s = (int)P.u(W_PASS, k) + 1;
    if (s == L.spp) p.accum[(size_t)P.u(W_IY, k) * p.W + P.u(W_IX, k)] = P.acc(k);
    P.setu(W_PASS, k, (uint32_t)s);
    P.setu(W_CTL, k, F_FRESH);
    return s == L.spp ? Q_FREE : Q_START;
  };
  // The shadow ray of path k is traced: its fragment, then the main ray or
  // the pass's end.
  auto end_shadow = [&](const RenderParams &p, int k, uint32_t ctl, bool occluded) -> int {
    if (!occluded || (ctl & F_SPLIT)) {
      const float clampMax = 10.f * (float)(1 + L.accumIdStart + (int)P.u(W_PASS, k));
      const vec3 frag = vmin(P.f(W_SMIS, k) * from_half(P.half3(W_STP, k)), vec3(clampMax));
      if (ctl & F_SPLIT) {
        log_fragment(L, P.u(W_REC, k), (int)((ctl >> 8) & 0xffu) - 1, occluded ? vec3(0.f) : frag);
      } else {
        float4 acc = P.acc(k);
        accum_add(acc, frag);
        P.setacc(k, acc);
      }
    }
    if (!(ctl & F_ALIVE)) return end_pass(p, k, ctl);
    P.setu(W_CTL, k, ctl & ~F_SHADOW);
    return (int)Q_READY;
  };
  // The volume is traced for the ray of path k (hit: at t, colour rgb).
  auto end_trace = [&](const RenderParams &p, int k, bool hit, float t, vec3 rgb) -> int {
    const uint32_t ctl = P.u(W_CTL, k);
    const bool search = Iso && (!p.isoFirst || (ctl & F_ISOBOX));
    if (ctl & F_SHADOW) {
      // an occluded shadow ray stays so whatever the surface does
      return search && !hit ? (int)Q_ISO : end_shadow(p, k, ctl, hit);
    }
    if (hit) {
      P.setf(W_HT, k, t);
      P.setv3(W_HRGB, k, rgb);
      if (Iso) P.setu(W_CTL, k, ctl | F_VOLHIT);
    }
    return search ? (int)Q_ISO : hit ? (int)Q_HIT : (int)Q_START;
  };

  int idle = 0;  // polls without work
  while (true) {
    // ---- choose a stage ----
    const int nStart = P.waiting(Q_START), nHit = P.waiting(Q_HIT), nReady = P.waiting(Q_READY);
    const int nIso = Iso ? P.waiting(Q_ISO) : 0;
    const int nFree = poolDone ? 0 : P.waiting(Q_FREE);
    const int held = __popc(__ballot_sync(FULL, cur >= 0));
    const int nTrace = nReady + held, nOpen = nStart + nFree;
    enum { S_NONE, S_TRACE, S_HIT, S_START, S_ISO };
    int stage;
    const int most = max(max(nHit, nOpen), nIso);
    bool shading = P.shading();
    if (shading && most < kFull) {
      P.set_shading(0u);
      shading = false;
    }
    if (most >= kFull && (shading || nTrace < kFull)) {
      // One order for all warps: those that share a stage share its code.
      // Passes are started before hits are shaded, which keeps rays coming
      // (against the longest queue first: U8 853x479 x 8 passes 0.316 -> 0.287
      // ms, 512^3 x 16 passes 7.56 -> 7.40, 64 scenes x 8 passes 5.12 -> 5.04;
      // hits first 0.335, 7.43, 4.98); with an iso-surface the searches first,
      // then the hits (4.46 -> 4.38 ms).
      if (Iso) stage = nIso >= kFull ? S_ISO : nHit >= kFull ? S_HIT : S_START;
      else stage = nOpen >= kFull ? S_START : S_HIT;
    }
    else if (nTrace >= most) stage = nTrace ? S_TRACE : S_NONE;
    else stage = nHit == most ? S_HIT : Iso && nIso == most ? S_ISO : S_START;
    if (stage == S_NONE) {
      // Nothing waits: the block is done, or its paths are with other warps.
      // What becomes of them may need this warp (it may hold a tile whose
      // pixels wait for slots), so it looks again; each path ends, so does this.
      if (poolDone && P.waiting(Q_FREE) == L.slots) break;
      if (++idle > L.idlePolls) {  // pixels of its tile may be missing
        if (lane == 0) {
          GBV_COUNT(cnt, caps);
          if (L.capFlag) *L.capFlag = 1;
        }
        break;
      }
      __nanosleep(idle < 64 ? 200 : 1000);
      continue;
    }
    idle = 0;
    const long long c0 = (Count && L.profile) ? clock64() : 0;
    int phase;
    if (stage == S_TRACE) {
      // ---- trace: seek and sample until too few lanes are left ----
      phase = 1;
      while (true) {
        unsigned act = __ballot_sync(FULL, cur >= 0);
        const int idleLanes = 32 - __popc(act);
        int ended = -1;  // path whose volume trace ended in this iteration
        bool endHit = false;
        vec3 rgb(0.f);
        // refill in batches: the ray set-up runs for the new rays alone
        int more = 0;
        if (idleLanes > 0) {
          more = P.waiting(Q_READY);
          if (min(more, idleLanes) < (idleLanes > 24 ? 1 : kRefillMin)) more = -more;
        }
        if (more > 0) {
          int n;
          const int got = P.take(Q_READY, idleLanes, rot, n);
          const int k = __shfl_sync(FULL, got, __popc(~act & lt));
          if (cur < 0 && __popc(~act & lt) < n) {
            const uint32_t ctl = P.u(W_CTL, k);
            const bool shadow = ctl & F_SHADOW;
            const RenderParams &p = Batch ? items[P.u(W_ITEM, k)] : p0;
            const int o = shadow ? W_SORG : W_ORG, sw = shadow ? W_SSEED : W_SEED;
            const vec3 org = P.v3(o, k), dir = P.v3(o + 3, k);
            const float tmax = shadow ? P.f(W_STMAX, k) : (ctl & 0xff00u) ? INF : 1e30f;
            RNGSeed seed;
            seed.state = P.u64(sw, k);
            if (Iso) {
              uint32_t isoBit = 0;
              if (p.isoFirst) {
                // the surface's instance first: its box test and stream now, its
                // search once the volume's collision is known (iso_trace_after)
                uint64_t isoRng = 0;
                if (iso_begin(p, org, dir, tmax, seed, isoRng)) {
                  isoBit = F_ISOBOX;
                  P.setu64(W_ISORNG, k, isoRng);
                }
              }
              if (!p.hasVolume) GBV_COUNT(cnt, rays);
              P.setu(W_CTL, k, (ctl & ~(F_ISOBOX | kHitMask)) | isoBit);
            }
            const bool active = (!Iso || p.hasVolume) &&
                                trace_begin(p.F, p.G, p.rcpMc, org, dir, tmax, seed, T, cnt,
                                            Iso ? p.volHash : kVolumeStreamHash);
            P.setu64(sw, k, seed.state);
            if (active) cur = k;
            else ended = k;
          }
          act = __ballot_sync(FULL, cur >= 0);
        }
        if (cur >= 0) {
          const RenderParams &p = Batch ? items[P.u(W_ITEM, cur)] : p0;
          if (T.inCell != 2) {
            if constexpr (Batch) {
              const MCGridDev G = p.G;  // in registers while it seeks
              if (trace_seek(G, T, cnt, L.skip, false, L.capFlag) == TR_MISS) ended = cur;
            } else {
              if (trace_seek(p.G, T, cnt, L.skip, L.maskWords > 0, L.capFlag) == TR_MISS) ended = cur;
            }
          }
          __syncwarp(act);  // the lanes with a position sample together
          if (T.inCell == 2) {
            Hit h;
            if (trace_sample(p.F, make_store<Store>(p), p.xf, T, h, cnt) == TR_HIT) {
              ended = cur;
              endHit = true;
              rgb = h.rgb;
            }
          }
        }
        if (Count && L.profile && lane == 0) {
          simt[0]++;
          simt[1] += __popc(act);
        }
        if (ended >= 0) {
          P.publish(end_trace(Batch ? items[P.u(W_ITEM, ended)] : p0, ended, endHit, T.t, rgb), ended);
          if (ended == cur) cur = -1;
        }
        const int n = __popc(__ballot_sync(FULL, cur >= 0));
        if (more == 0 && n == 0) break;
        const bool low = more <= 0 && n * 100 < 32 * L.threshold;
        if (low || P.shading()) {
          if (P.waiting(Q_HIT) >= kFull || P.waiting(Q_START) >= kFull || (Iso && P.waiting(Q_ISO) >= kFull)) {
            P.set_shading(1u);
            break;
          }
        }
      }
    } else if (stage == S_HIT) {
      // ---- shade hits (bounce(), shadeRays.cu:477-878) ----
      phase = 2;
      int n;
      const int k = P.take(Q_HIT, 32, rot, n);
      if (Count && L.profile && lane == 0) {
        simt[2]++;
        simt[3] += n;
      }
      ShadeOut so;
      uint32_t ctl = 0u;
      bool shadow = false;
      if (k >= 0) {
        const RenderParams &p = Batch ? items[P.u(W_ITEM, k)] : p0;
        ctl = P.u(W_CTL, k);
        const int gen = (int)((ctl >> 8) & 0xffu);
        PathRay ray;
        ray.org = P.v3(W_ORG, k);
        ray.dir = P.v3(W_DIR, k);
        ray.seed.state = P.u64(W_SEED, k);
        ray.tp = P.half3(W_TP, k);
        const uint32_t bounces = P.u(W_TP + 1, k) >> 16;
        ray.numVolumeBounces = (int)(bounces & 0xffu);
        ray.numDiffuseBounces = (int)(bounces >> 8);
        ray.misWeight = P.f(W_MIS, k);
        ray.tMax = 1.f;
        Hit h;
        h.hit = !Iso || !(ctl & F_SURFHIT);
        h.t = P.f(W_HT, k);
        h.rgb = P.v3(W_HRGB, k);
        Random rnd = Random::derive(ray.seed, (uint64_t)hit_hash(h.t));
        EnvPick pick;
        if (p.hasEnv) {
          pick = env_pick_coords(p, rnd);
          const float4 t = tex2D(p.env, pick.sx, pick.sy);
          pick.radiance = p.env.scale * vec3(t.x, t.y, t.z);
        }
        const int accumID = L.accumIdStart + (int)P.u(W_PASS, k);
        if (!Batch && gen == 0 && (p.depth || p.primId || p.instId || p.objId))
          write_aux(p, (size_t)P.u(W_IY, k) * p.W + P.u(W_IX, k), accumID, h.t, h.hit ? 1 : 2);
        // a hit's own fragment is zero; the first generation's alpha is one
        if (gen == 0 && !(ctl & F_SPLIT)) {
          if (accumID == 0) P.setacc(k, make_float4(0.f, 0.f, 0.f, 1.f));
          else P.setf(W_ACC + 3, k, P.f(W_ACC + 3, k) + 1.f);
        }
        // setVolumeHit's P = obj_org + t * obj_dir (MCAccelerator.h:79), the
        // trace direction's zero components replaced as trace_begin does
        vec3 tdir = ray.dir;
        if (tdir.x == 0.f) tdir.x = 1e-6f;
        if (tdir.y == 0.f) tdir.y = 1e-6f;
        if (tdir.z == 0.f) tdir.z = 1e-6f;
        const vec3 hitP = ray.org + h.t * tdir;
        if (Iso && !h.hit) bounce_surface_hit(p, ray, P.half3(W_HN, k), h.t, hitP, gen, rnd, pick, so);
        else bounce_volume_hit(p, ray, h, hitP, gen, rnd, pick, so);
        shadow = so.shadowValid && so.shadow.tMax > 0.f;
        const bool alive = ray.tMax > 0.f;
        if (alive) {
          P.setv3(W_ORG, k, ray.org);
          P.setv3(W_DIR, k, ray.dir);
          P.setu64(W_SEED, k, ray.seed.state);
          P.sethalf3(W_TP, k, ray.tp, (uint32_t)ray.numVolumeBounces | ((uint32_t)ray.numDiffuseBounces << 8));
          P.setf(W_MIS, k, ray.misWeight);
        }
        ctl = (ctl & F_SPLIT) | (shadow ? F_SHADOW : 0u) | (alive ? F_ALIVE : 0u) | ((uint32_t)(gen + 1) << 8);
        if ((ctl & F_SPLIT) && shadow) P.setu(W_MASK, k, P.u(W_MASK, k) | (1u << gen));
      }
      // A split path's shadow ray is traced beside its bounce ray when a slot
      // is free for it (the log orders their fragments).
      const bool lone = (ctl & (F_SPLIT | F_SHADOW | F_ALIVE)) == (F_SPLIT | F_SHADOW | F_ALIVE) && k >= 0;
      const unsigned wants = __ballot_sync(FULL, lone);
      int home = k;  // the slot of the shadow ray
      if (wants) {
        int m;
        const int got = P.take(Q_FREE, __popc(wants), rot, m);
        const int r = __popc(wants & lt);
        const int slot = __shfl_sync(FULL, got, r);
        if (lone && r < m) {
          home = slot;
          P.setu(W_REC, home, P.u(W_REC, k));
          P.setu(W_PASS, home, P.u(W_PASS, k));
          if (Batch) P.setu(W_ITEM, home, P.u(W_ITEM, k));
          P.setu(W_CTL, home, (ctl & ~F_ALIVE) | F_LONE);
          ctl &= ~F_SHADOW;
        }
      }
      if (k >= 0) {
        if (shadow) {
          P.setv3(W_SORG, home, so.shadow.org);
          P.setv3(W_SDIR, home, so.shadow.dir);
          P.setf(W_STMAX, home, so.shadow.tMax);
          P.setu64(W_SSEED, home, so.shadow.seed.state);
          P.sethalf3(W_STP, home, so.shadow.tp);
          P.setf(W_SMIS, home, so.shadow.misWeight);
        }
        if (home != k) P.publish(Q_READY, home);
        int q = Q_READY;
        if (ctl & (F_SHADOW | F_ALIVE)) P.setu(W_CTL, k, ctl);
        else q = end_pass(Batch ? items[P.u(W_ITEM, k)] : p0, k, ctl);
        P.publish(q, k);
      }
    } else if (stage == S_START) {
      // ---- start passes (_generateRays) and shade misses ----
      // A new primary ray that misses the field's bounds is shaded at once,
      // and a warp most of whose paths end this way (background) goes on with
      // their next passes.  Free slots take new pixels.
      phase = 0;
      int n;
      int k = nStart ? P.take(Q_START, 32, rot, n) : (n = 0, -1);
      bool mine = k >= 0, fresh = false;
      int ix = 0, iy = 0, s = 0, gen = 0, item = 0;
      uint32_t split = 0u, rec = 0u, mask = 0u;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      vec3 dir(0.f), weight(0.f);  // weight: the path's throughput (later generations)
      float mis = 0.f;
      if (mine) {
        const uint32_t ctl = P.u(W_CTL, k);
        fresh = ctl & F_FRESH;
        split = ctl & F_SPLIT;
        ix = (int)P.u(W_IX, k);
        iy = (int)P.u(W_IY, k);
        s = (int)P.u(W_PASS, k);
        acc = P.acc(k);
        rec = P.u(W_REC, k);
        mask = P.u(W_MASK, k);
        if (Batch) item = (int)P.u(W_ITEM, k);
        if (!fresh) {
          gen = (int)((ctl >> 8) & 0xffu);
          dir = P.v3(W_DIR, k);
          weight = from_half(P.half3(W_TP, k));
          mis = P.f(W_MIS, k);
        }
      }
      if (n < 32 && !poolDone) {
        int m;
        const int got = P.take(Q_FREE, 32 - n, rot, m);
        const int slot = __shfl_sync(FULL, got, lane - n);
        if (lane >= n && lane < n + m) k = slot;
      }
      // the warp's tile, kept in shared memory between its visits here
      uint32_t *const own = P.queue(Q_COUNT) + 1 + 6 * warp;
      int tile = (int)own[0], tileTaken = (int)own[1], tileItem = (int)own[2], tilePass = (int)own[3];
      uint32_t tileRec = own[4];  // log record of a split tile's first pixel
      bool tileSplit = own[5] & 1u;
      while (true) {
        // pixels for the lanes that hold a free slot
        while (true) {
          const unsigned need = __ballot_sync(FULL, k >= 0 && !mine);
          if (!need || poolDone) break;
          if (tileTaken == 32) {
            int t = 0;
            if (lane == 0) t = atomicAdd(pool, 1);
            t = __shfl_sync(FULL, t, 0);
            if (t >= launch_tiles(L)) {
              poolDone = true;
              break;
            }
            const long long j = t - L.whole;
            tileTaken = 0;
            tilePass = 0;
            long long idx = t;
            tileSplit = j >= 0;
            if (tileSplit) {
              tileRec = (uint32_t)j * 32u;
              tilePass = (int)((uint32_t)j % (uint32_t)L.spp);
              idx = L.whole + (uint32_t)j / (uint32_t)L.spp;
            }
            if (Batch) {  // the item whose tiles idx falls in
              tileItem = tile_item_warp(tileStart, numItems, idx);
              idx -= tileStart[tileItem];
            }
            tile = inner_tile(Batch ? items[tileItem] : p0, (int)idx);
          }
          const RenderParams &tp = Batch ? items[tileItem] : p0;
          int tx, ty;
          tile_corner<Batch>(L, tp, tile, tx, ty);
          const int r = __popc(need & lt), take = min(__popc(need), 32 - tileTaken);
          if (k >= 0 && !mine && r < take) {
            const int at = tileTaken + r;
            const int px = tx + (at & 7), py = ty + (at >> 3);
            if (px < tp.W && py < tp.H) {
              mine = fresh = true;
              ix = px;
              iy = py;
              s = tilePass;
              split = tileSplit ? F_SPLIT : 0u;
              rec = tileRec + (uint32_t)at;
              mask = 0u;
              acc = L.accumIdStart == 0 || tileSplit ? make_float4(0.f, 0.f, 0.f, 0.f)
                                                     : tp.accum[(size_t)py * tp.W + px];
              item = tileItem;
            }
          }
          tileTaken += take;
        }
        const RenderParams &p = Batch ? items[item] : p0;
        bool missed = mine && !fresh;
        if (mine && fresh) {
          PathRay ray;
          gen = 0;
          generate_primary(p, ix, iy, L.accumIdStart + s, ray);
          vec3 tdir = ray.dir;
          if (tdir.x == 0.f) tdir.x = 1e-6f;
          if (tdir.y == 0.f) tdir.y = 1e-6f;
          if (tdir.z == 0.f) tdir.z = 1e-6f;
          float tLo = 0.f, tHi = ray.tMax;
          if (box_test(ray.org, tdir, tLo, tHi, p.F.boundsLo, p.F.boundsHi)) {
            P.setv3(W_ORG, k, ray.org);
            P.setv3(W_DIR, k, ray.dir);
            P.setu64(W_SEED, k, ray.seed.state);
            P.sethalf3(W_TP, k, ray.tp);
            P.setf(W_MIS, k, ray.misWeight);
            if (split) {
              P.setu(W_REC, k, rec);
              P.setu(W_MASK, k, 0u);
            } else {
              P.setacc(k, acc);
            }
            P.setu(W_PASS, k, (uint32_t)s);
            P.setu(W_IX, k, (uint32_t)ix);
            P.setu(W_IY, k, (uint32_t)iy);
            if (Batch) P.setu(W_ITEM, k, (uint32_t)item);
            P.setu(W_CTL, k, F_ALIVE | split);
            P.publish(Q_READY, k);
            mine = false;
            k = -1;
          } else {
            GBV_COUNT(cnt, rays);
            dir = ray.dir;
            missed = true;
          }
        }
        if (missed) {
          const int accumID = L.accumIdStart + s;
          if (!Batch && gen == 0 && (p.depth || p.primId || p.instId || p.objId))
            write_aux(p, (size_t)iy * p.W + ix, accumID, 1e30f, 0);
          vec3 frag;
          float alpha = 1.f;
          if (gen == 0) {
            const float4 m = primary_miss(p, iy, dir, accumID);
            frag = vec3(m.x, m.y, m.z);
            alpha = m.w;
          } else {
            vec3 env(p.ambient);
            if (p.hasEnv) {
              const float2 uv = env_miss_coords(p, dir);
              const float4 t = tex2D(p.env, uv.x, uv.y);
              env = p.env.scale * vec3(t.x, t.y, t.z);
            }
            frag = vmin(weight * env * mis, vec3(10.f * (float)(1 + accumID)));
          }
          if (split) {
            log_fragment(L, rec, gen, frag);
            log_end(L, rec, mask | (1u << gen) | (gen == 0 ? kLogMissed : 0u), alpha);
            mine = false;
          } else {
            if (gen == 0) add_miss(acc, make_float4(frag.x, frag.y, frag.z, alpha), accumID);
            else accum_add(acc, frag);
            if (++s == L.spp) {
              p.accum[(size_t)iy * p.W + ix] = acc;
              mine = false;
            }
          }
          fresh = true;
        }
        if (__popc(__ballot_sync(FULL, mine || (k >= 0 && !poolDone))) < kRepeatMin) break;
      }
      __syncwarp();
      if (lane == 0) {
        own[0] = (uint32_t)tile;
        own[1] = (uint32_t)tileTaken;
        own[2] = (uint32_t)tileItem;
        own[3] = (uint32_t)tilePass;
        own[4] = tileRec;
        own[5] = tileSplit ? 1u : 0u;
      }
      if (mine) {
        P.setacc(k, acc);
        P.setu(W_PASS, k, (uint32_t)s);
        P.setu(W_IX, k, (uint32_t)ix);
        P.setu(W_IY, k, (uint32_t)iy);
        if (Batch) P.setu(W_ITEM, k, (uint32_t)item);
        P.setu(W_CTL, k, F_FRESH);
      }
      if (k >= 0) P.publish(mine ? Q_START : Q_FREE, k);
    } else {
      // ---- the iso-surface's search, after the volume's trace ----
      phase = 2;
      int n;
      const int k = P.take(Q_ISO, 32, rot, n);
      if (k >= 0) {
        const RenderParams &p = p0;
        const uint32_t ctl = P.u(W_CTL, k);
        const bool shadow = ctl & F_SHADOW, volHit = ctl & F_VOLHIT;
        const int o = shadow ? W_SORG : W_ORG, sw = shadow ? W_SSEED : W_SEED;
        const vec3 org = P.v3(o, k), dir = P.v3(o + 3, k);
        const float tmax = shadow ? P.f(W_STMAX, k) : (ctl & 0xff00u) ? INF : 1e30f;
        float sT = 0.f;
        vec3h sN{0, 0, 0};
        bool hit;
        if (p.isoFirst) {
          // the surface's search, up to the volume's first collision
          hit = iso_trace_after<Store>(p, org, dir, tmax, volHit ? P.f(W_HT, k) : INF, P.u64(W_ISORNG, k),
                                       !shadow, sT, sN);
        } else {
          // the iso-surface after the volume, up to the volume's hit
          RNGSeed seed;
          seed.state = P.u64(sw, k);
          hit = iso_trace<Store>(p, org, dir, volHit ? P.f(W_HT, k) : tmax, seed, !shadow, sT, sN);
          P.setu64(sw, k, seed.state);
        }
        int q;
        if (shadow) {
          q = end_shadow(p, k, ctl, hit);
        } else {
          if (hit) {
            P.setf(W_HT, k, sT);
            P.sethalf3(W_HN, k, sN);
            P.setu(W_CTL, k, (ctl & ~kHitMask) | F_SURFHIT);
          }
          q = hit || volHit ? Q_HIT : Q_START;
        }
        P.publish(q, k);
      }
    }
    __syncwarp();
    if (Count && L.profile && lane == 0) cyc[phase] += (unsigned long long)(clock64() - c0);
  }
  if (Count && L.counters) {
    unsigned long long v[12] = {cnt.samples, cnt.mcs, cnt.rays, cnt.caps, cnt.cells, cyc[0], cyc[1], cyc[2],
                                simt[0], simt[1], simt[2], simt[3]};
    // (per-lane counts are 32-bit; a lane processes far fewer than 2^32 events)
#pragma unroll
    for (int k = 0; k < 12; k++) {
      unsigned long long x = v[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(FULL, x, o);
      if (lane == 0 && x) atomicAdd(L.counters + k, x);
    }
  }
}

// A lane's pixel of a warp tile; false past the frame's edge
template <bool Batch>
__device__ __forceinline__ bool tile_pixel(const RenderParams &L, const RenderParams &p, int tile, int lane, int &ix,
                                           int &iy) {
  tile_corner<Batch>(L, p, tile, ix, iy);
  ix += lane & 7;
  iy += lane >> 3;
  return ix < p.W && iy < p.H;
}
// What the frame kernel leaves of a frame: the outer tiles, whose rays see
// nothing of the field, and the sums of the split tiles' fragments.  A lane
// per pixel, a warp per tile, passes in order.  It is launched with the frame
// kernel (programmatic stream serialization): its blocks start on the SMs
// that run out of paths first and fill them with the outer tiles (taken from
// pool[1]) until the last path has ended; then they add up the log.
//
// As stages of the frame kernel the outer tiles took path slots, registers and
// instruction cache from the rest: 64 scenes of 8 passes 5.52 -> 5.20 ms, 1080p
// 512^3 of one pass 0.76 -> 0.70 ms without them there.  Taken one by one, the
// counter they are taken from bounds them (64 scenes of one pass 0.79 ms, in
// groups 0.73 ms).  The sums are bound by the log's reads, one round trip per
// kAhead passes (64 scenes of 8 passes: 5.14 -> 5.12 ms, 256^2 of 16 passes 0.142
// -> 0.138 ms from 4 passes at a time; 8 at a time the same).
constexpr int kFinishThreads = 256;
template <bool Batch>
static __global__ void __launch_bounds__(kFinishThreads)
    finish_kernel(const __grid_constant__ RenderParams L, const RenderParams *__restrict__ items,
                  const long long *__restrict__ tileStart, int numItems, int *__restrict__ pool, int group) {
  const int lane = threadIdx.x & 31;
  while (L.outer > 0) {
    int t = 0;
    if (lane == 0) t = atomicAdd(pool + 1, group);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= L.outer) break;
    for (const int end = (int)min((long long)t + group, L.outer); t < end; t++) {
      long long idx = t;
      int item = 0;
      if (Batch) {
        item = tile_item_warp(tileStart + numItems + 1, numItems, idx);
        idx -= tileStart[numItems + 1 + item];
      }
      const RenderParams &p = Batch ? items[item] : L;
      int ix, iy;
      const bool inside = tile_pixel<Batch>(L, p, outer_tile(p, (int)idx), lane, ix, iy);
      if (L.counters) {
        const int rays = __popc(__ballot_sync(0xffffffffu, inside));
        if (lane == 0) atomicAdd(L.counters + 2, (unsigned long long)rays * L.spp);
      }
      if (inside) {
        const size_t at = (size_t)iy * p.W + ix;
        float4 acc = L.accumIdStart == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : p.accum[at];
        for (int s = 0; s < L.spp; s++) {
          const int accumID = L.accumIdStart + s;
          PathRay ray;
          if (p.hasEnv) generate_primary(p, ix, iy, accumID, ray);
          if (!Batch && (p.depth || p.primId || p.instId || p.objId)) write_aux(p, at, accumID, 1e30f, 0);
          add_miss(acc, primary_miss(p, iy, ray.dir, accumID), accumID);
        }
        p.accum[at] = acc;
      }
      __syncwarp();
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the frame kernel is complete
  const long long warps = (long long)gridDim.x * (kFinishThreads / 32);
  for (long long k = ((long long)blockIdx.x * kFinishThreads + threadIdx.x) >> 5; k < L.split; k += warps) {
    const long long t = L.whole + k;
    const int item = Batch ? tile_item_warp(tileStart, numItems, t) : 0;
    const RenderParams &p = Batch ? items[item] : L;
    int ix, iy;
    if (!tile_pixel<Batch>(L, p, inner_tile(p, (int)(Batch ? t - tileStart[item] : t)), lane, ix, iy)) continue;
    float4 *out = p.accum + (size_t)iy * p.W + ix;
    float4 acc = L.accumIdStart == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *out;
    const int words = log_words(L.logHits);
    const uint32_t *r = L.log + ((size_t)k * L.spp * 32 + lane) * words;
    // kAhead records at a time, all their first words asked for at once (a
    // path's first fragment is the only one of most records; where it logged
    // none its words are not used)
    constexpr int kAhead = 4;
    for (int s0 = 0; s0 < L.spp; s0 += kAhead, r += (size_t)kAhead * 32 * words) {
      uint32_t head[kAhead][5];
#pragma unroll
      for (int a = 0; a < kAhead; a++)
#pragma unroll
        for (int w = 0; w < 5; w++) head[a][w] = s0 + a < L.spp ? r[(size_t)a * 32 * words + w] : 0u;
#pragma unroll
      for (int a = 0; a < kAhead; a++) {
        if (s0 + a >= L.spp) break;
        // (no bit past the record's fragments: a pass that a warp gave up on,
        // see idlePolls, has logged nothing)
        uint32_t mask = head[a][0] & (kLogMissed | ((1u << L.logHits) - 1u));
        const float alpha = __uint_as_float(head[a][1]);
        const vec3 first(__uint_as_float(head[a][2]), __uint_as_float(head[a][3]), __uint_as_float(head[a][4]));
        if (L.accumIdStart + s0 + a == 0) {
          acc = make_float4(0.f, 0.f, 0.f, alpha);
          if (mask & kLogMissed) {
            acc.x = first.x;
            acc.y = first.y;
            acc.z = first.z;
            continue;
          }
        } else if (alpha > 0.f) {
          acc.w += alpha;
        }
        if (mask & 1u) accum_add(acc, first);
        for (mask &= ~(kLogMissed | 1u); mask; mask &= mask - 1) {
          const float *g = reinterpret_cast<const float *>(r + (size_t)a * 32 * words + 2) + 3 * (__ffs(mask) - 1);
          accum_add(acc, vec3(g[0], g[1], g[2]));
        }
      }
    }
    *out = acc;
  }
}
// After the frame kernel of the same launch.
template <bool Batch>
inline gbv_status launch_finish(const RenderParams &L, const RenderParams *items, const long long *tileStart, int numItems,
                                int *pool, cudaStream_t stream) {
  if (L.outer + L.split == 0) return GBV_OK;
  int dev = 0, sms = 0;
  gbv_status st = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (st == GBV_OK) st = check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
  if (st != GBV_OK) return st;
  const int warps = kFinishThreads / 32;
  const long long tiles = L.outer > L.split ? L.outer : L.split, most = (long long)sms * 8;
  const long long blocks = (tiles + warps - 1) / warps;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(blocks < most ? blocks : most));
  cfg.blockDim = dim3(kFinishThreads);
  cfg.stream = stream;
  cudaLaunchAttribute serial;
  serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  serial.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &serial;
  cfg.numAttrs = 1;
  // outer tiles a warp takes at a time: a few turns for each warp of the GPU
  const long long turns = L.outer / (most * warps * 2);
  const int group = (int)(turns < 1 ? 1 : turns > 16 ? 16 : turns);
  return check_cuda(cudaLaunchKernelEx(&cfg, finish_kernel<Batch>, L, items, tileStart, numItems, pool, group),
                    "finish_kernel");
}

// Fragments a path of this world can log: one per hit (its shadow ray) or
// the miss that ends it.  A volume hit of the single-scatter build ends the
// path; with isotropic scattering every hit ends it or counts against
// maxVolumeBounces; else (a scatter of vanishing pdf leaves the ray alive and
// counts nothing) only the path depth (10) bounds the hits.
inline int path_hits(const RenderParams &p) {
  if (p.isoOn || (p.multi && !(fabsf(p.aniso) < 1e-3f))) return 11;
  if (!p.multi || !p.volMS) return 1;
  return p.maxVB < 0 ? 1 : p.maxVB < 10 ? p.maxVB + 1 : 11;
}
// Log memory of a launch (of a batch) at most.  512^3, 1080p, 64 passes: not
// in parts, a log for a tenth of the inner tiles 40.5 ms; in parts with 256 MB
// 32.7 ms (31.0 with the 96-register budget), 512 MB 32.4 (30.5), 1 GB 31.5
// (29.5), 3 GB 31.1 (29.2).
constexpr size_t kLogBytes = (size_t)512 << 20, kBatchLogBytes = (size_t)256 << 20;
constexpr int kBatchLogPasses = 16;
// The rectangle of warp tiles the field's bounds project to (p.rx, ...);
// returns the number of tiles in it.  A tile outside it provably sees nothing
// of the field: the bounds' projection is the hull of its corners'
// projections, taken here in double, and the tile's pixels keep a margin of
// two pixels from the hull's rectangle, at least 2e-5 rad where a pixel spans
// 1e-5 rad or more.  A ray's float direction is within 1e-6 rad of its exact
// one, and rotating a ray by d changes the ratio of two slab distances by
// sqrt(2) d or more, against a rounding error of 1e-6 in the float slab test.
// Where that does not hold (a corner behind or beside the camera, finer
// pixels, values that are not finite) the rectangle is the whole frame; where
// every corner lies behind the plane through the camera, by 1e-3 rad or more,
// no ray of the frame, all of which lead ahead of it, sees the field (256^3,
// 1080p, 4 passes, env map: 107 us, 364 as a frame of inner tiles).  A
// launch of a rank's share of the tiles has no rectangle: rw = 0, every tile
// is an inner one.
inline long long plan_rect(RenderParams &p) {
  const long long tx = ((long long)p.W + 7) >> 3, ty = ((long long)p.H + 3) >> 2;
  p.rx = p.ry = p.rw = p.rh = 0;
  if (p.numRanks > 1) return warp_tile_count(p);
  struct D3 { double x, y, z; };
  auto dotd = [](D3 a, vec3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; };
  const double aspect = (double)p.W / p.H;
  const D3 d00{p.dir00.x, p.dir00.y, p.dir00.z};
  const double dd = dotd(d00, p.dir00);  // dir00 is 1 / (2 tan(fovy / 2)) long, du and dv are unit vectors
  // the smallest angle a pixel spans, at the frame's corners
  const double corner2 = dd + .25 * aspect * aspect + .25;
  bool whole = !(sqrt(dd) / corner2 / p.H > 1e-5);
  double x0 = 1e30, x1 = -1e30, y0 = 1e30, y1 = -1e30;
  bool behind = !whole;  // every corner lies behind the camera
  for (int k = 0; k < 8; k++) {
    const D3 d{(double)(k & 1 ? p.F.boundsHi.x : p.F.boundsLo.x) - p.lens00.x,
               (double)(k & 2 ? p.F.boundsHi.y : p.F.boundsLo.y) - p.lens00.y,
               (double)(k & 4 ? p.F.boundsHi.z : p.F.boundsLo.z) - p.lens00.z};
    const double t = dotd(d, p.dir00) / dd, len = sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
    whole = whole || !(t * sqrt(dd) > 1e-3 * len);
    behind = behind && t * sqrt(dd) < -1e-3 * len;
    const double x = (.5 + dotd(d, p.du) / t / aspect) * p.W, y = (.5 + dotd(d, p.dv) / t) * p.H;
    whole = whole || !(fabs(x) < 1e9 && fabs(y) < 1e9);
    x0 = x < x0 ? x : x0;
    x1 = x > x1 ? x : x1;
    y0 = y < y0 ? y : y0;
    y1 = y > y1 ? y : y1;
  }
  if (behind) {  // nothing of the field is seen: one inner tile, so that rw > 0
    p.rw = p.rh = 1;
    return 1;
  }
  if (whole) {
    p.rw = (int)tx;
    p.rh = (int)ty;
    return tx * ty;
  }
  // tiles that overlap [x0 - 2, x1 + 2] x [y0 - 2, y1 + 2]
  auto tiles = [](double lo, double hi, int pixels, int edge, int &first, int &count) {
    const long long a = clampv((long long)floor(lo - 2.), 0ll, (long long)pixels) / edge;
    const long long b = (clampv((long long)ceil(hi + 2.), 0ll, (long long)pixels) + edge - 1) / edge;
    first = (int)a;
    count = (int)(b - a);
  };
  tiles(x0, x1, p.W, 8, p.rx, p.rw);
  tiles(y0, y1, p.H, 4, p.ry, p.rh);
  if (p.rw <= 0 || p.rh <= 0) {  // the frame sees nothing of the field: one inner tile, so that rw > 0
    p.rx = p.ry = 0;
    p.rw = p.rh = 1;
  }
  return (long long)p.rw * p.rh;
}

// Passes a launch renders at most: a frame of more passes than the log holds
// for all of its inner tiles is rendered in parts that it does hold, as long as
// a part has kPartPasses passes or more (the frame continues from the
// accumulation buffer as progressive frames do).
constexpr int kPartPasses = 4;
inline int part_passes(const RenderParams &p, long long inner, int hits) {
  const long long most = (long long)(kLogBytes / ((size_t)inner * 32 * log_words(hits) * sizeof(uint32_t)));
  if (p.depth || p.primId || p.instId || p.objId || most < kPartPasses || p.spp <= most) return p.spp;
  const long long parts = (p.spp + most - 1) / most;
  return (int)((p.spp + parts - 1) / parts);
}

// What a launch over `inner` + `outer` tiles splits: as many of the last
// inner tiles as `room` bytes of log hold.  Returns the log's bytes.
inline size_t plan_split(RenderParams &p, long long inner, long long outer, int hits, size_t room) {
  const size_t perTile = (size_t)p.spp * 32 * log_words(hits) * sizeof(uint32_t);
  long long split = (long long)(room / perTile);
  if (split > inner) split = inner;
  // a pixel's depth channel is the running minimum of its passes in order
  if (p.depth || p.primId || p.instId || p.objId) split = 0;
  if (split * 16 < inner || inner + outer + split * p.spp >= (1ll << 31) - (1ll << 24)) split = 0;
  p.whole = inner - split;
  p.split = split;
  p.outer = outer;
  p.logHits = hits;
  p.log = nullptr;
  return (size_t)split * perTile;
}

// 32-bit words of dynamic shared memory the staged tables take
inline size_t staged_words(const RenderParams &p) {
  long long end = p.maskWords;
  if (p.cdfYOff >= 0) end = end > p.cdfYOff + p.env.H ? end : p.cdfYOff + p.env.H;
  if (p.pivOff >= 0) end = end > p.pivOff + (long long)p.env.H * p.pivPerRow ? end : p.pivOff + (long long)p.env.H * p.pivPerRow;
  if (p.rowOff >= 0) end = end > p.rowOff + 2LL * p.env.H ? end : p.rowOff + 2LL * p.env.H;
  return (size_t)end;
}

using RenderKernelFn = void (*)(const RenderParams, const RenderParams *, const long long *, int, int *);

// The words plan_staging places at most (64 KB of tables, the row terms on top
// where the bitmask fills them), and the shared memory a launch may ask for:
// the kernel's limit is always set to this, whatever one launch needs, since
// another host thread may set it for its own scene before this one's launch.
constexpr int kMaxStagedWords = 16 * 1024 + 2 * 1024 + 4;
template <bool Iso> constexpr size_t kMaxDynamicSmem = (kMaxStagedWords + PathPool<Iso>::kStride) * sizeof(uint32_t);
static_assert(kMaxDynamicSmem<true> + 1024 <= 227 * 1024, "a block's tables and path pool");

// Places the block's path pool behind the `staged` words of tables; returns
// the block's dynamic shared memory in bytes.
template <bool Iso> inline size_t plan_pool(RenderParams &p, size_t staged) {
  p.poolOff = (int)((staged + 3) & ~(size_t)3);
  return ((size_t)p.poolOff + PathPool<Iso>::kStride) * sizeof(uint32_t);
}

// Persistent grid of a launch over `tiles` warp tiles: one block per SM, and
// the path slots each block uses: no more than its share of the pixels, so
// that no block holds pixels that another would be idle without.
inline gbv_status plan_grid(RenderParams &p, RenderKernelFn kernel, size_t smemLimit, long long tiles,
                            long long &blocks) {
  int dev = 0, sms = 0;
  gbv_status st = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (st == GBV_OK) st = check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
  if (st == GBV_OK)
    st = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemLimit),
                    "render_kernel: shared-memory size");
  if (st != GBV_OK) return st;
  blocks = tiles < sms ? tiles : sms;
  if (blocks < 1) blocks = 1;
  const long long share = (p.split ? 64 : 32) * ((tiles + blocks - 1) / blocks);
  p.slots = (int)(share < kSlots ? share : kSlots);
  return GBV_OK;
}

// The one-scene render kernels of a launch: with and without event
// counting, for a volume-only world or (with the 128-register budget) one
// with an iso-surface.
template <class Store, int Budget>
inline void render_kernels(const RenderParams &p, RenderKernelFn &counting, RenderKernelFn &plain) {
  counting = render_kernel<Store, Budget, false, true>;
  plain = render_kernel<Store, Budget, false, false>;
  if constexpr (Budget == 4) {
    if (p.isoOn) {
      counting = render_kernel<Store, 4, false, true, true>;
      plain = render_kernel<Store, 4, false, false, true>;
    }
  }
}

template <class Store, int Budget>
inline gbv_status launch_render_t(const RenderParams &p, const Store &store, cudaStream_t stream) {
  RenderKernelFn kCount, kPlain;
  render_kernels<Store, Budget>(p, kCount, kPlain);
  const RenderKernelFn kernel = p.counters ? kCount : kPlain;
  RenderParams q = p;
  const size_t smem = p.isoOn ? plan_pool<true>(q, staged_words(p)) : plan_pool<false>(q, staged_words(p));
  const size_t limit = p.isoOn ? kMaxDynamicSmem<true> : kMaxDynamicSmem<false>;
  long long blocks = 0;
  gbv_status st = GBV_OK;
  // the tile pool counter, the majorant bitmask and the log live in
  // stream-ordered scratch memory (the mask at a 256-byte offset: 16-byte
  // aligned for the bulk copy)
  int *pool = nullptr;
  const long long inner = plan_rect(q), outer = warp_tile_count(p) - inner;
  const int hits = path_hits(p), most = part_passes(p, inner, hits);
  q.spp = most;
  size_t logBytes = plan_split(q, inner, outer, hits, kLogBytes);
  const size_t maskBytes = ((size_t)p.maskWords * 4 + 255) & ~(size_t)255;
  if (logBytes && scratch_alloc((void **)&pool, 256 + maskBytes + logBytes, stream) != cudaSuccess) {
    cudaGetLastError();  // no room for the log: no tile is split
    logBytes = 0;
  }
  if (!logBytes) st = check_cuda(scratch_alloc((void **)&pool, 256 + maskBytes, stream), "tile pool scratch");
  if (st != GBV_OK) return st;
  if (p.maskWords > 0 && p.maskSrc == nullptr && p.maskMode == 0) {
    uint32_t *mask = reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(pool) + 256);
    const int nmc = p.G.M[0] * p.G.M[1] * p.G.M[2];
    majorant_mask_kernel<<<(unsigned)((p.maskWords + 7) / 8), 256, 0, stream>>>(p.G.maj, nmc, p.maskWords, mask);
    st = check_launch("majorant_mask_kernel");
    q.maskSrc = mask;
  }
  const int step = logBytes ? most : p.spp;
  for (int done = 0; st == GBV_OK && done < p.spp; done += step) {
    q.accumIdStart = p.accumIdStart + done;
    q.spp = p.spp - done < step ? p.spp - done : step;
    if (plan_split(q, inner, outer, logBytes ? hits : 1, logBytes ? kLogBytes : 0))
      q.log = reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(pool) + 256 + maskBytes);
    st = plan_grid(q, kernel, limit, launch_tiles(q), blocks);
    if (st == GBV_OK)
      st = check_cuda(cudaMemsetAsync(pool, 0, 2 * sizeof(int), stream), "render_kernel: clearing the tile pool");
    if (st == GBV_OK) {
      kernel<<<(unsigned)blocks, block_threads(Budget), smem, stream>>>(q, nullptr, nullptr, 0, pool);
      st = check_launch("render_kernel");
    }
    if (st == GBV_OK) st = launch_finish<false>(q, nullptr, nullptr, 0, pool, stream);
  }
  const gbv_status fst = check_cuda(cudaFreeAsync(pool, stream), "cudaFreeAsync(tile pool)");
  return st != GBV_OK ? st : fst;
}

// Launch settings resolved from a gbv_render_config (gbv_render_ex): the
// register budget and the shared-memory staging mode.  The traversal settings
// (skip, threshold) and the profile switch travel in RenderParams; skip is here
// too, to tell a setting from the default.
struct LaunchChoice {
  int occ = 0;   // 0: default_budget
  int skip = 0;  // 0: the default (kSkipDefault, or kFilledSkip with default_budget)
  int stage = GBV_STAGE_DEFAULT;
  int mode = GBV_RENDER_PERSISTENT;
};

// Shared-memory staging (same results either way).  GBV_STAGE_DEFAULT: the
// bitmask of non-zero majorants, one bit per macrocell, when it takes at
// most 8 KB per block (64 Ki macrocells; 4 KB for the 32^3 grid of the 512^3
// frame): the empty-cell test of the traversal becomes a shared-memory load
// (measured +1.8%); with an env map of at most 1024 rows also the row terms
// of its pdf (8 bytes a row).  GBV_STAGE_ALL also stages the env-map cdf_y
// and the per-row pivots of cdf_x (up to 64 KB per block; measured slower:
// the shared memory comes out of L1, which spills and CDF loads use).
// GBV_STAGE_NONE stages nothing.
inline void plan_staging(RenderParams &p, int stage) {
  const long long nmc = (long long)p.G.M[0] * p.G.M[1] * p.G.M[2];
  const bool any = stage != GBV_STAGE_NONE, all = stage == GBV_STAGE_ALL;
  p.maskMode = stage == GBV_STAGE_BALLOT ? 1 : 0;
  const int budget = (all ? 64 : 8) * 1024 / 4;
  int used = 0;
  p.maskWords = 0;
  p.cdfYOff = p.pivOff = p.rowOff = -1;
  p.pivPerRow = 0;
  p.maskSrc = nullptr;
  if (any && nmc > 0 && p.hasVolume && (((nmc + 31) / 32 + 3) & ~3ll) <= budget) {
    p.maskWords = (int)(((nmc + 31) / 32 + 3) & ~3ll);  // whole 16-byte units (one bulk copy)
    used = p.maskWords;
  }
  if (any && p.hasEnv && p.env.H >= 1 && p.env.H <= 1024) {
    used = (used + 1) & ~1;  // float2 entries
    p.rowOff = used;
    used += 2 * p.env.H;
  }
  if (all && p.hasEnv && p.env.W >= 2) {
    if (used + p.env.H <= budget) {
      p.cdfYOff = used;
      used += p.env.H;
    }
    const int per = (p.env.W - 1 + 31) / 32;  // segments holding entries 0..W-2
    if ((long long)used + (long long)p.env.H * per <= budget) {
      p.pivOff = used;
      p.pivPerRow = per;
      used += p.env.H * per;
    }
  }
}

// The register budget of a launch that asks for none: 20 warps of 96
// registers for frames long enough to be bound by their middle (kManyPaths or
// more paths that may see the field: 512^3 1080p 64 passes 32.4 -> 30.5 ms,
// U8 1080p 32 passes 3.98 -> 3.73; 256^3 2560x1440 4 passes 3.77 -> 3.71), 16
// of 128 for shorter ones, whose end waits for single paths (256^3 720p 1 pass
// 0.50 ms, 0.60 with 20 warps; 853x479 8 passes 0.35, 0.40), for NanoVDB grids
// (8.8 ms, 9.5) and iso-surfaces.
//
// Long single-scatter frames that the field fills -- a camera inside it, or one
// that sees nothing but the field -- are rays through all of it, alike from
// pixel to pixel, which a lane a pixel traced faster: 24 warps of 80 registers
// and longer seeks give most of that back.  256^3 and U8 512^3 from inside,
// 1080p, 4 passes: a lane a pixel 4.98 and 5.83 ms, 20 warps and 4 rounds 5.26
// and 6.25, 24 and 4 5.14 and 6.08, 24 and kFilledSkip 5.13 and 5.78 (a frame of
// 0.05 degrees: 4.97, 5.55, 5.38, 5.25).
constexpr long long kManyPaths = 4ll << 20;
constexpr int kFilledSkip = 8;
template <class Store> inline int default_budget(RenderParams p, bool &filled) {
  filled = false;
  if (std::is_same<Store, StoreNanoVDB>::value || p.isoOn) return 4;
  const long long inner = plan_rect(p);
  if (inner * 32 * p.spp < kManyPaths) return 4;
  filled = !p.multi && p.numRanks == 1 && inner == warp_tile_count(p);
  return filled ? 6 : 5;
}

template <class Store>
inline gbv_status launch_render(RenderParams p, const Store &store, cudaStream_t stream, const LaunchChoice &lc) {
  plan_staging(p, lc.stage);
  if (!p.counters) p.profile = 0;
  bool filled = false;
  const int budget = p.isoOn ? 4 : lc.occ ? lc.occ : default_budget<Store>(p, filled);
  if (filled && !lc.skip) p.skip = kFilledSkip;
  if (budget <= 4) return launch_render_t<Store, 4>(p, store, stream);
  if (budget >= 6) return launch_render_t<Store, 6>(p, store, stream);
  return launch_render_t<Store, 5>(p, store, stream);
}

template <class Store>
inline gbv_status launch_render_noalloc(RenderParams p, const Store &store, cudaStream_t stream, int *pool) {
  // fixed launch settings (results do not depend on them): the 128-register
  // budget, the default traversal settings, no shared-memory staging
  p.skip = kSkipDefault;
  p.threshold = kThresholdDefault;
  p.idlePolls = kIdlePolls;
  p.maskWords = 0;
  p.cdfYOff = p.pivOff = p.rowOff = -1;
  p.pivPerRow = 0;
  p.profile = 0;
  // no tile is split: a log would be an allocation
  const long long inner = plan_rect(p);
  plan_split(p, inner, warp_tile_count(p) - inner, 1, 0);
  RenderKernelFn kCount, kPlain;
  render_kernels<Store, 4>(p, kCount, kPlain);
  const RenderKernelFn kernel = p.counters ? kCount : kPlain;
  const size_t smem = p.isoOn ? plan_pool<true>(p, 0) : plan_pool<false>(p, 0);
  long long blocks = 0;
  gbv_status st = plan_grid(p, kernel, p.isoOn ? kMaxDynamicSmem<true> : kMaxDynamicSmem<false>, launch_tiles(p),
                            blocks);
  if (st != GBV_OK) return st;
  st = check_cuda(cudaMemsetAsync(pool, 0, 2 * sizeof(int), stream), "gbv_render_noalloc: clearing the tile pool");
  if (st != GBV_OK) return st;
  kernel<<<(unsigned)blocks, block_threads(4), smem, stream>>>(p, nullptr, nullptr, 0, pool);
  st = check_launch("render_kernel (noalloc)");
  return st != GBV_OK ? st : launch_finish<false>(p, nullptr, nullptr, 0, pool, stream);
}

}  // namespace gbv

struct gbv_batch {
  int count;
  int format, layout;
  gbv::RenderParams *d_items;  // device copy of the per-item parameters
  long long *d_tileStart;      // prefix sums of the items' inner 8x4 tiles, then of their outer ones
  int *d_pool;                 // tile-pool counter
  long long innerTiles, outerTiles;
  int occ, threshold, skip;
  int device;
  int hits;          // most fragments a path of any item can log
  uint32_t *d_log;   // log of the split tiles (null: none are split)
  size_t logBytes;
};

namespace gbv {

template <class Store, int Budget>
inline gbv_status batch_launch_t(const gbv_batch *b, RenderParams L, cudaStream_t stream) {
  const RenderKernelFn kernel = L.counters ? render_kernel<Store, Budget, true, true>
                                           : render_kernel<Store, Budget, true, false>;
  const size_t smem = plan_pool<false>(L, 0);
  long long blocks = 0;
  // One pass each has no passes to split, and many scenes' pixels fill the GPU
  // by themselves: 64 scenes 0.82 -> 0.80 ms without the log
  const size_t room = L.spp > 1 ? b->logBytes : 0;
  if (plan_split(L, b->innerTiles, b->outerTiles, b->hits, room)) L.log = b->d_log;
  gbv_status st = plan_grid(L, kernel, kMaxDynamicSmem<false>, launch_tiles(L), blocks);
  if (st == GBV_OK) st = check_cuda(cudaMemsetAsync(b->d_pool, 0, 2 * sizeof(int), stream), "gbv_batch_render: pool");
  if (st != GBV_OK) return st;
  kernel<<<(unsigned)blocks, block_threads(Budget), smem, stream>>>(L, b->d_items, b->d_tileStart, b->count, b->d_pool);
  st = check_launch("render_kernel (batch)");
  if (st == GBV_OK) st = launch_finish<true>(L, b->d_items, b->d_tileStart, b->count, b->d_pool, stream);
  return st;
}
template <class Store>
inline gbv_status batch_launch(const gbv_batch *b, const RenderParams &L, cudaStream_t stream) {
  switch (b->occ) {
    case 4: return batch_launch_t<Store, 4>(b, L, stream);
    case 6: return batch_launch_t<Store, 6>(b, L, stream);
    default: return batch_launch_t<Store, 5>(b, L, stream);
  }
}

#define GBV_DECLARE_STORE_LAUNCHERS(NAME)                                                        \
  gbv_status render_launch_##NAME(const RenderParams &p, cudaStream_t s, const LaunchChoice &lc); \
  gbv_status render_launch_noalloc_##NAME(const RenderParams &p, cudaStream_t s, int *pool);    \
  gbv_status batch_launch_##NAME(const gbv_batch *b, const RenderParams &L, cudaStream_t s);

GBV_DECLARE_STORE_LAUNCHERS(linear)
GBV_DECLARE_STORE_LAUNCHERS(f32)
GBV_DECLARE_STORE_LAUNCHERS(f16)
GBV_DECLARE_STORE_LAUNCHERS(bf16)
GBV_DECLARE_STORE_LAUNCHERS(u8)
GBV_DECLARE_STORE_LAUNCHERS(nvdb)

}  // namespace gbv

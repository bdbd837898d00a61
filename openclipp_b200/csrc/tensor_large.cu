// Tensor-core ImageProximity for templates larger than 64 x 64.
//
// The reference serves large templates with its FFT path
// (C++/programs/ImageProximityFFT.cpp:112-210: an FFT correlation plus the
// window statistics of cl-files/ImageProximityFFT.cl:55-147 from a
// SqrIntegral). Here the product term is split over template tiles of at
// most 64 x 64, with the tile's offset folded into the window anchor. All tiles
// run in one launch of the tcgen05 kernel (groups of them where their maps would
// take more than kMapBytes), each writing a map of its own: FP32 sums, or int32
// (i8 MMA, exact). The scoring pass adds the tiles' sums in FP64, in tile order,
// and forms the measure from them, the window energy (the row energies of
// row_energy.cu summed in FP64 over th rows, by blocks of 16 output rows) and
// the template energy, with the same formulas as the one-launch kernel's
// epilogue: U8 results are bit-identical to the plain path's, F32 and U16
// within its split-BF16 error.
//
// One launch a tile, adding to an F64 map, gave each launch bands of 86 rows
// with 63 rows of ramp (2048 x 1536, 200 x 120: 8 tiles, 144 CTAs a launch) and
// 16 bytes of map traffic per output and tile. All tiles at once take bands of
// 768 rows, and 8 bytes. CrossCorr_Norm of that image and template: 887 us
// with a launch a tile, 499 so.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "host.h"
#include "internal.h"
#include "row_energy.h"
#include "tensor.h"

namespace ocipb {
namespace {

constexpr size_t kMapBytes = size_t(256) << 20;  // maps of the tiles of one launch

// Template energy sum T^2 per channel, FP64 (exact for integer templates): one
// block of 32 warps per channel, a warp per template row.
template <typename ET>
__global__ void __launch_bounds__(1024)
    template_energy_f64_kernel(const char* tmpl, size_t pitch, int tw, int th, int nch, double* out) {
  const int c = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double e = 0.0;
  for (int h = warp; h < th; h += 32) {
    const ET* row = reinterpret_cast<const ET*>(tmpl + (size_t)h * pitch) + c;
    for (int w0 = lane; w0 < tw; w0 += 256) {
      ET v[8];  // in flight together
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = w0 + 32 * j < tw ? __ldg(row + (size_t)(w0 + 32 * j) * nch) : ET(0);
#pragma unroll
      for (int j = 0; j < 8; ++j) e = fma((double)v[j], (double)v[j], e);
    }
  }
  __shared__ double part[32];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) e += __shfl_xor_sync(0xffffffffu, e, d);
  if (lane == 0) part[warp] = e;
  __syncthreads();
  if (warp == 0) {
    e = part[lane];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) e += __shfl_xor_sync(0xffffffffu, e, d);
    if (lane == 0) out[c] = e;
  }
}

// The tiles' maps: FP32 or int32 sums, tile i and channel c at
// maps + (i nch + c) * plane; and, with more tiles than fit, the FP64 sums of the
// groups before (one plane per channel).
struct TileMaps {
  const char* maps;
  size_t pitch, plane;
  int n;
  double* before;   // null: none
  size_t before_pitch, before_plane;  // bytes
};

constexpr int kCols = 4;         // columns of a thread (16-byte loads)
constexpr int kGroups = 16;      // rows of a block (one a thread), 128 columns wide
constexpr int kBlockCols = 32 * kCols;

template <typename RT>
__device__ __forceinline__ void load4(const char* p, RT (&v)[kCols]) {
  const uint4 q = __ldcs(reinterpret_cast<const uint4*>(p));
  memcpy(v, &q, sizeof(v));
}

// The sums of kCols columns from x of one row, tile by tile in order; the loads of
// eight tiles are in flight together. Columns past the last read the rows'
// pitch (a multiple of 32 values).
template <typename RT>
__device__ __forceinline__ void tile_sums(const TileMaps& t, int nch, int c, int y, int x,
                                          double (&s)[kCols]) {
#pragma unroll
  for (int k = 0; k < kCols; ++k) s[k] = 0.0;
  if (t.before) {
    const double* b = reinterpret_cast<const double*>(reinterpret_cast<const char*>(t.before) +
                                                      c * t.before_plane +
                                                      (size_t)y * t.before_pitch) + x;
#pragma unroll
    for (int k = 0; k < kCols; ++k) s[k] = b[k];
  }
  const char* p = t.maps + c * t.plane + (size_t)y * t.pitch + (size_t)x * 4;
  const size_t step = nch * t.plane;
  for (int i0 = 0; i0 < t.n; i0 += 8, p += 8 * step) {
    RT v[8][kCols];
    if (t.n - i0 >= 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) load4<RT>(p + i * step, v[i]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k < kCols; ++k) s[k] += static_cast<double>(v[i][k]);
    } else {
#pragma unroll
      for (int i = 0; i < 7; ++i)
        if (i < t.n - i0) load4<RT>(p + i * step, v[i]);
#pragma unroll
      for (int i = 0; i < 7; ++i)
        if (i < t.n - i0) {
#pragma unroll
          for (int k = 0; k < kCols; ++k) s[k] += static_cast<double>(v[i][k]);
        }
    }
  }
}

// FP64 sums of a group of tiles that is not the last one.
template <typename RT>
__global__ void __launch_bounds__(32 * kGroups)
    tile_sum_kernel(const TileMaps t, int W, int H, int nch, double* out, size_t pitch, size_t plane) {
  const int x = blockIdx.x * kBlockCols + threadIdx.x * kCols;
  const int y = blockIdx.y * kGroups + threadIdx.y;
  if (x >= W || y >= H) return;
  double s[kCols];
  tile_sums<RT>(t, nch, blockIdx.z, y, x, s);
  double* o = reinterpret_cast<double*>(reinterpret_cast<char*>(out) + blockIdx.z * plane +
                                        (size_t)y * pitch) + x;  // (row pitch: as the maps')
#pragma unroll
  for (int k = 0; k < kCols; ++k) o[k] = s[k];
}

struct ScoreParams {
  TileMaps c;           // product sums
  const char* rmap;     // row energies (int32 for U8, FP32 otherwise), one plane per channel
  size_t r_pitch, r_plane;
  const double* et;     // template energy per channel
  char* dst;
  size_t dst_pitch;
  int dst_f64;
  int W, H, nch;
  int th, ay;
  int measure;
  int u8_float;         // U8 _Norm in float arithmetic (the plain path's float sums are exact)
};

// A block takes 128 columns x 16 output rows of a channel, a thread 4 columns of a
// row. The window energy of the block's first row is a sum of th row energies,
// a sixteenth of them a thread; the rows below it differ by the row energies that
// enter and leave, prefix-summed down the column (FP64, exact for U8). Threads
// that walked down single columns with a running sum, 4-byte loads a row apart, took
// 90 us for 2048 x 1536 with 8 tiles; this takes 35.
template <bool SPLIT>
__global__ void __launch_bounds__(32 * kGroups) large_score_kernel(const ScoreParams p) {
  typedef typename std::conditional<SPLIT, float, int>::type RT;
  __shared__ __align__(16) double part[kGroups][kBlockCols], step[kGroups][kBlockCols];
  const int c = blockIdx.z, g = threadIdx.y, xs = threadIdx.x * kCols;
  const int x0 = blockIdx.x * kBlockCols + xs;
  const int yb = blockIdx.y * kGroups, y = yb + g;
  const bool in_x = x0 < p.W, in = in_x && y < p.H;
  double cc4[kCols] = {}, e4[kCols] = {};
  if (in) tile_sums<RT>(p.c, p.nch, c, y, x0, cc4);
  const bool need_e = p.measure != kCrossCorr;
  const double et = p.et[c];
  if (need_e) {
    const char* rplane = p.rmap + c * p.r_plane + (size_t)x0 * 4;
    auto r_at = [&](int r, RT (&v)[kCols]) {
      if (in_x && r >= 0 && r < p.H) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(rplane + (size_t)r * p.r_pitch));
        memcpy(v, &q, sizeof(v));
      } else {
#pragma unroll
        for (int k = 0; k < kCols; ++k) v[k] = RT(0);
      }
    };
    // Rows of the first window: first + g, first + g + 16, ...
    const int first = yb - p.ay;
    for (int r0 = g; r0 < p.th; r0 += 4 * kGroups) {
      RT v[4][kCols];  // in flight together
#pragma unroll
      for (int i = 0; i < 4; ++i) r_at(r0 + i * kGroups < p.th ? first + r0 + i * kGroups : -1, v[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < kCols; ++k) e4[k] += static_cast<double>(v[i][k]);
    }
    // Change of the window energy from row y - 1 to row y (none into row yb).
    RT rin[kCols], rout[kCols];
    r_at(g > 0 ? y - p.ay + p.th - 1 : -1, rin);
    r_at(g > 0 ? y - p.ay - 1 : -1, rout);
#pragma unroll
    for (int k = 0; k < kCols; ++k) {
      part[g][xs + k] = e4[k];
      step[g][xs + k] = static_cast<double>(rin[k]) - static_cast<double>(rout[k]);
    }
    __syncthreads();
    // A thread per column (adjacent ones: no bank conflicts) turns the steps into
    // the rows' window energies.
    const int j = threadIdx.y * 32 + threadIdx.x;
    if (j < kBlockCols) {
      double e = 0.0, d[kGroups];
#pragma unroll
      for (int i = 0; i < kGroups; ++i) d[i] = step[i][j];
#pragma unroll
      for (int i = 0; i < kGroups; ++i) e += part[i][j];
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        e += d[i];  // d[0] is 0
        step[i][j] = e;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kCols; ++k) e4[k] = step[g][xs + k];
  }
  if (!in) return;
#pragma unroll
  for (int u = 0; u < kCols; ++u) {
    const int x = x0 + u;
    if (x >= p.W) break;
    const double cc = cc4[u], e = e4[u];
    double v;
    float vf;
    if (SPLIT) {
      const double num = (p.measure == kCrossCorr || p.measure == kCrossCorrNorm)
                             ? cc
                             : e - 2.0 * cc + et;
      v = (p.measure == kCrossCorr || p.measure == kSqrDistance) ? num : num * rsqrt(e * et);
      vf = (float)v;
    } else {
      // Exact integers in FP64; the plain path's float or double formulas.
      const double num = (p.measure == kCrossCorr || p.measure == kCrossCorrNorm)
                             ? cc
                             : e - 2.0 * cc + et;
      if (p.measure == kCrossCorr || p.measure == kSqrDistance) {
        v = num;
        vf = (float)num;
      } else if (p.u8_float) {
        vf = __fdiv_rn((float)num, __fsqrt_rn(__fmul_rn((float)e, (float)et)));
        v = vf;
      } else {
        v = __ddiv_rn(num, __dsqrt_rn(__dmul_rn(e, et)));
        vf = (float)v;
      }
    }
    char* orow = p.dst + (size_t)y * p.dst_pitch;
    if (p.dst_f64)
      reinterpret_cast<double*>(orow)[(size_t)x * p.nch + c] = v;
    else
      reinterpret_cast<float*>(orow)[(size_t)x * p.nch + c] = vf;
  }
}

}  // namespace

cudaError_t launch_proximity_tensor_large(Context& ctx, Measure m, const DevImage& src,
                                          const DevImage& tmpl, const DevImage& dst) {
  const int tw = tmpl.width, th = tmpl.height, nch = src.nch;
  const int ax = tw / 2, ay = th / 2;
  const int es = type_bytes(tmpl.type);
  const TensorPlanes planes = tensor_source_planes(ctx, src);
  // Tiles of at most 64 x 64, balanced: rows [i th / ntr, (i + 1) th / ntr).
  const int ntr = (th + 63) / 64, ntc = (tw + 63) / 64;
  std::vector<TensorTile> tiles;
  for (int i = 0; i < ntr; ++i) {
    const int r0 = (int)((long long)i * th / ntr), r1 = (int)((long long)(i + 1) * th / ntr);
    for (int j = 0; j < ntc; ++j) {
      const int c0 = (int)((long long)j * tw / ntc), c1 = (int)((long long)(j + 1) * tw / ntc);
      TensorTile t;
      t.tmpl = tmpl;
      t.tmpl.ptr = (char*)tmpl.ptr + (size_t)r0 * tmpl.pitch + (size_t)c0 * nch * es;
      t.tmpl.width = c1 - c0;
      t.tmpl.height = r1 - r0;
      t.ax = ax - c0;
      t.ay = ay - r0;
      tiles.push_back(t);
    }
  }
  // Maps of one launch's tiles, and FP64 sums where there are more launches.
  TileMaps c;
  c.pitch = row_energy_pitch(src.width);
  c.plane = c.pitch * src.height;
  const int group = (int)std::max<size_t>(
      1, std::min<size_t>({(size_t)tensor_max_tiles(), tiles.size(), kMapBytes / (c.plane * nch)}));
  const size_t d_pitch = 2 * c.pitch, d_plane = d_pitch * src.height;
  const bool more = tiles.size() > (size_t)group;
  const size_t map_bytes = c.plane * nch * group;
  char* maps = reinterpret_cast<char*>(
      ctx.scratch(Context::kProductMap, map_bytes + (more ? d_plane * nch : 0)));
  c.maps = maps;
  c.before = nullptr;
  c.before_pitch = d_pitch;
  c.before_plane = d_plane;
  for (size_t at = 0; at < tiles.size(); at += group) {
    const size_t end = std::min(tiles.size(), at + group);
    const std::vector<TensorTile> part(tiles.begin() + at, tiles.begin() + end);
    const cudaError_t e = launch_tensor_tiles(ctx, src, part, planes, maps, c.pitch);
    if (e != cudaSuccess) return e;
    c.n = (int)part.size();
    if (end == tiles.size()) break;  // the scoring pass adds the last group
    double* sums = reinterpret_cast<double*>(maps + map_bytes);
    const dim3 grid((src.width + kBlockCols - 1) / kBlockCols, (src.height + kGroups - 1) / kGroups,
                    nch);
    if (src.type == U8)
      tile_sum_kernel<int><<<grid, dim3(32, kGroups), 0, ctx.stream>>>(c, src.width, src.height, nch, sums,
                                                         d_pitch, d_plane);
    else
      tile_sum_kernel<float><<<grid, dim3(32, kGroups), 0, ctx.stream>>>(c, src.width, src.height, nch, sums,
                                                           d_pitch, d_plane);
    count_launches(1);
    c.before = sums;
  }
  // Row energies of the whole template width (measures other than CrossCorr).
  const size_t r_pitch = row_energy_pitch(src.width), r_plane = r_pitch * src.height;
  char* rmap = nullptr;
  if (m != kCrossCorr) {
    rmap = reinterpret_cast<char*>(ctx.scratch(Context::kEnergyMap, r_plane * nch));
    const RowEnergyJob job{planes.ptr, planes.pitch, planes.bytes, rmap,  r_pitch, r_plane,
                           src.width,  src.height,   nch,          tw,    ax};
    const cudaError_t e =
        launch_row_energies(src.type, tw, job, nullptr, 1, src.width, src.height, ctx.stream);
    if (e != cudaSuccess) return e;
    count_launches(1);
  }
  double* et = reinterpret_cast<double*>(ctx.scratch(Context::kTemplateStats, 64));
  if (m != kCrossCorr) {
    auto kern = tmpl.type == U8    ? template_energy_f64_kernel<uint8_t>
                : tmpl.type == U16 ? template_energy_f64_kernel<uint16_t>
                                   : template_energy_f64_kernel<float>;
    kern<<<nch, 1024, 0, ctx.stream>>>((const char*)tmpl.ptr, tmpl.pitch, tw, th, nch, et);
    count_launches(1);
  }
  ScoreParams p;
  p.c = c;
  p.rmap = rmap;
  p.r_pitch = r_pitch;
  p.r_plane = r_plane;
  p.et = et;
  p.dst = (char*)dst.ptr;
  p.dst_pitch = dst.pitch;
  p.dst_f64 = dst.type == F64;
  p.W = src.width;
  p.H = src.height;
  p.nch = nch;
  p.th = th;
  p.ay = ay;
  p.measure = m;
  p.u8_float = (double)tw * th * 65025.0 <= 16777216.0;
  const dim3 grid((src.width + kBlockCols - 1) / kBlockCols, (src.height + kGroups - 1) / kGroups,
                    nch);
  if (src.type == U8)
    large_score_kernel<false><<<grid, dim3(32, kGroups), 0, ctx.stream>>>(p);
  else
    large_score_kernel<true><<<grid, dim3(32, kGroups), 0, ctx.stream>>>(p);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace ocipb

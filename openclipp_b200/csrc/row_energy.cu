// Row energies of the ImageProximity windows, for the tensor-core path.
//
// R(x, r, c) = sum_{w < tw} S(x + w - ax, r, c)^2 (zero outside the image):
// the energy of the template-wide row segment of source row r that output
// column x's window covers. The window energy of output (x, y) -- the
// counterpart of the reference's AreaSqSum over a SqrIntegral
// (cl-files/ImageProximityFFT.cl:55-84) and of the sum S^2 accumulator of
// the direct _Norm kernels (cl-files/ImageProximity.cl:122-211, 375-466) --
// is then the sum of R over the th rows y - ay .. y - ay + th - 1, which the
// tensor kernel's epilogue keeps as a running sum (FP64; int32 for U8) while it
// walks down the rows. Rows are independent here, so every warp streams its own row
// segment with all its loads in flight.
//
// R is stored as FP32 for F32 and U16 sources (a difference of FP64 prefix
// sums rounded once: 2^-24 of it and, for F32, about 2^-50 of its segment's
// energy) and as int32 for U8 sources (exact). An FP64 running sum of FP32
// values adds and later removes each value exactly while their exponents lie
// within 2^29 of one another, less log2 th: always for U16, and for F32 down to
// energies of about 2^-24 of the brightest window's. Beyond that an F32 window can
// keep a residue of what is beside or above it, up to 2^-50 of that energy (a
// window of zeros a finite score instead of NaN). Bound: HBM (the source read
// once, 4 bytes written per output column and source row).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "internal.h"
#include "row_energy.h"

namespace ocipb {
namespace {

constexpr int kWarps = 8;        // one row segment per warp
constexpr int kSeg = 256;        // output columns per segment (8 per lane)
constexpr int kMaxTw = 1024;  // 256 + tw - 1 <= 32 * 41

template <typename ET>
struct RowSumOf {
  // Prefix sums, exact for integers: int32 for 8-bit sources (at most
  // 1279 * 255^2 < 2^31), FP64 otherwise (16-bit: below 2^53; F32: squares
  // exact, sums rounded in FP64).
  typedef typename std::conditional<sizeof(ET) == 1, int, double>::type A;
  // Stored: int32 for 8-bit sources, FP32 otherwise.
  typedef typename std::conditional<sizeof(ET) == 1, int, float>::type R;
};

// One warp per (source row, 256 output columns) of one plane of one job. The n =
// 256 + tw - 1 source pixels the segment's windows cover are staged raw in
// shared memory with 16-byte loads (from the 16-byte group at or below the
// first, so `sh` pixels lead); lane l squares its K contiguous entries and
// turns them into prefix sums (local prefix plus a warp scan of the lanes'
// totals), P(i) = sum of squares [0, i) stored at entry i - 1; output column
// x0 + j (j = lane + 32 u) is then P(j + tw) - P(j): two conflict-free reads,
// and the warp's stores are 128-byte rows.
//
// Channels come as planes (the tensor kernels' copies): reading them
// interleaved, one channel per block, took 96 us for 3840 x 2160 x 4 U16
// where the planes take 57 (under the profiler).
//
// TABLE: block z takes plane z mod nch of job z / nch of a device table, else plane z
// of the one job (with the choice made at run time 4096 x 4096 F32 took 39 us, so
// 36, under the profiler). A batch's 42 maps of 1024 x 1024 U8 took 5 us each in
// launches of their own, 74 us in all in two.
template <typename ET, int K, bool TABLE>
__global__ void __launch_bounds__(kWarps * 32)
    row_energy_kernel(const __grid_constant__ RowEnergyJob one, const RowEnergyJob* jobs) {
  typedef typename RowSumOf<ET>::A A;
  typedef typename RowSumOf<ET>::R RT;
  constexpr int kInner = 16 / (int)sizeof(ET);                      // pixels per group
  constexpr int kRawGroups = (32 * K + kInner - 1) / kInner + 1;     // covers sh + 32 K
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  cudaTriggerProgrammaticLaunchCompletion();  // the tensor kernel may start in the tail
  RowEnergyJob entry;
  if (TABLE) entry = jobs[blockIdx.z / one.nch];
  const RowEnergyJob& p = TABLE ? entry : one;
  const int c = TABLE ? blockIdx.z % one.nch : blockIdx.z;
  const int r = blockIdx.y * kWarps + warp;
  const int x0 = blockIdx.x * kSeg;
  if (r >= p.H || x0 >= p.W) return;  // whole warp
  A* buf = reinterpret_cast<A*>(smem) + warp * (32 * K);
  ET* raw = reinterpret_cast<ET*>(smem + (size_t)kWarps * 32 * K * sizeof(A)) +
            warp * (kRawGroups * kInner);
  const ET* row =
      reinterpret_cast<const ET*>(p.src + c * p.src_plane + (size_t)r * p.src_pitch);
  const int n = kSeg + p.tw - 1;
  const int xs0 = x0 - p.ax;
  const int xa = xs0 >= 0 ? xs0 - xs0 % kInner : -((-xs0 + kInner - 1) / kInner) * kInner;
  const int sh = xs0 - xa;
  // Raw pixels xa .. xa + kRawGroups * kInner - 1, zero outside the image:
  // whole groups inside the row with one 16-byte load, the rest per pixel.
  for (int g = lane; g < kRawGroups; g += 32) {
    const int x = xa + g * kInner;
    uint4 v;
    if (x >= 0 && x + kInner <= p.W) {
      v = __ldg(reinterpret_cast<const uint4*>(row + x));
    } else {
      ET e[kInner];
#pragma unroll
      for (int i = 0; i < kInner; ++i) e[i] = (x + i >= 0 && x + i < p.W) ? row[x + i] : ET(0);
      memcpy(&v, e, sizeof(v));
    }
    reinterpret_cast<uint4*>(raw)[g] = v;
  }
  __syncwarp();
  // Lane l: staged entries K l .. K l + K - 1 (pixel xs0 + i is raw[sh + i]).
  A loc[K];
  A tot = A(0);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = K * lane + k;
    const A e = i < n ? static_cast<A>(raw[sh + i]) : A(0);
    tot += e * e;
    loc[k] = tot;
  }
  A incl = tot;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const A o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  const A excl = incl - tot;
#pragma unroll
  for (int k = 0; k < K; ++k) buf[K * lane + k] = excl + loc[k];
  __syncwarp();
  RT* dst = reinterpret_cast<RT*>(p.dst + c * p.dst_plane + (size_t)r * p.dst_pitch);
#pragma unroll
  for (int u = 0; u < kSeg / 32; ++u) {
    const int j = lane + 32 * u;
    const int x = x0 + j;
    if (x < p.W) {
      const A hi = buf[j + p.tw - 1];
      const A lo = j > 0 ? buf[j - 1] : A(0);
      dst[x] = static_cast<RT>(hi - lo);
    }
  }
}

// `n` jobs (a device table), or the one given.
template <typename ET, int K>
cudaError_t launch_k(const RowEnergyJob& one, const RowEnergyJob* jobs, int n, int W, int H,
                     cudaStream_t st) {
  typedef typename RowSumOf<ET>::A A;
  constexpr int kInner = 16 / (int)sizeof(ET);
  constexpr int kRawGroups = (32 * K + kInner - 1) / kInner + 1;
  const size_t smem = (size_t)kWarps * (32 * K * sizeof(A) + kRawGroups * 16);
  auto launch = [&](auto kern, dim3 grid, const RowEnergyJob* table) {
    if (smem > 48 * 1024) {
      const cudaError_t e =
          cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    kern<<<grid, kWarps * 32, smem, st>>>(one, table);
    return cudaGetLastError();
  };
  const unsigned nx = (W + kSeg - 1) / kSeg, ny = (H + kWarps - 1) / kWarps;
  if (!jobs) return launch(row_energy_kernel<ET, K, false>, dim3(nx, ny, one.nch), nullptr);
  // Grid dimension z holds 65535 planes.
  const int most = 65535 / one.nch;
  for (int i = 0; i < n; i += most) {
    const cudaError_t e = launch(row_energy_kernel<ET, K, true>,
                                 dim3(nx, ny, one.nch * (n - i < most ? n - i : most)), jobs + i);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Staged entries per lane for a template width: 32 K >= 256 + tw - 1.
constexpr int k_for(int tw) {
  const int n = kSeg + tw - 1;
  return n <= 32 * 9 ? 9 : n <= 32 * 11 ? 11 : n <= 32 * 17 ? 17 : 41;
}

template <typename ET>
cudaError_t launch_typed(int tw, const RowEnergyJob& one, const RowEnergyJob* jobs, int n, int W,
                         int H, cudaStream_t st) {
  switch (k_for(tw)) {
    case 9: return launch_k<ET, 9>(one, jobs, n, W, H, st);
    case 11: return launch_k<ET, 11>(one, jobs, n, W, H, st);
    case 17: return launch_k<ET, 17>(one, jobs, n, W, H, st);
    default: return launch_k<ET, 41>(one, jobs, n, W, H, st);
  }
}

}  // namespace

size_t row_energy_pitch(int width) { return ((size_t)width * 4 + 127) / 128 * 128; }

cudaError_t launch_row_energies(int type, int tw_max, const RowEnergyJob& one,
                                const RowEnergyJob* jobs, int n, int W, int H,
                                cudaStream_t stream) {
  if (tw_max < 1 || tw_max > kMaxTw) return cudaErrorInvalidValue;
  // The kernels read 16-byte groups of pixels and write 4-byte sums. (A table's
  // planes have passed the check that its tensor maps make.)
  if (!jobs && (((uintptr_t)one.src | one.src_pitch | one.src_plane) % 16 ||
                ((uintptr_t)one.dst | one.dst_pitch | one.dst_plane) % 4))
    return cudaErrorInvalidValue;
  switch (type) {
    case U8: return launch_typed<uint8_t>(tw_max, one, jobs, n, W, H, stream);
    case U16: return launch_typed<uint16_t>(tw_max, one, jobs, n, W, H, stream);
    case F32: return launch_typed<float>(tw_max, one, jobs, n, W, H, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ocipb

// Row energies of the ImageProximity windows (row_energy.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace ocipb {

// Row pitch (bytes) of a row-energy map: 4 bytes per column, 128-byte rows.
size_t row_energy_pitch(int width);

// R(x, r) = sum_{w < tw} S(x + w - ax, r)^2 (zero outside the image) of every
// plane of an image: int32 for U8, FP32 for U16 and F32. Source rows start on
// 16 bytes.
struct RowEnergyJob {
  const char* src;
  size_t src_pitch, src_plane;  // bytes between rows, between channel planes
  char* dst;
  size_t dst_pitch, dst_plane;
  int W, H, nch;
  int tw, ax;
};

// One launch for the job `one` (jobs null, n = 1) or for `n` jobs of a device
// table with one type and channel count (one.nch): W, H and tw_max are the
// largest of any job.
cudaError_t launch_row_energies(int type, int tw_max, const RowEnergyJob& one,
                                const RowEnergyJob* jobs, int n, int W, int H,
                                cudaStream_t stream);

}  // namespace ocipb

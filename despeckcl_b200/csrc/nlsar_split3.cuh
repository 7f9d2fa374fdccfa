// Definitions shared by the 3x3 (PolSAR) NL-SAR kernels, and the interface of
// their two-kernel path (nlsar_split3.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "nlsar_common.cuh"
#include "nlsar_plan.h"

namespace dcl {

// planes of the nine similarity reals within the 18 covariance planes
__host__ __device__ constexpr int sim_plane(int k) {
  return k == 0 ? 0 : k == 1 ? 8 : k == 2 ? 16 : k == 3 ? 2 : k == 4 ? 3 : k == 5 ? 4 : k == 6 ? 5 : k == 7 ? 10 : 11;
}
// planes of the diagonal intensities
__host__ __device__ constexpr int diag_plane(int d) { return 8 * d; }

// sim_measures.h:78-97 with a = {a00, a11, a22, Re a01, Im a01, Re a02, Im a02, Re a12, Im a12}
__host__ __device__ __forceinline__ float det3f(const float* a) {
  return a[0] * a[1] * a[2] - a[0] * (a[7] * a[7] + a[8] * a[8]) - a[1] * (a[5] * a[5] + a[6] * a[6]) -
         a[2] * (a[3] * a[3] + a[4] * a[4]) +
         2.0f * (a[3] * a[7] * a[5] - a[4] * a[8] * a[5] + a[3] * a[8] * a[6] + a[4] * a[7] * a[6]);
}

struct Scene3 {
  const float* c18;             // [18][Hp][pitch]
  const float* s9[kMaxScales];  // [9][Hp][pitch] per scale slot
  const float* ld[kMaxScales];  // [Hp][pitch] per scale slot
  float* out;                   // [18][H][W]
  int H, W, vH, vW, pitch, tiles_x;
  int tile_skip;                // scene tiles before block 0 of the launch (row bands)
  size_t plane;                 // Hp * pitch
};

// The two-kernel path of a 3x3 call: segments whose similarity and word
// volumes fit a budget.
struct Split3 {
  int rows = 0, cols = 0;           // virtual rows and columns per segment; rows 0: the call is not served
  int pitch = 0, spitch = 0;        // words, similarities per volume row
  bool exact = false;               // the settings and arithmetic of nlsar3_kernel
  size_t sim_bytes = 0, vol_bytes = 0;  // similarities of one scale, then the words of every pass
};
// Whether nlsar3_fast_kernel has a call's shapes (nlsar_dim3.cu).
bool fast3_supported(const FilterParams& F);
// Sizes the segments for `budget` bytes: runs of whole rows where two rows of
// the tallest tiles fit, else cut in columns too; rows 0 where the plan has no
// kernels or one tile column of that does not fit.
Split3 split3_layout(const Plan& pl, const Scene3& S, size_t budget);
// Filters virtual rows [vy0, vy1) (at most L.rows) and columns [vx0, vx1) (at
// most L.cols, vx0 a multiple of it) with the volumes at `vol`.
cudaError_t launch_split3(const Plan& pl, const FilterParams& F, const Scene3& S, int Hp, int Wp, const Split3& L,
                          char* vol, int vy0, int vy1, int vx0, int vx1, int sms, cudaStream_t st);

}  // namespace dcl

// Host interface of the two-kernel NL-SAR path (nlsar_split.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

#include "nlsar_common.cuh"
#include "nlsar_plan.h"

namespace dcl {

// Volume of weight indices held at a time, at most.
constexpr size_t kSplitBudgetBytes = size_t(2) << 30;
constexpr size_t kSplitMinBudgetBytes = size_t(32) << 20;  // not tried smaller when memory is short
// kSplitBudgetBytes, or what DESPECKCL_B200_VOLUME_MIB=n caps it to (0: no
// call takes the two-kernel path).
size_t split_budget();
constexpr size_t kSplitSmem = 227 * 1024;
constexpr int kSplitShapes = 2;  // different pass shapes of one call

// A rectangle of virtual pixels of one scene with its volume: per pass words
// [half-window offset][rows][pitch] of one byte per patch size (three: four).
struct SplitSeg {
  int scene;
  int vy0, vy1;        // virtual rows filtered
  int vx0;             // first virtual column filtered, on a tile column
  int row0, rows;      // virtual row of the volume's first row (vy0 - wsh), row count
  int pitch;           // words per row; volume column c is virtual column vx0 + c - wsh
  int tiles_x, tile_begin;  // mean kernel: tiles per row, first tile in the chunk
  int idx_begin[kSplitShapes], idx_bx[kSplitShapes], idx_R[kSplitShapes];  // index kernel: blocks, columns, rows
  size_t vol, pass[kMaxPasses];  // first byte, and of each pass from there
};

// Segments filtered together: one index launch per pass shape, one mean launch.
struct SplitChunk {
  int seg0, seg1;
  int th, tiles;  // mean kernel: tile rows, tiles
  int idx_blocks[kSplitShapes], idx_z[kSplitShapes];
  size_t idx_smem[kSplitShapes];
};

// Passes of one shape.
struct PassList {
  int n;
  int id[kMaxPasses];
};

// Virtual rows [row0, row1) of a scene, row0 on a tile row.
struct SplitJob {
  int scene, row0, row1;
};

struct SplitLayout {
  std::vector<SplitSeg> segs;
  std::vector<SplitChunk> chunks;
  size_t vol_bytes;
  int nshape, shape[kSplitShapes];
  PassList passes[kSplitShapes];
};

// Whether the two-kernel path serves a call: the specialised kernel's shapes
// in its default arithmetic, or other windows with passes of the same patch
// sizes or {3,5}; tables that fit byte codes.
bool split_supported(const Plan& pl);
// Whether the weight tables of a plan's passes fit byte codes.
bool split_tables_ok(const Plan& pl);
bool split_layout(const Plan& pl, const std::vector<SceneGeom>& geo, const std::vector<SplitJob>& jobs,
                  size_t budget, int sms, SplitLayout& out);
// Kernels a layout launches.
int split_launches(const SplitLayout& lay);
// Launches chunk `chunk`: index kernels, then the mean kernel.
cudaError_t launch_split(const Plan& pl, const FilterParams& F, const SplitLayout& lay, int chunk,
                         const SceneDesc* d_scenes, const SplitSeg* d_segs, char* vol, cudaStream_t st);

// All chunks of a layout (nlsar_host.cu), timed as one launch by the profile.
int launch_split_all(const Plan& pl, const FilterParams& F, const SplitLayout& lay, const SceneDesc* d_scenes,
                     const SplitSeg* d_segs, char* vol, cudaStream_t st);

}  // namespace dcl

// Host interface of the basin form of the batched TFCE sweep (tfce_basin.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace tfgb {

struct CleanLists;
struct BasinPlan;  // tiles, neighbour slices, boundary tables and workspaces of one adjacency handle

// What one tfce_sweep_batch call asks for (device pointers).
struct BasinRequest {
  const float* stats;
  int64_t map_stride;
  int32_t n_maps;
  int32_t signs;
  const float* vdensity;
  float* out_max;
  float* out_maps;
  int32_t out_mode;
  bool exact;         // the reference's float accumulation where vertex values are needed
  bool potentials;    // keep the potentials for maxima-only launches too
  int32_t dense;      // 1: more items resident with less shared state each; 0: fewer, larger
  const int32_t* thr_group;
  const float* d_H;
  const int64_t* d_seg_off;
  const int32_t* seg_rank;
  int32_t* err;
};

// Tiles of cleaned lists, seg [n_seg+1].  *out stays NULL (and TFCE_OK is returned) for graphs
// that the form does not take.
int basin_plan_create(const CleanLists& lists, const std::vector<int64_t>& seg, BasinPlan** out);
void basin_plan_destroy(BasinPlan* p);
// Tables of extent^E of the segments' exponents (host array of n_seg).
int basin_plan_set_exponents(BasinPlan* p, const float* E);
// Whether the request can run in this form (the vertex values of the
// reference's arithmetic need a node table that grows with the segment).
bool basin_takes(const BasinPlan* p, const BasinRequest& r);
// *refused: there was no memory for the workspace, and nothing was launched.
int basin_sweep(BasinPlan* p, const BasinRequest& r, cudaStream_t st, bool* refused);
int64_t basin_launched(const BasinPlan* p);  // kernels, so far
// Items that a launch of many sweeps at once.
int basin_resident_items(const BasinPlan* p, bool dense);

}  // namespace tfgb

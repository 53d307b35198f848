// Fused execution of recognised step phases (TE_MODE_FUSED).
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "te_dims.cuh"

namespace te {

struct Op;
struct Plan;
class StepDeps;

// A step's op list rewritten into segments: runs of exact per-dispatch kernels and
// fused phase kernels that produce bit-identical prognostic fields.
struct FusedSegment {
  int kind = 0;  // 0 = exact ops [first, last]; >0 = a fused phase
  int first = 0, last = 0;
  int aux[16] = {0};
};

struct FusedStep {
  std::vector<FusedSegment> segs;
  void* data = nullptr;  // kernel arguments of the fused segments
  // with keep_scratch every word of memory ends as the op sequence leaves it: a phase whose
  // fused kernels skip scratch stores runs per dispatch unless the step stores them again later
  void build(Plan& P, std::vector<Op>& ops, bool keep_scratch);
  // the whole step; with deps (during a capture) each kernel after those it depends on only
  void launch(Plan& P, std::vector<Op>& ops, StepDeps* deps);
  // one segment; part = -1 for all of its kernels, else the index of one of them
  void launch_segment(Plan& P, std::vector<Op>& ops, int seg, int part);
  // the same for a caller that plays a segment on its own: a whole substep then starts from and
  // ends in its fields, halos filled, wherever it stands in a run of them
  void play_segment(Plan& P, std::vector<Op>& ops, int seg, int part);
  static bool chains_substeps(const std::vector<Op>& ops);  // a run of substeps that wants Plan::work
  int kernels(int seg) const;  // launches of a fused segment (0: a run of exact ops)
  void release();
};

// ops[i], ops[i + 1] are bc_periodic_x(f) then bc_periodic_y(f) over the standard halo
// grids (4 x (ny + 7) x (nz + 1), 4 x (nx + 7) x (nz + 1)): sets *f, returns true.
bool periodic_halo_pair(const std::vector<Op>& ops, size_t i, float** f);

// The final state of such pairs for nf <= 4 distinct fields in one launch: every halo point
// of levels 0..nz holds the interior value at (i mod nx, j mod ny).
void launch_periodic_halos(const Dims& g, float* const* f, int nf, cudaStream_t s);

}  // namespace te

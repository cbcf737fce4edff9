// Shape of the node-step kernel's CTAs (node_step.cu): shared-memory layout for the largest
// rollout of a plan.
#pragma once
#include "mc_internal.cuh"

namespace mc {

constexpr int kNodeStepMaxThreads = 768;  // 80 registers each: the phases spill with fewer

struct NodeStepShape {
  int threads, bytes;                       // per CTA
  int teams, rod_warps, longest;            // rods at a time, warps each, nodes of the longest rod
  int bars;                                 // named barriers per team
  int hash;                                 // hash entries (more than the contributions, a multiple of 4)
  int pos, vel, nvl, delta, w, slot, rw, rn, hcell, hrun, shared;  // offsets in shared memory
};

void launch_node_step(const RDesc* d, int n, int* tdev, const NodeStepShape& shape, int parity, int main, int next,
                      cudaStream_t s);
cudaError_t node_step_set_smem(size_t bytes);

}  // namespace mc

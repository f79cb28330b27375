// Device-side hyper-parameter block of the Lion kernels.
#pragma once

#include <stdint.h>

#include "kaon_device.cuh"
#include "kaon_plan.h"

namespace kaon {

struct LionDev {
  float lr, b1, w1, b2, w2, wd;
  int cautious, gc, sr, has_wd;
  uint32_t step, k0, k1;
  uint32_t rk0[KAON_PHILOX_ROUNDS], rk1[KAON_PHILOX_ROUNDS];  // Philox round keys (k + r * Weyl), from the host
  int kahan;
};

// lion_warp.cu: the cautious step as warp units.  lion_warp_tensor: whether a tensor can take it; lion_warp_units: the
// units of the plan's eligible tensors, MAIN and APPLY in the order they are claimed, and each one's number of MAIN units.
bool lion_warp_tensor(const DevTensor& t, int momentum_kind);
int lion_warp_units(const std::vector<DevTensor>& tensors, const std::vector<char>& elig, std::vector<Task>& out, std::vector<int>& n_main);
int launch_lion_warp(kaon_plan* pl, const PlanView& base, const LionDev& hp, cudaStream_t s);

}  // namespace kaon

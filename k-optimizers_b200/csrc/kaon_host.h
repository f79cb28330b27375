// Host-only helpers shared by the translation units of libkaon_b200.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

struct kaon_plan;

namespace kaon {

int fail(int code, const char* fmt, ...);           // records the message, returns code
int cuda_fail(cudaError_t e, const char* what);     // KAON_E_CUDA with the runtime's message
size_t momentum_bytes_per_cap(int momentum_kind);   // bytes of momentum storage per CAP elements
int configure_launch(kaon_plan* pl, const cudaDeviceProp& prop);  // Lion: grid + dynamic shared memory
int configure_launch_adakaon(kaon_plan* pl, const cudaDeviceProp& prop, int max_cols);
// bf16_method == KAHAN with bf16 weights needs every tensor's shift buffer: KAON_OK or an error
int check_kahan(const kaon_plan* pl, int bf16_method);
// the calling thread's current device must be the one the plan was built on: KAON_OK or KAON_E_INVALID
int check_device(const kaon_plan* pl);

#define KAON_CUDA(call)                                              \
  do {                                                               \
    cudaError_t e__ = (call);                                        \
    if (e__ != cudaSuccess) return ::kaon::cuda_fail(e__, #call);    \
  } while (0)

// A launch that may begin while the launch before it on the stream drains (programmatic stream serialization): the kernel calls
// after_launch_before() ahead of the first access to what that launch writes, or, where the two have nothing to do with
// each other, at its end.  Not with reserved multiprocessors (`early` false): its blocks would find room on those first, while
// the others are full, and either sit there or, as they should, leave, all of them, with the work undone.
template <typename... P, typename... A>
cudaError_t launch_early(bool early, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace kaon

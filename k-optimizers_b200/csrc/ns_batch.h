// Newton-Schulz over a batch of matrices (ns.cu), as AdaMuon runs it.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <vector>

#include "ns_share.h"

namespace kaon {

// One matrix: [R, C] as stored.  Scratch matrices have row strides padded to eight elements (TMA describes them
// whatever C is); `out` is dense.
struct NsMat {
  long long R, C, ld, lr;
  __nv_bfloat16 *x0, *xb, *A, *B, *out;   // x0: the unnormalised matrix, left by the caller
  float* scal;                            // {s*s, 0, s, s}, s = 1 / norm
  int tensor;                             // its place in the gradient column
};

struct NsScale { int begin, end; float* scal; };   // partial sums of squares of one matrix

struct NsStage { int prob0, tile0, begin0, grid; bool pair; };   // (grid: CTAs, or pairs of CTAs)

struct NsBatch {
  std::vector<NsStage> stages;        // three per iteration (iterations share their tiles)
  std::vector<unsigned char> host;    // device tables: products, tiles, tile ranges
  size_t bytes = 0, off_tiles = 0, off_begin = 0;
};

size_t ns_scratch_bytes(long long R, long long C);
void ns_scratch_layout(NsMat& m, unsigned char* base);
int ns_batch_build(const std::vector<NsMat>& mats, int steps, NsShares& shares, NsBatch& out);
int ns_batch_run(const NsBatch& b, const unsigned char* dev, const void* const* grads, unsigned* status, cudaStream_t s, long long* launches);
void ns_batch_scale(const NsScale* mats, int n, const double* part, cudaStream_t s);

}  // namespace kaon

// Newton–Schulz orthogonalisation (reference src/kaon/adamuon.py:97-149) as a chain of tcgen05 GEMMs.
//
//   X = M / (||M||_F + 1e-7);  steps x { A = X X^T;  B = b A + c A A;  X = a X + B X }
// run on the matrix in its stored orientation: for a wide matrix [r, k] (r <= k) X is used as stored;
// for a tall one [k, r] the stored matrix is X^T, A = (X^T)^T (X^T) takes both operands MN-major and
// X^T <- a X^T + X^T B uses that B is symmetric.  The 1/norm scaling is folded into the epilogues of
// the first iteration (A = s^2 M M^T, X1 = s (a M + B M)), so the unnormalised bf16 matrix is read
// directly and no normalisation pass exists.  Every product rounds to bf16 once, after the fused fp32
// epilogue (the reference rounds after every op; both sit within its own 2e-2 tolerance).
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "kaon_host.h"
#include "ns_batch.h"
#include "ns_gemm.cuh"

namespace kaon {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Tensor map of a row-major bf16 matrix [outer, inner] with row stride ld (elements), box = [box_outer, 64].
static int make_map(CUtensorMap* m, const void* base, long long inner, long long outer, long long ld, int box_outer) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(KAON_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)box_outer};
  cuuint32_t es[2] = {1u, 1u};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(KAON_E_CUDA, "cuTensorMapEncodeTiled failed with %d (inner %lld outer %lld ld %lld)", (int)r, inner, outer, ld);
  return KAON_OK;
}

// Plain fp32-accumulate GEMM for shapes TMA cannot describe (row stride not a multiple of 16 bytes).
__global__ void ns_gemm_simple_kernel(const __nv_bfloat16* A, int a_mn, long long lda, const __nv_bfloat16* B,
                                      int b_mn, long long ldb, GemmParams p) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= (long long)p.M * p.N) return;
  const int i = (int)(idx / p.N), j = (int)(idx % p.N);
  float acc = 0.0f;
  for (int k = 0; k < p.K; ++k) {
    const float a = __bfloat162float(a_mn ? A[(long long)k * lda + i] : A[(long long)i * lda + k]);
    const float b = __bfloat162float(b_mn ? B[(long long)k * ldb + j] : B[(long long)j * ldb + k]);
    acc += a * b;
  }
  const float alpha = p.dev_scale ? p.alpha * p.dev_scale[0] : p.alpha;
  const float beta = p.dev_scale ? p.beta * p.dev_scale[1] : p.beta;
  const float x = p.aux ? __bfloat162float(p.aux[(long long)i * p.ld_aux + j]) : 0.0f;
  p.out[(long long)i * p.ld_out + j] = __float2bfloat16_rn(acc * alpha + beta * x);
}

// always the shared memory of the widest tile: one CTA per SM, whose tensor-memory allocation (all 512
// columns) then never waits for a neighbour
constexpr size_t G2_SMEM = 1024 + (size_t)G2_RING + (size_t)G2_EPI_WARPS * G2_STAGE_OUT;

static std::atomic<int> g_gemm_sms[64];  // multiprocessors per device, once the kernel's shared-memory limit is set

static int gemm_sms(int* out) {
  int dev = 0;
  KAON_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(KAON_E_UNSUPPORTED, "device index %d", dev);
  if (!g_gemm_sms[dev].load()) {
    KAON_CUDA(cudaFuncSetAttribute((const void*)ns_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G2_SMEM));
    KAON_CUDA(cudaFuncSetAttribute((const void*)ns_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G2_SMEM));
    KAON_CUDA(cudaFuncSetAttribute((const void*)ns_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G2_SMEM));
    int sms = 0;
    KAON_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    g_gemm_sms[dev].store(sms);
  }
  *out = g_gemm_sms[dev].load();
  return KAON_OK;
}

// (a pair's CTA loads half of a tile's columns)
static int operand_maps(NsProblem& pr, const __nv_bfloat16* A, long long lda, const __nv_bfloat16* B, long long ldb, bool pair = false) {
  const GemmParams& p = pr.p;
  int rc = p.a_mn ? make_map(&pr.a, A, p.M, p.K, lda, 64) : make_map(&pr.a, A, p.K, p.M, lda, G_BM);
  if (rc) return rc;
  return p.b_mn ? make_map(&pr.b, B, p.N, p.K, ldb, 64) : make_map(&pr.b, B, p.K, p.N, ldb, pair ? p.BN / 2 : p.BN);
}

// out[M,N] = bf16(alpha * A(m,:) . B(n,:) + beta * aux)
static int launch_ns_gemm(const __nv_bfloat16* A, bool a_mn, long long lda, const __nv_bfloat16* B, bool b_mn, long long ldb,
                   int M, int N, int K, float alpha, float beta, const float* dev_scale, const __nv_bfloat16* aux,
                   long long ld_aux, __nv_bfloat16* out, long long ld_out, unsigned* status, cudaStream_t stream,
                   long long* launches, bool sym = false) {
  GemmParams p{};
  p.sym = sym && M == N ? 1 : 0;
  p.M = M; p.N = N; p.K = K; p.a_mn = a_mn; p.b_mn = b_mn;
  p.alpha = alpha; p.beta = aux ? beta : 0.0f; p.dev_scale = dev_scale;
  p.aux = aux; p.ld_aux = ld_aux; p.out = out; p.ld_out = ld_out;
  const bool tma_ok = (lda % 8 == 0) && (ldb % 8 == 0) && ((uintptr_t)A % 16 == 0) && ((uintptr_t)B % 16 == 0);
  if (launches) *launches += 1;
  if (!tma_ok) {
    const long long total = (long long)M * N;
    ns_gemm_simple_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(A, a_mn, lda, B, b_mn, ldb, p);
    KAON_CUDA(cudaGetLastError());
    return KAON_OK;
  }
  p.BN = N >= 256 ? 256 : (N > 64 ? 128 : 64);
  NsProblem pr{};
  pr.p = p;
  if (int rc = operand_maps(pr, A, lda, B, ldb)) return rc;
  int sms = 0;
  if (int rc = gemm_sms(&sms)) return rc;
  // computed tiles: all of them, or in symmetric mode those that reach the diagonal
  const int tm = ns_tiles(M, G_BM), tn = ns_tiles(N, p.BN);
  int total = 0;
  for (int mi = 0; mi < tm; ++mi) total += tn - (p.sym ? std::min(tn, (mi * G_BM) / p.BN) : 0);
  ns_gemm_kernel<false><<<std::min(total, sms), G2_THREADS, G2_SMEM, stream>>>(pr, NsWork{total, nullptr, nullptr, nullptr, nullptr, status});
  KAON_CUDA(cudaGetLastError());
  return KAON_OK;
}

// sum of squares of a bf16 matrix -> scal = {s*s, 0, s, s} with s = 1 / bf16(bf16(||x||) + 1e-7)
__global__ void ns_sumsq_kernel(const __nv_bfloat16* x, long long n, double* partial) {
  __shared__ double red[8];
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = __bfloat162float(x[i]);
    acc += (double)v * (double)v;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
}

__global__ void ns_scale_kernel(const double* partial, int n, float* scal) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < n; ++i) t += partial[i];
    const float nrm = round_bf16((float)sqrt(t));
    const float den = round_bf16(nrm + 1e-7f);
    const float s = 1.0f / den;
    scal[0] = s * s; scal[1] = 0.0f; scal[2] = s; scal[3] = s;
  }
}

constexpr int NS_PARTIALS = 296;

static size_t ns_workspace_bytes(long long R, long long C) {
  const long long r = std::min(R, C);
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  return up((size_t)R * C * 2) + 2 * up((size_t)r * r * 2) + up(NS_PARTIALS * 8) + 256;
}

// x_in [R,C] bf16 (unnormalised) -> out [R,C] bf16.  out may not alias x_in.  ws >= ns_workspace_bytes.
static int ns_run(const __nv_bfloat16* x_in, long long R, long long C, int steps, __nv_bfloat16* out, void* ws,
           unsigned* status, cudaStream_t stream, long long* launches) {
  const bool tall = R > C;             // stored matrix is X^T (k rows, r columns)
  const long long r = tall ? C : R, k = tall ? R : C;
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  unsigned char* w = reinterpret_cast<unsigned char*>(ws);
  __nv_bfloat16* xb = reinterpret_cast<__nv_bfloat16*>(w); w += up((size_t)R * C * 2);
  __nv_bfloat16* Am = reinterpret_cast<__nv_bfloat16*>(w); w += up((size_t)r * r * 2);
  __nv_bfloat16* Bm = reinterpret_cast<__nv_bfloat16*>(w); w += up((size_t)r * r * 2);
  double* partial = reinterpret_cast<double*>(w); w += up(NS_PARTIALS * 8);
  float* scal = reinterpret_cast<float*>(w);
  ns_sumsq_kernel<<<NS_PARTIALS, 256, 0, stream>>>(x_in, R * C, partial);
  ns_scale_kernel<<<1, 32, 0, stream>>>(partial, NS_PARTIALS, scal);
  KAON_CUDA(cudaGetLastError());
  if (launches) *launches += 2;
  const float a = 3.4445f, b = -4.7750f, c = 2.0315f;
  // ping-pong so that the last iteration lands in `out`
  const __nv_bfloat16* cur = x_in;
  for (int it = 0; it < steps; ++it) {
    __nv_bfloat16* nxt = ((steps - 1 - it) % 2 == 0) ? out : xb;
    const float* sc_a = it == 0 ? scal : nullptr;
    const float* sc_x = it == 0 ? scal + 2 : nullptr;
    int rc;
    // A = X X^T  [r, r]
    // (symmetric: only the tiles on and above the diagonal are computed)
    if (tall) rc = launch_ns_gemm(cur, true, C, cur, true, C, (int)r, (int)r, (int)k, 1.0f, 0.0f, sc_a, nullptr, 0, Am, r, status, stream, launches, true);
    else      rc = launch_ns_gemm(cur, false, C, cur, false, C, (int)r, (int)r, (int)k, 1.0f, 0.0f, sc_a, nullptr, 0, Am, r, status, stream, launches, true);
    if (rc) return rc;
    // B = b A + c A A   (A symmetric: A A = A A^T, both operands K-major)
    rc = launch_ns_gemm(Am, false, r, Am, false, r, (int)r, (int)r, (int)r, c, b, nullptr, Am, r, Bm, r, status, stream, launches, true);
    if (rc) return rc;
    // X <- a X + B X
    if (tall)  // X^T <- a X^T + X^T B : out[kk, j] = sum_i X^T[kk, i] B[j, i]
      rc = launch_ns_gemm(cur, false, C, Bm, false, r, (int)k, (int)r, (int)r, 1.0f, a, sc_x, cur, C, nxt, C, status, stream, launches);
    else       // out[i, j] = sum_l B[i, l] X[l, j] : second operand MN-major
      rc = launch_ns_gemm(Bm, false, r, cur, true, C, (int)r, (int)k, (int)r, 1.0f, a, sc_x, cur, C, nxt, C, status, stream, launches);
    if (rc) return rc;
    cur = nxt;
  }
  return KAON_OK;
}

// ---------------------------------------------------------------------------------------------------
// A batch of matrices: every matrix at the same stage of the iteration in one grouped launch.

// scal of every matrix from its partial sums of squares: one CTA per matrix, partials in a fixed order.
__global__ void __launch_bounds__(256) ns_batch_scale_kernel(const NsScale* mats, const double* part) {
  __shared__ double red[8];
  const NsScale m = mats[blockIdx.x];
  double acc = 0.0;
  for (int i = m.begin + threadIdx.x; i < m.end; i += 256) acc += part[i];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w];
    const float den = round_bf16(round_bf16((float)sqrt(t)) + 1e-7f);
    const float s = 1.0f / den;
    m.scal[0] = s * s; m.scal[1] = 0.0f; m.scal[2] = s; m.scal[3] = s;
  }
}

void ns_batch_scale(const NsScale* mats, int n, const double* part, cudaStream_t s) {
  ns_batch_scale_kernel<<<n, 256, 0, s>>>(mats, part);
}

static long long pad8(long long x) { return (x + 7) / 8 * 8; }

size_t ns_scratch_bytes(long long R, long long C) {
  const long long r = std::min(R, C);
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  return 2 * up((size_t)R * pad8(C) * 2) + 2 * up((size_t)r * pad8(r) * 2) + 256;
}

void ns_scratch_layout(NsMat& m, unsigned char* base) {
  const long long r = std::min(m.R, m.C);
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  m.ld = pad8(m.C); m.lr = pad8(r);
  m.x0 = reinterpret_cast<__nv_bfloat16*>(base); base += up((size_t)m.R * m.ld * 2);
  m.xb = reinterpret_cast<__nv_bfloat16*>(base); base += up((size_t)m.R * m.ld * 2);
  m.A = reinterpret_cast<__nv_bfloat16*>(base); base += up((size_t)r * m.lr * 2);
  m.B = reinterpret_cast<__nv_bfloat16*>(base); base += up((size_t)r * m.lr * 2);
  m.scal = reinterpret_cast<float*>(base);
}

// The launches of a batch's iterations: products and tensor maps per iteration, tiles per stage.
int ns_batch_build(const std::vector<NsMat>& mats, int steps, NsShares& shares, NsBatch& out) {
  out = NsBatch{};
  if (mats.empty()) return KAON_OK;
  int sms = 0;
  if (int rc = gemm_sms(&sms)) return rc;
  NsShares::Key key;
  for (const NsMat& m : mats) key.push_back({m.R, m.C});
  const std::array<NsShare, 3>& share = shares.get(key, sms);
  const float a = 3.4445f, b = -4.7750f, c = 2.0315f;
  std::vector<NsProblem> probs;
  std::vector<NsTile> tiles;
  std::vector<int> begin;
  int tile0[3], begin0[3];
  for (int stage = 0; stage < 3; ++stage) {
    tile0[stage] = (int)tiles.size();
    begin0[stage] = (int)begin.size();
    tiles.insert(tiles.end(), share[stage].tiles.begin(), share[stage].tiles.end());
    begin.insert(begin.end(), share[stage].begin.begin(), share[stage].begin.end());
  }
  for (int it = 0; it < steps; ++it) {
    for (int stage = 0; stage < 3; ++stage) {
      out.stages.push_back(NsStage{(int)probs.size(), tile0[stage], begin0[stage], (int)share[stage].begin.size() - 1, share[stage].pair});
      for (const NsMat& m : mats) {
        const bool tall = m.R > m.C;   // the stored matrix is X^T (k rows, r columns)
        // ping-pong; the last iteration lands in `out`
        const bool last = it == steps - 1;
        const __nv_bfloat16* cur = (it & 1) ? m.xb : m.x0;
        __nv_bfloat16* nxt = last ? m.out : (it & 1) ? m.x0 : m.xb;
        const NsShape sh = ns_stage_shape(stage, m.R, m.C);
        NsProblem pr{};
        GemmParams& p = pr.p;
        p.M = sh.M; p.N = sh.N; p.K = sh.K; p.sym = sh.sym;
        p.BN = ns_tile_cols(share[stage].bn, sh.N, share[stage].pair);
        pr.tensor = m.tensor;
        const __nv_bfloat16 *A, *B;
        long long lda, ldb;
        if (stage == 0) {          // A = X X^T
          A = B = cur; lda = ldb = m.ld;
          p.a_mn = tall; p.b_mn = tall; p.alpha = 1.0f;
          p.dev_scale = it == 0 ? m.scal : nullptr;
          p.out = m.A; p.ld_out = m.lr;
        } else if (stage == 1) {   // B = b A + c A A   (A symmetric: A A = A A^T, both operands K-major)
          A = B = m.A; lda = ldb = m.lr;
          p.alpha = c; p.beta = b;
          p.aux = m.A; p.ld_aux = m.lr; p.out = m.B; p.ld_out = m.lr;
        } else {                   // X <- a X + B X; stored transposed: X^T <- a X^T + X^T B
          A = tall ? cur : m.B; lda = tall ? m.ld : m.lr;
          B = tall ? m.B : cur; ldb = tall ? m.lr : m.ld;
          p.b_mn = !tall; p.alpha = 1.0f; p.beta = a;
          p.dev_scale = it == 0 ? m.scal + 2 : nullptr;
          p.aux = cur; p.ld_aux = m.ld; p.out = nxt; p.ld_out = last ? m.C : m.ld;
        }
        if (int rc = operand_maps(pr, A, lda, B, ldb, share[stage].pair)) return rc;
        probs.push_back(pr);
      }
    }
  }
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t o_t = up(sizeof(NsProblem) * probs.size()), o_b = o_t + up(sizeof(NsTile) * tiles.size());
  out.bytes = o_b + up(sizeof(int) * begin.size());
  out.host.assign(out.bytes, 0);
  std::memcpy(out.host.data(), probs.data(), sizeof(NsProblem) * probs.size());
  std::memcpy(out.host.data() + o_t, tiles.data(), sizeof(NsTile) * tiles.size());
  std::memcpy(out.host.data() + o_b, begin.data(), sizeof(int) * begin.size());
  out.off_tiles = o_t;
  out.off_begin = o_b;
  return KAON_OK;
}

// One grouped launch per stage, from the tables at `dev` (the bytes of NsBatch::host).  `grads`: the gradient column where
// some matrix of the batch has none (its products are passed over), null where all have one.
int ns_batch_run(const NsBatch& b, const unsigned char* dev, const void* const* grads, unsigned* status, cudaStream_t s, long long* launches) {
  const NsProblem none{};
  for (const NsStage& st : b.stages) {
    NsWork w{};
    w.probs = reinterpret_cast<const NsProblem*>(dev) + st.prob0;
    w.tiles = reinterpret_cast<const NsTile*>(dev + b.off_tiles) + st.tile0;
    w.begin = reinterpret_cast<const int*>(dev + b.off_begin) + st.begin0;
    w.grads = grads;
    w.status = status;
    if (st.pair) ns_pair_kernel<<<2 * st.grid, G2_THREADS, G2_SMEM, s>>>(w);
    else ns_gemm_kernel<true><<<st.grid, G2_THREADS, G2_SMEM, s>>>(none, w);
    *launches += 1;
  }
  KAON_CUDA(cudaGetLastError());
  return KAON_OK;
}

}  // namespace kaon

using namespace kaon;

extern "C" int64_t kaon_newton_schulz_workspace_bytes(int64_t rows, int64_t cols) {
  return (int64_t)ns_workspace_bytes(rows, cols) + 256;
}

extern "C" int kaon_newton_schulz(const void* x_bf16, int64_t rows, int64_t cols, int steps, void* out_bf16,
                                  void* workspace, int64_t workspace_bytes, void* stream) {
  if (!x_bf16 || !out_bf16 || !workspace || rows <= 0 || cols <= 0 || steps < 1) return fail(KAON_E_INVALID, "kaon_newton_schulz: bad argument");
  if (x_bf16 == out_bf16) return fail(KAON_E_INVALID, "kaon_newton_schulz: output may not alias the input");
  if (workspace_bytes < kaon_newton_schulz_workspace_bytes(rows, cols)) return fail(KAON_E_INVALID, "kaon_newton_schulz: workspace too small");
  if (rows >= (1ll << 31) || cols >= (1ll << 31)) return fail(KAON_E_UNSUPPORTED, "matrix too large");
  // the first 4 bytes of the workspace are the status word of this call
  unsigned* status = reinterpret_cast<unsigned*>(workspace);
  KAON_CUDA(cudaMemsetAsync(status, 0, 4, (cudaStream_t)stream));
  return ns_run(reinterpret_cast<const __nv_bfloat16*>(x_bf16), rows, cols, steps,
                reinterpret_cast<__nv_bfloat16*>(out_bf16), reinterpret_cast<unsigned char*>(workspace) + 256,
                status, (cudaStream_t)stream, nullptr);
}

// bf16 GEMM for the Newton–Schulz iteration on sm_100a tensor cores:
//   out[M,N] = bf16( alpha * sum_k A(m,k) * B(n,k)  +  beta * aux[M,N] )
// tcgen05.mma (cta_group::1, kind::f16, M=128, N<=256, K=16) issued by one thread, operands staged in
// shared memory by TMA (128-byte swizzle, no multicast), fp32 accumulators in tensor memory, read back
// with tcgen05.ld for the fused epilogue.  Either operand may be K-major (matrix stored [MN, K], K
// contiguous) or MN-major (stored [K, MN], MN contiguous), which is what lets the iteration run on a
// matrix in its native orientation without ever transposing it in memory.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kaon_stage.cuh"
#include "ns_share.h"

namespace kaon {

constexpr int G_BM = NS_TILE_M;    // rows of the output tile = UMMA M
constexpr int G_BK = NS_TILE_K;    // K elements per stage (one 128-byte swizzle atom of bf16)
constexpr int G_A_BYTES = G_BM * G_BK * 2;  // 16 KiB
constexpr int G_MAX_BN = 256;
constexpr unsigned G_WAIT_LIMIT = 1u << 22;

struct GemmParams {
  int M, N, K;
  int a_mn, b_mn;    // 0 = K-major operand, 1 = MN-major operand
  int BN;            // 64, 128, 192 or 256
  float alpha, beta;
  const float* dev_scale;    // optional device pair {alpha multiplier, beta multiplier} (e.g. 1/norm)
  const __nv_bfloat16* aux;  // [M, ld_aux] or null (beta ignored)
  long long ld_aux;
  __nv_bfloat16* out;        // [M, ld_out]
  long long ld_out;
  int sym;                   // the product is symmetric (M == N, same operand on both sides): tiles that lie
                             // wholly below the diagonal are not computed; every computed tile also stores
                             // its transpose, which fills them
};

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// A tensor map in global memory is read through a proxy of its own: what was written there since (the host's copy of
// the next tables into the same allocation) has to be acquired before a block's first load with it.
__device__ __forceinline__ void tensormap_acquire(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
}

// 64-bit shared-memory matrix descriptor, 128-byte swizzle.
//  K-major : rows of 128 B (64 bf16 of K), 8-row groups 1024 B apart (SBO); LBO unused (1).
//  MN-major: K rows of 128 B (64 bf16 of MN), 8-K-row groups 1024 B apart (SBO), the next 64 MN
//            elements LBO bytes further (one 64x64 TMA box = 8192 B).
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, bool mn_major) {
  const uint64_t lbo = mn_major ? (8192u >> 4) : 1u;
  const uint64_t sbo = 1024u >> 4;
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (lbo << 16) | (sbo << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ uint32_t umma_idesc(int n, bool a_mn, bool b_mn, int m = G_BM) {
  return (1u << 4) /* D = f32 */ | (1u << 7) /* A = bf16 */ | (1u << 10) /* B = bf16 */ |
         ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_c, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_c), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t v[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32"
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15,"
      " %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}

// ---- persistent, warp-specialised kernel ----
// One CTA per SM walks the output tiles (128 x BN) in a fixed stride.  Warp 0 (one lane) feeds a ring of
// G2_STAGES shared-memory stages by TMA; warp 1 (one lane) issues the MMAs into one of two accumulators in
// tensor memory (2 x 256 columns, allocated once per CTA); warps 2-9 drain the other accumulator
// (tcgen05.ld, fused epilogue, bf16 stores), so that a tile's epilogue runs under the next tile's MMAs.
// In symmetric mode only the tiles that reach the diagonal are enumerated.
// Every wait is bounded: a wait that runs out raises a flag in shared memory, every role leaves its
// loops when it sees the flag, the CTA records the status code and frees its tensor memory.

constexpr int G2_EPI_WARPS = 8;       // two for each quarter of the accumulator's lanes, half the columns each
constexpr int G2_THREADS = 64 + 32 * G2_EPI_WARPS;
constexpr int G2_STAGES = 4;
constexpr int G2_RING = G2_STAGES * (G_A_BYTES + G_MAX_BN * G_BK * 2);   // bytes of the operands' ring
constexpr int G2_STAGE_OUT = 2048;   // bytes an epilogue warp passes its rows through
constexpr int G2_ACC_COLS = 256;   // tensor-memory columns of one accumulator

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// wait with a poll limit, giving up early when another role has failed
__device__ __forceinline__ bool mbar_wait_or_fail(uint64_t* bar, unsigned parity, volatile int* fail) {
  for (unsigned i = 0; i < G_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u && *fail) return false;
  }
  *fail = 1;
  return false;
}

// computed-tile index c -> tile coordinates (rows of tiles are walked in order; in symmetric mode a row
// starts at the first tile that reaches the diagonal)
__device__ __forceinline__ void tile_coords(const GemmParams& p, int tn, int c, int& mi, int& ni) {
  mi = 0;
  while (true) {
    const int skip = p.sym ? min(tn, (mi * G_BM) / p.BN) : 0;
    const int cnt = tn - skip;
    if (c < cnt) { ni = skip + c; return; }
    c -= cnt;
    ++mi;
  }
}

// One product of a grouped launch, in device memory.
struct alignas(128) NsProblem {
  CUtensorMap a, b;
  GemmParams p;
  int tensor;   // whose gradient decides whether it is computed (NsWork::grads)
};

// What a launch works on.  One product (a Newton-Schulz call on its own): `one` is a kernel argument, CTA b takes tiles
// b, b + grid, ...  GROUPED (every matrix of a batch at the same stage of the iteration): the products lie in device
// memory and CTA b takes tiles[begin[b]] .. tiles[begin[b + 1]], shared out by the host so that all finish together; with
// `grads` set, the tiles of matrices without a gradient are passed over.
struct NsWork {
  int total;
  const NsProblem* probs;
  const NsTile* tiles;
  const int* begin;
  const void* const* grads;
  unsigned* status;
};

// The fused epilogue of a tile: a warp stores its 32 rows, from row0 on, of half the tile's columns, from the accumulator's
// lanes at `tmem`.  A lane holds a row; rows go through the warp's 2 KB of shared memory (16-byte pieces, swizzled
// against bank conflicts), so that global memory sees eight rows of 64 consecutive bytes an instruction: straight from the
// lanes, 32 rows of 16 bytes, and of a symmetric product's mirror image 64 bytes, it was the epilogue that the tensor cores
// waited for (DiT list of four blocks, all products: 9.2 ms, and 7.6 without its stores).
__device__ __forceinline__ void store_tile(const GemmParams& p, const uint32_t tmem, const unsigned row0, const int n0, const int half, const float alpha,
                                           const float beta, unsigned char* stage, const int lane) {
  const unsigned row = row0 + lane, M = p.M, N = p.N;
  // (rows of `out` off the 16-byte grid, those of the last product where the length is no multiple of eight, go out as
  // 32 consecutive elements an instruction)
  const bool vec_out = ((reinterpret_cast<uintptr_t>(p.out) | (uintptr_t)(p.ld_out * 2)) & 15) == 0;
  const bool vec_aux = ((reinterpret_cast<uintptr_t>(p.aux) | (uintptr_t)(p.aux ? p.ld_aux * 2 : 0)) & 15) == 0;
  const int pr = lane >> 2, ps = lane & 3;   // the row (of eight) and the piece of it that this lane moves to and from memory
  auto piece = [&](int r, int s) { return reinterpret_cast<uint4*>(stage + r * 64 + ((s ^ ((r >> 1) & 3)) << 4)); };
  for (int c0 = half * (p.BN / 2); c0 < (half + 1) * (p.BN / 2); c0 += 32) {
    const unsigned col = (unsigned)n0 + c0;
    uint32_t v[32];
    tmem_ld32(tmem + (uint32_t)c0, v);
    const bool full = vec_aux && col + 32 <= N && (!p.sym || (vec_out && row0 + 32 <= M));   // (the warp's)
    uint4 x[4];
    if (full && p.aux) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned r = row0 + i * 8 + pr;
        x[i] = r < M ? *reinterpret_cast<const uint4*>(p.aux + (long long)r * p.ld_aux + col + ps * 8) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (full) {
      uint32_t w[16];
      if (p.aux) {
#pragma unroll
        for (int i = 0; i < 4; ++i) *piece(i * 8 + pr, ps) = x[i];
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = *piece(lane, q);
        __syncwarp();
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const uint32_t xw = (&x[e >> 2].x)[e & 3];
        w[e] = pack_bf16_rn(__uint_as_float(v[2 * e]) * alpha + beta * bf16lo(xw), __uint_as_float(v[2 * e + 1]) * alpha + beta * bf16hi(xw));
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) *piece(lane, q) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
      __syncwarp();
      if (vec_out) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned r = row0 + i * 8 + pr;
          const uint4 o = *piece(i * 8 + pr, ps);
          if (r < M) *reinterpret_cast<uint4*>(p.out + (long long)r * p.ld_out + col + ps * 8) = o;
        }
      } else {
        unsigned short* orow = reinterpret_cast<unsigned short*>(p.out + (long long)row0 * p.ld_out + col) + lane;
        const int rows = (int)min(32u, M > row0 ? M - row0 : 0u);
#pragma unroll 4
        for (int i = 0; i < rows; ++i, orow += p.ld_out) *orow = reinterpret_cast<const unsigned short*>(piece(i, lane >> 3))[lane & 7];
      }
      __syncwarp();
      if (p.sym) {   // the mirror image: out[col + j, row0 ..], a column of the block a row of it
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          reinterpret_cast<unsigned short*>(piece(2 * e, lane >> 3))[lane & 7] = (unsigned short)(w[e] & 0xffffu);
          reinterpret_cast<unsigned short*>(piece(2 * e + 1, lane >> 3))[lane & 7] = (unsigned short)(w[e] >> 16);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(p.out + (long long)(col + i * 8 + pr) * p.ld_out + row0 + ps * 8) = *piece(i * 8 + pr, ps);
        __syncwarp();
      }
    } else if (row < M && col < N) {   // a ragged end: element by element
      __nv_bfloat16* orow = p.out + (long long)row * p.ld_out + col;
      const __nv_bfloat16* arow = p.aux ? p.aux + (long long)row * p.ld_aux + col : nullptr;
      const int left = (int)min(32u, N - col);
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        if (e >= left) break;
        const float a = arow ? __bfloat162float(arow[e]) : 0.0f;
        const __nv_bfloat16 r = __float2bfloat16_rn(__uint_as_float(v[e]) * alpha + beta * a);
        orow[e] = r;
        if (p.sym) p.out[(long long)(col + e) * p.ld_out + row] = r;
      }
    }
  }
}

template <bool GROUPED>
__global__ void __launch_bounds__(G2_THREADS, 1)
ns_gemm_kernel(const __grid_constant__ NsProblem one, const __grid_constant__ NsWork work) {
  extern __shared__ __align__(1024) unsigned char gsm[];
  __shared__ __align__(8) uint64_t full_bar[G2_STAGES];
  __shared__ __align__(8) uint64_t empty_bar[G2_STAGES];
  __shared__ __align__(8) uint64_t accf_bar[2];   // accumulator complete (MMA -> epilogue)
  __shared__ __align__(8) uint64_t acce_bar[2];   // accumulator drained (epilogue -> MMA)
  __shared__ uint32_t tmem_base_s;
  __shared__ int fail_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int stage_bytes = G_A_BYTES + G_MAX_BN * G_BK * 2;
  // 1024-byte aligned tile base (the swizzle pattern is a function of address bits 4..9)
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gsm) + 1023) & ~uintptr_t(1023));
  const int c_first = GROUPED ? work.begin[blockIdx.x] : (int)blockIdx.x;
  const int c_end = GROUPED ? work.begin[blockIdx.x + 1] : work.total, c_step = GROUPED ? 1 : (int)gridDim.x;
  // the product and the tile with number c
  auto tile_of = [&](int c, int& mi, int& ni) -> const NsProblem* {
    if constexpr (GROUPED) {
      const NsTile t = work.tiles[c];
      mi = t.mi; ni = t.ni;
      return work.probs + t.prob;
    } else {
      tile_coords(one.p, ns_tiles(one.p.N, one.p.BN), c, mi, ni);
      return &one;
    }
  };
  auto passed_over = [&](const NsProblem* pr) { return GROUPED && work.grads && work.grads[pr->tensor] == nullptr; };
  volatile int* fail = &fail_s;

  if (tid == 0) {
    for (int s = 0; s < G2_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&accf_bar[b], 1); mbar_init(&acce_bar[b], G2_EPI_WARPS); }
    fail_s = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(2u * G2_ACC_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_s;

  if (warp == 0) {
    // ---- TMA producer ----
    if (lane == 0) {
      unsigned it = 0;
      const NsProblem* last = nullptr;
      for (int c = c_first; c < c_end && !*fail; c += c_step) {
        int mi, ni;
        const NsProblem* pr = tile_of(c, mi, ni);
        if (passed_over(pr)) continue;
        const CUtensorMap *mapA = &pr->a, *mapB = &pr->b;
        if (GROUPED && pr != last) {   // (the one product's maps are kernel parameters)
          tensormap_acquire(mapA);
          tensormap_acquire(mapB);
          last = pr;
        }
        const int kblocks = ns_tiles(pr->p.K, G_BK), BN = pr->p.BN;
        const bool a_mn = pr->p.a_mn != 0, b_mn = pr->p.b_mn != 0;
        const unsigned tx = (unsigned)(G_A_BYTES + BN * G_BK * 2);
        const int m0 = mi * G_BM, n0 = ni * BN;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % G2_STAGES;
          const unsigned use = it / G2_STAGES;
          if (use > 0 && !mbar_wait_or_fail(&empty_bar[s], (use - 1u) & 1u, fail)) break;
          unsigned char* a_dst = tiles + (size_t)s * stage_bytes;
          unsigned char* b_dst = a_dst + G_A_BYTES;
          mbar_expect_tx(&full_bar[s], tx);
          const int k0 = kb * G_BK;
          if (a_mn) {
            for (int j = 0; j < G_BM / 64; ++j) tma_load_2d(a_dst + j * 8192, mapA, m0 + 64 * j, k0, &full_bar[s]);
          } else {
            tma_load_2d(a_dst, mapA, k0, m0, &full_bar[s]);
          }
          if (b_mn) {
            for (int j = 0; j < BN / 64; ++j) tma_load_2d(b_dst + j * 8192, mapB, n0 + 64 * j, k0, &full_bar[s]);
          } else {
            tma_load_2d(b_dst, mapB, k0, n0, &full_bar[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----
    if (lane == 0) {
      unsigned it = 0, tcount = 0;
      for (int c = c_first; c < c_end && !*fail; c += c_step) {
        int mi, ni;
        const NsProblem* pr = tile_of(c, mi, ni);
        if (passed_over(pr)) continue;
        const int kblocks = ns_tiles(pr->p.K, G_BK);
        const bool a_mn = pr->p.a_mn != 0, b_mn = pr->p.b_mn != 0;
        const uint32_t idesc = umma_idesc(pr->p.BN, a_mn, b_mn);
        const unsigned buf = tcount & 1u, use = tcount >> 1;
        ++tcount;
        if (use > 0 && !mbar_wait_or_fail(&acce_bar[buf], (use - 1u) & 1u, fail)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_acc = tmem_base + buf * G2_ACC_COLS;
        bool ok = true;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % G2_STAGES;
          if (!mbar_wait_or_fail(&full_bar[s], (it / G2_STAGES) & 1u, fail)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = smem_u32(tiles + (size_t)s * stage_bytes);
          const uint32_t b_addr = a_addr + G_A_BYTES;
#pragma unroll
          for (int k = 0; k < G_BK / 16; ++k) {
            const uint64_t da = umma_desc(a_addr + (a_mn ? k * 2048 : k * 32), a_mn);
            const uint64_t db = umma_desc(b_addr + (b_mn ? k * 2048 : k * 32), b_mn);
            umma_f16(tmem_acc, da, db, idesc, (kb | k) ? 1u : 0u);
          }
          umma_commit(&empty_bar[s]);  // frees the stage once these MMAs have read it
        }
        if (!ok) break;
        umma_commit(&accf_bar[buf]);   // accumulator complete
      }
    }
  } else {
    // ---- epilogue: warps 2..9; a warp may touch the 32 tensor-memory lanes of its quarter (warp % 4) ----
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    unsigned tcount = 0;
    for (int c = c_first; c < c_end; c += c_step) {
      int mi, ni;
      const NsProblem* pr = tile_of(c, mi, ni);
      if (passed_over(pr)) continue;
      const GemmParams& p = pr->p;
      const float alpha = p.dev_scale ? p.alpha * p.dev_scale[0] : p.alpha;
      const float beta = p.dev_scale ? p.beta * p.dev_scale[1] : p.beta;
      const int m0 = mi * G_BM, n0 = ni * p.BN;
      const unsigned buf = tcount & 1u, use = tcount >> 1;
      ++tcount;
      if (!mbar_wait_or_fail(&accf_bar[buf], use & 1u, fail)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_acc = tmem_base + buf * G2_ACC_COLS;
      const unsigned row0 = (unsigned)m0 + quarter * 32;   // (beyond 2^31 in the last tile of the tallest matrix)
      store_tile(p, tmem_acc + ((uint32_t)(quarter * 32) << 16), row0, n0, half, alpha, beta, tiles + G2_RING + (warp - 2) * G2_STAGE_OUT, lane);
      // this warp has read its part of the accumulator: hand the buffer back to the MMA issuer
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acce_bar[buf]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && fail_s) atomicCAS(work.status, 0u, 20001u);
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * G2_ACC_COLS) : "memory");
  }
}

// ---- pairs of CTAs ----
// The grouped launch of large batches: a cluster of two CTAs computes tiles of 256 x BN (tcgen05 cta_group::2).  Each CTA
// keeps 128 rows of A, HALF of B's columns, and its 128 rows of the accumulator, so that a k-block brings 32 KB into
// its shared memory where a tile of one CTA takes 48, and the MMAs read as much less of it.  What that saves is energy: alone
// on the machine both take the same time (DiT list of four blocks, all products: 8.4 and 8.3 ms), but long products run at
// the power limit, and a step with pairs takes 10.9 ms, with single CTAs 11.4.
// Both CTAs' loads (no multicast) complete on the LEADER's full barrier; its MMA thread multiplies for both and commits to
// both CTAs' barriers; both CTAs' epilogue warps hand the accumulator back to the leader.  Roles, bounds of the waits and
// the share-out of tiles as above.
constexpr int P_MAX_B = 128 * G_BK * 2;                    // bytes of a CTA's half of B at BN = 256
constexpr int P_STAGES = 6;
static_assert(P_STAGES * (G_A_BYTES + P_MAX_B) <= G2_RING, "a pair's ring lies where a single CTA's does");

__device__ __forceinline__ uint32_t leader_addr(const void* p) {   // this shared-memory address in the pair's first CTA
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_c, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_c), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {   // to the barrier at this address in both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((unsigned short)3)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// Wait with a poll limit (a poll suspends for about a microsecond at most: a second in all), giving up early when another role
// has failed; what the other CTA wrote before it arrived is visible.
constexpr unsigned P_WAIT_LIMIT = 1u << 20;
__device__ __forceinline__ bool pair_wait(uint64_t* bar, unsigned parity, volatile int* fail) {
  for (unsigned i = 0; i < P_WAIT_LIMIT; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(1000u) : "memory");
    if (ok) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  return false;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G2_THREADS, 1) ns_pair_kernel(const __grid_constant__ NsWork work) {
  extern __shared__ __align__(1024) unsigned char gsm[];
  __shared__ __align__(8) uint64_t full_bar[P_STAGES];    // (the leader's are used)
  __shared__ __align__(8) uint64_t empty_bar[P_STAGES];
  __shared__ __align__(8) uint64_t accf_bar[2];
  __shared__ __align__(8) uint64_t acce_bar[2];           // (the leader's are used)
  __shared__ uint32_t tmem_base_s;
  __shared__ int fail_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  constexpr int stage_bytes = G_A_BYTES + P_MAX_B;
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gsm) + 1023) & ~uintptr_t(1023));
  const int pair = (int)(blockIdx.x >> 1);
  const int c_first = work.begin[pair], c_end = work.begin[pair + 1];
  auto passed_over = [&](const NsProblem* pr) { return work.grads && work.grads[pr->tensor] == nullptr; };
  volatile int* fail = &fail_s;

  if (tid == 0) {
    for (int s = 0; s < P_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&accf_bar[b], 1); mbar_init(&acce_bar[b], 2 * G2_EPI_WARPS); }
    fail_s = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(2u * G2_ACC_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();   // both CTAs' barriers are set up and their tensor memory is there
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_s;

  if (warp == 0) {
    // ---- TMA producer, one in each CTA: its rows of A, its half of B ----
    if (lane == 0) {
      unsigned it = 0;
      const NsProblem* last = nullptr;
      bool ok = true;
      for (int c = c_first; ok && c < c_end && !*fail; ++c) {
        const NsTile t = work.tiles[c];
        const NsProblem* pr = work.probs + t.prob;
        if (passed_over(pr)) continue;
        const CUtensorMap *mapA = &pr->a, *mapB = &pr->b;
        if (pr != last) {
          tensormap_acquire(mapA);
          tensormap_acquire(mapB);
          last = pr;
        }
        const int kblocks = ns_tiles(pr->p.K, G_BK), half = pr->p.BN / 2;
        const bool a_mn = pr->p.a_mn != 0, b_mn = pr->p.b_mn != 0;
        const unsigned tx = 2u * (unsigned)(G_A_BYTES + half * G_BK * 2);   // both CTAs'
        const int m0 = t.mi * (2 * G_BM) + (int)rank * G_BM, n0 = t.ni * pr->p.BN + (int)rank * half;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % P_STAGES;
          const unsigned use = it / P_STAGES;
          if (use > 0 && !pair_wait(&empty_bar[s], (use - 1u) & 1u, fail)) { ok = false; break; }
          unsigned char* a_dst = tiles + (size_t)s * stage_bytes;
          unsigned char* b_dst = a_dst + G_A_BYTES;
          if (rank == 0) mbar_expect_tx(&full_bar[s], tx);
          const uint32_t bar = leader_addr(&full_bar[s]);
          const int k0 = kb * G_BK;
          if (a_mn) {
            for (int j = 0; j < G_BM / 64; ++j) tma_load_2d_pair(a_dst + j * 8192, mapA, m0 + 64 * j, k0, bar);
          } else {
            tma_load_2d_pair(a_dst, mapA, k0, m0, bar);
          }
          if (b_mn) {
            for (int j = 0; j < half / 64; ++j) tma_load_2d_pair(b_dst + j * 8192, mapB, n0 + 64 * j, k0, bar);
          } else {
            tma_load_2d_pair(b_dst, mapB, k0, n0, bar);
          }
        }
      }
      // until the last commits have arrived here: this CTA stays while the pair's MMAs read its shared memory
      for (unsigned j = it > P_STAGES ? it - P_STAGES : 0u; ok && j < it; ++j)
        ok = pair_wait(&empty_bar[j % P_STAGES], (j / P_STAGES) & 1u, fail);
    }
  } else if (warp == 1) {
    // ---- MMA issuer of the pair ----
    if (rank == 0 && lane == 0) {
      unsigned it = 0, tcount = 0;
      for (int c = c_first; c < c_end && !*fail; ++c) {
        const NsProblem* pr = work.probs + work.tiles[c].prob;
        if (passed_over(pr)) continue;
        const int kblocks = ns_tiles(pr->p.K, G_BK);
        const bool a_mn = pr->p.a_mn != 0, b_mn = pr->p.b_mn != 0;
        const uint32_t idesc = umma_idesc(pr->p.BN, a_mn, b_mn, 2 * G_BM);
        const unsigned buf = tcount & 1u, use = tcount >> 1;
        ++tcount;
        if (use > 0 && !pair_wait(&acce_bar[buf], (use - 1u) & 1u, fail)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_acc = tmem_base + buf * G2_ACC_COLS;
        bool ok = true;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % P_STAGES;
          if (!pair_wait(&full_bar[s], (it / P_STAGES) & 1u, fail)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = smem_u32(tiles + (size_t)s * stage_bytes);
          const uint32_t b_addr = a_addr + G_A_BYTES;
#pragma unroll
          for (int k = 0; k < G_BK / 16; ++k) {
            const uint64_t da = umma_desc(a_addr + (a_mn ? k * 2048 : k * 32), a_mn);
            const uint64_t db = umma_desc(b_addr + (b_mn ? k * 2048 : k * 32), b_mn);
            umma_f16_pair(tmem_acc, da, db, idesc, (kb | k) ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[s]);
        }
        if (!ok) break;
        umma_commit_pair(&accf_bar[buf]);
      }
    }
  } else {
    // ---- epilogue of this CTA's 128 rows: warps 2..9 ----
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    unsigned tcount = 0;
    for (int c = c_first; c < c_end; ++c) {
      const NsTile t = work.tiles[c];
      const NsProblem* pr = work.probs + t.prob;
      if (passed_over(pr)) continue;
      const GemmParams& p = pr->p;
      const float alpha = p.dev_scale ? p.alpha * p.dev_scale[0] : p.alpha;
      const float beta = p.dev_scale ? p.beta * p.dev_scale[1] : p.beta;
      const unsigned buf = tcount & 1u, use = tcount >> 1;
      ++tcount;
      if (!pair_wait(&accf_bar[buf], use & 1u, fail)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned row0 = (unsigned)t.mi * (2u * G_BM) + rank * G_BM + quarter * 32;
      store_tile(p, tmem_base + buf * G2_ACC_COLS + ((uint32_t)(quarter * 32) << 16), row0, t.ni * p.BN, half, alpha, beta,
                 tiles + G2_RING + (warp - 2) * G2_STAGE_OUT, lane);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_addr(&acce_bar[buf]));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && fail_s) atomicCAS(work.status, 0u, 20001u);
  cluster_sync();   // neither CTA leaves, or frees its tensor memory, before the other is done with both
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * G2_ACC_COLS) : "memory");
  }
}

}  // namespace kaon

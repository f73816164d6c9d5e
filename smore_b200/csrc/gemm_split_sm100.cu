// fp32-accurate matrix products on the bf16 tensor cores, for dot-product scoring against a shared list.
//
// Every fp32 operand is split once, ahead of the product, into three bf16 planes whose sum is the operand
// (8 + 8 + 8 significant bits); the product is the sum of plane products.  A GEMM that splits its operands
// inside the main loop repeats that work for every tile that reads them and keeps the tensor cores waiting
// for it: the three products of a 4096 x 8192 x 1000 step took 2.09 ms that way.  Here the main loop only
// moves bf16 tiles (TMA) and issues tcgen05.mma.
//
//   split_planes_kernel   fp32 [rows, cols] -> planes [3][rows][ld] and / or transposed [3][cols][ld_t]; all
//                         products then have both operands K-major, and one GEMM kernel serves them
//   split_gemm_kernel     D[M, N] = A . B^T, A planes [3][M][K], B planes [3][N][K]; one 128 x 256 tile per
//                         CTA at a time, a fixed set of CTAs walks the tiles.  Warp 0 issues the TMA loads,
//                         warp 1 the MMAs, warps 2..9 own the result.
//   sum_parts_kernel      adds the parts of a reduction that was cut to fill the SMs
//
// Precision.  Six of the nine plane products are taken: with round-to-nearest planes the other three (second
// by third, third by second and third by third plane) are together below 2^-25 of the operands' product, half of
// what rounding it to fp32 may cost.  The error comes from the additions instead: a tensor-memory accumulator
// is added to once per 16 products, with truncation, so it takes the small products first and holds kChunk = 32
// of the reduction; it is then added, rounding to nearest, to the running sums in the registers of warps 2..9,
// while the MMAs go on in a second accumulator; in reductions of more than kNoFlush chunks those
// go to a tile of scratch in L2 every kFlush, so no
// chain of additions is long.  Relative error (2-norm) of the scores of 4096 x 8192 x 1000 against 64 bits:
// 1.5e-7 with the splitting template, 3.2e-7 with nine products in chunks of 64, 1.2e-7 like this; its
// gradients 2.8e-7 and 4.1e-7, 3.4e-7 and 3.7e-7, 1.1e-7 and 1.2e-7.  The three products take 0.97 ms (nine
// products in chunks of 64: 1.19; the scratch costs 0.07, without it the gradients are at 2.1e-7 and 3.0e-7).  A reduction of
// up to kNoFlush chunks stays in registers, which is below the template's error too.
//
// Every wait on an mbarrier is bounded; one that runs out sets kStatusCopyWait and lets the CTA finish.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "bulk_copy.cuh"
#include "common.cuh"
#include "gemm_split.cuh"

namespace smore {

static __device__ int g_split_status = 0;

// ----------------------------------------------------------------------------------------
// planes
// ----------------------------------------------------------------------------------------

constexpr int kSplitTile = 64;

__device__ __forceinline__ void split3(float x, __nv_bfloat16 (&p)[3]) {
  p[0] = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(p[0]);        // exact
  p[1] = __float2bfloat16_rn(r);
  p[2] = __float2bfloat16_rn(r - __bfloat162float(p[1]));
}

// One 64 x 64 block per CTA, the blocks of a row of blocks next to each other.  plain: [3][rows][ld],
// transposed: [3][cols][ld_t]; either may be nullptr.  x: [rows, cols], ld_x floats from row to row.
__global__ void __launch_bounds__(256)
    split_planes_kernel(const float* __restrict__ x, size_t ld_x, int rows, int cols, __nv_bfloat16* __restrict__ plain,
                        size_t ld, __nv_bfloat16* __restrict__ transposed, size_t ld_t) {
  __shared__ float tile[kSplitTile][kSplitTile + 1];
  const unsigned col_blocks = (unsigned)(cols + kSplitTile - 1) / kSplitTile;
  const int r0 = (int)(blockIdx.x / col_blocks) * kSplitTile, c0 = (int)(blockIdx.x % col_blocks) * kSplitTile;
  const int t = threadIdx.x;
  {
    // 4 floats per thread and pass; cols is a multiple of 4
    const int c = c0 + (t & 15) * 4;
    for (int r = t >> 4; r < kSplitTile; r += 16) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r0 + r < rows && c < cols) v = __ldg(reinterpret_cast<const float4*>(x + (size_t)(r0 + r) * ld_x + c));
      float* d = &tile[r][(t & 15) * 4];
      d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
  }
  __syncthreads();
  // a thread writes two consecutive elements of each plane
  auto write = [&](__nv_bfloat16* out, size_t stride, size_t plane, int a0, int n_a, int b0, int n_b, bool flip) {
    const int b = (t & 31) * 2;
    for (int a = t >> 5; a < kSplitTile; a += 8) {
      if (a0 + a >= n_a || b0 + b >= n_b) continue;
      __nv_bfloat16 u[3], v[3];
      split3(flip ? tile[b][a] : tile[a][b], u);
      split3(flip ? tile[b + 1][a] : tile[a][b + 1], v);
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        __nv_bfloat162 w;
        w.x = u[p];
        w.y = v[p];
        // (the row pitch is even and at least n_b: the second element of an odd end lands in the padding)
        *reinterpret_cast<__nv_bfloat162*>(out + p * plane + (size_t)(a0 + a) * stride + b0 + b) = w;
      }
    }
  };
  if (plain) write(plain, ld, (size_t)rows * ld, r0, rows, c0, cols, false);
  if (transposed) write(transposed, ld_t, (size_t)cols * ld_t, c0, cols, r0, rows, true);
}

// ----------------------------------------------------------------------------------------
// the product
// ----------------------------------------------------------------------------------------

constexpr int kTileM = 128, kTileN = 256;
constexpr int kBlockK = 32;                      // reduction per pipeline stage: 64-byte rows, 64-byte swizzle
constexpr int kChunk = 32;                       // reduction per tensor-memory accumulator
constexpr int kBlocksPerChunk = kChunk / kBlockK;
constexpr int kFlush = 16, kNoFlush = 32;        // chunks whose sum is kept in registers; of a whole reduction
constexpr int kStages = 3;
constexpr int kPlaneA = kTileM * kBlockK * 2, kPlaneB = kTileN * kBlockK * 2;    // bytes
constexpr int kStageBytes = 3 * (kPlaneA + kPlaneB);                             // 72 KB
constexpr int kGemmThreads = 320, kResultThreads = 256;
constexpr int kGemmSmem = kStages * kStageBytes + 1024 /* alignment */;

struct GemmArgs {
  float* d;              // [M, N] row-major
  size_t ld_d;           // floats from row to row of d
  float* spill;          // [CTAs][128 x 256], for reductions longer than kNoFlush chunks
  float* part_sums;      // [parts][M][N] when the reduction is cut, else nullptr
  int M, N;
  bool add;              // add to d
  int k_blocks;          // stages of the whole reduction
  int parts;             // parts the reduction is cut into
  int tiles_m, tiles_n;
};

__device__ __forceinline__ bool wait_bar(uint64_t* bar, unsigned parity) {
  if (bulk::barrier_wait(bar, parity)) return true;
  atomicOr(&g_split_status, kStatusCopyWait);
  return false;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          bulk::smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bulk::smem_addr(bar))
      : "memory");
}

// shared-memory descriptor of a K-major operand tile with 64-byte rows: 64-byte swizzle, 8-row groups 512 B apart
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem) {
  return (uint64_t)((smem & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)4 << 61);
}

// What a product does with the buffer the tensor core reads A through: neighbours with the same A tile read it once.
enum KeepA { kOnce, kFill, kUse, kLastUse };
template <int KEEP>
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
#define SMORE_MMA(QUALIFIER)                                                    \
  asm volatile(                                                                 \
      "{\n\t.reg .pred p;\n\t"                                                  \
      "setp.ne.b32 p, %4, 0;\n\t"                                               \
      "tcgen05.mma.cta_group::1.kind::f16" QUALIFIER " [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), \
      "l"(a), "l"(b), "r"(idesc), "r"((unsigned)accumulate)                     \
      : "memory")
  if constexpr (KEEP == kFill) SMORE_MMA(".collector::a::fill");
  else if constexpr (KEEP == kUse) SMORE_MMA(".collector::a::use");
  else if constexpr (KEEP == kLastUse) SMORE_MMA(".collector::a::lastuse");
  else SMORE_MMA("");
#undef SMORE_MMA
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bulk::smem_addr(bar))
               : "memory");
}

__device__ __forceinline__ void barrier_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bulk::smem_addr(bar)) : "memory");
}

// adds 16 consecutive columns of this warp's 32 tensor-memory lanes
__device__ __forceinline__ void tmem_add16(uint32_t addr, float* sum) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) sum[i] += __uint_as_float(r[i]);
}

__device__ __forceinline__ void store_sector(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
               "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// the part of the work item `item` covers: tile, range of stages, part of the reduction
struct Item {
  int m0, n0, k_begin, k_end, part;
};
__device__ __forceinline__ Item item_of(const GemmArgs& g, int item) {
  // parts outermost, then tiles row by row of B's tiles: CTAs that run together share operand rows in L2
  const int tiles = g.tiles_m * g.tiles_n;
  const int part = item / tiles, t = item - part * tiles;
  const int tn = t / g.tiles_m, tm = t - tn * g.tiles_m;
  // parts are whole chunks
  const int chunks = (g.k_blocks + kBlocksPerChunk - 1) / kBlocksPerChunk;
  const int per = (chunks + g.parts - 1) / g.parts;
  return {tm * kTileM, tn * kTileN, min(g.k_blocks, part * per * kBlocksPerChunk),
          min(g.k_blocks, (part + 1) * per * kBlocksPerChunk), part};
}

__global__ void __launch_bounds__(kGemmThreads, 1)
    split_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, GemmArgs g) {
  extern __shared__ unsigned char gemm_smem[];
  __shared__ uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2], drained;
  __shared__ uint32_t tmem_base_sh;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gemm_smem) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      bulk::barrier_init(full + s, 1);
      bulk::barrier_init(empty + s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      bulk::barrier_init(acc_full + i, 1);
      bulk::barrier_init(acc_empty + i, 8);   // one arrival per result warp
    }
    bulk::barrier_init(&drained, 1);
    bulk::fence_barrier_init();
  }
  if (warp == 1) {
    // both accumulators: all 512 columns of the SM's tensor memory (one CTA per SM)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bulk::smem_addr(&tmem_base_sh)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_sh;
  const int items = g.tiles_m * g.tiles_n * g.parts;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      unsigned parity = 0;
      long long loads = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const Item it = item_of(g, item);
        for (int kb = it.k_begin; kb < it.k_end; ++kb) {
          ok = wait_bar(empty + stage, parity ^ 1u);
          if (!ok) break;
          unsigned char* a = ring + (size_t)stage * kStageBytes;
          bulk::barrier_expect(full + stage, kStageBytes);
          tma_load_3d(a, &map_a, kb * kBlockK, it.m0, 0, full + stage);
          tma_load_3d(a + 3 * kPlaneA, &map_b, kb * kBlockK, it.n0, 0, full + stage);
          ++loads;
          if (++stage == kStages) {
            stage = 0;
            parity ^= 1u;
          }
        }
      }
      // no copy of this CTA is still in flight when it ends, whatever became of its readers
      for (long long l = loads > kStages ? loads - kStages : 0; l < loads; ++l)
        wait_bar(full + l % kStages, (unsigned)(l / kStages) & 1u);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // D fp32, A and B bf16, both K-major, N / 8, M / 16
      constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kTileN / 8) << 17) | ((kTileM / 16) << 24);
      int stage = 0, acc = 0;
      unsigned parity = 0, acc_parity = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const Item it = item_of(g, item);
        for (int kb0 = it.k_begin; kb0 < it.k_end && ok; kb0 += kBlocksPerChunk) {
          ok = wait_bar(acc_empty + acc, acc_parity ^ 1u);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t d = tmem + acc * kTileN;
          for (int kb = kb0; kb < min(it.k_end, kb0 + kBlocksPerChunk); ++kb) {
            ok = wait_bar(full + stage, parity);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = bulk::smem_addr(ring + (size_t)stage * kStageBytes), b = a + 3 * kPlaneA;
            auto product = [&](auto keep, int k, int pa, int pb, bool add) {
              mma_bf16<decltype(keep)::value>(d, operand_desc(a + pa * kPlaneA + k * 32), operand_desc(b + pb * kPlaneB + k * 32),
                                              kIdesc, add);
            };
            using Once = std::integral_constant<int, kOnce>;
            using Fill = std::integral_constant<int, kFill>;
            using Use = std::integral_constant<int, kUse>;
            using Last = std::integral_constant<int, kLastUse>;
            // plane products, the large ones last; those that share an A tile next to each other: shared memory
            // is read at 96 bytes a cycle otherwise, next to the copies that fill it at 48
            product(Once{}, 0, 2, 0, kb > kb0);
            product(Fill{}, 0, 1, 1, true);
            product(Last{}, 0, 1, 0, true);
            product(Once{}, 1, 2, 0, true);
            product(Fill{}, 1, 1, 1, true);
            product(Last{}, 1, 1, 0, true);
            product(Fill{}, 0, 0, 2, true);
            product(Last{}, 0, 0, 1, true);
            product(Fill{}, 1, 0, 2, true);
            product(Use{}, 1, 0, 1, true);
            product(Last{}, 1, 0, 0, true);
            product(Once{}, 0, 0, 0, true);
            mma_commit(empty + stage);
            if (++stage == kStages) {
              stage = 0;
              parity ^= 1u;
            }
          }
          mma_commit(acc_full + acc);
          if (++acc == 2) {
            acc = 0;
            acc_parity ^= 1u;
          }
        }
      }
      mma_commit(&drained);      // nor is a product
      wait_bar(&drained, 0);
    }
  } else {
    // a warp reads the tensor-memory lanes (result rows) of its quarter, and half of the tile's columns
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    int acc = 0;
    unsigned acc_parity = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const Item it = item_of(g, item);
      // the running sums leave for this CTA's tile of `spill` now and then, laid out so that a warp's
      // accesses are contiguous
      float4* spill = reinterpret_cast<float4*>(g.spill) + (size_t)blockIdx.x * (kTileM * kTileN / 4) + (threadIdx.x - 64);
      const int run = (it.k_end - it.k_begin > kNoFlush * kBlocksPerChunk ? kFlush : kNoFlush) * kBlocksPerChunk;
#pragma unroll 1
      for (int kb1 = it.k_begin; kb1 < it.k_end && ok; kb1 += run) {
        float sum[kTileN / 2];
#pragma unroll
        for (int i = 0; i < kTileN / 2; ++i) sum[i] = 0.f;
#pragma unroll 1
        for (int kb0 = kb1; kb0 < min(it.k_end, kb1 + run); kb0 += kBlocksPerChunk) {
          ok = wait_bar(acc_full + acc, acc_parity);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int c = 0; c < kTileN / 2; c += 16)
            tmem_add16(tmem + lanes + acc * kTileN + half * (kTileN / 2) + c, sum + c);
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) barrier_arrive(acc_empty + acc);
          if (++acc == 2) {
            acc = 0;
            acc_parity ^= 1u;
          }
        }
        const bool first = kb1 == it.k_begin;
        if (kb1 + run < it.k_end) {
          if (first) {
#pragma unroll
            for (int c = 0; c < kTileN / 2; c += 4)
              __stcg(spill + c / 4 * kResultThreads, make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]));
          } else {
#pragma unroll
            for (int c = 0; c < kTileN / 2; c += 4)
              atomicAdd(spill + c / 4 * kResultThreads, make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]));
          }
          continue;
        }
        if (!first) {
#pragma unroll
          for (int c = 0; c < kTileN / 2; c += 4) {
            const float4 v = __ldcg(spill + c / 4 * kResultThreads);
            sum[c] += v.x;
            sum[c + 1] += v.y;
            sum[c + 2] += v.z;
            sum[c + 3] += v.w;
          }
        }
        const int m = it.m0 + quarter * 32 + lane, n0 = it.n0 + half * (kTileN / 2);
        float* out = g.part_sums ? g.part_sums + ((size_t)it.part * g.M + m) * g.N + n0 : g.d + (size_t)m * g.ld_d + n0;
        const int n = ok && m < g.M ? g.N - n0 : 0;     // columns of the result here; N is a multiple of 4
        const bool add = g.add && !g.part_sums;
        const bool sectors = !add && ((reinterpret_cast<uintptr_t>(out) & 31) | (n & 7)) == 0;
        // A thread owns a row of the tile, so a warp's stores go to 32 rows, and the MMAs wait for them: a whole
        // 32-byte sector per store where rows are aligned (scores of 4096 x 8192 x 1000: 393 -> 351 us, of
        // 4096 x 8192 x 128: 114 -> 68 us), else 16 bytes.
        if (sectors) {
#pragma unroll
          for (int c = 0; c < kTileN / 2; c += 8)
            if (c < n) store_sector(out + c, sum + c);
        }
#pragma unroll
        for (int c = 0; c < kTileN / 2; c += 4) {
          if (sectors || c >= n) continue;
          const float4 v = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
          if (add) atomicAdd(reinterpret_cast<float4*>(out + c), v);
          else *reinterpret_cast<float4*>(out + c) = v;
        }
        __syncwarp();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// d (+)= the parts' sums, in the order of the parts
__global__ void __launch_bounds__(256) sum_parts_kernel(const float* __restrict__ part_sums, int parts, float* __restrict__ d,
                                                        size_t ld_d, int M, int N, bool add) {
  const size_t n4 = (size_t)N >> 2, total = (size_t)M * n4;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t m = i / n4, c = i - m * n4;
    float4 s = __ldcg(reinterpret_cast<const float4*>(part_sums) + i);
    for (int p = 1; p < parts; ++p) {
      const float4 v = __ldcg(reinterpret_cast<const float4*>(part_sums) + p * total + i);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    float4* out = reinterpret_cast<float4*>(d + m * ld_d) + c;
    if (add) {
      const float4 v = *out;
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *out = s;
  }
}

// ----------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiled encode_tiled() {
  static EncodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiled>(p);
  }();
  return fn;
}

size_t split_pitch(size_t k) { return (k + 7) & ~(size_t)7; }
size_t split_plane_bytes(size_t rows, size_t k) { return (3 * rows * split_pitch(k) * 2 + 1023) & ~(size_t)1023; }

int split_planes(const float* x, size_t ld_x, size_t rows, size_t cols, void* plain, void* transposed, cudaStream_t st) {
  const size_t blocks = ((cols + kSplitTile - 1) / kSplitTile) * ((rows + kSplitTile - 1) / kSplitTile);
  if (blocks > 0x7fffffff) return fail(SMORE_ERR_TOO_LARGE, "dot: operand of %zu x %zu is too large", rows, cols);
  split_planes_kernel<<<(unsigned)blocks, 256, 0, st>>>(x, ld_x, (int)rows, (int)cols, static_cast<__nv_bfloat16*>(plain),
                                                        split_pitch(cols), static_cast<__nv_bfloat16*>(transposed),
                                                        split_pitch(rows));
  return check_launch("split_planes_kernel");
}

// map of planes [3][rows][pitch(k)]: boxes of kBlockK x box_rows x 3
static int plane_map(CUtensorMap* map, const void* planes, size_t rows, size_t k, int box_rows) {
  const size_t pitch = split_pitch(k) * 2;
  const cuuint64_t dims[3] = {k, rows, 3}, strides[2] = {pitch, pitch * rows};
  const cuuint32_t box[3] = {(cuuint32_t)kBlockK, (cuuint32_t)box_rows, 3}, ones[3] = {1, 1, 1};
  EncodeTiled encode = encode_tiled();
  if (!encode) return fail(SMORE_ERR_CUDA, "dot: cuTensorMapEncodeTiled is not available");
  const CUresult rc = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(planes), dims, strides, box, ones,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return fail(SMORE_ERR_CUDA, "dot: cuTensorMapEncodeTiled failed (%d)", (int)rc);
  return SMORE_OK;
}

// Parts of the reduction: where the tiles leave at least half of the SMs without one, as many as there are SMs
// for, each at least kFlush chunks long.  The parts' sums then fit one tile per SM.
static int reduction_parts(size_t M, size_t N, size_t K) {
  const size_t tiles = ((M + kTileM - 1) / kTileM) * ((N + kTileN - 1) / kTileN);
  const size_t flushes = (K + kChunk - 1) / kChunk / kFlush;
  return (int)std::max<size_t>(1, std::min<size_t>((size_t)sm_count() / tiles, flushes));
}

static size_t spill_bytes(size_t K) {
  return K > (size_t)kChunk * kNoFlush ? (size_t)sm_count() * kTileM * kTileN * sizeof(float) : 0;
}

size_t split_gemm_scratch_bytes(size_t M, size_t N, size_t K) {
  const int parts = reduction_parts(M, N, K);
  return spill_bytes(K) + (parts > 1 ? (parts * M * N * sizeof(float) + 1023) & ~(size_t)1023 : 0);
}

int split_gemm(const void* a_planes, const void* b_planes, float* d, size_t ld_d, bool add, size_t M, size_t N, size_t K,
               void* scratch, cudaStream_t st) {
  CUtensorMap map_a, map_b;
  if (int rc = plane_map(&map_a, a_planes, M, K, kTileM)) return rc;
  if (int rc = plane_map(&map_b, b_planes, N, K, kTileN)) return rc;
  GemmArgs g;
  g.d = d;
  g.ld_d = ld_d;
  g.M = (int)M;
  g.N = (int)N;
  g.add = add;
  g.k_blocks = (int)((K + kBlockK - 1) / kBlockK);
  g.tiles_m = (int)((M + kTileM - 1) / kTileM);
  g.tiles_n = (int)((N + kTileN - 1) / kTileN);
  g.parts = reduction_parts(M, N, K);
  // (parts are rounded up to whole chunks, so the last ones may be empty)
  const int chunks = (g.k_blocks + kBlocksPerChunk - 1) / kBlocksPerChunk, per = (chunks + g.parts - 1) / g.parts;
  g.parts = (chunks + per - 1) / per;
  g.spill = static_cast<float*>(scratch);
  g.part_sums = g.parts > 1 ? reinterpret_cast<float*>(static_cast<unsigned char*>(scratch) + spill_bytes(K)) : nullptr;
  if (int rc = allow_large_smem(split_gemm_kernel, kGemmSmem)) return rc;
  const size_t items = (size_t)g.tiles_m * g.tiles_n * g.parts;
  const unsigned grid = (unsigned)std::min(items, (size_t)sm_count());
  split_gemm_kernel<<<grid, kGemmThreads, kGemmSmem, st>>>(map_a, map_b, g);
  if (int rc = check_launch("split_gemm_kernel")) return rc;
  if (g.parts == 1) return SMORE_OK;
  const size_t ctas = std::min<size_t>((M * (N / 4) + 255) / 256, (size_t)sm_count() * 8);
  sum_parts_kernel<<<(unsigned)ctas, 256, 0, st>>>(g.part_sums, g.parts, d, ld_d, g.M, g.N, add);
  return check_launch("sum_parts_kernel");
}

}  // namespace smore

using namespace smore;

extern "C" {

int smore_split_status(int* status) {   // not part of the public header; smore_async_status adds it in
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_split_status, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status: cannot read the status word");
  *status = v;
  return SMORE_OK;
}

int smore_split_status_clear(void) {
  const int zero = 0;
  if (cudaMemcpyToSymbol(g_split_status, &zero, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status_clear: cannot write the status word");
  return SMORE_OK;
}

}  // extern "C"

// Kernels for the shared-candidate shape: one set of K candidate rows scored against every one of
// B queries (entity [1, K, W] or table + idx[K]; query [B, 1, dim]) — the reference's
// `--share_negative` training shape and its full-table evaluation shape.
//
// Every (query, candidate) pair re-uses rows that other pairs also use, so this shape is bound by
// fp32 ALU throughput and on-chip bandwidth, not by HBM: B*K*dim term evaluations against only
// (B + K)*dim*4 bytes.  The forward kernel is tiled like a SIMT matrix product (a 32 x 64 tile of
// cells per CTA, operands staged through shared memory, 4 x 4 cells per thread); the backward
// kernel evaluates every term once for both gradients: candidate-row gradients are summed in a fixed
// order (registers, then across a thread-block cluster), query gradients by floating-point
// reductions in L2.
//
// The reference runs this shape through the same three kernels as every other shape
// (smore/common/torchext/common_kernel.h:33-123): one warp per cell re-reading both rows from L2
// in the forward pass, and column-strided walks (one 32-byte sector per 4 useful bytes) in the
// backward pass.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "dist_terms.cuh"

namespace smore {

// One tile of scores: kTileB queries x kTileK candidate rows by kTileThreads threads, kCellsB x kCellsK
// cells each.  32 queries per tile because that is what an evaluation batch and the ragged end of a
// training batch have (64 left half the tile empty at 32 queries); a row of cells per thread re-uses
// every operand four times from registers, which keeps shared-memory reads at 12 per 320 arithmetic
// instructions (box distances).
constexpr int kTileB = 32;
constexpr int kTileK = 64;
constexpr int kTileThreads = 128;
constexpr int kCellsB = 4, kCellsK = 4;
constexpr int kTileTx = kTileK / kCellsK;                 // thread columns: candidates tx + kTileTx * j
constexpr int kTileTy = kTileThreads / kTileTx;           // thread rows: queries ty + kTileTy * i
constexpr int kTileD = 32;                                // embedding dims staged per step
constexpr int kTileStride = kTileD + 4;                   // floats per staged row: rows stay 16-byte aligned
                                                          // and eight consecutive ones cover all 32 banks
static_assert(kTileTy * kCellsB == kTileB && kTileTx * kCellsK == kTileK, "tile shape");

struct SharedArgs {
  const float* ent;        // [K, W] or table when idx != nullptr
  const int64_t* idx;      // nullable [K]
  const float* first;      // [B, dim]
  const float* second;     // [B, dim]
  int B, K, dim;           // dim % 4 == 0
  long long n_rows;        // rows of `ent` when idx != nullptr (0: ids are not checked)
};

// Device status word of the distance kernels (kStatus* bits): a bulk-copy wait that gave up, a row
// id outside the table.  Either makes the results of the launch invalid; smore_async_status reads
// it.  (Defined here because this header is part of exactly one translation unit, dist_kernels.cu.)
__device__ int g_async_status = 0;

// Shared memory of one tile: two stages of kTileD dims, filled by asynchronous copies while the other
// one is being used.
template <class Term>
struct TileStage {
  float q0[kTileB][kTileStride];
  float q1[Term::kNQ == 2 ? kTileB : 1][kTileStride];
  float e[Term::kMul][kTileK][kTileStride];
};
template <class Term>
struct TileSmem {
  TileStage<Term> stage[2];
  long long rows[kTileK];       // table rows of the tile's candidates; -1: an id outside the table
};

__device__ __forceinline__ void copy16_async(void* smem, const void* gmem, bool ok) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int bytes = ok ? 16 : 0;   // 0: zero-fill, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}

// Scores of the tile (queries b0.., candidates k0..) into acc: thread (ty, tx) owns queries
// b0 + ty + kTileTy * i and candidates k0 + tx + kTileTx * j.  Every cell accumulates its terms in the
// order of the embedding dim, one after the other, so a (query, candidate) pair gets the same value
// wherever it falls in a tile and whatever the tile's neighbours are.  All threads of the CTA call this;
// it starts with a barrier (the previous tile's shared memory is free again) and sets sm.rows.
// (32 queries x 10.76M rows of dim 400, box distances: 57.3 ms with 64 x 64 tiles of half-empty query
// rows, see kTileB.)
template <class Term>
__device__ __forceinline__ void tile_scores(const SharedArgs& a, TileSmem<Term>& sm, int b0, int k0,
                                            float (&acc)[kCellsB][kCellsK][Term::kNOut]) {
  const int tx = threadIdx.x % kTileTx, ty = threadIdx.x / kTileTx;
  const int dim4 = a.dim >> 2;
  const size_t w4 = (size_t)dim4 * Term::kMul;
  __syncthreads();
  if (threadIdx.x < kTileK) {
    const int k = k0 + threadIdx.x;
    sm.rows[threadIdx.x] = k >= a.K ? 0 : a.idx ? checked_row_id(a.idx, k, a.n_rows, &g_async_status) : (long long)k;
  }
  __syncthreads();
  // staging role: the 16-byte pieces lc of rows lr, lr + 16, ... of every operand
  constexpr int kPieces = kTileD / 4, kRowsPerPass = kTileThreads / kPieces;
  const int lc = threadIdx.x % kPieces, lr = threadIdx.x / kPieces;
  const float4* ent4 = reinterpret_cast<const float4*>(a.ent);
  const float4* first4 = reinterpret_cast<const float4*>(a.first);
  const float4* second4 = reinterpret_cast<const float4*>(a.second);
  auto stage = [&](int which, int d0) {
    TileStage<Term>& st = sm.stage[which];
    const int d4 = (d0 >> 2) + lc;
    const bool d_ok = d4 < dim4;
#pragma unroll
    for (int r = lr; r < kTileB; r += kRowsPerPass) {
      const bool ok = d_ok && b0 + r < a.B;
      const size_t at = ok ? (size_t)(b0 + r) * dim4 + d4 : 0;
      copy16_async(&st.q0[r][lc * 4], first4 + at, ok);
      if (Term::kNQ == 2) copy16_async(&st.q1[r][lc * 4], second4 + at, ok);
    }
#pragma unroll
    for (int r = lr; r < kTileK; r += kRowsPerPass) {
      const bool ok = d_ok && k0 + r < a.K;
      const size_t at = ok ? (size_t)max(sm.rows[r], 0LL) * w4 + d4 : 0;
      copy16_async(&st.e[0][r][lc * 4], ent4 + at, ok);
      if (Term::kMul == 2) copy16_async(&st.e[Term::kMul - 1][r][lc * 4], ent4 + (ok ? at + dim4 : 0), ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < kCellsB; ++i)
#pragma unroll
    for (int j = 0; j < kCellsK; ++j)
#pragma unroll
      for (int o = 0; o < Term::kNOut; ++o) acc[i][j][o] = 0.f;

  stage(0, 0);
  int cur = 0;
  for (int d0 = 0; d0 < a.dim; d0 += kTileD, cur ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // this stage has landed for everyone, and nobody reads the other one any more
    if (d0 + kTileD < a.dim) stage(cur ^ 1, d0 + kTileD);
    const TileStage<Term>& st = sm.stage[cur];
    const int pieces = min(kPieces, dim4 - (d0 >> 2));
#pragma unroll 1
    for (int p = 0; p < pieces; ++p) {
      float4 q0[kCellsB], q1[kCellsB], e0[kCellsK], e1[kCellsK];
#pragma unroll
      for (int i = 0; i < kCellsB; ++i) {
        q0[i] = *reinterpret_cast<const float4*>(&st.q0[ty + kTileTy * i][p * 4]);
        q1[i] = Term::kNQ == 2 ? *reinterpret_cast<const float4*>(&st.q1[ty + kTileTy * i][p * 4]) : q0[i];
      }
#pragma unroll
      for (int j = 0; j < kCellsK; ++j) {
        e0[j] = *reinterpret_cast<const float4*>(&st.e[0][tx + kTileTx * j][p * 4]);
        e1[j] = Term::kMul == 2 ? *reinterpret_cast<const float4*>(&st.e[Term::kMul - 1][tx + kTileTx * j][p * 4]) : e0[j];
      }
#pragma unroll
      for (int i = 0; i < kCellsB; ++i)
#pragma unroll
        for (int j = 0; j < kCellsK; ++j) {
          Term::fwd(e0[j].x, e1[j].x, q0[i].x, q1[i].x, acc[i][j]);
          Term::fwd(e0[j].y, e1[j].y, q0[i].y, q1[i].y, acc[i][j]);
          Term::fwd(e0[j].z, e1[j].z, q0[i].z, q1[i].z, acc[i][j]);
          Term::fwd(e0[j].w, e1[j].w, q0[i].w, q1[i].w, acc[i][j]);
        }
    }
  }
}

// Grid: one CTA per tile, query tiles of the same candidates next to each other (they share the rows in L2).
template <class Term>
__global__ void __launch_bounds__(kTileThreads)
    shared_forward_kernel(SharedArgs a, float* __restrict__ dst0, float* __restrict__ dst1) {
  extern __shared__ __align__(16) unsigned char tile_smem[];
  TileSmem<Term>& sm = *reinterpret_cast<TileSmem<Term>*>(tile_smem);
  const int tx = threadIdx.x % kTileTx, ty = threadIdx.x / kTileTx;
  const int q_tiles = (a.B + kTileB - 1) / kTileB;
  const int b0 = (int)(blockIdx.x % q_tiles) * kTileB, k0 = (int)(blockIdx.x / q_tiles) * kTileK;
  float acc[kCellsB][kCellsK][Term::kNOut];
  tile_scores<Term>(a, sm, b0, k0, acc);
#pragma unroll
  for (int i = 0; i < kCellsB; ++i) {
    const int b = b0 + ty + kTileTy * i;
    if (b >= a.B) continue;
#pragma unroll
    for (int j = 0; j < kCellsK; ++j) {
      const int k = k0 + tx + kTileTx * j;
      if (k < a.K) {
        const bool bad = sm.rows[tx + kTileTx * j] < 0;
        dst0[(size_t)b * a.K + k] = bad ? NAN : acc[i][j][0];
        if (Term::kNOut == 2) dst1[(size_t)b * a.K + k] = bad ? NAN : acc[i][j][Term::kNOut - 1];
      }
    }
  }
}

struct SharedGradArgs {
  const float* gout0;         // [B, K]
  const float* gout1;         // [B, K] (two-output term only)
  float* g_ent;               // dense [K, W], or nullptr when slot != nullptr
  const int32_t* slot;        // [K] -> row of g_rows (< 0: skip)
  const int32_t* slot_count;  // nullable: nullptr = accumulate everywhere
  float* g_rows;
  float* g_first;             // [B, dim]
  float* g_second;            // [B, dim]
};

// ---- both gradients of the shared-candidate shape from ONE evaluation of every term ----
//
// Thread = one embedding dim d; CTA = KT candidate rows x a segment of the queries x blockDim.x
// dims.  The thread keeps e[k, d] and its gradient for the KT rows in registers and walks the
// segment's queries: per query it loads q[b, d], evaluates the KT terms (upstream gradients
// broadcast from shared memory) and sends the query's partial gradient (the sum over the CTA's KT
// rows) to g_first / g_second with one coalesced reduction per warp, so those must be zero at
// launch.  The CTAs that share rows and dims but hold different query segments form one
// thread-block cluster: at the end they add their row gradients through distributed shared memory
// in rank order (deterministic) and each rank writes KT / cluster-size of the rows.
constexpr int kBwdChunkB = 64;    // queries whose upstream gradients are staged at a time
constexpr int kBwdAhead = 4;      // query rows loaded ahead of the one being used
constexpr int kBwdMaxThreads = 512;

template <class Term, int KT>
__global__ void __launch_bounds__(kBwdMaxThreads)
    shared_backward_tile_kernel(SharedArgs a, SharedGradArgs ga, int seg_b) {
  static_assert((KT * Term::kNOut) % 4 == 0, "a query's upstream gradients are read 16 bytes at a time");
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int NO = Term::kNOut, M = Term::kMul;
  __shared__ __align__(16) float gs[kBwdChunkB][KT][NO];
  __shared__ long long rows_sh[KT];
  extern __shared__ float tile_red[];   // [KT * M][blockDim.x]
  float* red = tile_red;

  const int tid = threadIdx.x, T = blockDim.x;
  const int k0 = blockIdx.x * KT;
  const int d = blockIdx.z * T + tid;
  const bool d_ok = d < a.dim;
  const bool warp_live = blockIdx.z * T + (tid & ~31) < a.dim;   // warps past the last dim only take part in barriers
  const unsigned rank = cluster.block_rank(), n_ranks = cluster.num_blocks();
  const int b_begin = min(a.B, (int)rank * seg_b), b_end = min(a.B, b_begin + seg_b);

  if (tid < KT) {
    const int k = k0 + tid;
    rows_sh[tid] = k < a.K ? (a.idx ? checked_row_id(a.idx, k, a.n_rows, &g_async_status) : (long long)k) : -1;
  }
  __syncthreads();
  const size_t W = (size_t)a.dim * M;
  float e0[KT], e1[KT], ge0[KT], ge1[KT];
#pragma unroll
  for (int j = 0; j < KT; ++j) {
    const long long r = rows_sh[j];
    const bool ok = r >= 0 && d_ok;
    e0[j] = ok ? __ldg(a.ent + (size_t)r * W + d) : 0.f;
    e1[j] = (M == 2 && ok) ? __ldg(a.ent + (size_t)r * W + a.dim + d) : e0[j];
    ge0[j] = 0.f;
    ge1[j] = 0.f;
  }
  const float* __restrict__ q0p = a.first + d;
  const float* __restrict__ q1p = a.second + d;

  for (int bs = b_begin; bs < b_end; bs += kBwdChunkB) {
    const int nb = min(kBwdChunkB, b_end - bs);
    __syncthreads();   // the previous chunk's gradients are no longer being read
    // upstream gradients of the chunk; zero for rows that do not exist, so their terms add nothing
    for (int i = tid; i < nb * KT; i += T) {
      const int bb = i / KT, j = i % KT;
      const bool ok = rows_sh[j] >= 0;
      const size_t at = (size_t)(bs + bb) * a.K + k0 + j;
      gs[bb][j][0] = ok ? __ldg(ga.gout0 + at) : 0.f;
      if (NO == 2) gs[bb][j][NO - 1] = ok ? __ldg(ga.gout1 + at) : 0.f;
    }
    __syncthreads();
    if (!warp_live) continue;
    float q0n[kBwdAhead], q1n[kBwdAhead];
#pragma unroll
    for (int u = 0; u < kBwdAhead; ++u) {
      const bool ok = d_ok && u < nb;
      q0n[u] = ok ? __ldg(q0p + (size_t)(bs + u) * a.dim) : 0.f;
      q1n[u] = (Term::kNQ == 2 && ok) ? __ldg(q1p + (size_t)(bs + u) * a.dim) : q0n[u];
    }
    for (int bb0 = 0; bb0 < nb; bb0 += kBwdAhead) {
      float q0c[kBwdAhead], q1c[kBwdAhead];
#pragma unroll
      for (int u = 0; u < kBwdAhead; ++u) {
        q0c[u] = q0n[u];
        q1c[u] = q1n[u];
        const int bn = bb0 + kBwdAhead + u;
        const bool ok = d_ok && bn < nb;
        q0n[u] = ok ? __ldg(q0p + (size_t)(bs + bn) * a.dim) : 0.f;
        q1n[u] = (Term::kNQ == 2 && ok) ? __ldg(q1p + (size_t)(bs + bn) * a.dim) : q0n[u];
      }
#pragma unroll
      for (int u = 0; u < kBwdAhead; ++u) {
        const int bb = bb0 + u;
        if (bb >= nb) break;
        float gq0 = 0.f, gq1 = 0.f;
        // the query's KT x NO upstream gradients: a few 16-byte broadcast loads instead of one load per value
        float gl[KT * NO];
        const float4* g4 = reinterpret_cast<const float4*>(&gs[bb][0][0]);
#pragma unroll
        for (int i = 0; i < KT * NO / 4; ++i) {
          const float4 t = g4[i];
          gl[4 * i + 0] = t.x; gl[4 * i + 1] = t.y; gl[4 * i + 2] = t.z; gl[4 * i + 3] = t.w;
        }
#pragma unroll
        for (int j = 0; j < KT; ++j) Term::bwd(&gl[j * NO], e0[j], e1[j], q0c[u], q1c[u], ge0[j], ge1[j], gq0, gq1);
        if (d_ok) {
          const size_t at = (size_t)(bs + bb) * a.dim + d;
          atomicAdd(ga.g_first + at, gq0);
          if (Term::kNQ == 2) atomicAdd(ga.g_second + at, gq1);
        }
      }
    }
  }

  // row gradients: sum over the cluster's query segments in rank order
#pragma unroll
  for (int j = 0; j < KT; ++j) {
    red[(j * M) * T + tid] = ge0[j];
    if (M == 2) red[(j * M + M - 1) * T + tid] = ge1[j];
  }
  cluster.sync();
  for (int j = (int)rank; j < KT; j += (int)n_ranks) {
    const int k = k0 + j;
    if (k >= a.K || rows_sh[j] < 0 || !d_ok) continue;
    float s0 = 0.f, s1 = 0.f;
    for (unsigned r = 0; r < n_ranks; ++r) {
      const float* remote = cluster.map_shared_rank(red, r);
      s0 += remote[(j * M) * T + tid];
      if (M == 2) s1 += remote[(j * M + M - 1) * T + tid];
    }
    if (ga.slot == nullptr) {
      ga.g_ent[(size_t)k * W + d] = s0;
      if (M == 2) ga.g_ent[(size_t)k * W + a.dim + d] = s1;
    } else {
      const int32_t s = ga.slot[k];
      if (s < 0) continue;
      float* out = ga.g_rows + (size_t)s * W + d;
      if (ga.slot_count != nullptr && ga.slot_count[s] == 1) {
        out[0] = s0;
        if (M == 2) out[a.dim] = s1;
      } else {
        atomicAdd(out, s0);
        if (M == 2) atomicAdd(out + a.dim, s1);
      }
    }
  }
  cluster.sync();   // no CTA leaves while another still reads its shared memory
}

}  // namespace smore

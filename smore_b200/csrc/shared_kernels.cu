// Kernels for the shared-candidate shape: one set of K candidate rows scored against every one of
// B queries (entity [1, K, W] or table + idx[K]; query [B, 1, dim]) — the reference's
// `--share_negative` training shape and its full-table evaluation shape — and the same with the roles of
// the operands' leading dims swapped (entity [K, 1, W], query [1, B, dim]), where only the result is
// laid out differently.
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
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "dist_common.cuh"
#include "rank_common.cuh"

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
  int B, K, dim;
  long long n_rows;        // rows of `ent` when idx != nullptr (0: ids are not checked)
  size_t at_b, at_k;       // result and upstream gradient of (b, k) lie at b * at_b + k * at_k
};

static __device__ int g_shared_status = 0;   // kStatusBadRowId: a row id lay outside the table

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

// V floats of a row to shared memory; zeros, and nothing read, where !ok
template <int V>
__device__ __forceinline__ void copy_async(float* smem, const float* gmem, bool ok) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int bytes = ok ? 4 * V : 0;
  if (V == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}

template <class Term>
__device__ __forceinline__ void tile_term(float e0, float e1, float q0, float q1, float* acc) {
  if constexpr (Term::kFast) Term::fwd_fast(e0, e1, q0, q1, acc);
  else Term::fwd(e0, e1, q0, q1, acc);
}

// First output of one cell with Term::fwd, in the order of the dims as everywhere.
template <class Term>
__device__ __noinline__ float exact_cell(const SharedArgs& a, int b, long long row) {
  const float* e = a.ent + (size_t)row * a.dim * Term::kMul;
  const float *q0 = a.first + (size_t)b * a.dim, *q1 = Term::kNQ == 2 ? a.second + (size_t)b * a.dim : q0;
  float acc[Term::kNOut] = {};
  for (int d = 0; d < a.dim; ++d) Term::fwd(e[d], Term::kMul == 2 ? e[a.dim + d] : e[d], q0[d], q1[d], acc);
  return acc[0];
}

// Scores of the tile (queries b0.., candidates k0..) into acc: thread (ty, tx) owns queries
// b0 + ty + kTileTy * i and candidates k0 + tx + kTileTx * j.  Every cell accumulates its terms in the
// order of the embedding dim, one after the other, so a (query, candidate) pair gets the same value
// wherever it falls in a tile and whatever the tile's neighbours are.  All threads of the CTA call this;
// it starts with a barrier (the previous tile's shared memory is free again) and sets sm.rows.
// V: floats per asynchronous copy, 4 where rows are 16-byte aligned, else 1.
// (32 queries x 10.76M rows of dim 400, box distances: 57.3 ms with 64 x 64 tiles of half-empty query
// rows and six instructions per term, 27.4 ms like this: 6.05 instructions per term and thread, issue
// slots 82 % busy.)
template <class Term, int V>
__device__ __forceinline__ void tile_scores(const SharedArgs& a, TileSmem<Term>& sm, int b0, int k0,
                                            float (&acc)[kCellsB][kCellsK][Term::kNOut]) {
  const int tx = threadIdx.x % kTileTx, ty = threadIdx.x / kTileTx;
  const size_t width = (size_t)a.dim * Term::kMul;
  __syncthreads();
  if (threadIdx.x < kTileK) {
    const int k = k0 + threadIdx.x;
    sm.rows[threadIdx.x] = k >= a.K ? 0 : a.idx ? checked_row_id(a.idx, k, a.n_rows, &g_shared_status) : (long long)k;
  }
  __syncthreads();
  // staging role: the V-float pieces lc of rows lr, lr + kRowsPerPass, ... of every operand
  constexpr int kPieces = kTileD / V, kRowsPerPass = kTileThreads / kPieces;
  const int lc = threadIdx.x % kPieces, lr = threadIdx.x / kPieces;
  auto stage = [&](int which, int d0) {
    TileStage<Term>& st = sm.stage[which];
    const int d = d0 + lc * V;
    const bool d_ok = d < a.dim;
#pragma unroll
    for (int r = lr; r < kTileB; r += kRowsPerPass) {
      const bool ok = d_ok && b0 + r < a.B;
      const size_t at = ok ? (size_t)(b0 + r) * a.dim + d : 0;
      copy_async<V>(&st.q0[r][lc * V], a.first + at, ok);
      if (Term::kNQ == 2) copy_async<V>(&st.q1[r][lc * V], a.second + at, ok);
    }
#pragma unroll
    for (int r = lr; r < kTileK; r += kRowsPerPass) {
      const bool ok = d_ok && k0 + r < a.K;
      const size_t at = ok ? (size_t)max(sm.rows[r], 0LL) * width + d : 0;
      copy_async<V>(&st.e[0][r][lc * V], a.ent + at, ok);
      if (Term::kMul == 2) copy_async<V>(&st.e[Term::kMul - 1][r][lc * V], a.ent + (ok ? at + a.dim : 0), ok);
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
    const int quads = min(kTileD, a.dim - d0) >> 2;
#pragma unroll 1
    for (int p = 0; p < quads; ++p) {
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
          tile_term<Term>(e0[j].x, e1[j].x, q0[i].x, q1[i].x, acc[i][j]);
          tile_term<Term>(e0[j].y, e1[j].y, q0[i].y, q1[i].y, acc[i][j]);
          tile_term<Term>(e0[j].z, e1[j].z, q0[i].z, q1[i].z, acc[i][j]);
          tile_term<Term>(e0[j].w, e1[j].w, q0[i].w, q1[i].w, acc[i][j]);
        }
    }
    if (V == 1) {   // the up to three last dims of a row whose length is no multiple of four
#pragma unroll 1
      for (int d = quads * 4; d < min(kTileD, a.dim - d0); ++d)
#pragma unroll
        for (int i = 0; i < kCellsB; ++i) {
          const float q0 = st.q0[ty + kTileTy * i][d], q1 = Term::kNQ == 2 ? st.q1[ty + kTileTy * i][d] : q0;
#pragma unroll
          for (int j = 0; j < kCellsK; ++j) {
            const float e0 = st.e[0][tx + kTileTx * j][d];
            tile_term<Term>(e0, Term::kMul == 2 ? st.e[Term::kMul - 1][tx + kTileTx * j][d] : e0, q0, q1, acc[i][j]);
          }
        }
    }
  }
  if constexpr (Term::kFast) {   // cells with NaN operands (or an infinite distance to an infinite box)
#pragma unroll
    for (int i = 0; i < kCellsB; ++i)
#pragma unroll
      for (int j = 0; j < kCellsK; ++j)
        if (acc[i][j][0] != acc[i][j][0] && b0 + ty + kTileTy * i < a.B)
          acc[i][j][0] = exact_cell<Term>(a, b0 + ty + kTileTy * i, max(sm.rows[tx + kTileTx * j], 0LL));
  }
}

// Grid: one CTA per tile, query tiles of the same candidates next to each other (they share the rows in L2).
template <class Term, int V>
__global__ void __launch_bounds__(kTileThreads)
    shared_forward_kernel(SharedArgs a, float* __restrict__ dst0, float* __restrict__ dst1) {
  extern __shared__ __align__(16) unsigned char tile_smem[];
  TileSmem<Term>& sm = *reinterpret_cast<TileSmem<Term>*>(tile_smem);
  const int tx = threadIdx.x % kTileTx, ty = threadIdx.x / kTileTx;
  const int q_tiles = (a.B + kTileB - 1) / kTileB;
  const int b0 = (int)(blockIdx.x % q_tiles) * kTileB, k0 = (int)(blockIdx.x / q_tiles) * kTileK;
  float acc[kCellsB][kCellsK][Term::kNOut];
  tile_scores<Term, V>(a, sm, b0, k0, acc);
#pragma unroll
  for (int i = 0; i < kCellsB; ++i) {
    const int b = b0 + ty + kTileTy * i;
    if (b >= a.B) continue;
#pragma unroll
    for (int j = 0; j < kCellsK; ++j) {
      const int k = k0 + tx + kTileTx * j;
      if (k < a.K) {
        const bool bad = sm.rows[tx + kTileTx * j] < 0;
        const size_t at = b * a.at_b + k * a.at_k;
        dst0[at] = bad ? NAN : acc[i][j][0];
        if (Term::kNOut == 2) dst1[at] = bad ? NAN : acc[i][j][Term::kNOut - 1];
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
    rows_sh[tid] = k < a.K ? (a.idx ? checked_row_id(a.idx, k, a.n_rows, &g_shared_status) : (long long)k) : -1;
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
      const size_t at = (bs + bb) * a.at_b + (size_t)(k0 + j) * a.at_k;
      gs[bb][j][0] = ok ? __ldg(ga.gout0 + at) : 0.f;
      if (NO == 2) gs[bb][j][NO - 1] = ok ? __ldg(ga.gout1 + at) : 0.f;
    }
    __syncthreads();
    if (!warp_live) continue;
    float q0n[kBwdAhead], q1n[kBwdAhead];
    auto fetch = [&](int u, int bb) {
      const bool ok = d_ok && bb < nb;
      q0n[u] = ok ? Term::prep(__ldg(q0p + (size_t)(bs + bb) * a.dim)) : 0.f;
      q1n[u] = (Term::kNQ == 2 && ok) ? __ldg(q1p + (size_t)(bs + bb) * a.dim) : 1.f;
    };
#pragma unroll
    for (int u = 0; u < kBwdAhead; ++u) fetch(u, u);
    for (int bb0 = 0; bb0 < nb; bb0 += kBwdAhead) {
      float q0c[kBwdAhead], q1c[kBwdAhead];
#pragma unroll
      for (int u = 0; u < kBwdAhead; ++u) {
        q0c[u] = q0n[u];
        q1c[u] = q1n[u];
        fetch(u, bb0 + kBwdAhead + u);
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
        // (the cheaper rule where every lane's offset allows it: all of a trained model's do)
        if (Term::kPositive && __all_sync(0xffffffffu, q1c[u] > 0.f)) {
#pragma unroll
          for (int j = 0; j < KT; ++j) Term::bwd_pos(&gl[j * NO], e0[j], e1[j], q0c[u], q1c[u], ge0[j], ge1[j], gq0, gq1);
        } else {
#pragma unroll
          for (int j = 0; j < KT; ++j) Term::bwd(&gl[j * NO], e0[j], e1[j], q0c[u], q1c[u], ge0[j], ge1[j], gq0, gq1);
        }
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

// ----------------------------------------------------------------------------------------
// Evaluation: scores of a batch of queries against EVERY entity, ranked on the fly.
// The reference's test step (smore/training/train_process.py:104-146) materialises the [Q, N] logits,
// argsorts them and scatters ranks; smore_filtered_ranks already replaces the sort by counting but
// still reads a logits matrix.  Here the scoring tile never leaves the registers: every cell is
// turned into the model's logit with the arithmetic torch would use on the distances
// (custom_cal_logit: gamma - d_out - cen * d_in for Query2box, box.py:157-164; gamma - d for GQE and
// RotatE; the similarity itself for ComplEx / DistMult), compared with the query's worst answer and,
// if it is ahead of it, placed among the query's sorted answers (binary search, one histogram
// increment).  The answers' own logits come from the same tile code run on the answers' rows, so a
// candidate that is an answer meets exactly its own value.
// ----------------------------------------------------------------------------------------

// acc over the 4 components of one 16-byte piece
template <class Term>
__device__ __forceinline__ void fwd4(const float4& e0, const float4& e1, const float4& q0,
                                     const float4& q1, float* acc) {
  Term::fwd(e0.x, e1.x, q0.x, q1.x, acc);
  Term::fwd(e0.y, e1.y, q0.y, q1.y, acc);
  Term::fwd(e0.z, e1.z, q0.z, q1.z, acc);
  Term::fwd(e0.w, e1.w, q0.w, q1.w, acc);
}

enum LogitKind { kLogitGammaMinus = 0, kLogitGammaMinusSqrt = 1, kLogitIdentity = 2 };

template <int NOUT>
__device__ __forceinline__ float logit_of(const float* acc, int kind, float gamma, float cen) {
  if (NOUT == 2) return __fsub_rn(__fsub_rn(gamma, acc[0]), __fmul_rn(cen, acc[NOUT - 1]));
  if (kind == kLogitGammaMinus) return __fsub_rn(gamma, acc[0]);
  if (kind == kLogitGammaMinusSqrt) return __fsub_rn(gamma, sqrtf(acc[0]));
  return acc[0];
}

// The answers' own logits, [n_answers] in the order of answer_ids.  A cell's terms have to be added one
// after the other, as tile_scores does, so an answer is one thread's serial sum; the rows it reads are
// first brought to shared memory by the whole CTA, kAnswersPerCta answers of one query at a time.
// (960 answers of 32 queries, dim 400: 72 us when the scoring tile computed every query against every
// answer, for the diagonal.)
constexpr int kAnswersPerCta = 8;
constexpr int kAnswerDims = 512;    // dims staged at a time

template <class Term>
__global__ void __launch_bounds__(128)
    answer_logits_kernel(SharedArgs a, const int64_t* __restrict__ answer_ptr, int kind, float gamma, float cen,
                         float* __restrict__ logits) {
  __shared__ __align__(16) float q[2][kAnswerDims];
  __shared__ __align__(16) float e[kAnswersPerCta][Term::kMul][kAnswerDims + 4];
  const int b = (int)(blockIdx.x % a.B);
  const long long begin = answer_ptr[b] + (long long)(blockIdx.x / a.B) * kAnswersPerCta;
  const int n = (int)max(0LL, min((long long)kAnswersPerCta, answer_ptr[b + 1] - begin));
  if (n == 0) return;
  float acc[Term::kNOut];
#pragma unroll
  for (int o = 0; o < Term::kNOut; ++o) acc[o] = 0.f;
  bool bad = false;
  for (int d0 = 0; d0 < a.dim; d0 += kAnswerDims) {
    const int n4 = min(kAnswerDims, a.dim - d0) >> 2;
    __syncthreads();
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
      reinterpret_cast<float4*>(q[0])[i] = __ldg(reinterpret_cast<const float4*>(a.first + (size_t)b * a.dim + d0) + i);
      if (Term::kNQ == 2)
        reinterpret_cast<float4*>(q[1])[i] = __ldg(reinterpret_cast<const float4*>(a.second + (size_t)b * a.dim + d0) + i);
    }
    for (int i = threadIdx.x; i < n * Term::kMul * n4; i += blockDim.x) {
      const int r = i / (Term::kMul * n4), rem = i - r * Term::kMul * n4, part = rem / n4, c = rem - part * n4;
      const long long row = max(checked_row_id(a.idx, begin + r, a.n_rows, &g_shared_status), 0LL);
      reinterpret_cast<float4*>(e[r][part])[c] =
          __ldg(reinterpret_cast<const float4*>(a.ent + ((size_t)row * Term::kMul + part) * a.dim + d0) + c);
    }
    __syncthreads();
    if (threadIdx.x < n) {
      const int r = threadIdx.x;
      bad = checked_row_id(a.idx, begin + r, a.n_rows, &g_shared_status) < 0;
      for (int i = 0; i < n4; ++i) {
        const float4 e0 = reinterpret_cast<const float4*>(e[r][0])[i], e1 = reinterpret_cast<const float4*>(e[r][Term::kMul - 1])[i];
        const float4 q0 = reinterpret_cast<const float4*>(q[0])[i];
        const float4 q1 = Term::kNQ == 2 ? reinterpret_cast<const float4*>(q[1])[i] : q0;
        fwd4<Term>(e0, e1, q0, q1, acc);
      }
    }
  }
  if (threadIdx.x < n) logits[begin + threadIdx.x] = bad ? NAN : logit_of<Term::kNOut>(acc, kind, gamma, cen);
}

// Scores the queries against every row of the table and counts, per answer, the candidates whose first
// answer behind them it is.  A fixed number of CTAs walks the tiles; the answers of a CTA's queries (keys,
// ids, counts) stay in shared memory while they fit (`cap` answers), and the counts go to `hist` once.
// A CTA keeps one query tile (blockIdx.y) and takes candidate tiles blockIdx.x, + gridDim.x, ...
template <class Term>
__global__ void __launch_bounds__(kTileThreads)
    score_rank_kernel(SharedArgs a, int kind, float gamma, float cen, const int64_t* __restrict__ answer_ptr,
                      const uint32_t* __restrict__ sorted_logit, const int64_t* __restrict__ sorted_id,
                      int32_t* __restrict__ hist, int cap) {
  extern __shared__ __align__(16) unsigned char tile_smem[];
  TileSmem<Term>& sm = *reinterpret_cast<TileSmem<Term>*>(tile_smem);
  uint32_t* key = reinterpret_cast<uint32_t*>(tile_smem + sizeof(TileSmem<Term>));   // [cap]
  int32_t* id = reinterpret_cast<int32_t*>(key + cap);                               // [cap]
  int32_t* count = id + cap;                                                         // [cap]
  __shared__ int q_at[kTileB], q_count[kTileB];       // a query's first answer, relative to the tile's; how many
  const int tx = threadIdx.x % kTileTx, ty = threadIdx.x / kTileTx;
  const int b0 = blockIdx.y * kTileB;
  const long long first_answer = answer_ptr[b0];
  const int n_tile = (int)(answer_ptr[min(a.B, b0 + kTileB)] - first_answer);
  const bool local = n_tile <= cap;
  if (threadIdx.x < kTileB) {
    const int b = b0 + threadIdx.x;
    q_at[threadIdx.x] = b < a.B ? (int)(answer_ptr[b] - first_answer) : 0;
    q_count[threadIdx.x] = b < a.B ? (int)(answer_ptr[b + 1] - answer_ptr[b]) : 0;
  }
  if (local) {
    for (int i = threadIdx.x; i < n_tile; i += kTileThreads) {
      key[i] = sorted_logit[first_answer + i];
      id[i] = (int32_t)sorted_id[first_answer + i];
      count[i] = 0;
    }
  }
  const int k_tiles = (a.K + kTileK - 1) / kTileK;
  for (int kt = blockIdx.x; kt < k_tiles; kt += gridDim.x) {
    float acc[kCellsB][kCellsK][Term::kNOut];
    const int k0 = kt * kTileK;
    tile_scores<Term, 4>(a, sm, b0, k0, acc);      // (its barriers also order the writes above)
#pragma unroll
    for (int i = 0; i < kCellsB; ++i) {
      const int bl = ty + kTileTy * i;
      const int A = q_count[bl];
      if (A == 0) continue;
      const int at = q_at[bl];
#pragma unroll
      for (int j = 0; j < kCellsK; ++j) {
        const int k = k0 + tx + kTileTx * j;
        if (k >= a.K) continue;
        const uint32_t x = rank_key(logit_of<Term::kNOut>(acc[i][j], kind, gamma, cen));
        int lo = 0, hi = A;       // first answer this candidate is ahead of; A: it is ahead of none
        if (local) {
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (rank_ahead(x, k, key[at + mid], id[at + mid])) hi = mid;
            else lo = mid + 1;
          }
          if (lo < A) atomicAdd(count + at + lo, 1);
        } else {
          const uint32_t* gk = sorted_logit + first_answer + at;
          const int64_t* gi = sorted_id + first_answer + at;
          if (!rank_ahead(x, k, gk[A - 1], gi[A - 1])) continue;
          --hi;
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (rank_ahead(x, k, gk[mid], gi[mid])) hi = mid;
            else lo = mid + 1;
          }
          atomicAdd(hist + first_answer + at + lo, 1);
        }
      }
    }
  }
  if (local) {
    __syncthreads();
    for (int i = threadIdx.x; i < n_tile; i += kTileThreads)
      if (count[i]) atomicAdd(hist + first_answer + i, count[i]);
  }
}

// ----------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------

// Which of the two layouts of the shape: entity [1, K, W] with queries [B, 1, dim] (result [B, K]), or entity
// [K, 1, W] with queries [1, B, dim] (result [K, B]).
static bool list_form(const Shape& s) { return s.be == 1 && s.ne == s.num && s.bc == s.bsize && s.nc == 1; }
static bool swapped_form(const Shape& s) { return s.be == s.bsize && s.ne == 1 && s.bc == 1 && s.nc == s.num; }

static SharedArgs shared_args(const Shape& s, const float* ent, const int64_t* idx, const float* first, const float* second) {
  if (list_form(s)) return {ent, idx, first, second, (int)s.bsize, (int)s.num, (int)s.dim, (long long)s.n_rows, s.num, 1};
  return {ent, idx, first, second, (int)s.num, (int)s.bsize, (int)s.dim, (long long)s.n_rows, 1, s.num};
}

bool shared_covers(const Shape& s) {
  if (!list_form(s) && !swapped_form(s)) return false;
  return s.bsize >= 8 && s.num >= 8 && s.bsize < ((size_t)1 << 24) && s.num < ((size_t)1 << 30) &&
         s.dim < ((size_t)1 << 20) &&
         ((s.bsize + kTileB - 1) / kTileB) * ((s.num + kTileK - 1) / kTileK) <= (size_t)INT_MAX;   // tiles: grid.x
}

static bool rows16(const SharedArgs& a) {
  return (a.dim & 3) == 0 && aligned16(a.ent) && aligned16(a.first) && aligned16(a.second);
}

template <class Term>
static int launch_shared_forward(const Shape& s, const ForwardArgs& f, cudaStream_t st) {
  const SharedArgs a = shared_args(s, f.ent, f.idx, f.first, Term::kNQ == 2 ? f.second : f.first);
  const size_t tiles = ((size_t)(a.K + kTileK - 1) / kTileK) * ((a.B + kTileB - 1) / kTileB);
  // A tile is a serial walk over the dims (13 us at dim 400); with a handful of tiles one warp per cell over
  // the whole device is done sooner.
  if (tiles < (size_t)sm_count() / 8) return cell_forward(Term::kId, s, f, st);
  auto kern = rows16(a) ? shared_forward_kernel<Term, 4> : shared_forward_kernel<Term, 1>;
  if (int rc = allow_large_smem(kern, (int)sizeof(TileSmem<Term>))) return rc;
  kern<<<(unsigned)tiles, kTileThreads, sizeof(TileSmem<Term>), st>>>(a, f.dst0, f.dst1);
  return check_launch("shared_forward_kernel");
}

int shared_forward(int term, const Shape& s, const ForwardArgs& a, cudaStream_t st) {
  SMORE_DISPATCH_BOTH(term, launch_shared_forward<Term>(s, a, st));
}

// Both gradients of the shared-candidate shape from one evaluation of every term
// (shared_backward_tile_kernel): a cluster of up to 8 CTAs per (KT candidate rows, 128 dims) splits
// the queries; the query gradients are reduced into zeroed buffers.  The device runs about one
// 8-CTA cluster per SM at a time whatever the CTA's size, so CTAs are 4 warps wide.
template <class Term, int KT>
static int launch_shared_backward_kt(const SharedArgs& a, const SharedGradArgs& ga, cudaStream_t st) {
  const size_t B = a.B, K = a.K, dim = a.dim;
  const size_t qbytes = B * dim * sizeof(float);
  if (cudaMemsetAsync(ga.g_first, 0, qbytes, st) != cudaSuccess ||
      (Term::kNQ == 2 && cudaMemsetAsync(ga.g_second, 0, qbytes, st) != cudaSuccess))
    return fail(SMORE_ERR_CUDA, "dist_backward: cudaMemsetAsync failed");
  // dims per CTA: whole warps, at most 128 (a warp past the last dim idles at the barriers only)
  const int threads = (int)std::min<size_t>(128, ((dim + 31) / 32) * 32);
  const unsigned dchunks = (unsigned)((dim + threads - 1) / threads);
  unsigned split = 1;   // query segments = CTAs per cluster: enough CTAs to fill the device, >= 32 queries each
  const size_t base_ctas = ((K + KT - 1) / KT) * dchunks;
  while (split < 8 && B / (split * 2) >= 32 && base_ctas * split * threads < (size_t)sm_count() * 2048 * 4) split *= 2;
  const int seg_b = (int)((B + split - 1) / split);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((K + KT - 1) / KT), split, dchunks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)KT * Term::kMul * threads * sizeof(float);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = split;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, shared_backward_tile_kernel<Term, KT>, a, ga, seg_b) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "shared_backward_tile_kernel: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
  return check_launch("shared_backward_tile_kernel");
}

template <class Term>
static int launch_shared_backward(const Shape& s, const BackwardArgs& b, cudaStream_t st) {
  const SharedArgs a = shared_args(s, b.ent, b.idx, b.first, Term::kNQ == 2 ? b.second : b.first);
  const SharedGradArgs ga{b.gout0, b.gout1, b.g_ent, b.slot, b.slot_count, b.g_rows, b.g_first,
                          Term::kNQ == 2 ? b.g_second : b.g_first};
  // rows of one part are cheap to keep next to the per-query loads and reductions: twice the rows per
  // thread halves those
  if (Term::kMul == 1 && a.K >= 16) return launch_shared_backward_kt<Term, 16>(a, ga, st);
  return launch_shared_backward_kt<Term, 8>(a, ga, st);
}

int shared_backward(int term, const Shape& s, const BackwardArgs& a, cudaStream_t st) {
  SMORE_DISPATCH_BOTH(term, launch_shared_backward<Term>(s, a, st));
}

// One call of the evaluation step; ranks of all answers, or (hard_ptr given) the sorted ranks of the hard ones.
static int score_filtered_ranks_impl(int dist_id, const float* table, size_t n_candidates, const float* first,
                                     const float* second, size_t n_queries, size_t dim, double gamma, double cen,
                                     const int64_t* answer_ptr, const int64_t* answer_ids, size_t n_answers,
                                     size_t max_answers, const int64_t* hard_ptr, int64_t* ranks, void* workspace,
                                     size_t workspace_bytes, void* stream) {
  if (n_queries == 0 || n_answers == 0) return SMORE_OK;
  const bool both = dist_id == SMORE_DIST_BOX_BOTH;
  if (!both && (dist_id < 0 || dist_id >= SMORE_DIST_COUNT))
    return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", dist_id);
  if (dist_id == SMORE_DIST_BOX_OUT || dist_id == SMORE_DIST_BOX_IN)
    return fail(SMORE_ERR_BAD_DIST, "score_filtered_ranks: Query2box logits need both distances (SMORE_DIST_BOX_BOTH)");
  const bool two = both || needs_second(dist_id);
  if (!table || !first || (two && !second) || !answer_ptr || !answer_ids || !ranks || !workspace)
    return fail(SMORE_ERR_NULL, "score_filtered_ranks: NULL pointer");
  if (workspace_bytes < smore_score_filtered_ranks_workspace_bytes(n_queries, n_answers) ||
      (reinterpret_cast<uintptr_t>(workspace) & 255))
    return fail(SMORE_ERR_WORKSPACE, "score_filtered_ranks: workspace too small or not 256-byte aligned");
  if (!second) second = first;
  const Shape s_all{n_queries, n_candidates, 1, n_candidates, n_queries, 1, dim, 0};
  if (int rc = validate_shape(s_all)) return rc;
  if (!shared_covers(s_all) || (dim & 3) || !aligned16(table) || !aligned16(first) || !aligned16(second) || n_answers < 8 || max_answers == 0)
    return fail(SMORE_ERR_BAD_SHAPE,
                "score_filtered_ranks: needs 16-byte aligned operands, dim a multiple of 4, at least 8 queries, "
                "8 candidates and 8 answers in all");
  const RankWorkspace w = carve_rank_workspace(workspace, n_answers);
  float* logits = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + w.bytes);
  const int kind = (dist_id == SMORE_DIST_COMPLEX || dist_id == SMORE_DIST_DISTMULT) ? kLogitIdentity
                   : dist_id == SMORE_DIST_L2 ? kLogitGammaMinusSqrt : kLogitGammaMinus;
  cudaStream_t st = (cudaStream_t)stream;
  SharedArgs a_ans{table, answer_ids, first, second, (int)n_queries, (int)n_answers, (int)dim, (long long)n_candidates, 0, 0};
  SharedArgs a_all{table, nullptr, first, second, (int)n_queries, (int)n_candidates, (int)dim, 0, 0, 0};
  const size_t grid_ans = n_queries * ((max_answers + kAnswersPerCta - 1) / kAnswersPerCta);
  if (grid_ans > (size_t)INT_MAX) return fail(SMORE_ERR_TOO_LARGE, "score_filtered_ranks: too many answers");
  const size_t q_tiles = (n_queries + kTileB - 1) / kTileB, k_tiles = (n_candidates + kTileK - 1) / kTileK;
  // answers of a query tile kept on the SM: four CTAs per SM leave room for about a thousand (12 bytes each)
  const int cap = 1024;
#define SCORE_RANK(TERM)                                                                                             \
  {                                                                                                                  \
    answer_logits_kernel<TERM><<<(unsigned)grid_ans, 128, 0, st>>>(a_ans, answer_ptr, kind, (float)gamma, (float)cen, logits); \
    count_launches(1);                                                                                               \
    if (int rc = rank_sort_answers(logits, n_answers, answer_ptr, answer_ids, true, n_queries, n_answers,            \
                                   max_answers, w, st))                                                              \
      return rc;                                                                                                     \
    const size_t smem = sizeof(TileSmem<TERM>) + (size_t)cap * 12;                                                   \
    auto kern = score_rank_kernel<TERM>;                                                                             \
    if (int rc = allow_large_smem(kern, (int)smem)) return rc;                                                       \
    int per_sm = 0;                                                                                                  \
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kTileThreads, smem) != cudaSuccess || per_sm < 1) \
      per_sm = 1;                                                                                                    \
    const size_t ctas = std::max<size_t>(1, (size_t)sm_count() * per_sm / q_tiles);                                  \
    const dim3 grid((unsigned)std::min(ctas, k_tiles), (unsigned)q_tiles);                                           \
    kern<<<grid, kTileThreads, smem, st>>>(a_all, kind, (float)gamma, (float)cen, answer_ptr, w.sorted_logit,        \
                                           w.sorted_id, w.hist, cap);                                                \
  }
  if (both) SCORE_RANK(TermBoxBoth)
  else if (dist_id == SMORE_DIST_ROTATE) SCORE_RANK(TermRotate)
  else if (dist_id == SMORE_DIST_L1) SCORE_RANK(TermL1)
  else if (dist_id == SMORE_DIST_L2) SCORE_RANK(TermL2)
  else if (dist_id == SMORE_DIST_COMPLEX) SCORE_RANK(TermComplex)
  else SCORE_RANK(TermDistmult)
#undef SCORE_RANK
  if (int rc = check_launch("score_rank_kernel")) return rc;
  return rank_finalize(answer_ptr, w, hard_ptr, max_answers, ranks, n_queries, st);
}

}  // namespace smore

using namespace smore;

extern "C" {

size_t smore_score_filtered_ranks_workspace_bytes(size_t n_queries, size_t n_answers) {
  (void)n_queries;
  return carve_rank_workspace(nullptr, n_answers).bytes + ((n_answers * sizeof(float) + 255) / 256) * 256 + 256;
}

int smore_score_filtered_ranks(int dist_id, const float* table, size_t n_candidates, const float* first,
                               const float* second, size_t n_queries, size_t dim, double gamma, double cen,
                               const int64_t* answer_ptr, const int64_t* answer_ids, size_t n_answers,
                               size_t max_answers, int64_t* ranks, void* workspace, size_t workspace_bytes,
                               void* stream) {
  return score_filtered_ranks_impl(dist_id, table, n_candidates, first, second, n_queries, dim, gamma, cen, answer_ptr,
                                   answer_ids, n_answers, max_answers, nullptr, ranks, workspace, workspace_bytes, stream);
}

int smore_score_hard_ranks(int dist_id, const float* table, size_t n_candidates, const float* first, const float* second,
                           size_t n_queries, size_t dim, double gamma, double cen, const int64_t* answer_ptr,
                           const int64_t* answer_ids, size_t n_answers, size_t max_answers, const int64_t* hard_ptr,
                           int64_t* hard_ranks, void* workspace, size_t workspace_bytes, void* stream) {
  if (!hard_ptr) return fail(SMORE_ERR_NULL, "score_hard_ranks: hard_ptr is NULL");
  return score_filtered_ranks_impl(dist_id, table, n_candidates, first, second, n_queries, dim, gamma, cen, answer_ptr,
                                   answer_ids, n_answers, max_answers, hard_ptr, hard_ranks, workspace, workspace_bytes,
                                   stream);
}

int smore_shared_status(int* status) {   // not part of the public header; smore_async_status adds it in
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_shared_status, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status: cannot read the status word");
  *status = v;
  return SMORE_OK;
}

int smore_shared_status_clear(void) {
  const int zero = 0;
  if (cudaMemcpyToSymbol(g_shared_status, &zero, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status_clear: cannot write the status word");
  return SMORE_OK;
}

}  // extern "C"

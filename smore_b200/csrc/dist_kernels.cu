// Distance-op kernels for sm_100a and their C entry points.
//
// The "row-stream" kernels take the training shape in which every query owns its own candidate
// rows (entity [B, K, W] or table + idx[B, K]; query [B, 1, dim]).  A CTA keeps one query
// in registers and streams a block of that query's candidate rows, several rows in flight per
// warp; backward produces the row gradients and the query gradient in the same pass.  This is
// the HBM-bound hot path.  Rows whose length is a multiple of four floats move in 16-byte pieces,
// others in 8- or 4-byte pieces.  Other shapes: shared_kernels.cu, cell_kernels.cu.
//
// Replaces smore/common/torchext/common_kernel.h:33-145 (the three reference kernels and their
// launchers) and the dispatch of smore/common/torchext/ext_cuda_kernel.cu:25-77.
#include <cuda_runtime.h>

#include <type_traits>

#include "bulk_copy.cuh"
#include "dist_common.cuh"
#include "update_math.cuh"

namespace smore {

// Device status word of this file's kernels (kStatus* bits): a bulk-copy wait that gave up, a row id
// outside the table.  Either makes the results of the launch invalid; smore_async_status reads it.
static __device__ int g_async_status = 0;

// ----------------------------------------------------------------------------------------
// row-stream kernels (per-query candidate rows)
// ----------------------------------------------------------------------------------------

constexpr int kUnionBranches = 2;   // query branches the fused union kernels take
constexpr int kRowCtaThreads = 256;
constexpr int kRowCtaWarps = kRowCtaThreads / kWarp;

struct RowArgs {
  const float* ent;        // dense [B*K, W] or table [N, W] when idx != nullptr
  const int64_t* idx;      // nullable [B*K]
  const float* first;      // [B, dim]
  const float* second;     // [B, dim]
  int K;                   // candidate rows per query
  int dim;                 // multiple of 4
  int rows_per_cta;        // multiple of kRowCtaWarps * wrows
  int chunks;              // CTAs per query
  int wrows;               // rows a warp takes per sweep (<= 32)
  long long n_rows;        // rows of `ent` when idx != nullptr (0: ids are not checked)
  // Ragged form (bulk-copy kernels): query q has the seg[q].y candidate rows whose ids are
  // idx[seg[q].x ...]; results and upstream gradients are indexed by the same compact positions.
  // One CTA per query; K, rows_per_cta and chunks are not used.
  const int2* seg;
  // Ragged form on the owner of a row shard: query q belongs to rank q / seg_per_rank, and the
  // result / upstream gradient of compact position p lives at positions[p] in THAT rank's arrays
  // (peer memory): out_ptrs / up_ptrs hold one base pointer per rank and output.  positions ==
  // nullptr: results and upstream gradients are local arrays indexed by compact position.
  // With NB branches per query the rank's arrays are [query][branch][K]: positions[p] names branch 0,
  // branch u sits u * branch_stride (= that rank's K) further.
  const int32_t* positions;
  int seg_per_rank;
  int branch_stride;
  float* const* out_ptrs[2];
  const float* const* up_ptrs[2];
};

// The block of candidate rows a CTA of the row-stream kernels works on.
struct RowBlock {
  int b;            // query
  int r_begin, r_end;
  size_t pos_base;  // position of the query's row 0 in idx / results
};

__device__ __forceinline__ RowBlock row_block(const RowArgs& a) {
  RowBlock rb;
  if (a.seg != nullptr) {
    const int2 s = a.seg[blockIdx.x];
    rb.b = (int)blockIdx.x;
    rb.r_begin = 0;
    rb.r_end = s.y;
    rb.pos_base = (size_t)s.x;
  } else {
    rb.b = blockIdx.x / a.chunks;
    const int c = blockIdx.x - rb.b * a.chunks;
    rb.r_begin = c * a.rows_per_cta;
    rb.r_end = min(a.K, rb.r_begin + a.rows_per_cta);
    rb.pos_base = (size_t)rb.b * a.K;
  }
  return rb;
}

// First float of the block's NB query rows in `first` / `second` / the query-gradient arrays.  Dense
// form: query b's rows start at b * NB * dim.  Ragged form: rank r's queries occupy seg_per_rank * dim
// floats starting at r * seg_per_rank * dim, query q of that rank at q * NB * dim inside them.
template <int NB>
__device__ __forceinline__ size_t query_offset(const RowArgs& a, int b) {
  if (a.seg == nullptr) return (size_t)b * NB * a.dim;
  const int rank = b / a.seg_per_rank, q = b - rank * a.seg_per_rank;
  return ((size_t)rank * a.seg_per_rank + (size_t)q * NB) * a.dim;
}

__device__ __forceinline__ float4 ld_row4(const float4* p) { return __ldg(p); }

// acc over the 4 components of one 16-byte chunk
template <class Term, bool FAST>
__device__ __forceinline__ void fwd1(float e0, float e1, float q0, float q1, float* acc) {
  if constexpr (FAST) Term::fwd_fast(e0, e1, q0, q1, acc);
  else Term::fwd(e0, e1, q0, q1, acc);
}
template <class Term, bool FAST = false>
__device__ __forceinline__ void fwd4(const float4& e0, const float4& e1, const float4& q0,
                                     const float4& q1, float* acc) {
  fwd1<Term, FAST>(e0.x, e1.x, q0.x, q1.x, acc);
  fwd1<Term, FAST>(e0.y, e1.y, q0.y, q1.y, acc);
  fwd1<Term, FAST>(e0.z, e1.z, q0.z, q1.z, acc);
  fwd1<Term, FAST>(e0.w, e1.w, q0.w, q1.w, acc);
}

// POS: every q1 of the query is positive (see Term::kPositive)
template <class Term, bool POS>
__device__ __forceinline__ void bwd1(const float* g, float e0, float e1, float q0, float q1, float& ge0, float& ge1,
                                     float& gq0, float& gq1) {
  if (POS) Term::bwd_pos(g, e0, e1, q0, q1, ge0, ge1, gq0, gq1);
  else Term::bwd(g, e0, e1, q0, q1, ge0, ge1, gq0, gq1);
}

template <class Term, bool POS>
__device__ __forceinline__ void bwd4(const float* g, const float4& e0, const float4& e1,
                                     const float4& q0, const float4& q1, float4& ge0, float4& ge1,
                                     float4& gq0, float4& gq1) {
  bwd1<Term, POS>(g, e0.x, e1.x, q0.x, q1.x, ge0.x, ge1.x, gq0.x, gq1.x);
  bwd1<Term, POS>(g, e0.y, e1.y, q0.y, q1.y, ge0.y, ge1.y, gq0.y, gq1.y);
  bwd1<Term, POS>(g, e0.z, e1.z, q0.z, q1.z, ge0.z, ge1.z, gq0.z, gq1.z);
  bwd1<Term, POS>(g, e0.w, e1.w, q0.w, q1.w, ge0.w, ge1.w, gq0.w, gq1.w);
}

template <class Term>
__device__ __forceinline__ float4 prep4(const float4& q) {
  return make_float4(Term::prep(q.x), Term::prep(q.y), Term::prep(q.z), Term::prep(q.w));
}
__device__ __forceinline__ bool positive4(const float4& q) { return q.x > 0.f && q.y > 0.f && q.z > 0.f && q.w > 0.f; }

// V consecutive floats of a row: the unit in which the kernels of any row length move data
template <int V>
struct alignas(4 * V) Piece {
  float v[V];
};
template <int V>
__device__ __forceinline__ Piece<V> piece_load(const float* p) {
  Piece<V> r;
  if constexpr (V == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(p));
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
  } else if constexpr (V == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(p));
    r.v[0] = t.x; r.v[1] = t.y;
  } else {
    r.v[0] = __ldg(p);
  }
  return r;
}
template <int V>
__device__ __forceinline__ void piece_add(float* p, const Piece<V>& x) {
  if constexpr (V == 4) atomicAdd(reinterpret_cast<float4*>(p), make_float4(x.v[0], x.v[1], x.v[2], x.v[3]));
  else if constexpr (V == 2) atomicAdd(reinterpret_cast<float2*>(p), make_float2(x.v[0], x.v[1]));
  else atomicAdd(p, x.v[0]);
}
template <int V>
__device__ __forceinline__ void piece_store(float* p, const Piece<V>& x) { *reinterpret_cast<Piece<V>*>(p) = x; }

template <class Term, int NCH, int R>
__global__ void __launch_bounds__(kRowCtaThreads)
    row_forward_kernel(RowArgs a, float* __restrict__ dst0, float* __restrict__ dst1) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x / a.chunks, c = blockIdx.x - b * a.chunks;
  const int dim4 = a.dim >> 2;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);

  float4 q0[NCH], q1[NCH];
  {
    const float4* p0 = reinterpret_cast<const float4*>(a.first + (size_t)b * a.dim);
    const float4* p1 = reinterpret_cast<const float4*>(a.second + (size_t)b * a.dim);
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      const int d4 = lane + 32 * j;
      q0[j] = d4 < dim4 ? __ldg(p0 + d4) : z4;
      q1[j] = (Term::kNQ == 2 && d4 < dim4) ? __ldg(p1 + d4) : z4;
    }
  }

  const int r_begin = c * a.rows_per_cta;
  const int r_end = min(a.K, r_begin + a.rows_per_cta);
  const size_t w4 = (size_t)dim4 * Term::kMul;
  const float4* ent4 = reinterpret_cast<const float4*>(a.ent);

  for (int base = r_begin + warp * a.wrows; base < r_end; base += kRowCtaWarps * a.wrows) {
    const int n = min(a.wrows, r_end - base);
    const size_t pos = (size_t)b * a.K + base + lane;
    long long myrow = 0;   // -1: an id outside the table (row 0 is read instead, the result is NaN)
    if (lane < n) myrow = a.idx ? checked_row_id(a.idx, pos, a.n_rows, &g_async_status) : (long long)pos;
    float out0 = 0.f, out1 = 0.f;
    for (int t = 0; t < n; t += R) {
      float4 e[R][Term::kMul][NCH];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const long long row = max(__shfl_sync(0xffffffffu, myrow, min(t + r, n - 1)), 0LL);
        const float4* pe = ent4 + (size_t)row * w4;
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
          const int d4 = lane + 32 * j;
          if (d4 < dim4) {
            e[r][0][j] = ld_row4(pe + d4);
            if (Term::kMul == 2) e[r][Term::kMul - 1][j] = ld_row4(pe + dim4 + d4);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float acc[Term::kNOut];
#pragma unroll
        for (int o = 0; o < Term::kNOut; ++o) acc[o] = 0.f;
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
          if (lane + 32 * j < dim4) fwd4<Term>(e[r][0][j], e[r][Term::kMul - 1][j], q0[j], q1[j], acc);
        }
#pragma unroll
        for (int o = 0; o < Term::kNOut; ++o) acc[o] = warp_sum(acc[o]);
        if (lane == t + r) {
          out0 = acc[0];
          out1 = acc[Term::kNOut - 1];
        }
      }
    }
    if (lane < n) {
      dst0[pos] = myrow < 0 ? NAN : out0;
      if (Term::kNOut == 2) dst1[pos] = myrow < 0 ? NAN : out1;
    }
  }
}

struct RowGradArgs {
  const float* gout0;         // [B, K]
  const float* gout1;         // [B, K] (two-output term only)
  float* g_ent;               // dense [B*K, W], or nullptr when slot != nullptr
  const int32_t* slot;        // [B*K] -> row of g_rows, < 0 to skip
  const int32_t* slot_count;  // contributors per slot over the whole step
  float* g_rows;              // [capacity, W]
  float* g_first;             // [B, dim]
  float* g_second;            // [B, dim]
  int query_atomic;           // several CTAs share one query: accumulate into zeroed g_first/second
};

__device__ __forceinline__ void add4(float4& a, const float4& b) {
  a.x += b.x;
  a.y += b.y;
  a.z += b.z;
  a.w += b.w;
}

// Forward for rows that cannot move in 16-byte pieces, or are too long for the kernels above: the query
// sits in shared memory, a warp takes R rows at a time and walks their columns in V-float pieces.
// (333 x 101 rows of 250 floats: 17 us with one warp per row and one 4-byte load in flight per lane.)
template <class Term, int V>
__global__ void __launch_bounds__(kRowCtaThreads)
    row_forward_any_kernel(RowArgs a, float* __restrict__ dst0, float* __restrict__ dst1) {
  constexpr int R = 4;
  extern __shared__ __align__(16) float sq_any[];   // [kNQ][dim]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x / a.chunks, c = blockIdx.x - b * a.chunks;
  for (int i = threadIdx.x; i < a.dim; i += kRowCtaThreads) {
    sq_any[i] = __ldg(a.first + (size_t)b * a.dim + i);
    if (Term::kNQ == 2) sq_any[a.dim + i] = __ldg(a.second + (size_t)b * a.dim + i);
  }
  __syncthreads();
  const int r_begin = c * a.rows_per_cta, r_end = min(a.K, r_begin + a.rows_per_cta);
  const size_t width = (size_t)a.dim * Term::kMul;
  for (int base = r_begin + warp * a.wrows; base < r_end; base += kRowCtaWarps * a.wrows) {
    const int n = min(a.wrows, r_end - base);
    const size_t pos = (size_t)b * a.K + base + lane;
    long long myrow = 0;   // -1: an id outside the table (row 0 is read instead, the result is NaN)
    if (lane < n) myrow = a.idx ? checked_row_id(a.idx, pos, a.n_rows, &g_async_status) : (long long)pos;
    float out0 = 0.f, out1 = 0.f;
    for (int t = 0; t < n; t += R) {
      const float* pe[R];
      float acc[R][Term::kNOut];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        pe[r] = a.ent + (size_t)max(__shfl_sync(0xffffffffu, myrow, min(t + r, n - 1)), 0LL) * width;
#pragma unroll
        for (int o = 0; o < Term::kNOut; ++o) acc[r][o] = 0.f;
      }
#pragma unroll 2
      for (int d = lane * V; d < a.dim; d += 32 * V) {
        Piece<V> e0[R], e1[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          e0[r] = piece_load<V>(pe[r] + d);
          e1[r] = Term::kMul == 2 ? piece_load<V>(pe[r] + a.dim + d) : e0[r];
        }
        const Piece<V> q0 = *reinterpret_cast<const Piece<V>*>(sq_any + d);
        const Piece<V> q1 = Term::kNQ == 2 ? *reinterpret_cast<const Piece<V>*>(sq_any + a.dim + d) : q0;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int i = 0; i < V; ++i) Term::fwd(e0[r].v[i], e1[r].v[i], q0.v[i], q1.v[i], acc[r]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int o = 0; o < Term::kNOut; ++o) acc[r][o] = warp_sum(acc[r][o]);
        if (lane == t + r) {
          out0 = acc[r][0];
          out1 = acc[r][Term::kNOut - 1];
        }
      }
    }
    if (lane < n) {
      dst0[pos] = myrow < 0 ? NAN : out0;
      if (Term::kNOut == 2) dst1[pos] = myrow < 0 ? NAN : out1;
    }
  }
}

// Backward of the row-stream shape.  The gradient of a row element needs no reduction over the
// embedding dim, so the CTA is laid out by columns: `tpr` consecutive threads (a multiple of 32)
// own the V-float columns of a row and `groups` such thread groups take alternate rows of the
// CTA's block; rows of more than kRowCtaThreads columns are cut into column blocks (blockIdx.y).
// A thread keeps only its column of the query and of the query gradient in
// registers (a handful of registers: high occupancy), has U row loads in flight, and writes its
// column of each row gradient.  Per-row scalars (row offset, output gradients, destination) are
// fetched 32 rows at a time by the lanes of each warp into a warp-private shared-memory table, so
// the inner loop is one broadcast read, one add and one access of V floats per operand: the kernel
// has to stay well under the SM's issue rate to be bound by HBM instead.
template <class Term, int U, int V>
__global__ void __launch_bounds__(kRowCtaThreads)
    col_backward_kernel(RowArgs a, RowGradArgs ga, int tpr, int groups) {
  extern __shared__ __align__(16) float red[];  // [groups][kNQ][cols of the block][V]
  __shared__ size_t meta_src[kRowCtaWarps][32];
  __shared__ long long meta_dst[kRowCtaWarps][32];
  __shared__ float2 meta_g[kRowCtaWarps][32];
  __shared__ int meta_single[kRowCtaWarps][32];
  const int lane = threadIdx.x & 31;
  const int grp = threadIdx.x / tpr, lcol = threadIdx.x - grp * tpr;
  const int b = blockIdx.x / a.chunks, c = blockIdx.x - b * a.chunks;
  const int cols = min(kRowCtaThreads, a.dim / V - (int)blockIdx.y * kRowCtaThreads);   // of this column block
  const bool active = grp < groups && lcol < cols;
  const size_t at = ((size_t)blockIdx.y * kRowCtaThreads + lcol) * V;                   // first float of the column
  const size_t width = (size_t)a.dim * Term::kMul;
  float* gbase = ga.slot ? ga.g_rows : ga.g_ent;

  Piece<V> q0 = {}, q1 = {}, gq0 = {}, gq1 = {};
  bool pos_ok = true;
  if (active) {
    q0 = piece_load<V>(a.first + (size_t)b * a.dim + at);
    if (Term::kNQ == 2) q1 = piece_load<V>(a.second + (size_t)b * a.dim + at);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      q0.v[i] = Term::prep(q0.v[i]);
      pos_ok = pos_ok && q1.v[i] > 0.f;
    }
  }
  const bool positive = Term::kPositive && __syncthreads_and(pos_ok);

  const int r_begin = c * a.rows_per_cta;
  const int r_end = min(a.K, r_begin + a.rows_per_cta);
  auto walk = [&](auto pos_tag) {
    constexpr bool POS = decltype(pos_tag)::value;
    // this group's rows: r_begin + grp + groups * t, t = 0, 1, ...
    const int n_mine = (r_end - r_begin - grp + groups - 1) / groups;
    const int warp = threadIdx.x >> 5;
    for (int t0 = 0; t0 < n_mine; t0 += 32) {
      const int n = min(32, n_mine - t0);
      // Each warp keeps its own copy of the next 32 rows' scalars in shared memory: where the row
      // starts, where its gradient goes, the output gradients, and whether the destination is stored or
      // accumulated.
      __syncwarp();
      {
        const int l = lane < n ? lane : 0;   // surplus lanes repeat the tile's first row: harmless loads
        const size_t pos = (size_t)b * a.K + r_begin + grp + (size_t)groups * (t0 + l);
        const long long row = a.idx ? checked_row_id(a.idx, pos, a.n_rows, &g_async_status) : (long long)pos;
        long long dst = (long long)pos;
        int single = 1;
        if (ga.slot) {
          const int32_t s = ga.slot[pos];
          dst = s;
          single = (s >= 0 && ga.slot_count != nullptr) ? (ga.slot_count[s] == 1) : 0;
        }
        // an id outside the table: row 0 is read, no gradient is written and, with the output
        // gradients zeroed, nothing reaches the query gradient either
        const bool bad = row < 0;
        meta_src[warp][lane] = bad ? 0 : (size_t)row * width;
        meta_dst[warp][lane] = (dst < 0 || bad) ? -1 : dst * (long long)width;
        meta_g[warp][lane] = bad ? make_float2(0.f, 0.f)
                                 : make_float2(ga.gout0[pos], Term::kNOut == 2 ? ga.gout1[pos] : 0.f);
        meta_single[warp][lane] = single;
      }
      __syncwarp();
      for (int t = 0; t < n; t += U) {
        Piece<V> e0[U], e1[U];
        if (active) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float* pe = a.ent + meta_src[warp][t + u] + at;
            e0[u] = piece_load<V>(pe);
            e1[u] = Term::kMul == 2 ? piece_load<V>(pe + a.dim) : e0[u];
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (t + u < n) {
              const float2 g2 = meta_g[warp][t + u];
              const long long dst = meta_dst[warp][t + u];
              float g[Term::kNOut];
              g[0] = g2.x;
              if (Term::kNOut == 2) g[Term::kNOut - 1] = g2.y;
              Piece<V> ge0 = {}, ge1 = {};
#pragma unroll
              for (int i = 0; i < V; ++i)
                bwd1<Term, POS>(g, e0[u].v[i], e1[u].v[i], q0.v[i], q1.v[i], ge0.v[i], ge1.v[i], gq0.v[i], gq1.v[i]);
              if (dst >= 0) {
                float* out = gbase + dst + at;
                if (meta_single[warp][t + u]) {
                  piece_store(out, ge0);
                  if (Term::kMul == 2) piece_store(out + a.dim, ge1);
                } else {
                  piece_add(out, ge0);
                  if (Term::kMul == 2) piece_add(out + a.dim, ge1);
                }
              }
            }
          }
        }
      }
    }
  };
  if (grp < groups) {
    if (positive) walk(std::true_type{});
    else walk(std::false_type{});
  }

  // fold the groups' query gradients in group order (fixed order: deterministic per CTA)
  Piece<V>* fold = reinterpret_cast<Piece<V>*>(red);
  if (active) {
    fold[(size_t)grp * Term::kNQ * cols + lcol] = gq0;
    if (Term::kNQ == 2) fold[(size_t)grp * Term::kNQ * cols + cols + lcol] = gq1;
  }
  __syncthreads();
  if (grp == 0 && active) {
    for (int gi = 1; gi < groups; ++gi) {
      const Piece<V> x0 = fold[(size_t)gi * Term::kNQ * cols + lcol];
#pragma unroll
      for (int i = 0; i < V; ++i) gq0.v[i] += x0.v[i];
      if (Term::kNQ == 2) {
        const Piece<V> x1 = fold[(size_t)gi * Term::kNQ * cols + cols + lcol];
#pragma unroll
        for (int i = 0; i < V; ++i) gq1.v[i] += x1.v[i];
      }
    }
    float* gf = ga.g_first + (size_t)b * a.dim + at;
    float* gs = ga.g_second + (size_t)b * a.dim + at;
    if (ga.query_atomic) {
      piece_add(gf, gq0);
      if (Term::kNQ == 2) piece_add(gs, gq1);
    } else {
      piece_store(gf, gq0);
      if (Term::kNQ == 2) piece_store(gs, gq1);
    }
  }
}

// ----------------------------------------------------------------------------------------
// Row-stream forward with the rows staged through shared memory by bulk asynchronous copies.
// Each warp owns a ring of `stages` row slots and one mbarrier per slot; lane 0 keeps `stages`
// row copies (one instruction per row) in flight ahead of the row the warp is reducing, so the
// bytes in flight per SM no longer depend on registers or on how many warps are resident.
// Work split: the CTA's block of rows is cut into one contiguous run per warp.
// ----------------------------------------------------------------------------------------

__host__ __device__ inline size_t bulk_ring_offset(int stages) {
  return ((size_t)kRowCtaWarps * stages * sizeof(uint64_t) + 127) & ~(size_t)127;
}

// A lane's share of a row: 16-byte pieces lane, lane + 32, ... of every part.  With TAIL the last of the
// NCH pieces of a warp covers at most 32 floats and is taken one float per lane: rows of 400 floats are
// 3 pieces and 16 floats, a quarter of the work of a fourth piece with 4 of 32 lanes busy.
template <int NCH, bool TAIL>
struct LanePieces {
  static constexpr int kFull = TAIL ? NCH - 1 : NCH;
  // f4(j, index of the piece within a part), then f1(index of the float)
  template <class F4, class F1>
  __device__ __forceinline__ static void each(int lane, int dim, F4&& f4, F1&& f1) {
#pragma unroll
    for (int j = 0; j < kFull; ++j) {
      const int d4 = lane + 32 * j;
      if (TAIL || d4 < (dim >> 2)) f4(j, d4);
    }
    if (TAIL) {
      const int d = 128 * kFull + lane;
      if (d < dim) f1(d);
    }
  }
};
// pieces and tail of a row of `dim` floats per part
inline bool row_tail(size_t dim, int nch) { return dim > 128 * (size_t)(nch - 1) && dim <= 128 * (size_t)(nch - 1) + 32; }

// NB: query branches scored against every row (union queries; results [query][branch][row]).
template <class Term, int NB, int NCH, bool TAIL>
__global__ void __launch_bounds__(kRowCtaThreads)
    row_forward_bulk_kernel(RowArgs a, float* __restrict__ dst0, float* __restrict__ dst1, int stages) {
  extern __shared__ __align__(128) unsigned char bulk_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const RowBlock rb = row_block(a);
  if (rb.r_end <= rb.r_begin) return;    // (ragged form: a query without rows here)
  const int b = rb.b;
  const int dim4 = a.dim >> 2;
  const unsigned row_bytes = (unsigned)dim4 * Term::kMul * 16u;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  uint64_t* bars = reinterpret_cast<uint64_t*>(bulk_smem) + warp * stages;
  unsigned char* ring = bulk_smem + bulk_ring_offset(stages) + (size_t)warp * stages * row_bytes;
  if (lane == 0) {
    for (int s = 0; s < stages; ++s) bulk::barrier_init(bars + s, 1);
    bulk::fence_barrier_init();
  }
  __syncthreads();

  using Lanes = LanePieces<NCH, TAIL>;
  float4 q0[NB][Lanes::kFull], q1[NB][Lanes::kFull];
  float t0[NB], t1[NB];                    // the tail's floats
  {
    const size_t q_off = query_offset<NB>(a, b);
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      const float* p0 = a.first + q_off + (size_t)u * a.dim;
      const float* p1 = a.second + q_off + (size_t)u * a.dim;
#pragma unroll
      for (int j = 0; j < Lanes::kFull; ++j) q0[u][j] = q1[u][j] = z4;
      t0[u] = t1[u] = 0.f;
      Lanes::each(lane, a.dim,
                  [&](int j, int d4) {
                    q0[u][j] = __ldg(reinterpret_cast<const float4*>(p0) + d4);
                    if (Term::kNQ == 2) q1[u][j] = __ldg(reinterpret_cast<const float4*>(p1) + d4);
                  },
                  [&](int d) {
                    t0[u] = __ldg(p0 + d);
                    if (Term::kNQ == 2) t1[u] = __ldg(p1 + d);
                  });
    }
  }

  const int r_begin = rb.r_begin, r_end = rb.r_end;
  const int per_warp = (r_end - r_begin + kRowCtaWarps - 1) / kRowCtaWarps;
  const int w_begin = r_begin + warp * per_warp;
  const int n = max(0, min(r_end, w_begin + per_warp) - w_begin);
  const size_t pos0 = rb.pos_base + w_begin;
  const unsigned char* ent = reinterpret_cast<const unsigned char*>(a.ent);

  // row ids of a batch of 32 rows, one per lane; -1 marks an id outside the table (row 0 is copied
  // in its place and the result written for it is NaN)
  auto batch_ids = [&](int first_t) -> long long {
    const int t = first_t + lane;
    if (t >= n) return 0;
    return a.idx ? checked_row_id(a.idx, pos0 + t, a.n_rows, &g_async_status) : (long long)(pos0 + t);
  };
  long long cur = batch_ids(0), nxt = 0;
  // prologue: fill the ring
  const int ahead = min(stages, n);
  for (int t = 0; t < ahead; ++t) {
    const long long row = max(__shfl_sync(0xffffffffu, cur, t), 0LL);
    if (lane == 0) {
      bulk::barrier_expect(bars + t, row_bytes);
      bulk::load(ring + (size_t)t * row_bytes, ent + (size_t)row * row_bytes, row_bytes, bars + t);
    }
  }
  int slot = 0;
  unsigned parity = 0;
  float out0[NB], out1[NB];
#pragma unroll
  for (int u = 0; u < NB; ++u) out0[u] = out1[u] = 0.f;
  for (int t = 0; t < n; ++t) {
    const int tl = t & 31;
    if (tl == 0) nxt = batch_ids(t + 32);
    bool ok = bulk::barrier_wait(bars + slot, parity);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      // give up: let the copies still in flight land (bounded), flag the failure, stop
      if (lane == 0) atomicOr(&g_async_status, kStatusCopyWait);
      for (int k = 1; k < stages && t + k < n; ++k) {
        const int s2 = (slot + k) % stages;
        bulk::barrier_wait(bars + s2, s2 > slot ? parity : parity ^ 1u);
      }
      break;
    }
    const float* row = reinterpret_cast<const float*>(ring + (size_t)slot * row_bytes);
    const float4* row4 = reinterpret_cast<const float4*>(row);
    float acc[NB][Term::kNOut];
    auto score = [&](auto fast_tag) {
      constexpr bool FAST = decltype(fast_tag)::value;
#pragma unroll
      for (int u = 0; u < NB; ++u)
#pragma unroll
        for (int o = 0; o < Term::kNOut; ++o) acc[u][o] = 0.f;
      Lanes::each(lane, a.dim,
                  [&](int j, int d4) {
                    const float4 e0 = row4[d4];
                    const float4 e1 = Term::kMul == 2 ? row4[dim4 + d4] : e0;
#pragma unroll
                    for (int u = 0; u < NB; ++u) fwd4<Term, FAST>(e0, e1, q0[u][j], q1[u][j], acc[u]);
                  },
                  [&](int d) {
                    const float e0 = row[d], e1 = Term::kMul == 2 ? row[a.dim + d] : e0;
#pragma unroll
                    for (int u = 0; u < NB; ++u) fwd1<Term, FAST>(e0, e1, t0[u], t1[u], acc[u]);
                  });
#pragma unroll
      for (int u = 0; u < NB; ++u)
#pragma unroll
        for (int o = 0; o < Term::kNOut; ++o) acc[u][o] = warp_sum(acc[u][o]);
    };
    score(std::integral_constant<bool, Term::kFast>{});
    if constexpr (Term::kFast) {     // NaN operands: again, with the exact rule (every lane holds the same sums)
      bool nan = false;
#pragma unroll
      for (int u = 0; u < NB; ++u) nan = nan || acc[u][0] != acc[u][0];
      if (nan) score(std::false_type{});
    }
    // the sums above consumed every lane's reads of the slot: it may be refilled
    __syncwarp();
    const int tn = t + stages;
    if (tn < n) {
      const long long row = max(__shfl_sync(0xffffffffu, (tn >> 5) == (t >> 5) ? cur : nxt, tn & 31), 0LL);
      if (lane == 0) {
        bulk::barrier_expect(bars + slot, row_bytes);
        bulk::load(ring + (size_t)slot * row_bytes, ent + (size_t)row * row_bytes, row_bytes, bars + slot);
      }
    }
    if (lane == tl) {
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        out0[u] = acc[u][0];
        out1[u] = acc[u][Term::kNOut - 1];
      }
    }
    if (tl == 31 || t == n - 1) {
      if (lane <= tl) {
        const size_t o = pos0 + (t - tl) + lane;
        if (a.positions != nullptr) {          // straight into the requesting rank's result arrays
          const int rank = b / a.seg_per_rank;
          const size_t at = (size_t)a.positions[o];
#pragma unroll
          for (int u = 0; u < NB; ++u) {
            a.out_ptrs[0][rank][at + (size_t)u * a.branch_stride] = cur < 0 ? NAN : out0[u];
            if (Term::kNOut == 2) a.out_ptrs[1][rank][at + (size_t)u * a.branch_stride] = cur < 0 ? NAN : out1[u];
          }
        } else {                                // local result arrays ([query][branch][row])
#pragma unroll
          for (int u = 0; u < NB; ++u) {
            const size_t at = NB == 1 ? o : ((size_t)b * NB + u) * a.K + (o - (size_t)b * a.K);
            dst0[at] = cur < 0 ? NAN : out0[u];
            if (Term::kNOut == 2) dst1[at] = cur < 0 ? NAN : out1[u];
          }
        }
      }
      cur = nxt;
    }
    if (++slot == stages) {
      slot = 0;
      parity ^= 1u;
    }
  }
}

// ----------------------------------------------------------------------------------------
// Row-stream backward on the same bulk-copy ring.  A warp takes a contiguous run of rows; each
// row is copied into a ring slot, its gradient is computed IN PLACE over the row (every lane
// overwrites exactly the 16-byte pieces it read), and lane 0 sends the slot to the gradient
// buffer with one bulk store - or one bulk floating-point add where several positions of the
// step share the destination row.  The slot is refilled once that transfer has read it.
// NB query branches (union queries) are applied to every row; their row gradients are summed in
// registers before the slot is written.  The query gradients stay in registers over the warp's
// run and are folded over the CTA's warps through the ring at the end, in warp order.
// ----------------------------------------------------------------------------------------

template <class Term, int NB, int NCH>
__global__ void __launch_bounds__(kRowCtaThreads, 2)
    row_backward_bulk_kernel(RowArgs a, RowGradArgs ga, int stages) {
  constexpr int NG = NB * Term::kNOut;
  extern __shared__ __align__(128) unsigned char bulk_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x / a.chunks, c = blockIdx.x - b * a.chunks;
  const int dim4 = a.dim >> 2;
  const unsigned row_bytes = (unsigned)dim4 * Term::kMul * 16u;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  uint64_t* bars = reinterpret_cast<uint64_t*>(bulk_smem) + warp * stages;
  float4* sq = reinterpret_cast<float4*>(bulk_smem + bulk_ring_offset(stages));   // [kNQ][NB][dim4]
  unsigned char* ring_all = reinterpret_cast<unsigned char*>(sq + (size_t)Term::kNQ * NB * dim4);
  unsigned char* ring = ring_all + (size_t)warp * stages * row_bytes;
  if (lane == 0) {
    for (int s = 0; s < stages; ++s) bulk::barrier_init(bars + s, 1);
    bulk::fence_barrier_init();
  }
  bool pos_ok = true;
  {
    const float4* p0 = reinterpret_cast<const float4*>(a.first + (size_t)b * NB * a.dim);
    const float4* p1 = reinterpret_cast<const float4*>(a.second + (size_t)b * NB * a.dim);
    for (int i = threadIdx.x; i < NB * dim4; i += kRowCtaThreads) {
      sq[i] = prep4<Term>(__ldg(p0 + i));
      if (Term::kNQ == 2) {
        sq[NB * dim4 + i] = __ldg(p1 + i);
        pos_ok = pos_ok && positive4(sq[NB * dim4 + i]);
      }
    }
  }
  const bool positive = __syncthreads_and(pos_ok) && Term::kPositive;
  const float4* sq0 = sq;
  const float4* sq1 = Term::kNQ == 2 ? sq + NB * dim4 : sq;

  float4 gq0[NB][NCH], gq1[NB][NCH];
#pragma unroll
  for (int u = 0; u < NB; ++u)
#pragma unroll
    for (int j = 0; j < NCH; ++j) gq0[u][j] = gq1[u][j] = z4;

  const int r_begin = c * a.rows_per_cta;
  const int r_end = min(a.K, r_begin + a.rows_per_cta);
  const int per_warp = (r_end - r_begin + kRowCtaWarps - 1) / kRowCtaWarps;
  const int w_begin = r_begin + warp * per_warp;
  const int n = max(0, min(r_end, w_begin + per_warp) - w_begin);
  const size_t pos0 = (size_t)b * a.K + w_begin;
  const unsigned char* ent = reinterpret_cast<const unsigned char*>(a.ent);
  unsigned char* gbase = reinterpret_cast<unsigned char*>(ga.slot ? ga.g_rows : ga.g_ent);

  // per-lane scalars of one batch of 32 rows: source row, destination row (-1: none), whether the
  // destination is written by this position alone, output gradients of every branch
  struct Meta {
    long long src, dst;
    int single;
    float g[NG];
  };
  auto load_meta = [&](int first_t) {
    Meta m;
    m.src = 0;
    m.dst = -1;
    m.single = 1;
#pragma unroll
    for (int i = 0; i < NG; ++i) m.g[i] = 0.f;
    const int t = first_t + lane;
    if (t < n) {
      const size_t pos = pos0 + t;
      m.src = a.idx ? checked_row_id(a.idx, pos, a.n_rows, &g_async_status) : (long long)pos;
      m.dst = (long long)pos;
      if (ga.slot) {
        const int32_t sl = ga.slot[pos];
        m.dst = sl;
        m.single = (sl >= 0 && ga.slot_count != nullptr) ? (ga.slot_count[sl] == 1) : 0;
      }
      if (m.src < 0) {
        // an id outside the table: row 0 is copied, nothing is written for it and its output
        // gradients stay zero, so the query gradients see nothing of it either
        m.src = 0;
        m.dst = -1;
      } else {
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const size_t o = ((size_t)b * NB + u) * a.K + (w_begin + t);
          m.g[u * Term::kNOut] = ga.gout0[o];
          if (Term::kNOut == 2) m.g[u * Term::kNOut + Term::kNOut - 1] = ga.gout1[o];
        }
      }
    }
    return m;
  };
  Meta cur = load_meta(0), nxt = cur;

  const int ahead = min(stages - 1, n);   // one slot always belongs to the store in flight
  for (int t = 0; t < ahead; ++t) {
    const long long row = __shfl_sync(0xffffffffu, cur.src, t);
    if (lane == 0) {
      bulk::barrier_expect(bars + t, row_bytes);
      bulk::load(ring + (size_t)t * row_bytes, ent + (size_t)row * row_bytes, row_bytes, bars + t);
    }
  }
  auto walk = [&](auto pos_tag) {
  constexpr bool POS = decltype(pos_tag)::value;
  int slot = 0;
  unsigned parity = 0;
  for (int t = 0; t < n; ++t) {
    const int tl = t & 31;
    if (tl == 0) nxt = load_meta(t + 32);
    bool ok = bulk::barrier_wait(bars + slot, parity);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0) atomicOr(&g_async_status, kStatusCopyWait);
      for (int k = 1; k < stages - 1 && t + k < n; ++k) {
        const int s2 = (slot + k) % stages;
        bulk::barrier_wait(bars + s2, s2 > slot ? parity : parity ^ 1u);
      }
      break;
    }
    float g[NG];
#pragma unroll
    for (int i = 0; i < NG; ++i) g[i] = __shfl_sync(0xffffffffu, cur.g[i], tl);
    const long long dst = __shfl_sync(0xffffffffu, cur.dst, tl);
    const int single = __shfl_sync(0xffffffffu, cur.single, tl);
    float4* row4 = reinterpret_cast<float4*>(ring + (size_t)slot * row_bytes);
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      const int d4 = lane + 32 * j;
      if (d4 < dim4) {
        const float4 e0 = row4[d4];
        const float4 e1 = Term::kMul == 2 ? row4[dim4 + d4] : e0;
        float4 ge0 = z4, ge1 = z4;
#pragma unroll
        for (int u = 0; u < NB; ++u)
          bwd4<Term, POS>(g + u * Term::kNOut, e0, e1, sq0[u * dim4 + d4], sq1[u * dim4 + d4], ge0, ge1, gq0[u][j],
                     gq1[u][j]);
        row4[d4] = ge0;
        if (Term::kMul == 2) row4[dim4 + d4] = ge1;
      }
    }
    bulk::fence_async_shared();   // the gradient row is visible to the copy engine
    __syncwarp();
    // refill target: the slot of the previous row, whose transfer was committed one row ago
    const int tn = t + stages - 1;
    const long long next_row = __shfl_sync(0xffffffffu, (tn >> 5) == (t >> 5) ? cur.src : nxt.src, tn & 31);
    if (lane == 0) {
      if (dst >= 0) {
        unsigned char* out = gbase + (size_t)dst * row_bytes;
        if (single) bulk::store(out, row4, row_bytes);
        else bulk::reduce_add_f32(out, row4, row_bytes);
      }
      bulk::commit_group();
      if (tn < n) {
        bulk::wait_group_read<1>();   // all transfers but the one just committed have read their slots
        const int s2 = slot == 0 ? stages - 1 : slot - 1;
        bulk::barrier_expect(bars + s2, row_bytes);
        bulk::load(ring + (size_t)s2 * row_bytes, ent + (size_t)next_row * row_bytes, row_bytes, bars + s2);
      }
    }
    if (tl == 31) cur = nxt;
    if (++slot == stages) {
      slot = 0;
      parity ^= 1u;
    }
  }
  };
  if (positive) walk(std::true_type{});
  else walk(std::false_type{});
  if (lane == 0) bulk::wait_group<0>();   // every gradient row has left shared memory and landed
  __syncthreads();

  // fold the warps' query gradients through the (now idle) ring, in warp order
  float4* red = reinterpret_cast<float4*>(ring_all);
  const size_t per_warp4 = (size_t)NB * Term::kNQ * dim4;
#pragma unroll
  for (int u = 0; u < NB; ++u)
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      const int d4 = lane + 32 * j;
      if (d4 < dim4) {
        red[warp * per_warp4 + (size_t)u * Term::kNQ * dim4 + d4] = gq0[u][j];
        if (Term::kNQ == 2) red[warp * per_warp4 + (size_t)u * Term::kNQ * dim4 + dim4 + d4] = gq1[u][j];
      }
    }
  __syncthreads();
  for (size_t i = threadIdx.x; i < per_warp4; i += kRowCtaThreads) {
    float4 acc = red[i];
    for (int w = 1; w < kRowCtaWarps; ++w) add4(acc, red[w * per_warp4 + i]);
    const size_t u = i / ((size_t)Term::kNQ * dim4), rem = i - u * Term::kNQ * dim4;
    const bool second = rem >= (size_t)dim4;
    float* base = second ? ga.g_second : ga.g_first;
    float4* out = reinterpret_cast<float4*>(base + ((size_t)b * NB + u) * a.dim) + (rem - (second ? dim4 : 0));
    if (ga.query_atomic) atomicAdd(out, acc);
    else *out = acc;
  }
}

// ----------------------------------------------------------------------------------------
// Row-stream backward with the optimizer step folded in (Adam, row-wise second moment).
//
// Most rows a step touches are touched by exactly one (query, candidate) position (about 95 % at
// the Freebase-scale benchmark).  For such a row the gradient this kernel computes IS the step's
// merged gradient, so writing it to the gradient buffer only to have the update kernel read it
// back - together with the parameter row this kernel has just read - is wasted traffic: per row
// 1.6 KB written and 3.2 KB read again.  Here the warp that owns the row also copies the row of
// the first moment into the ring (same bulk copy group as the parameter row), applies the update
// in shared memory and sends both rows back with bulk stores; the row's entry in the step's list
// of distinct rows is complemented (~row, negative), which the update kernel skips.  Rows with
// several contributors take the ordinary route (bulk floating-point add into the gradient buffer,
// updated afterwards by smore_sparse_update_rows).
// Safe because a row with a single contributor is read by no other position of the backward pass
// and the forward pass has finished.  The arithmetic is that of adam_rows_reg_kernel.
// ----------------------------------------------------------------------------------------

// (rows of 2 KB and more fill the shared memory of an SM with one CTA: no need to save registers for two)
template <class Term, int NB, int NCH, bool TAIL>
__global__ void __launch_bounds__(kRowCtaThreads, NCH > 4 || Term::kMul == 2 ? 1 : 2)
    row_backward_adam_bulk_kernel(RowArgs a, RowGradArgs ga, UpdateArgs ua, int64_t* __restrict__ uniq_rw, int stages) {
  constexpr int NG = NB * Term::kNOut;
  extern __shared__ __align__(128) unsigned char bulk_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const RowBlock rb = row_block(a);
  const int b = rb.b;
  const int dim4 = a.dim >> 2;
  const unsigned row_bytes = (unsigned)dim4 * Term::kMul * 16u;
  const unsigned stage_bytes = 2u * row_bytes;          // [parameter row | first-moment row]
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t q_off = query_offset<NB>(a, b);
  if (rb.r_end <= rb.r_begin) {
    // (ragged form: a query without rows here) its query gradient is zero.  A rank has room for
    // seg_per_rank / NB queries of NB rows: the segment slots beyond that are never used and own no
    // part of the query-gradient array (their offset would fall into the next rank's part).
    const bool has_slot = a.seg == nullptr || ((b % a.seg_per_rank) + 1) * NB <= a.seg_per_rank;
    if (has_slot) {
      for (int i = threadIdx.x; i < NB * dim4; i += kRowCtaThreads) {
        reinterpret_cast<float4*>(ga.g_first + q_off)[i] = z4;
        if (Term::kNQ == 2) reinterpret_cast<float4*>(ga.g_second + q_off)[i] = z4;
      }
    }
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(bulk_smem) + warp * stages;
  float4* sq = reinterpret_cast<float4*>(bulk_smem + bulk_ring_offset(stages));   // [kNQ][NB][dim4]
  unsigned char* ring_all = reinterpret_cast<unsigned char*>(sq + (size_t)Term::kNQ * NB * dim4);
  unsigned char* ring = ring_all + (size_t)warp * stages * stage_bytes;
  if (lane == 0) {
    for (int s = 0; s < stages; ++s) bulk::barrier_init(bars + s, 1);
    bulk::fence_barrier_init();
  }
  bool pos_ok = true;
  {
    const float4* p0 = reinterpret_cast<const float4*>(a.first + q_off);
    const float4* p1 = reinterpret_cast<const float4*>(a.second + q_off);
    for (int i = threadIdx.x; i < NB * dim4; i += kRowCtaThreads) {
      sq[i] = prep4<Term>(__ldg(p0 + i));
      if (Term::kNQ == 2) {
        sq[NB * dim4 + i] = __ldg(p1 + i);
        pos_ok = pos_ok && positive4(sq[NB * dim4 + i]);
      }
    }
  }
  const bool positive = __syncthreads_and(pos_ok) && Term::kPositive;
  load_dyn(ua);
  const float4* sq0 = sq;
  const float4* sq1 = Term::kNQ == 2 ? sq + NB * dim4 : sq;
  const float *sf0 = reinterpret_cast<const float*>(sq0), *sf1 = reinterpret_cast<const float*>(sq1);

  using Lanes = LanePieces<NCH, TAIL>;
  constexpr int NF = Lanes::kFull;
  float4 gq0[NB][NF], gq1[NB][NF];
  float tq0[NB], tq1[NB];                  // query gradients of the tail's floats
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    tq0[u] = tq1[u] = 0.f;
#pragma unroll
    for (int j = 0; j < NF; ++j) gq0[u][j] = gq1[u][j] = z4;
  }

  const int r_begin = rb.r_begin, r_end = rb.r_end;
  const int per_warp = (r_end - r_begin + kRowCtaWarps - 1) / kRowCtaWarps;
  const int w_begin = r_begin + warp * per_warp;
  const int n = max(0, min(r_end, w_begin + per_warp) - w_begin);
  const size_t pos0 = rb.pos_base + w_begin;
  const unsigned char* ent = reinterpret_cast<const unsigned char*>(a.ent);
  const unsigned char* mom = reinterpret_cast<const unsigned char*>(ua.m);
  unsigned char* gbase = reinterpret_cast<unsigned char*>(ga.g_rows);

  struct Meta {
    long long src, dst;
    int single;
    float v;          // second moment of a row that is updated here
    float g[NG];
  };
  auto load_meta = [&](int first_t) {
    Meta m;
    m.src = 0;
    m.dst = -1;
    m.single = 0;
    m.v = 0.f;
#pragma unroll
    for (int i = 0; i < NG; ++i) m.g[i] = 0.f;
    const int t = first_t + lane;
    if (t < n) {
      const size_t pos = pos0 + t;
      m.src = checked_row_id(a.idx, pos, a.n_rows, &g_async_status);
      const int32_t sl = ga.slot[pos];
      m.dst = sl;
      m.single = (sl >= 0 && ga.slot_count != nullptr) ? (ga.slot_count[sl] == 1) : 0;
      if (m.src < 0) {
        m.src = 0;
        m.dst = -1;
        m.single = 0;
      } else {
        if (m.single) m.v = ua.v[m.src];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          if (a.positions != nullptr) {        // from the requesting rank's arrays ([query][branch][row])
            const int rank = b / a.seg_per_rank;
            const size_t at = (size_t)a.positions[pos] + (size_t)u * a.branch_stride;
            m.g[u * Term::kNOut] = a.up_ptrs[0][rank][at];
            if (Term::kNOut == 2) m.g[u * Term::kNOut + Term::kNOut - 1] = a.up_ptrs[1][rank][at];
            continue;
          }
          // (ragged form with local arrays: upstream gradients sit at the rows' compact positions)
          const size_t o = a.seg != nullptr ? pos : ((size_t)b * NB + u) * a.K + (w_begin + t);
          m.g[u * Term::kNOut] = ga.gout0[o];
          if (Term::kNOut == 2) m.g[u * Term::kNOut + Term::kNOut - 1] = ga.gout1[o];
        }
      }
    }
    return m;
  };
  // lane 0: start the copies of one row (and, for a row updated here, of its first-moment row)
  auto issue = [&](int s, long long row, int single) {
    unsigned char* dst = ring + (size_t)s * stage_bytes;
    bulk::barrier_expect(bars + s, single ? stage_bytes : row_bytes);
    bulk::load(dst, ent + (size_t)row * row_bytes, row_bytes, bars + s);
    if (single) bulk::load(dst + row_bytes, mom + (size_t)row * row_bytes, row_bytes, bars + s);
  };
  Meta cur = load_meta(0), nxt = cur;

  const int ahead = min(stages - 1, n);   // one slot always belongs to the stores in flight
  for (int t = 0; t < ahead; ++t) {
    const long long row = __shfl_sync(0xffffffffu, cur.src, t);
    const int single = __shfl_sync(0xffffffffu, (cur.dst >= 0) ? cur.single : 0, t);
    if (lane == 0) issue(t, row, single);
  }
  auto walk = [&](auto pos_tag) {
  constexpr bool POS = decltype(pos_tag)::value;
  int slot = 0;
  unsigned parity = 0;
  for (int t = 0; t < n; ++t) {
    const int tl = t & 31;
    if (tl == 0) nxt = load_meta(t + 32);
    bool ok = bulk::barrier_wait(bars + slot, parity);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0) atomicOr(&g_async_status, kStatusCopyWait);
      for (int k = 1; k < stages - 1 && t + k < n; ++k) {
        const int s2 = (slot + k) % stages;
        bulk::barrier_wait(bars + s2, s2 > slot ? parity : parity ^ 1u);
      }
      break;
    }
    float g[NG];
#pragma unroll
    for (int i = 0; i < NG; ++i) g[i] = __shfl_sync(0xffffffffu, cur.g[i], tl);
    const long long dst = __shfl_sync(0xffffffffu, cur.dst, tl);
    const long long row = __shfl_sync(0xffffffffu, cur.src, tl);
    const int single = dst >= 0 ? __shfl_sync(0xffffffffu, cur.single, tl) : 0;
    float* row1 = reinterpret_cast<float*>(ring + (size_t)slot * stage_bytes);
    float* mom1 = reinterpret_cast<float*>(ring + (size_t)slot * stage_bytes + row_bytes);
    float4 *row4 = reinterpret_cast<float4*>(row1), *mom4 = reinterpret_cast<float4*>(mom1);
    float4 ge[Term::kMul][NF];
    float te[Term::kMul];
    float sumsq = 0.f;
#pragma unroll
    for (int part = 0; part < Term::kMul; ++part) {
      te[part] = 0.f;
#pragma unroll
      for (int k = 0; k < NF; ++k) ge[part][k] = z4;
    }
    Lanes::each(lane, a.dim,
                [&](int k, int d4) {
                  const float4 e0 = row4[d4];
                  const float4 e1 = Term::kMul == 2 ? row4[dim4 + d4] : e0;
                  float4 ge0 = z4, ge1 = z4;
#pragma unroll
                  for (int u = 0; u < NB; ++u)
                    bwd4<Term, POS>(g + u * Term::kNOut, e0, e1, sq0[u * dim4 + d4], sq1[u * dim4 + d4], ge0, ge1, gq0[u][k],
                                    gq1[u][k]);
                  ge[0][k] = ge0;
                  sumsq += ge0.x * ge0.x + ge0.y * ge0.y + ge0.z * ge0.z + ge0.w * ge0.w;
                  if (Term::kMul == 2) {
                    ge[Term::kMul - 1][k] = ge1;
                    sumsq += ge1.x * ge1.x + ge1.y * ge1.y + ge1.z * ge1.z + ge1.w * ge1.w;
                  }
                },
                [&](int d) {
                  const float e0 = row1[d], e1 = Term::kMul == 2 ? row1[a.dim + d] : e0;
                  float ge0 = 0.f, ge1 = 0.f;
#pragma unroll
                  for (int u = 0; u < NB; ++u)
                    bwd1<Term, POS>(g + u * Term::kNOut, e0, e1, sf0[u * a.dim + d], sf1[u * a.dim + d], ge0, ge1, tq0[u], tq1[u]);
                  te[0] = ge0;
                  sumsq += ge0 * ge0;
                  if (Term::kMul == 2) {
                    te[Term::kMul - 1] = ge1;
                    sumsq += ge1 * ge1;
                  }
                });
    float v_new = 0.f;
    const float v_old = __shfl_sync(0xffffffffu, cur.v, tl);
    if (single) {
      // the row's Adam step, in place: the slot holds the parameter row and the first-moment row
      const float g2mean = warp_sum(sumsq) / (float)ua.width;
      v_new = v_old * ua.beta2 + g2mean * ua.omb2;
      const RowDenom denom = rowwise_denom(v_new, ua);
      Lanes::each(lane, a.dim,
                  [&](int k, int d4) {
#pragma unroll
                    for (int part = 0; part < Term::kMul; ++part) {
                      float4 p = row4[part * dim4 + d4], m = mom4[part * dim4 + d4];
                      const float4 gg = ge[part][k];
                      adam_elem_rowwise(gg.x, p.x, m.x, denom, ua);
                      adam_elem_rowwise(gg.y, p.y, m.y, denom, ua);
                      adam_elem_rowwise(gg.z, p.z, m.z, denom, ua);
                      adam_elem_rowwise(gg.w, p.w, m.w, denom, ua);
                      row4[part * dim4 + d4] = p;
                      mom4[part * dim4 + d4] = m;
                    }
                  },
                  [&](int d) {
#pragma unroll
                    for (int part = 0; part < Term::kMul; ++part) {
                      float p = row1[part * a.dim + d], m = mom1[part * a.dim + d];
                      adam_elem_rowwise(te[part], p, m, denom, ua);
                      row1[part * a.dim + d] = p;
                      mom1[part * a.dim + d] = m;
                    }
                  });
    } else {
      Lanes::each(lane, a.dim,
                  [&](int k, int d4) {
                    row4[d4] = ge[0][k];
                    if (Term::kMul == 2) row4[dim4 + d4] = ge[Term::kMul - 1][k];
                  },
                  [&](int d) {
                    row1[d] = te[0];
                    if (Term::kMul == 2) row1[a.dim + d] = te[Term::kMul - 1];
                  });
    }
    bulk::fence_async_shared();   // what the lanes wrote is visible to the copy engine
    __syncwarp();
    const int tn = t + stages - 1;
    const bool same = (tn >> 5) == (t >> 5);
    const long long next_row = __shfl_sync(0xffffffffu, same ? cur.src : nxt.src, tn & 31);
    const int next_single = __shfl_sync(0xffffffffu, same ? ((cur.dst >= 0) ? cur.single : 0)
                                                          : ((nxt.dst >= 0) ? nxt.single : 0), tn & 31);
    if (lane == 0) {
      if (single) {
        bulk::store(const_cast<unsigned char*>(ent) + (size_t)row * row_bytes, row4, row_bytes);
        bulk::store(const_cast<unsigned char*>(mom) + (size_t)row * row_bytes, mom4, row_bytes);
        ua.v[row] = v_old + (v_new - v_old);
        uniq_rw[dst] = ~(int64_t)row;       // this row's update is done: the update kernel skips it
      } else if (dst >= 0) {
        bulk::reduce_add_f32(gbase + (size_t)dst * row_bytes, row4, row_bytes);
      }
      bulk::commit_group();
      if (tn < n) {
        bulk::wait_group_read<1>();   // all transfers but the ones just committed have read their slots
        const int s2 = slot == 0 ? stages - 1 : slot - 1;
        issue(s2, next_row, next_single);
      }
    }
    if (tl == 31) cur = nxt;
    if (++slot == stages) {
      slot = 0;
      parity ^= 1u;
    }
  }
  };
  if (positive) walk(std::true_type{});
  else walk(std::false_type{});
  if (lane == 0) bulk::wait_group<0>();
  __syncthreads();

  // fold the warps' query gradients through the (now idle) ring, in warp order
  float4* red = reinterpret_cast<float4*>(ring_all);
  const size_t per_warp4 = (size_t)NB * Term::kNQ * dim4;
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    float4* mine = red + warp * per_warp4 + (size_t)u * Term::kNQ * dim4;
    Lanes::each(lane, a.dim,
                [&](int k, int d4) {
                  mine[d4] = gq0[u][k];
                  if (Term::kNQ == 2) mine[dim4 + d4] = gq1[u][k];
                },
                [&](int d) {
                  reinterpret_cast<float*>(mine)[d] = tq0[u];
                  if (Term::kNQ == 2) reinterpret_cast<float*>(mine)[a.dim + d] = tq1[u];
                });
  }
  __syncthreads();
  for (size_t i = threadIdx.x; i < per_warp4; i += kRowCtaThreads) {
    float4 acc = red[i];
    for (int w = 1; w < kRowCtaWarps; ++w) add4(acc, red[w * per_warp4 + i]);
    const size_t u = i / ((size_t)Term::kNQ * dim4), rem = i - u * Term::kNQ * dim4;
    const bool second = rem >= (size_t)dim4;
    float* base = second ? ga.g_second : ga.g_first;
    float4* out = reinterpret_cast<float4*>(base + q_off + u * a.dim) + (rem - (second ? dim4 : 0));
    if (ga.query_atomic) atomicAdd(out, acc);
    else *out = acc;
  }
}

// ----------------------------------------------------------------------------------------
// The same with a full second moment.  Nothing is reduced over a row then, so the rows need not be held
// whole: the layout is col_backward_kernel's, a thread owning one 16-byte column of every row its group
// takes.  It loads its column of the parameter row and, where this position is the row's only one, of both
// moments, and stores all three back; U rows are in flight.  Other rows take the gradient buffer.
// Per such row 12 row lengths of traffic instead of 20 (gradient written and read again, parameters read
// twice), and nothing at all for the update kernel.
// ----------------------------------------------------------------------------------------

template <int N>
struct alignas(4 * N) GoutVec {
  float v[N];
};

template <class Term, int NB, int U>
__global__ void __launch_bounds__(kRowCtaThreads, 2)
    col_backward_adam_kernel(RowArgs a, RowGradArgs ga, UpdateArgs ua, int64_t* __restrict__ uniq_rw, int tpr, int groups) {
  constexpr int NG = NB * Term::kNOut, M = Term::kMul;
  extern __shared__ float4 red4[];       // [groups][NB][kNQ][dim4]
  __shared__ size_t meta_src[kRowCtaWarps][32];
  __shared__ int meta_dst[kRowCtaWarps][32];
  __shared__ GoutVec<NG> meta_g[kRowCtaWarps][32];
  __shared__ int meta_single[kRowCtaWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = threadIdx.x / tpr, col = threadIdx.x - grp * tpr;
  const int b = blockIdx.x / a.chunks, c = blockIdx.x - b * a.chunks;
  const int dim4 = a.dim >> 2;
  const bool active = grp < groups && col < dim4;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t w4 = (size_t)dim4 * M;
  float4* table4 = reinterpret_cast<float4*>(ua.table);
  float4* m4 = reinterpret_cast<float4*>(ua.m);
  float4* v4 = reinterpret_cast<float4*>(ua.v);
  float4* gbase = reinterpret_cast<float4*>(ga.g_rows);
  load_dyn(ua);

  float4 q0[NB], q1[NB], gq0[NB], gq1[NB];
  bool pos_ok = true;
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    q0[u] = q1[u] = gq0[u] = gq1[u] = z4;
    if (active) {
      q0[u] = prep4<Term>(__ldg(reinterpret_cast<const float4*>(a.first + ((size_t)b * NB + u) * a.dim) + col));
      if (Term::kNQ == 2) q1[u] = __ldg(reinterpret_cast<const float4*>(a.second + ((size_t)b * NB + u) * a.dim) + col);
      pos_ok = pos_ok && positive4(q1[u]);
    }
  }
  const bool positive = __syncthreads_and(pos_ok) && Term::kPositive;

  const int r_begin = c * a.rows_per_cta;
  const int r_end = min(a.K, r_begin + a.rows_per_cta);
  auto walk = [&](auto pos_tag) {
    constexpr bool POS = decltype(pos_tag)::value;
    const int n_mine = (r_end - r_begin - grp + groups - 1) / groups;
    for (int t0 = 0; t0 < n_mine; t0 += 32) {
      const int n = min(32, n_mine - t0);
      __syncwarp();
      {
        const int l = lane < n ? lane : 0;   // surplus lanes repeat the tile's first row; their entries are not used
        const int k = r_begin + grp + groups * (t0 + l);
        const size_t pos = (size_t)b * a.K + k;
        const long long row = checked_row_id(a.idx, pos, a.n_rows, &g_async_status);
        const bool bad = row < 0;            // read row 0, write and contribute nothing
        const int32_t s = ga.slot[pos];
        meta_src[warp][lane] = bad ? 0 : (size_t)row * w4;
        meta_dst[warp][lane] = bad ? -1 : s;
        GoutVec<NG> g;
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const size_t o = ((size_t)b * NB + u) * a.K + k;
          g.v[u * Term::kNOut] = bad ? 0.f : ga.gout0[o];
          if (Term::kNOut == 2) g.v[u * Term::kNOut + Term::kNOut - 1] = bad ? 0.f : ga.gout1[o];
        }
        meta_g[warp][lane] = g;
        meta_single[warp][lane] = (!bad && s >= 0 && lane < n) ? (ga.slot_count[s] == 1) : 0;
      }
      __syncwarp();
      for (int t = 0; t < n; t += U) {
        if (!active) continue;
        float4 p[U][M], m[U][M], v[U][M];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const size_t at = meta_src[warp][t + u] + col;
          const bool single = meta_single[warp][t + u];
#pragma unroll
          for (int part = 0; part < M; ++part) {
            p[u][part] = table4[at + part * dim4];
            if (single) {
              m[u][part] = m4[at + part * dim4];
              v[u][part] = v4[at + part * dim4];
            }
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (t + u >= n) break;
          const GoutVec<NG> gv = meta_g[warp][t + u];
          float4 ge[2] = {z4, z4};
#pragma unroll
          for (int br = 0; br < NB; ++br) {
            float g[Term::kNOut];
            g[0] = gv.v[br * Term::kNOut];
            if (Term::kNOut == 2) g[Term::kNOut - 1] = gv.v[br * Term::kNOut + Term::kNOut - 1];
            bwd4<Term, POS>(g, p[u][0], p[u][M - 1], q0[br], q1[br], ge[0], ge[1], gq0[br], gq1[br]);
          }
          const int dst = meta_dst[warp][t + u];
          if (meta_single[warp][t + u]) {
            const size_t at = meta_src[warp][t + u] + col;
#pragma unroll
            for (int part = 0; part < M; ++part) {
              const float4 gg = ge[part];
              float4 pp = p[u][part], mm = m[u][part], vv = v[u][part];
              adam_elem(gg.x, pp.x, mm.x, vv.x, ua);
              adam_elem(gg.y, pp.y, mm.y, vv.y, ua);
              adam_elem(gg.z, pp.z, mm.z, vv.z, ua);
              adam_elem(gg.w, pp.w, mm.w, vv.w, ua);
              table4[at + part * dim4] = pp;
              m4[at + part * dim4] = mm;
              v4[at + part * dim4] = vv;
            }
            if (col == 0) uniq_rw[dst] = ~(int64_t)(meta_src[warp][t + u] / w4);   // the update kernel skips it
          } else if (dst >= 0) {
            float4* out = gbase + (size_t)dst * w4 + col;
#pragma unroll
            for (int part = 0; part < M; ++part) atomicAdd(out + part * dim4, ge[part]);
          }
        }
      }
    }
  };
  if (grp < groups) {
    if (positive) walk(std::true_type{});
    else walk(std::false_type{});
  }

  // fold the groups' query gradients in group order
  const size_t per_group = (size_t)NB * Term::kNQ * dim4;
  if (active) {
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      red4[grp * per_group + (size_t)u * Term::kNQ * dim4 + col] = gq0[u];
      if (Term::kNQ == 2) red4[grp * per_group + (size_t)u * Term::kNQ * dim4 + dim4 + col] = gq1[u];
    }
  }
  __syncthreads();
  if (grp == 0 && active) {
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      for (int gi = 1; gi < groups; ++gi) {
        add4(gq0[u], red4[gi * per_group + (size_t)u * Term::kNQ * dim4 + col]);
        if (Term::kNQ == 2) add4(gq1[u], red4[gi * per_group + (size_t)u * Term::kNQ * dim4 + dim4 + col]);
      }
      float4* gf = reinterpret_cast<float4*>(ga.g_first + ((size_t)b * NB + u) * a.dim) + col;
      float4* gs = reinterpret_cast<float4*>(ga.g_second + ((size_t)b * NB + u) * a.dim) + col;
      if (ga.query_atomic) {
        atomicAdd(gf, gq0[u]);
        if (Term::kNQ == 2) atomicAdd(gs, gq1[u]);
      } else {
        *gf = gq0[u];
        if (Term::kNQ == 2) *gs = gq1[u];
      }
    }
  }
}

// ----------------------------------------------------------------------------------------
// Union queries: NB branches of every query scored against the same candidate rows.
// The reference runs the op once per branch and stacks the results (a Python loop over the
// branch axis of a 4-D query operand); here one pass over the rows serves all branches, and the
// backward pass writes the sum of the branches' row gradients once.
// Operands: first / second [B, NB, dim]; outputs and output gradients [B, NB, K].
// ----------------------------------------------------------------------------------------

template <class Term, int NB, int NCH, int R>
__global__ void __launch_bounds__(kRowCtaThreads)
    row_forward_union_kernel(RowArgs a, float* __restrict__ dst0, float* __restrict__ dst1) {
  extern __shared__ float4 sq[];  // [2][NB][dim4]: the query's branches, first then second operand
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x / a.chunks, c = blockIdx.x - b * a.chunks;
  const int dim4 = a.dim >> 2;
  {
    const float4* p0 = reinterpret_cast<const float4*>(a.first + (size_t)b * NB * a.dim);
    const float4* p1 = reinterpret_cast<const float4*>(a.second + (size_t)b * NB * a.dim);
    for (int i = threadIdx.x; i < NB * dim4; i += kRowCtaThreads) {
      sq[i] = __ldg(p0 + i);
      if (Term::kNQ == 2) sq[NB * dim4 + i] = __ldg(p1 + i);
    }
  }
  __syncthreads();
  const float4* sq0 = sq;
  const float4* sq1 = Term::kNQ == 2 ? sq + NB * dim4 : sq;

  const int r_begin = c * a.rows_per_cta;
  const int r_end = min(a.K, r_begin + a.rows_per_cta);
  const size_t w4 = (size_t)dim4 * Term::kMul;
  const float4* ent4 = reinterpret_cast<const float4*>(a.ent);

  for (int base = r_begin + warp * a.wrows; base < r_end; base += kRowCtaWarps * a.wrows) {
    const int n = min(a.wrows, r_end - base);
    const size_t pos = (size_t)b * a.K + base + lane;
    long long myrow = 0;   // -1: an id outside the table (row 0 is read instead, the result is NaN)
    if (lane < n) myrow = a.idx ? checked_row_id(a.idx, pos, a.n_rows, &g_async_status) : (long long)pos;
    float out0[NB], out1[NB];
#pragma unroll
    for (int u = 0; u < NB; ++u) out0[u] = out1[u] = 0.f;
    for (int t = 0; t < n; t += R) {
      float4 e[R][Term::kMul][NCH];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const long long row = max(__shfl_sync(0xffffffffu, myrow, min(t + r, n - 1)), 0LL);
        const float4* pe = ent4 + (size_t)row * w4;
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
          const int d4 = lane + 32 * j;
          if (d4 < dim4) {
            e[r][0][j] = ld_row4(pe + d4);
            if (Term::kMul == 2) e[r][Term::kMul - 1][j] = ld_row4(pe + dim4 + d4);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          float acc[Term::kNOut];
#pragma unroll
          for (int o = 0; o < Term::kNOut; ++o) acc[o] = 0.f;
#pragma unroll
          for (int j = 0; j < NCH; ++j) {
            const int d4 = lane + 32 * j;
            if (d4 < dim4)
              fwd4<Term>(e[r][0][j], e[r][Term::kMul - 1][j], sq0[u * dim4 + d4], sq1[u * dim4 + d4], acc);
          }
#pragma unroll
          for (int o = 0; o < Term::kNOut; ++o) acc[o] = warp_sum(acc[o]);
          if (lane == t + r) {
            out0[u] = acc[0];
            out1[u] = acc[Term::kNOut - 1];
          }
        }
      }
    }
    if (lane < n) {
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const size_t o = ((size_t)b * NB + u) * a.K + base + lane;
        dst0[o] = myrow < 0 ? NAN : out0[u];
        if (Term::kNOut == 2) dst1[o] = myrow < 0 ? NAN : out1[u];
      }
    }
  }
}

template <class Term, int NB, int U>
__global__ void __launch_bounds__(kRowCtaThreads)
    col_backward_union_kernel(RowArgs a, RowGradArgs ga, int tpr, int groups) {
  constexpr int NG = NB * Term::kNOut;   // output gradients per row: 2 or 4
  extern __shared__ float4 red4[];       // [groups][NB][kNQ][dim4]
  __shared__ size_t meta_src[kRowCtaWarps][32];
  __shared__ long long meta_dst[kRowCtaWarps][32];
  __shared__ GoutVec<NG> meta_g[kRowCtaWarps][32];
  __shared__ int meta_single[kRowCtaWarps][32];
  const int lane = threadIdx.x & 31;
  const int grp = threadIdx.x / tpr, col = threadIdx.x - grp * tpr;
  const int b = blockIdx.x / a.chunks, c = blockIdx.x - b * a.chunks;
  const int dim4 = a.dim >> 2;
  const bool active = grp < groups && col < dim4;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t w4 = (size_t)dim4 * Term::kMul;
  const float4* ent4 = reinterpret_cast<const float4*>(a.ent);
  float4* gbase = reinterpret_cast<float4*>(ga.g_rows);

  float4 q0[NB], q1[NB], gq0[NB], gq1[NB];
  bool pos_ok = true;
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    q0[u] = q1[u] = gq0[u] = gq1[u] = z4;
    if (active) {
      q0[u] = prep4<Term>(__ldg(reinterpret_cast<const float4*>(a.first + ((size_t)b * NB + u) * a.dim) + col));
      if (Term::kNQ == 2)
        q1[u] = __ldg(reinterpret_cast<const float4*>(a.second + ((size_t)b * NB + u) * a.dim) + col);
      pos_ok = pos_ok && positive4(q1[u]);
    }
  }
  const bool positive = __syncthreads_and(pos_ok) && Term::kPositive;

  const int r_begin = c * a.rows_per_cta;
  const int r_end = min(a.K, r_begin + a.rows_per_cta);
  auto walk = [&](auto pos_tag) {
    constexpr bool POS = decltype(pos_tag)::value;
    const int n_mine = (r_end - r_begin - grp + groups - 1) / groups;
    const int warp = threadIdx.x >> 5;
    for (int t0 = 0; t0 < n_mine; t0 += 32) {
      const int n = min(32, n_mine - t0);
      __syncwarp();
      {
        const int l = lane < n ? lane : 0;
        const int k = r_begin + grp + groups * (t0 + l);
        const size_t pos = (size_t)b * a.K + k;
        const long long row = checked_row_id(a.idx, pos, a.n_rows, &g_async_status);
        const bool bad = row < 0;   // as in col_backward_kernel: read row 0, write and contribute nothing
        const int32_t s = ga.slot[pos];
        meta_src[warp][lane] = bad ? 0 : (size_t)row * w4;
        meta_dst[warp][lane] = (s < 0 || bad) ? -1 : s * (long long)w4;
        GoutVec<NG> g;
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const size_t o = ((size_t)b * NB + u) * a.K + k;
          g.v[u * Term::kNOut] = bad ? 0.f : ga.gout0[o];
          if (Term::kNOut == 2) g.v[u * Term::kNOut + Term::kNOut - 1] = bad ? 0.f : ga.gout1[o];
        }
        meta_g[warp][lane] = g;
        meta_single[warp][lane] = (s >= 0 && ga.slot_count != nullptr) ? (ga.slot_count[s] == 1) : 0;
      }
      __syncwarp();
      for (int t = 0; t < n; t += U) {
        float4 e0[U], e1[U];
        if (active) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float4* pe = ent4 + meta_src[warp][t + u] + col;
            e0[u] = ld_row4(pe);
            if (Term::kMul == 2) e1[u] = ld_row4(pe + dim4);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (t + u < n) {
              const GoutVec<NG> gv = meta_g[warp][t + u];
              const long long dst = meta_dst[warp][t + u];
              float4 ge0 = z4, ge1 = z4;
#pragma unroll
              for (int br = 0; br < NB; ++br) {
                float g[Term::kNOut];
                g[0] = gv.v[br * Term::kNOut];
                if (Term::kNOut == 2) g[Term::kNOut - 1] = gv.v[br * Term::kNOut + Term::kNOut - 1];
                bwd4<Term, POS>(g, e0[u], Term::kMul == 2 ? e1[u] : e0[u], q0[br], q1[br], ge0, ge1, gq0[br], gq1[br]);
              }
              if (dst >= 0) {
                float4* out = gbase + dst + col;
                if (meta_single[warp][t + u]) {
                  out[0] = ge0;
                  if (Term::kMul == 2) out[dim4] = ge1;
                } else {
                  atomicAdd(out, ge0);
                  if (Term::kMul == 2) atomicAdd(out + dim4, ge1);
                }
              }
            }
          }
        }
      }
    }
  };

  if (grp < groups) {
    if (positive) walk(std::true_type{});
    else walk(std::false_type{});
  }

  // fold the groups' query gradients in group order
  const size_t per_group = (size_t)NB * Term::kNQ * dim4;
  if (active) {
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      red4[grp * per_group + (size_t)u * Term::kNQ * dim4 + col] = gq0[u];
      if (Term::kNQ == 2) red4[grp * per_group + (size_t)u * Term::kNQ * dim4 + dim4 + col] = gq1[u];
    }
  }
  __syncthreads();
  if (grp == 0 && active) {
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      for (int gi = 1; gi < groups; ++gi) {
        add4(gq0[u], red4[gi * per_group + (size_t)u * Term::kNQ * dim4 + col]);
        if (Term::kNQ == 2) add4(gq1[u], red4[gi * per_group + (size_t)u * Term::kNQ * dim4 + dim4 + col]);
      }
      float4* gf = reinterpret_cast<float4*>(ga.g_first + ((size_t)b * NB + u) * a.dim) + col;
      float4* gs = reinterpret_cast<float4*>(ga.g_second + ((size_t)b * NB + u) * a.dim) + col;
      if (ga.query_atomic) {
        atomicAdd(gf, gq0[u]);
        if (Term::kNQ == 2) atomicAdd(gs, gq1[u]);
      } else {
        *gf = gq0[u];
        if (Term::kNQ == 2) *gs = gq1[u];
      }
    }
  }
}

// ----------------------------------------------------------------------------------------
// host side: validation, shape classification, launches
// ----------------------------------------------------------------------------------------

// row-stream launch plan; chunks == 0 means "not eligible", nch == 0 that the rows take the kernels of any
// row length (V floats at a time)
struct RowPlan {
  int nch, v, wrows, rows_per_cta, chunks;
};

// address bits of a set of pointers: what their common alignment leaves over
template <class... P>
static uintptr_t low_bits(const P*... ptr) {
  return (reinterpret_cast<uintptr_t>(ptr) | ...) & 15u;
}

static RowPlan plan_rows(const Shape& s, uintptr_t bits) {
  RowPlan p{0, 0, 0, 0, 0};
  const bool shape_ok = s.be == s.bsize && s.bc == s.bsize && s.ne == s.num && s.nc == 1;
  if (!shape_ok || s.dim > 4096 || s.num < 4 || s.num > (size_t)1 << 30 || s.bsize > (size_t)1 << 24) return p;
  const int dim4 = (int)(s.dim >> 2);
  p.v = (s.dim & 3) == 0 && bits == 0 ? 4 : (s.dim & 1) == 0 && (bits & 7) == 0 ? 2 : 1;
  if (p.v == 4 && s.dim <= 1024) p.nch = dim4 <= 32 ? 1 : dim4 <= 64 ? 2 : dim4 <= 128 ? 4 : 8;
  const size_t K = s.num;
  int wrows = 32;
  while (wrows > 4 && (size_t)wrows * kRowCtaWarps / 2 >= K) wrows >>= 1;
  p.wrows = wrows;
  const size_t sweep = (size_t)wrows * kRowCtaWarps;
  size_t sweeps_per_cta = 1;
  const size_t sweeps_total = (K + sweep - 1) / sweep;
  // keep the grid within a few dozen waves; larger blocks of rows amortise the query load
  const size_t max_ctas = (size_t)sm_count() * 32;
  while (s.bsize * ((sweeps_total + sweeps_per_cta - 1) / sweeps_per_cta) > max_ctas &&
         sweeps_per_cta < sweeps_total)
    sweeps_per_cta *= 2;
  p.rows_per_cta = (int)std::min<size_t>(sweep * sweeps_per_cta, (size_t)1 << 30);
  p.chunks = (int)((K + p.rows_per_cta - 1) / p.rows_per_cta);
  return p;
}

// Launches row_backward_bulk_kernel when the row width suits it.  Returns 1 when launched, 0 when
// the caller should use another kernel, a negative status on failure.
template <class Term, int NB>
static int launch_backward_bulk(const Shape& s, RowArgs a, RowGradArgs ga, int nch, cudaStream_t st) {
  // Measured on B200: ahead of the column-thread kernel for rows of 2 KB and more (RotatE rows of
  // 4000 B: 1.59 ms against 1.67 ms per 1M rows); for 1600-byte rows it executes more instructions
  // per row (waits, per-row scalars) than that kernel and ends level with it, so those stay there.
  const size_t row_bytes = s.dim * Term::kMul * sizeof(float);
  if ((nch != 4 && nch != 8) || row_bytes < 2048) return 0;
  const int need = (NB * Term::kNQ + Term::kMul - 1) / Term::kMul;   // ring must hold the final fold
  const int stages = std::max(3, need);
  const size_t q_bytes = (size_t)NB * Term::kNQ * s.dim * sizeof(float);
  const size_t smem = bulk_ring_offset(stages) + q_bytes + (size_t)kRowCtaWarps * stages * row_bytes;
  if (smem > 110 * 1024) return 0;
  a.rows_per_cta = (int)std::min<size_t>(s.num, 512);
  a.chunks = (int)((s.num + a.rows_per_cta - 1) / a.rows_per_cta);
  ga.query_atomic = a.chunks > 1;
  if (a.chunks > 1) {
    const size_t bytes = s.bsize * NB * s.dim * sizeof(float);
    if (cudaMemsetAsync(ga.g_first, 0, bytes, st) != cudaSuccess ||
        (Term::kNQ == 2 && cudaMemsetAsync(ga.g_second, 0, bytes, st) != cudaSuccess))
      return fail(SMORE_ERR_CUDA, "row_backward_bulk_kernel: cudaMemsetAsync failed");
  }
  auto kern = nch == 4 ? row_backward_bulk_kernel<Term, NB, 4> : row_backward_bulk_kernel<Term, NB, 8>;
  if (int rc = allow_large_smem(kern, 110 * 1024)) return rc;
  kern<<<(unsigned)(s.bsize * a.chunks), kRowCtaThreads, smem, st>>>(a, ga, stages);
  if (int rc = check_launch("row_backward_bulk_kernel")) return rc;
  return 1;
}

// Pieces per lane of the bulk-copy kernels and whether the last is the tail of a row (see LanePieces).
struct LaneShape {
  int nch;
  bool tail;
};
static LaneShape lane_shape(size_t dim, int nch) {
  if (nch == 4) return {4, row_tail(dim, 4)};
  if (nch == 8 && row_tail(dim, 7)) return {7, true};
  return {nch, false};
}

#define SMORE_LANES(ls, KERN, ...)                                              \
  ((ls).nch == 4 ? ((ls).tail ? KERN<__VA_ARGS__, 4, true> : KERN<__VA_ARGS__, 4, false>) \
                 : ((ls).tail ? KERN<__VA_ARGS__, 7, true> : KERN<__VA_ARGS__, 8, false>))

// Launches row_backward_adam_bulk_kernel (row-wise second moment) or col_backward_adam_kernel (full) when
// the shape suits it.  Returns 1 when launched, 0 when the caller should use the ordinary backward +
// update, a negative status on failure.
template <class Term, int NB>
static int launch_backward_adam(const Shape& s, RowArgs a, RowGradArgs ga, const UpdateArgs& ua, int64_t* uniq,
                                int nch, cudaStream_t st) {
  const size_t row_bytes = s.dim * Term::kMul * sizeof(float);
  const bool full = !ua.squeeze;
  if (!full && ((nch != 4 && nch != 8) || row_bytes < 1024)) return 0;
  if (full && nch == 0) return 0;
  int stages = 0, tpr = 0, groups = 0;
  size_t smem;
  if (full) {
    const int dim4 = (int)(s.dim >> 2);
    tpr = ((dim4 + 31) / 32) * 32;
    groups = kRowCtaThreads / tpr;
    smem = (size_t)groups * NB * Term::kNQ * s.dim * sizeof(float);
  } else {
    const int need = (NB * Term::kNQ + 2 * Term::kMul - 1) / (2 * Term::kMul);   // ring must hold the final fold
    const size_t q_bytes = (size_t)NB * Term::kNQ * s.dim * sizeof(float);
    // as many stages (3..5) as fit two CTAs per SM: every stage holds a parameter row and a moment row
    stages = 5;
    while (stages > 3 && bulk_ring_offset(stages) + q_bytes + (size_t)kRowCtaWarps * stages * 2 * row_bytes > 110 * 1024)
      --stages;
    stages = std::max(stages, need);
    smem = bulk_ring_offset(stages) + q_bytes + (size_t)kRowCtaWarps * stages * 2 * row_bytes;
    if (smem > 200 * 1024) return 0;      // wide rows (RotatE, 4000 bytes): one CTA per SM
  }
  if (a.seg != nullptr) {
    a.chunks = 1;         // ragged form: one CTA per query, s.bsize queries
  } else {
    a.rows_per_cta = (int)std::min<size_t>(s.num, 512);
    a.chunks = (int)((s.num + a.rows_per_cta - 1) / a.rows_per_cta);
  }
  ga.query_atomic = a.chunks > 1;
  if (a.chunks > 1) {
    const size_t bytes = s.bsize * NB * s.dim * sizeof(float);
    if (cudaMemsetAsync(ga.g_first, 0, bytes, st) != cudaSuccess ||
        (Term::kNQ == 2 && cudaMemsetAsync(ga.g_second, 0, bytes, st) != cudaSuccess))
      return fail(SMORE_ERR_CUDA, "backward_adam: cudaMemsetAsync failed");
  }
  const unsigned grid = (unsigned)(s.bsize * a.chunks);
  if (full) {
    // rows of two parts keep six 16-byte loads in flight per row
    constexpr int U = Term::kMul == 2 ? 2 : 4;
    col_backward_adam_kernel<Term, NB, U><<<grid, kRowCtaThreads, smem, st>>>(a, ga, ua, uniq, tpr, groups);
    if (int rc = check_launch("col_backward_adam_kernel")) return rc;
    return 1;
  }
  const LaneShape ls = lane_shape(s.dim, nch);
  auto kern = SMORE_LANES(ls, row_backward_adam_bulk_kernel, Term, NB);
  if (int rc = allow_large_smem(kern, 200 * 1024)) return rc;
  kern<<<grid, kRowCtaThreads, smem, st>>>(a, ga, ua, uniq, stages);
  if (int rc = check_launch("row_backward_adam_bulk_kernel")) return rc;
  return 1;
}

template <class Term>
static int backward_adam_common(size_t branches, const Shape& s, const float* gout0, const float* gout1, float* table,
                                const int64_t* idx, const float* first, const float* second, const int32_t* slot,
                                const int32_t* slot_count, float* g_rows, float* g_first, float* g_second,
                                const UpdateArgs& ua, int64_t* uniq, cudaStream_t st) {
  if (Term::kNQ == 1) {
    second = first;
    g_second = g_first;
  }
  const RowPlan p = plan_rows(s, low_bits(table, first, second, g_rows, g_first, g_second, ua.m) |
                                     (ua.squeeze ? 0 : low_bits(ua.v)));
  if (p.nch == 0) return 0;
  RowArgs a{table, idx, first, second, (int)s.num, (int)s.dim, p.rows_per_cta, p.chunks, p.wrows, (long long)s.n_rows};
  RowGradArgs ga{gout0, gout1, nullptr, slot, slot_count, g_rows, g_first, g_second, 0};
  if (branches == 1) return launch_backward_adam<Term, 1>(s, a, ga, ua, uniq, p.nch, st);
  return launch_backward_adam<Term, kUnionBranches>(s, a, ga, ua, uniq, p.nch, st);
}

// ---- ragged form: query q scores / differentiates the candidate rows idx[seg[q].x .. + seg[q].y) ----
// (the owner side of a row-sharded table: the queries of every rank against this shard's rows).
// Returns 1 when launched, 0 when the row width is outside the bulk-copy kernels' range.
static int ragged_nch(size_t dim, size_t mul) {
  const size_t dim4 = dim >> 2, row_bytes = dim * mul * sizeof(float);
  if ((dim & 3) || dim > 1024 || dim4 <= 64 || row_bytes < 1024) return 0;
  return dim4 <= 128 ? 4 : 8;
}

struct RaggedPeers {        // where results go / upstream gradients come from (see RowArgs)
  const int32_t* positions;
  size_t seg_per_rank;
  size_t branch_stride;
  float* const* out0;
  float* const* out1;
  const float* const* up0;
  const float* const* up1;
};

static void set_peers(RowArgs& a, const RaggedPeers& pr) {
  a.positions = pr.positions;
  a.seg_per_rank = (int)std::max<size_t>(pr.seg_per_rank, 1);
  a.branch_stride = (int)pr.branch_stride;
  a.out_ptrs[0] = pr.out0; a.out_ptrs[1] = pr.out1;
  a.up_ptrs[0] = pr.up0; a.up_ptrs[1] = pr.up1;
}

// Ring of the bulk-copy forward kernel: 2..8 slots per warp, about 96 KB of row copies in flight per SM at 32
// resident warps (more in flight measured slower), and at least 46 KB per CTA, which keeps the residency at
// four CTAs per SM whatever the register count: five and more (terms with few registers) put more row
// copies in flight than the memory system likes and measured up to 1.8x slower.
static int forward_stages(size_t row_bytes) {
  return (int)std::min<size_t>(8, std::max<size_t>(2, (96 * 1024 / 32 + row_bytes - 1) / row_bytes));
}
static size_t forward_smem(size_t row_bytes, int stages) {
  return std::max<size_t>(bulk_ring_offset(stages) + (size_t)kRowCtaWarps * stages * row_bytes, 46 * 1024);
}

template <class Term>
static int launch_forward_ragged(size_t branches, size_t n_seg, size_t dim, size_t n_rows, const float* table,
                                 const int64_t* rows, const float* first, const float* second, const int2* seg,
                                 float* out0, float* out1, const RaggedPeers& pr, cudaStream_t st) {
  if (Term::kNQ == 1) second = first;
  const int nch = ragged_nch(dim, Term::kMul);
  if (!nch || !aligned16(table) || !aligned16(first) || !aligned16(second)) return 0;
  const size_t row_bytes = dim * Term::kMul * sizeof(float);
  const int stages = forward_stages(row_bytes);
  const size_t smem = forward_smem(row_bytes, stages);
  if (smem > 110 * 1024) return 0;
  RowArgs a{table, rows, first, second, 0, (int)dim, 0, 1, 0, (long long)n_rows, seg};
  set_peers(a, pr);
  const LaneShape ls = lane_shape(dim, nch);
  auto kern = branches == 1 ? SMORE_LANES(ls, row_forward_bulk_kernel, Term, 1)
                            : SMORE_LANES(ls, row_forward_bulk_kernel, Term, kUnionBranches);
  if (int rc = allow_large_smem(kern, 110 * 1024)) return rc;
  kern<<<(unsigned)n_seg, kRowCtaThreads, smem, st>>>(a, out0, out1, stages);
  if (int rc = check_launch("row_forward_bulk_kernel")) return rc;
  return 1;
}

template <class Term>
static int launch_backward_adam_ragged(size_t branches, size_t n_seg, size_t dim, size_t n_rows, const float* gout0, const float* gout1,
                                       float* table, const int64_t* rows, const float* first, const float* second,
                                       const int2* seg, const int32_t* slot, const int32_t* slot_count, float* g_rows,
                                       float* g_first, float* g_second, const UpdateArgs& ua, int64_t* uniq,
                                       const RaggedPeers& pr, cudaStream_t st) {
  if (Term::kNQ == 1) {
    second = first;
    g_second = g_first;
  }
  const int nch = ragged_nch(dim, Term::kMul);
  if (!nch || !aligned16(table) || !aligned16(first) || !aligned16(second) || !aligned16(g_rows) || !aligned16(g_first) ||
      !aligned16(g_second) || !aligned16(ua.m))
    return 0;
  const Shape s{n_seg, 4, n_seg, 4, n_seg, 1, dim, n_rows};
  RowArgs a{table, rows, first, second, 0, (int)dim, 0, 1, 0, (long long)n_rows, seg};
  set_peers(a, pr);
  RowGradArgs ga{gout0, gout1, nullptr, slot, slot_count, g_rows, g_first, g_second, 0};
  if (branches == 1) return launch_backward_adam<Term, 1>(s, a, ga, ua, uniq, nch, st);
  return launch_backward_adam<Term, kUnionBranches>(s, a, ga, ua, uniq, nch, st);
}

template <class Term>
static int launch_forward(int term, const Shape& s, const float* ent, const int64_t* idx, const float* first,
                          const float* second, float* dst0, float* dst1, cudaStream_t st) {
  if (Term::kNQ == 1) second = first;
  const RowPlan p = plan_rows(s, low_bits(ent, first, second));
  if (p.chunks == 0) {
    const ForwardArgs fa{ent, idx, first, second, dst0, dst1};
    return shared_covers(s) ? shared_forward(term, s, fa, st) : cell_forward(term, s, fa, st);
  }
  RowArgs a{ent, idx, first, second, (int)s.num, (int)s.dim, p.rows_per_cta, p.chunks, p.wrows, (long long)s.n_rows};
  const unsigned grid = (unsigned)(s.bsize * p.chunks);
  if (p.nch == 0) {
    const size_t smem = Term::kNQ * s.dim * sizeof(float);
    auto kern = p.v == 4 ? row_forward_any_kernel<Term, 4> : p.v == 2 ? row_forward_any_kernel<Term, 2> : row_forward_any_kernel<Term, 1>;
    kern<<<grid, kRowCtaThreads, smem, st>>>(a, dst0, dst1);
    return check_launch("row_forward_any_kernel");
  }
  constexpr int R = 2;  // rows in flight per warp at 4 chunks per lane
  // Rows of 1 KB and more go through the bulk-copy kernel, CTAs of 512 rows.  It needs at least two CTAs
  // per SM to cover the reduction latency.
  const size_t row_bytes = s.dim * Term::kMul * sizeof(float);
  const int stages = forward_stages(row_bytes);
  const size_t bulk_smem = forward_smem(row_bytes, stages);
  if ((p.nch == 4 || p.nch == 8) && bulk_smem <= 110 * 1024) {
    RowArgs ab = a;
    ab.rows_per_cta = (int)std::min<size_t>(s.num, 512);
    ab.chunks = (int)((s.num + ab.rows_per_cta - 1) / ab.rows_per_cta);
    const LaneShape ls = lane_shape(s.dim, p.nch);
    auto kern = SMORE_LANES(ls, row_forward_bulk_kernel, Term, 1);
    if (int rc = allow_large_smem(kern, 110 * 1024)) return rc;
    kern<<<(unsigned)(s.bsize * ab.chunks), kRowCtaThreads, bulk_smem, st>>>(ab, dst0, dst1, stages);
    return check_launch("row_forward_bulk_kernel");
  }
  switch (p.nch) {
    case 1: row_forward_kernel<Term, 1, 4><<<grid, kRowCtaThreads, 0, st>>>(a, dst0, dst1); break;
    case 2: row_forward_kernel<Term, 2, 4><<<grid, kRowCtaThreads, 0, st>>>(a, dst0, dst1); break;
    case 4: row_forward_kernel<Term, 4, R><<<grid, kRowCtaThreads, 0, st>>>(a, dst0, dst1); break;
    default: row_forward_kernel<Term, 8, 1><<<grid, kRowCtaThreads, 0, st>>>(a, dst0, dst1); break;
  }
  return check_launch("row_forward_kernel");
}

template <class Term>
static int launch_backward(int term, const Shape& s, const float* gout0, const float* gout1, const float* ent,
                           const int64_t* idx, const float* first, const float* second, float* g_ent,
                           const int32_t* slot, const int32_t* slot_count, float* g_rows,
                           float* g_first, float* g_second, cudaStream_t st) {
  if (Term::kNQ == 1) {
    second = first;
    g_second = g_first;
  }
  float* gdst = slot ? g_rows : g_ent;
  const RowPlan p = plan_rows(s, low_bits(ent, first, second, gdst, g_first, g_second));
  if (p.chunks == 0) {
    const BackwardArgs ba{gout0, gout1, ent, idx, first, second, g_ent, slot, slot_count, g_rows, g_first, g_second};
    return shared_covers(s) ? shared_backward(term, s, ba, st) : cell_backward(term, s, ba, st);
  }
  RowArgs a{ent, idx, first, second, (int)s.num, (int)s.dim, p.rows_per_cta, p.chunks, p.wrows, (long long)s.n_rows};
  RowGradArgs ga{gout0, gout1, g_ent, slot, slot_count, g_rows, g_first, g_second, p.chunks > 1};
  if (p.nch) {
    if (int rc = launch_backward_bulk<Term, 1>(s, a, ga, p.nch, st)) return rc < 0 ? rc : SMORE_OK;
  }
  if (p.chunks > 1) {
    const size_t bytes = s.bsize * s.dim * sizeof(float);
    if (cudaMemsetAsync(g_first, 0, bytes, st) != cudaSuccess ||
        (Term::kNQ == 2 && cudaMemsetAsync(g_second, 0, bytes, st) != cudaSuccess))
      return fail(SMORE_ERR_CUDA, "dist_backward: cudaMemsetAsync failed");
  }
  const int cols = (int)s.dim / p.v;
  const dim3 grid((unsigned)(s.bsize * p.chunks), (unsigned)((cols + kRowCtaThreads - 1) / kRowCtaThreads));
  const int block_cols = std::min(cols, kRowCtaThreads);
  const int tpr = ((block_cols + 31) / 32) * 32;    // threads that own the columns of one row
  const int groups = kRowCtaThreads / tpr;          // row groups per CTA
  const size_t smem = (size_t)groups * Term::kNQ * block_cols * p.v * sizeof(float);
  constexpr int U = Term::kMul == 2 ? 4 : 8;
  if (p.v == 4) col_backward_kernel<Term, U, 4><<<grid, kRowCtaThreads, smem, st>>>(a, ga, tpr, groups);
  else if (p.v == 2) col_backward_kernel<Term, U, 2><<<grid, kRowCtaThreads, smem, st>>>(a, ga, tpr, groups);
  else col_backward_kernel<Term, U, 1><<<grid, kRowCtaThreads, smem, st>>>(a, ga, tpr, groups);
  return check_launch("col_backward_kernel");
}

static int check_union(const char* what, size_t branches, const Shape& s, uintptr_t bits, RowPlan* p) {
  if (branches != kUnionBranches)
    return fail(SMORE_ERR_BAD_SHAPE, "%s: %d branches per query are supported (run other counts branch by branch)",
                what, kUnionBranches);
  if (int rc = validate_shape(s)) return rc;
  *p = plan_rows(s, bits);
  if (p->nch == 0)
    return fail(SMORE_ERR_BAD_SHAPE,
                "%s: needs 16-byte aligned operands, dim a multiple of 4 and <= 1024, at least 4 rows per query", what);
  return SMORE_OK;
}

template <class Term>
static int launch_forward_union(size_t branches, const Shape& s, const float* table, const int64_t* idx,
                                const float* first, const float* second, float* dst0, float* dst1,
                                cudaStream_t st) {
  if (Term::kNQ == 1) second = first;
  RowPlan p;
  if (int rc = check_union("union_forward_rows", branches, s, low_bits(table, first, second), &p))
    return rc;
  RowArgs a{table, idx, first, second, (int)s.num, (int)s.dim, p.rows_per_cta, p.chunks, p.wrows, (long long)s.n_rows};
  constexpr int NB = kUnionBranches;
  const size_t row_bytes = s.dim * Term::kMul * sizeof(float);
  const int stages = forward_stages(row_bytes);
  const size_t bulk_smem = forward_smem(row_bytes, stages);
  if (p.nch >= 4 && bulk_smem <= 110 * 1024) {
    a.rows_per_cta = (int)std::min<size_t>(s.num, 512);
    a.chunks = (int)((s.num + a.rows_per_cta - 1) / a.rows_per_cta);
    const LaneShape ls = lane_shape(s.dim, p.nch);
    auto kern = SMORE_LANES(ls, row_forward_bulk_kernel, Term, NB);
    if (int rc = allow_large_smem(kern, 110 * 1024)) return rc;
    kern<<<(unsigned)(s.bsize * a.chunks), kRowCtaThreads, bulk_smem, st>>>(a, dst0, dst1, stages);
    return check_launch("row_forward_bulk_kernel");
  }
  const unsigned grid = (unsigned)(s.bsize * p.chunks);
  const size_t smem = (size_t)kUnionBranches * Term::kNQ * s.dim * sizeof(float);
  switch (p.nch) {
    case 1: row_forward_union_kernel<Term, NB, 1, 4><<<grid, kRowCtaThreads, smem, st>>>(a, dst0, dst1); break;
    case 2: row_forward_union_kernel<Term, NB, 2, 4><<<grid, kRowCtaThreads, smem, st>>>(a, dst0, dst1); break;
    case 4: row_forward_union_kernel<Term, NB, 4, 2><<<grid, kRowCtaThreads, smem, st>>>(a, dst0, dst1); break;
    default: row_forward_union_kernel<Term, NB, 8, 1><<<grid, kRowCtaThreads, smem, st>>>(a, dst0, dst1); break;
  }
  return check_launch("row_forward_union_kernel");
}

template <class Term>
static int launch_backward_union(size_t branches, const Shape& s, const float* gout0, const float* gout1,
                                 const float* table, const int64_t* idx, const float* first, const float* second,
                                 const int32_t* slot, const int32_t* slot_count, float* g_rows, float* g_first,
                                 float* g_second, cudaStream_t st) {
  if (Term::kNQ == 1) {
    second = first;
    g_second = g_first;
  }
  RowPlan p;
  if (int rc = check_union("union_backward_rows", branches, s, low_bits(table, first, second, g_rows, g_first, g_second), &p))
    return rc;
  constexpr int NB = kUnionBranches;
  RowArgs a{table, idx, first, second, (int)s.num, (int)s.dim, p.rows_per_cta, p.chunks, p.wrows, (long long)s.n_rows};
  RowGradArgs ga{gout0, gout1, nullptr, slot, slot_count, g_rows, g_first, g_second, p.chunks > 1};
  if (p.chunks > 1) {
    const size_t bytes = s.bsize * NB * s.dim * sizeof(float);
    if (cudaMemsetAsync(g_first, 0, bytes, st) != cudaSuccess ||
        (Term::kNQ == 2 && cudaMemsetAsync(g_second, 0, bytes, st) != cudaSuccess))
      return fail(SMORE_ERR_CUDA, "union_backward_rows: cudaMemsetAsync failed");
  }
  const unsigned grid = (unsigned)(s.bsize * p.chunks);
  const int dim4 = (int)(s.dim >> 2);
  const int tpr = ((dim4 + 31) / 32) * 32;
  const int groups = kRowCtaThreads / tpr;
  const size_t smem = (size_t)groups * NB * Term::kNQ * s.dim * sizeof(float);
  if (Term::kMul == 2)
    col_backward_union_kernel<Term, NB, 4><<<grid, kRowCtaThreads, smem, st>>>(a, ga, tpr, groups);
  else
    col_backward_union_kernel<Term, NB, 8><<<grid, kRowCtaThreads, smem, st>>>(a, ga, tpr, groups);
  return check_launch("col_backward_union_kernel");
}

static int forward_common(int id, const float* ent, const int64_t* idx, const float* first,
                          const float* second, float* dst, const Shape& s, void* stream) {
  if (id < 0 || id >= SMORE_DIST_COUNT) return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", id);
  if (!ent || !first || !dst || (needs_second(id) && !second))
    return fail(SMORE_ERR_NULL, "forward: required pointer is NULL");
  if (int rc = validate_shape(s)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  SMORE_DISPATCH(id, launch_forward<Term>(id, s, ent, idx, first, second, dst, dst, st));
}

static int backward_common(int id, const float* gout, const float* ent, const int64_t* idx,
                           const float* first, const float* second, float* g_ent, const int32_t* slot,
                           const int32_t* slot_count, float* g_rows, float* g_first, float* g_second,
                           const Shape& s, void* stream) {
  if (id < 0 || id >= SMORE_DIST_COUNT) return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", id);
  if (!gout || !ent || !first || !g_first || (needs_second(id) && (!second || !g_second)))
    return fail(SMORE_ERR_NULL, "backward: required pointer is NULL");
  if (slot ? !g_rows : !g_ent)
    return fail(SMORE_ERR_NULL, "backward: entity gradient destination is NULL");
  if (int rc = validate_shape(s)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  SMORE_DISPATCH(id, launch_backward<Term>(id, s, gout, gout, ent, idx, first, second, g_ent, slot, slot_count,
                                           g_rows, g_first, g_second, st));
}

}  // namespace smore

using namespace smore;

extern "C" {

int smore_dist_forward(int dist_id, const float* ent, const float* first, const float* second, float* dst,
                       size_t bsize, size_t num, size_t be, size_t ne, size_t bc, size_t nc, size_t dim,
                       void* stream) {
  return forward_common(dist_id, ent, nullptr, first, second, dst, Shape{bsize, num, be, ne, bc, nc, dim},
                        stream);
}

int smore_dist_backward(int dist_id, const float* gout, const float* ent, const float* first,
                        const float* second, float* g_ent, float* g_first, float* g_second, size_t bsize,
                        size_t num, size_t be, size_t ne, size_t bc, size_t nc, size_t dim, void* stream) {
  return backward_common(dist_id, gout, ent, nullptr, first, second, g_ent, nullptr, nullptr, nullptr,
                         g_first, g_second, Shape{bsize, num, be, ne, bc, nc, dim}, stream);
}

int smore_dist_forward_rows(int dist_id, const float* table, const int64_t* idx, size_t n_table_rows,
                            const float* first, const float* second, float* dst, size_t bsize, size_t num,
                            size_t be, size_t ne, size_t bc, size_t nc, size_t dim, void* stream) {
  if (!idx) return fail(SMORE_ERR_NULL, "forward_rows: idx is NULL");
  return forward_common(dist_id, table, idx, first, second, dst,
                        Shape{bsize, num, be, ne, bc, nc, dim, n_table_rows}, stream);
}

int smore_dist_backward_rows(int dist_id, const float* gout, const float* table, const int64_t* idx,
                             size_t n_table_rows, const float* first, const float* second, const int32_t* slot,
                             const int32_t* slot_count, float* g_rows, float* g_first, float* g_second,
                             size_t bsize, size_t num, size_t be, size_t ne, size_t bc, size_t nc,
                             size_t dim, void* stream) {
  if (!idx || !slot) return fail(SMORE_ERR_NULL, "backward_rows: idx or slot is NULL");
  return backward_common(dist_id, gout, table, idx, first, second, nullptr, slot, slot_count, g_rows,
                         g_first, g_second, Shape{bsize, num, be, ne, bc, nc, dim, n_table_rows}, stream);
}

int smore_box_forward(const float* ent, const int64_t* idx, size_t n_table_rows, const float* center,
                      const float* offset, float* dst_out, float* dst_in, size_t bsize, size_t num, size_t be,
                      size_t ne, size_t bc, size_t nc, size_t dim, void* stream) {
  if (!ent || !center || !offset || !dst_out || !dst_in)
    return fail(SMORE_ERR_NULL, "box_forward: required pointer is NULL");
  const Shape s{bsize, num, be, ne, bc, nc, dim, idx ? n_table_rows : 0};
  if (int rc = validate_shape(s)) return rc;
  return launch_forward<TermBoxBoth>(SMORE_DIST_BOX_BOTH, s, ent, idx, center, offset, dst_out, dst_in, (cudaStream_t)stream);
}

int smore_box_backward(const float* gout_out, const float* gout_in, const float* ent, const int64_t* idx,
                       size_t n_table_rows, const float* center, const float* offset, float* g_ent,
                       const int32_t* slot,
                       const int32_t* slot_count, float* g_rows, float* g_center, float* g_offset,
                       size_t bsize, size_t num, size_t be, size_t ne, size_t bc, size_t nc, size_t dim,
                       void* stream) {
  if (!gout_out || !gout_in || !ent || !center || !offset || !g_center || !g_offset)
    return fail(SMORE_ERR_NULL, "box_backward: required pointer is NULL");
  if (idx ? (!slot || !g_rows || g_ent) : (!g_ent || slot || g_rows))
    return fail(SMORE_ERR_NULL, "box_backward: pass g_ent (materialised) or slot/g_rows (indexed)");
  const Shape s{bsize, num, be, ne, bc, nc, dim, idx ? n_table_rows : 0};
  if (int rc = validate_shape(s)) return rc;
  return launch_backward<TermBoxBoth>(SMORE_DIST_BOX_BOTH, s, gout_out, gout_in, ent, idx, center, offset, g_ent, slot, slot_count,
                                      g_rows, g_center, g_offset, (cudaStream_t)stream);
}

int smore_union_forward_rows(int dist_id, const float* table, const int64_t* idx, size_t n_table_rows,
                             const float* first, const float* second, float* dst0, float* dst1, size_t branches,
                             size_t bsize, size_t num, size_t dim, void* stream) {
  const bool both = dist_id == SMORE_DIST_BOX_BOTH;
  if (!both && (dist_id < 0 || dist_id >= SMORE_DIST_COUNT))
    return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", dist_id);
  if (!table || !idx || !first || !dst0 || (both && !dst1) || ((both || needs_second(dist_id)) && !second))
    return fail(SMORE_ERR_NULL, "union_forward_rows: required pointer is NULL");
  const Shape s{bsize, num, bsize, num, bsize, 1, dim, n_table_rows};
  cudaStream_t st = (cudaStream_t)stream;
  if (both) return launch_forward_union<TermBoxBoth>(branches, s, table, idx, first, second, dst0, dst1, st);
  SMORE_DISPATCH(dist_id, launch_forward_union<Term>(branches, s, table, idx, first, second, dst0, dst0, st));
}

int smore_union_backward_rows(int dist_id, const float* gout0, const float* gout1, const float* table,
                              const int64_t* idx, size_t n_table_rows, const float* first, const float* second,
                              const int32_t* slot,
                              const int32_t* slot_count, float* g_rows, float* g_first, float* g_second,
                              size_t branches, size_t bsize, size_t num, size_t dim, void* stream) {
  const bool both = dist_id == SMORE_DIST_BOX_BOTH;
  if (!both && (dist_id < 0 || dist_id >= SMORE_DIST_COUNT))
    return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", dist_id);
  const bool two = both || needs_second(dist_id);
  if (!gout0 || (both && !gout1) || !table || !idx || !first || !slot || !g_rows || !g_first ||
      (two && (!second || !g_second)))
    return fail(SMORE_ERR_NULL, "union_backward_rows: required pointer is NULL");
  const Shape s{bsize, num, bsize, num, bsize, 1, dim, n_table_rows};
  cudaStream_t st = (cudaStream_t)stream;
  if (both)
    return launch_backward_union<TermBoxBoth>(branches, s, gout0, gout1, table, idx, first, second, slot, slot_count,
                                              g_rows, g_first, g_second, st);
  SMORE_DISPATCH(dist_id, launch_backward_union<Term>(branches, s, gout0, gout0, table, idx, first, second, slot,
                                                      slot_count, g_rows, g_first, g_second, st));
}

static int rows_backward_fused_adam(bool squeeze, int dist_id, const float* gout0, const float* gout1, float* table,
                                    const int64_t* idx, size_t n_table_rows, const float* first, const float* second,
                                    const int32_t* slot, const int32_t* slot_count, float* g_rows, float* g_first,
                                    float* g_second, size_t branches, size_t bsize, size_t num, size_t dim, float* m,
                                    float* v, int64_t* uniq, double lr, double beta1, double beta2, double eps,
                                    int64_t step, const float* step_scalars, void* stream) {
  const bool both = dist_id == SMORE_DIST_BOX_BOTH;
  if (!both && (dist_id < 0 || dist_id >= SMORE_DIST_COUNT))
    return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", dist_id);
  const bool two = both || needs_second(dist_id);
  if (!gout0 || (both && !gout1) || !table || !idx || !first || !slot || !slot_count || !g_rows || !g_first || !m ||
      !v || !uniq || (two && (!second || !g_second)))
    return fail(SMORE_ERR_NULL, "rows_backward_fused_adam: required pointer is NULL");
  if (branches != 1 && branches != (size_t)kUnionBranches)
    return fail(SMORE_ERR_BAD_SHAPE, "rows_backward_fused_adam: 1 or %d query branches", kUnionBranches);
  if (!step_scalars && step < 1) return fail(SMORE_ERR_BAD_SHAPE, "adam step must be >= 1");
  const Shape s{bsize, num, bsize, num, bsize, 1, dim, n_table_rows};
  if (int rc = validate_shape(s)) return rc;
  const size_t mul = (dist_id == SMORE_DIST_ROTATE || dist_id == SMORE_DIST_COMPLEX) ? 2 : 1;
  UpdateArgs ua;
  ua.table = table; ua.m = m; ua.v = v; ua.uniq = nullptr; ua.g_rows = nullptr; ua.n_unique = nullptr;
  ua.width = dim * mul;
  set_hyper(ua, lr, beta1, beta2, eps, step_scalars ? 1 : step, squeeze);
  ua.dyn = step_scalars;
  cudaStream_t st = (cudaStream_t)stream;
  int rc = 0;
  if (both) {
    rc = backward_adam_common<TermBoxBoth>(branches, s, gout0, gout1, table, idx, first, second, slot, slot_count, g_rows,
                                           g_first, g_second, ua, uniq, st);
  } else {
    switch (dist_id) {
#define FUSED_CASE(ID, TERM)                                                                                        \
  case ID:                                                                                                          \
    rc = backward_adam_common<TERM>(branches, s, gout0, gout0, table, idx, first, second, slot, slot_count, g_rows, \
                                    g_first, g_second, ua, uniq, st);                                               \
    break;
      FUSED_CASE(SMORE_DIST_BOX_OUT, TermBoxOut)
      FUSED_CASE(SMORE_DIST_BOX_IN, TermBoxIn)
      FUSED_CASE(SMORE_DIST_ROTATE, TermRotate)
      FUSED_CASE(SMORE_DIST_L1, TermL1)
      FUSED_CASE(SMORE_DIST_L2, TermL2)
      FUSED_CASE(SMORE_DIST_COMPLEX, TermComplex)
      FUSED_CASE(SMORE_DIST_DISTMULT, TermDistmult)
#undef FUSED_CASE
    }
  }
  if (rc < 0) return rc;
  if (rc == 0)
    return fail(SMORE_ERR_BAD_SHAPE,
                "rows_backward_fused_adam: shape not covered (dim a multiple of 4 up to 1024, with a row-wise second "
                "moment rows of 1 KB to about 4 KB, at least 4 rows per query, 16-byte aligned operands); use the "
                "separate backward and update calls");
  return SMORE_OK;
}

#define FUSED_PARAMS                                                                                                      \
  int dist_id, const float *gout0, const float *gout1, float *table, const int64_t *idx, size_t n_table_rows,             \
      const float *first, const float *second, const int32_t *slot, const int32_t *slot_count, float *g_rows,             \
      float *g_first, float *g_second, size_t branches, size_t bsize, size_t num, size_t dim, float *m, float *v,         \
      int64_t *uniq, double lr, double beta1, double beta2, double eps, int64_t step, const float *step_scalars,          \
      void *stream
#define FUSED_ARGS                                                                                                        \
  dist_id, gout0, gout1, table, idx, n_table_rows, first, second, slot, slot_count, g_rows, g_first, g_second, branches,  \
      bsize, num, dim, m, v, uniq, lr, beta1, beta2, eps, step, step_scalars, stream
int smore_rows_backward_fused_adam(FUSED_PARAMS) { return rows_backward_fused_adam(true, FUSED_ARGS); }
int smore_rows_backward_fused_adam_full(FUSED_PARAMS) { return rows_backward_fused_adam(false, FUSED_ARGS); }
#undef FUSED_PARAMS
#undef FUSED_ARGS

int smore_rows_forward_ragged(int dist_id, const float* table, const int64_t* rows, size_t n_table_rows,
                              const float* first, const float* second, const int32_t* segments, size_t n_segments,
                              size_t dim, float* out0, float* out1, const int32_t* positions,
                              size_t segments_per_rank, float* const* out0_ptrs, float* const* out1_ptrs,
                              size_t branches, size_t branch_stride, void* stream) {
  const bool both = dist_id == SMORE_DIST_BOX_BOTH;
  if (!both && (dist_id < 0 || dist_id >= SMORE_DIST_COUNT))
    return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", dist_id);
  if (!table || !rows || !first || !segments || ((both || needs_second(dist_id)) && !second))
    return fail(SMORE_ERR_NULL, "rows_forward_ragged: required pointer is NULL");
  if (positions ? (!out0_ptrs || (both && !out1_ptrs) || segments_per_rank == 0) : (!out0 || (both && !out1)))
    return fail(SMORE_ERR_NULL, "rows_forward_ragged: pass local result arrays, or positions with per-rank pointers");
  if (branches != 1 && (branches != (size_t)kUnionBranches || !positions))
    return fail(SMORE_ERR_BAD_SHAPE, "rows_forward_ragged: 1 branch, or %d with per-rank result arrays", kUnionBranches);
  const RaggedPeers pr{positions, segments_per_rank, branch_stride, out0_ptrs, both ? out1_ptrs : out0_ptrs, nullptr,
                       nullptr};
  if (n_segments == 0) return SMORE_OK;
  if (n_segments > (size_t)INT_MAX || dim == 0) return fail(SMORE_ERR_BAD_SHAPE, "rows_forward_ragged: bad sizes");
  cudaStream_t st = (cudaStream_t)stream;
  const int2* seg = reinterpret_cast<const int2*>(segments);
  int rc = 0;
  if (both) {
    rc = launch_forward_ragged<TermBoxBoth>(branches, n_segments, dim, n_table_rows, table, rows, first, second, seg, out0, out1, pr, st);
  } else {
    switch (dist_id) {
#define RAGGED_CASE(ID, TERM)                                                                                          \
  case ID:                                                                                                             \
    rc = launch_forward_ragged<TERM>(branches, n_segments, dim, n_table_rows, table, rows, first, second, seg, out0, out0, pr, st); \
    break;
      RAGGED_CASE(SMORE_DIST_BOX_OUT, TermBoxOut)
      RAGGED_CASE(SMORE_DIST_BOX_IN, TermBoxIn)
      RAGGED_CASE(SMORE_DIST_ROTATE, TermRotate)
      RAGGED_CASE(SMORE_DIST_L1, TermL1)
      RAGGED_CASE(SMORE_DIST_L2, TermL2)
      RAGGED_CASE(SMORE_DIST_COMPLEX, TermComplex)
      RAGGED_CASE(SMORE_DIST_DISTMULT, TermDistmult)
#undef RAGGED_CASE
    }
  }
  if (rc < 0) return rc;
  if (rc == 0)
    return fail(SMORE_ERR_BAD_SHAPE, "rows_forward_ragged: rows of 1 KB to about 6 KB, dim a multiple of 4 above 256, "
                                     "16-byte aligned operands");
  return SMORE_OK;
}

int smore_rows_backward_fused_adam_ragged(int dist_id, const float* gout0, const float* gout1, float* table,
                                          const int64_t* rows, size_t n_table_rows, const float* first,
                                          const float* second, const int32_t* segments, size_t n_segments,
                                          const int32_t* slot, const int32_t* slot_count, float* g_rows, float* g_first,
                                          float* g_second, size_t dim, float* m, float* v, int64_t* uniq, double lr,
                                          double beta1, double beta2, double eps, int64_t step,
                                          const float* step_scalars, const int32_t* positions,
                                          size_t segments_per_rank, const float* const* gout0_ptrs,
                                          const float* const* gout1_ptrs, size_t branches, size_t branch_stride,
                                          void* stream) {
  const bool both = dist_id == SMORE_DIST_BOX_BOTH;
  if (!both && (dist_id < 0 || dist_id >= SMORE_DIST_COUNT))
    return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", dist_id);
  const bool two = both || needs_second(dist_id);
  if (!table || !rows || !first || !segments || !slot || !slot_count || !g_rows || !g_first || !m || !v || !uniq ||
      (two && (!second || !g_second)))
    return fail(SMORE_ERR_NULL, "rows_backward_fused_adam_ragged: required pointer is NULL");
  if (positions ? (!gout0_ptrs || (both && !gout1_ptrs) || segments_per_rank == 0) : (!gout0 || (both && !gout1)))
    return fail(SMORE_ERR_NULL, "rows_backward_fused_adam_ragged: pass local upstream gradients, or positions with "
                                "per-rank pointers");
  if (branches != 1 && (branches != (size_t)kUnionBranches || !positions))
    return fail(SMORE_ERR_BAD_SHAPE, "rows_backward_fused_adam_ragged: 1 branch, or %d with per-rank upstream arrays",
                kUnionBranches);
  const RaggedPeers pr{positions, segments_per_rank, branch_stride, nullptr, nullptr, gout0_ptrs,
                       both ? gout1_ptrs : gout0_ptrs};
  if (!step_scalars && step < 1) return fail(SMORE_ERR_BAD_SHAPE, "adam step must be >= 1");
  if (n_segments == 0) return SMORE_OK;
  if (n_segments > (size_t)INT_MAX || dim == 0) return fail(SMORE_ERR_BAD_SHAPE, "rows_backward_fused_adam_ragged: bad sizes");
  const size_t mul = (dist_id == SMORE_DIST_ROTATE || dist_id == SMORE_DIST_COMPLEX) ? 2 : 1;
  UpdateArgs ua;
  ua.table = table; ua.m = m; ua.v = v; ua.uniq = nullptr; ua.g_rows = nullptr; ua.n_unique = nullptr;
  ua.width = dim * mul;
  set_hyper(ua, lr, beta1, beta2, eps, step_scalars ? 1 : step, 1);
  ua.dyn = step_scalars;
  cudaStream_t st = (cudaStream_t)stream;
  const int2* seg = reinterpret_cast<const int2*>(segments);
  int rc = 0;
  if (both) {
    rc = launch_backward_adam_ragged<TermBoxBoth>(branches, n_segments, dim, n_table_rows, gout0, gout1, table, rows, first, second,
                                                  seg, slot, slot_count, g_rows, g_first, g_second, ua, uniq, pr, st);
  } else {
    switch (dist_id) {
#define RAGGED_CASE(ID, TERM)                                                                                      \
  case ID:                                                                                                         \
    rc = launch_backward_adam_ragged<TERM>(branches, n_segments, dim, n_table_rows, gout0, gout0, table, rows, first, second, \
                                           seg, slot, slot_count, g_rows, g_first, g_second, ua, uniq, pr, st);    \
    break;
      RAGGED_CASE(SMORE_DIST_BOX_OUT, TermBoxOut)
      RAGGED_CASE(SMORE_DIST_BOX_IN, TermBoxIn)
      RAGGED_CASE(SMORE_DIST_ROTATE, TermRotate)
      RAGGED_CASE(SMORE_DIST_L1, TermL1)
      RAGGED_CASE(SMORE_DIST_L2, TermL2)
      RAGGED_CASE(SMORE_DIST_COMPLEX, TermComplex)
      RAGGED_CASE(SMORE_DIST_DISTMULT, TermDistmult)
#undef RAGGED_CASE
    }
  }
  if (rc < 0) return rc;
  if (rc == 0)
    return fail(SMORE_ERR_BAD_SHAPE, "rows_backward_fused_adam_ragged: rows of 1 KB to about 4 KB, dim a multiple of 4 "
                                     "above 256, 16-byte aligned operands");
  return SMORE_OK;
}

extern "C" int smore_peer_async_status(int* status);   // peer_kernels.cu (not part of the public header)
extern "C" int smore_rows_status(int* status);         // rows_kernels.cu (likewise)
extern "C" int smore_query_status(int* status);        // query_kernels.cu (likewise)
extern "C" int smore_shared_status(int* status);       // shared_kernels.cu (likewise)
extern "C" int smore_cell_status(int* status);         // cell_kernels.cu (likewise)
extern "C" int smore_split_status(int* status);        // gemm_split_sm100.cu (likewise)
extern "C" int smore_shared_status_clear(void);
extern "C" int smore_split_status_clear(void);
extern "C" int smore_cell_status_clear(void);
extern "C" int smore_peer_status_clear(void);
extern "C" int smore_rows_status_clear(void);
extern "C" int smore_query_status_clear(void);

int smore_async_status(int* status) {
  if (!status) return fail(SMORE_ERR_NULL, "async_status: NULL pointer");
  int v = 0, peer = 0, rows = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_async_status, sizeof(int));
  if (e != cudaSuccess) return fail(SMORE_ERR_CUDA, "async_status: %s", cudaGetErrorString(e));
  if (int rc = smore_peer_async_status(&peer)) return rc;   // the other files' kernels keep their own words
  if (int rc = smore_rows_status(&rows)) return rc;
  int query = 0, shared = 0, cell = 0, split = 0;
  if (int rc = smore_query_status(&query)) return rc;
  if (int rc = smore_shared_status(&shared)) return rc;
  if (int rc = smore_cell_status(&cell)) return rc;
  if (int rc = smore_split_status(&split)) return rc;
  *status = v | shared | cell | split | ((peer & 1) ? kStatusPeerWait : 0) | (peer & ~1) | rows | query;
  return SMORE_OK;
}

int smore_async_status_clear(void) {
  if (cudaDeviceSynchronize() != cudaSuccess) return fail(SMORE_ERR_CUDA, "async_status_clear: device error");
  const int zero = 0;
  if (cudaMemcpyToSymbol(g_async_status, &zero, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status_clear: cannot write the status word");
  if (int rc = smore_peer_status_clear()) return rc;
  if (int rc = smore_query_status_clear()) return rc;
  if (int rc = smore_shared_status_clear()) return rc;
  if (int rc = smore_cell_status_clear()) return rc;
  if (int rc = smore_split_status_clear()) return rc;
  return smore_rows_status_clear();
}

}  // extern "C"

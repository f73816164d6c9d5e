// Relation projection of a batch of path queries in one pass, for the additive geometries.
//
// The reference embeds a path query hop by hop (smore/models/kg_reasoning.py:229-236): every hop
// looks up the relation rows of the batch and adds them to the running embedding
// (GQE: vec.py:58-60; Query2box: box.py:126-129, where the box offset grows by the relation's
// offset row, optionally passed through relu).  Per hop that is two lookups, two additions and, in
// backward, two sort-based index_put kernels.  Here all H hops of a batch are one kernel each way:
//   center[b] = start_center[b] + sum_h rel[ids[b, h]]            (added in hop order)
//   offset[b] = start_offset[b] + sum_h act(off[ids[b, h]])       (Query2box only)
// and the backward pass adds the output gradients to the H relation rows of every query.
//
// A batch is a few million elements at most and every element is a short serial chain (row id, row, next
// hop): the work is cut into one thread per (query, piece of V dims), so that all chains are in flight at
// once.  (One warp per query walking the dims took 31 us forward and 60 us backward for 4096 queries of
// dim 1000, 34 us forward for 1024 three-hop queries of dim 400.)
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace smore {

// ----------------------------------------------------------------------------------------
// The general form: any geometry, and the path may start from table rows named by index, so that
// the anchor rows are never gathered into a tensor of their own and their gradient goes straight
// into the step's compact gradient buffer (kg_reasoning.py:217-250 with the models' hooks).
//   geometry 0  additive          GQE (vec.py:58-60), Query2box (box.py:126-129)
//   geometry 1  rotation          RotatE: relation rows are phases, each hop multiplies the complex
//                                 state by cos(phase) + i sin(phase), phase = row * phase_scale
//                                 (rotate.py:101-109)
//   geometry 2  complex product   ComplEx: relation rows [re | im] (complex.py:108-117, identity normaliser)
//   geometry 3  product           DistMult (distmult.py:106-111, identity normaliser)
// State rows of the multiplicative geometries are [re | im] (2 * dim floats), dim floats for DistMult.
// ----------------------------------------------------------------------------------------

constexpr int kMaxHops = 8;
__device__ int g_query_status = 0;   // kStatusBadRowId: a start-row id lay outside the table

struct EmbedArgs {
  int geometry;
  const float* start;          // [B, W] rows, or the table when start_idx != nullptr
  const int64_t* start_idx;    // nullable [B]
  long long n_start_rows;
  const float* start_offset;   // additive: [B, D] or nullptr
  const float* rel;            // [R, D] ([R, 2D] for geometry 2)
  const float* off;            // additive: [R, D] or nullptr
  const int64_t* ids;
  size_t id_stride, B, H, D, R;
  int relu_offset;
  float phase_scale;
};

template <int V>
struct alignas(4 * V) Piece {
  float v[V];
};
template <int V>
__device__ __forceinline__ Piece<V> piece_at(const float* p) {
  return *reinterpret_cast<const Piece<V>*>(p);
}
template <int V>
__device__ __forceinline__ void piece_add(float* p, const Piece<V>& x) {
  if constexpr (V == 4) atomicAdd(reinterpret_cast<float4*>(p), make_float4(x.v[0], x.v[1], x.v[2], x.v[3]));
  else atomicAdd(p, x.v[0]);
}

template <int V>
__device__ __forceinline__ void hop_pieces(const EmbedArgs& a, size_t r, size_t d, Piece<V>& c, Piece<V>& s) {
  if (a.geometry == 2) {
    c = piece_at<V>(a.rel + r * 2 * a.D + d);
    s = piece_at<V>(a.rel + r * 2 * a.D + a.D + d);
    return;
  }
  c = piece_at<V>(a.rel + r * a.D + d);
#pragma unroll
  for (int k = 0; k < V; ++k) {
    if (a.geometry == 1) {
      const float ph = c.v[k] * a.phase_scale;
      c.v[k] = cosf(ph);
      s.v[k] = sinf(ph);
    } else {
      s.v[k] = 0.f;
    }
  }
}

template <int V>
__global__ void __launch_bounds__(256)
    path_embed_forward_kernel(EmbedArgs a, float* __restrict__ out0, float* __restrict__ out1) {
  const bool two = a.geometry == 1 || a.geometry == 2;
  const size_t W = two ? 2 * a.D : a.D, cols = a.D / V, total = a.B * cols;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const size_t b = t / cols, d = (t - b * cols) * V;
    long long row = (long long)b;
    if (a.start_idx) row = checked_row_id(a.start_idx, b, a.n_start_rows, &g_query_status);
    const bool bad = row < 0;
    const float* x = a.start + (size_t)(bad ? 0 : row) * W;
    Piece<V> re = piece_at<V>(x + d), im = {};
    if (two) im = piece_at<V>(x + a.D + d);
    else if (a.geometry == 0 && a.start_offset) im = piece_at<V>(a.start_offset + b * a.D + d);
    for (size_t h = 0; h < a.H; ++h) {
      const size_t r = (size_t)a.ids[b * a.id_stride + h];
      if (r >= a.R) continue;   // out-of-range relation id: contributes nothing
      if (a.geometry == 0) {
        const Piece<V> c = piece_at<V>(a.rel + r * a.D + d);
#pragma unroll
        for (int k = 0; k < V; ++k) re.v[k] += c.v[k];
        if (a.off) {
          const Piece<V> o = piece_at<V>(a.off + r * a.D + d);
#pragma unroll
          for (int k = 0; k < V; ++k) im.v[k] += a.relu_offset ? fmaxf(o.v[k], 0.f) : o.v[k];
        }
        continue;
      }
      Piece<V> c, s;
      hop_pieces<V>(a, r, d, c, s);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        if (two) {
          const float nre = re.v[k] * c.v[k] - im.v[k] * s.v[k], nim = re.v[k] * s.v[k] + im.v[k] * c.v[k];
          re.v[k] = nre;
          im.v[k] = nim;
        } else {
          re.v[k] *= c.v[k];
        }
      }
    }
    if (bad) {
#pragma unroll
      for (int k = 0; k < V; ++k) re.v[k] = im.v[k] = NAN;
    }
    *reinterpret_cast<Piece<V>*>(out0 + b * a.D + d) = re;
    if (two || a.off) *reinterpret_cast<Piece<V>*>(out1 + b * a.D + d) = im;
  }
}

struct EmbedGradArgs {
  const float* g0;             // gradient of out0 [B, D]
  const float* g1;             // gradient of out1 [B, D] (nullable)
  float* g_rel;                // dense [R, D] ([R, 2D] for geometry 2), zeroed before the launch
  float* g_off;                // additive, nullable
  float* g_start;              // dense [B, W], or nullptr when slot != nullptr
  const int32_t* slot;         // [B] -> row of g_rows (< 0: skip)
  const int32_t* slot_count;   // nullable: nullptr = accumulate everywhere
  float* g_rows;
};

template <int V>
__global__ void __launch_bounds__(256) path_embed_backward_kernel(EmbedArgs a, EmbedGradArgs ga) {
  const bool two = a.geometry == 1 || a.geometry == 2;
  const size_t W = two ? 2 * a.D : a.D, cols = a.D / V, total = a.B * cols;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const size_t b = t / cols, d = (t - b * cols) * V;
    long long row = (long long)b;
    if (a.start_idx) row = checked_row_id(a.start_idx, b, a.n_start_rows, &g_query_status);
    if (row < 0) continue;      // a start row that does not exist: no gradient from it or for it
    float* gs = nullptr;
    bool store = true;
    if (ga.slot) {
      const int32_t sl = ga.slot[b];
      if (sl >= 0) {
        gs = ga.g_rows + (size_t)sl * W;
        store = ga.slot_count != nullptr && ga.slot_count[sl] == 1;
      }
    } else if (ga.g_start) {
      gs = ga.g_start + b * W;
    }
    Piece<V> gre = piece_at<V>(ga.g0 + b * a.D + d), gim = {};
    if (two && ga.g1) gim = piece_at<V>(ga.g1 + b * a.D + d);
    if (a.geometry == 0) {
      Piece<V> go = {};
      if (ga.g_off && ga.g1) go = piece_at<V>(ga.g1 + b * a.D + d);
      for (size_t h = 0; h < a.H; ++h) {
        const size_t r = (size_t)a.ids[b * a.id_stride + h];
        if (r >= a.R) continue;
        piece_add(ga.g_rel + r * a.D + d, gre);
        if (ga.g_off) {
          Piece<V> g = go;
          if (a.relu_offset) {
            const Piece<V> o = piece_at<V>(a.off + r * a.D + d);
#pragma unroll
            for (int k = 0; k < V; ++k)
              if (!(o.v[k] > 0.f)) g.v[k] = 0.f;
          }
          piece_add(ga.g_off + r * a.D + d, g);
        }
      }
    } else {
      // recompute the states before every hop, then walk the hops backwards
      const float* x = a.start + (size_t)row * W;
      Piece<V> xre[kMaxHops], xim[kMaxHops], cs[kMaxHops], sn[kMaxHops];
      Piece<V> re = piece_at<V>(x + d), im = {};
      if (two) im = piece_at<V>(x + a.D + d);
#pragma unroll
      for (int h = 0; h < kMaxHops; ++h) {
        if (h >= (int)a.H) break;
        xre[h] = re;
        xim[h] = im;
        const size_t r = (size_t)a.ids[b * a.id_stride + h];
        if (r >= a.R) continue;
        hop_pieces<V>(a, r, d, cs[h], sn[h]);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          if (two) {
            const float nre = re.v[k] * cs[h].v[k] - im.v[k] * sn[h].v[k];
            const float nim = re.v[k] * sn[h].v[k] + im.v[k] * cs[h].v[k];
            re.v[k] = nre;
            im.v[k] = nim;
          } else {
            re.v[k] *= cs[h].v[k];
          }
        }
      }
#pragma unroll
      for (int h = kMaxHops - 1; h >= 0; --h) {
        if (h >= (int)a.H) continue;
        const size_t r = (size_t)a.ids[b * a.id_stride + h];
        if (r >= a.R) continue;
        Piece<V> g_c, g_s, nre, nim;
#pragma unroll
        for (int k = 0; k < V; ++k) {
          g_c.v[k] = gre.v[k] * xre[h].v[k] + gim.v[k] * xim[h].v[k];
          g_s.v[k] = gim.v[k] * xre[h].v[k] - gre.v[k] * xim[h].v[k];
          nre.v[k] = gre.v[k] * cs[h].v[k] + gim.v[k] * sn[h].v[k];
          nim.v[k] = gim.v[k] * cs[h].v[k] - gre.v[k] * sn[h].v[k];
        }
        if (a.geometry == 1) {
          Piece<V> g_p;
#pragma unroll
          for (int k = 0; k < V; ++k) g_p.v[k] = (g_s.v[k] * cs[h].v[k] - g_c.v[k] * sn[h].v[k]) * a.phase_scale;
          piece_add(ga.g_rel + r * a.D + d, g_p);
        } else if (a.geometry == 2) {
          piece_add(ga.g_rel + r * 2 * a.D + d, g_c);
          piece_add(ga.g_rel + r * 2 * a.D + a.D + d, g_s);
        } else {
          piece_add(ga.g_rel + r * a.D + d, g_c);
        }
        gre = nre;
        gim = nim;
      }
    }
    if (gs != nullptr) {
      if (store) {
        *reinterpret_cast<Piece<V>*>(gs + d) = gre;
        if (two) *reinterpret_cast<Piece<V>*>(gs + a.D + d) = gim;
      } else {
        piece_add(gs + d, gre);
        if (two) piece_add(gs + a.D + d, gim);
      }
    }
  }
}

static int path_grid(size_t threads) {
  return (int)std::max<size_t>(1, std::min<size_t>((threads + 255) / 256, (size_t)sm_count() * 16));
}

template <class... P>
static bool all16(const P*... ptr) {
  return ((reinterpret_cast<uintptr_t>(ptr) | ...) & 15u) == 0;
}

}  // namespace smore

using namespace smore;

extern "C" {

static int embed_check(const char* what, int geometry, size_t n_relations, size_t id_stride, size_t hops, size_t dim) {
  if (geometry < 0 || geometry > 3) return fail(SMORE_ERR_BAD_DIST, "%s: unknown geometry %d", what, geometry);
  if (dim == 0 || hops == 0 || id_stride < hops || n_relations == 0)
    return fail(SMORE_ERR_BAD_SHAPE, "%s: dim, hops, n_relations must be positive, id_stride >= hops", what);
  if (geometry != 0 && hops > (size_t)kMaxHops)
    return fail(SMORE_ERR_TOO_LARGE, "%s: at most %d hops per call for the multiplicative geometries", what, kMaxHops);
  return SMORE_OK;
}

int smore_path_embed_forward(int geometry, const float* start, const int64_t* start_idx, size_t n_start_rows,
                             const float* start_offset, const float* rel_table, const float* off_table,
                             size_t n_relations, const int64_t* rel_ids, size_t id_stride, size_t n_queries,
                             size_t hops, size_t dim, int relu_offset, double phase_scale, float* out0, float* out1,
                             void* stream) {
  if (n_queries == 0) return SMORE_OK;
  if (int rc = embed_check("path_embed_forward", geometry, n_relations, id_stride, hops, dim)) return rc;
  const bool two = geometry == 1 || geometry == 2;
  if (!start || !rel_table || !rel_ids || !out0 || ((two || (geometry == 0 && off_table)) && !out1))
    return fail(SMORE_ERR_NULL, "path_embed_forward: NULL pointer");
  EmbedArgs a{geometry, start, start_idx, start_idx ? (long long)n_start_rows : 0,
              geometry == 0 && off_table ? start_offset : nullptr, rel_table, geometry == 0 ? off_table : nullptr,
              rel_ids, id_stride, n_queries, hops, dim, n_relations, relu_offset != 0, (float)phase_scale};
  if ((dim & 3) == 0 && all16(start, a.start_offset, rel_table, a.off, out0, out1))
    path_embed_forward_kernel<4><<<path_grid(n_queries * (dim / 4)), 256, 0, (cudaStream_t)stream>>>(a, out0, out1);
  else
    path_embed_forward_kernel<1><<<path_grid(n_queries * dim), 256, 0, (cudaStream_t)stream>>>(a, out0, out1);
  return check_launch("path_embed_forward_kernel");
}

int smore_path_embed_backward(int geometry, const float* g_out0, const float* g_out1, const float* start,
                              const int64_t* start_idx, size_t n_start_rows, const float* rel_table,
                              const float* off_table, size_t n_relations, const int64_t* rel_ids, size_t id_stride,
                              size_t n_queries, size_t hops, size_t dim, int relu_offset, double phase_scale,
                              float* g_rel_table, float* g_off_table, float* g_start, const int32_t* slot,
                              const int32_t* slot_count, float* g_rows, void* stream) {
  if (int rc = embed_check("path_embed_backward", geometry, n_relations, id_stride, hops, dim)) return rc;
  if (!g_rel_table) return fail(SMORE_ERR_NULL, "path_embed_backward: g_rel_table is NULL");
  if (slot ? (!g_rows || g_start) : (g_rows != nullptr))
    return fail(SMORE_ERR_NULL, "path_embed_backward: pass g_start (rows given as a tensor) or slot / g_rows (table rows)");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t rel_width = geometry == 2 ? 2 * dim : dim;
  if (cudaMemsetAsync(g_rel_table, 0, n_relations * rel_width * sizeof(float), st) != cudaSuccess ||
      (geometry == 0 && g_off_table &&
       cudaMemsetAsync(g_off_table, 0, n_relations * dim * sizeof(float), st) != cudaSuccess))
    return fail(SMORE_ERR_CUDA, "path_embed_backward: cudaMemsetAsync failed");
  if (n_queries == 0) return SMORE_OK;
  if (!g_out0 || !rel_ids || (geometry != 0 && (!start || !rel_table)) ||
      (geometry == 0 && g_off_table && relu_offset && !off_table))
    return fail(SMORE_ERR_NULL, "path_embed_backward: NULL pointer");
  EmbedArgs a{geometry, start, start_idx, start_idx ? (long long)n_start_rows : 0, nullptr, rel_table,
              geometry == 0 ? off_table : nullptr, rel_ids, id_stride, n_queries, hops, dim, n_relations,
              relu_offset != 0, (float)phase_scale};
  EmbedGradArgs ga{g_out0, g_out1, g_rel_table, geometry == 0 ? g_off_table : nullptr, g_start, slot, slot_count, g_rows};
  const bool vec = (dim & 3) == 0 && all16(start, rel_table, a.off, g_out0, g_out1, g_rel_table, ga.g_off, g_start, g_rows);
  if (vec) path_embed_backward_kernel<4><<<path_grid(n_queries * (dim / 4)), 256, 0, st>>>(a, ga);
  else path_embed_backward_kernel<1><<<path_grid(n_queries * dim), 256, 0, st>>>(a, ga);
  return check_launch("path_embed_backward_kernel");
}

int smore_path_project_forward(const float* start_center, const float* start_offset, const float* rel_table,
                               const float* off_table, size_t n_relations, const int64_t* rel_ids, size_t id_stride,
                               size_t n_queries, size_t hops, size_t dim, int relu_offset, float* center,
                               float* offset, void* stream) {
  return smore_path_embed_forward(0, start_center, nullptr, 0, start_offset, rel_table, off_table, n_relations, rel_ids,
                                  id_stride, n_queries, hops, dim, relu_offset, 1.0, center, offset, stream);
}

int smore_path_project_backward(const float* g_center, const float* g_offset, const float* off_table,
                                size_t n_relations, const int64_t* rel_ids, size_t id_stride, size_t n_queries,
                                size_t hops, size_t dim, int relu_offset, float* g_rel_table, float* g_off_table,
                                void* stream) {
  if (g_off_table && !g_offset) return fail(SMORE_ERR_NULL, "path_project_backward: NULL pointer");
  return smore_path_embed_backward(0, g_center, g_offset, nullptr, nullptr, 0, nullptr, off_table, n_relations, rel_ids,
                                   id_stride, n_queries, hops, dim, relu_offset, 1.0, g_rel_table, g_off_table, nullptr,
                                   nullptr, nullptr, nullptr, stream);
}

int smore_query_status(int* status) {    // not part of the public header; smore_async_status adds it in
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_query_status, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status: cannot read the status word");
  *status = v;
  return SMORE_OK;
}

int smore_query_status_clear(void) {
  const int zero = 0;
  if (cudaMemcpyToSymbol(g_query_status, &zero, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status_clear: cannot write the status word");
  return SMORE_OK;
}

}  // extern "C"

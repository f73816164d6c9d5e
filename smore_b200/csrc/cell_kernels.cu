// Distance kernels for shapes without a candidate list: one entity row per query (the positives of a
// training step, alone or against the branches of a union query), any other broadcast the op contract
// allows, any dim, fp32 or fp64.
//   cell_forward_kernel           one warp per output cell
//   pair_backward_kernel          one entity row per query row or per group of `num` query rows: both
//                                 gradients of every element by the thread that owns the element
//   cell_backward_*_kernel        anything: one thread per gradient element walks the cells that use it
//                                 in a fixed order (deterministic, coalesced over the embedding dim)
#include <cuda_runtime.h>

#include "dist_common.cuh"

namespace smore {

static __device__ int g_cell_status = 0;   // kStatusBadRowId: a row id lay outside the table

template <typename T>
struct CellArgs {
  const T* ent;        // [be*ne, mul*dim] or table when idx != nullptr
  const int64_t* idx;  // nullable: row ids into `ent`
  const T* first;      // [bc*nc, dim]
  const T* second;     // [bc*nc, dim] (== first for single-operand distances)
  size_t bsize, num, be, ne, bc, nc, dim;
  long long n_rows;    // rows of `ent` when idx != nullptr (0: ids are not checked)
};

// VEC: 16-byte loads (fp32, dim a multiple of four, aligned operands)
template <typename T, class Term, bool VEC>
__global__ void __launch_bounds__(256) cell_forward_kernel(CellArgs<T> a, T* __restrict__ dst0,
                                                           T* __restrict__ dst1) {
  const int lane = threadIdx.x & 31;
  const size_t warps_per_grid = (size_t)gridDim.x * (blockDim.x >> 5);
  const size_t cells = a.bsize * a.num;
  for (size_t cell = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); cell < cells;
       cell += warps_per_grid) {
    const size_t i = cell / a.num, j = cell - i * a.num;
    size_t row = (i % a.be) * a.ne + (j % a.ne);
    bool bad = false;
    if (a.idx) {
      const long long r = checked_row_id(a.idx, row, a.n_rows, &g_cell_status);
      bad = r < 0;
      row = bad ? 0 : (size_t)r;
    }
    const T* pe = a.ent + row * a.dim * Term::kMul;
    const size_t qrow = (i % a.bc) * a.nc + (j % a.nc);
    const T* p0 = a.first + qrow * a.dim;
    const T* p1 = a.second + qrow * a.dim;
    T acc[Term::kNOut];
#pragma unroll
    for (int o = 0; o < Term::kNOut; ++o) acc[o] = T(0);
    if constexpr (VEC) {
      const float4 *e4 = reinterpret_cast<const float4*>(pe), *q4 = reinterpret_cast<const float4*>(p0),
                   *r4 = reinterpret_cast<const float4*>(p1);
      const size_t dim4 = a.dim >> 2;
#pragma unroll 4
      for (size_t d = lane; d < dim4; d += kWarp) {
        const float4 e0 = __ldg(e4 + d), q0 = __ldg(q4 + d);
        const float4 e1 = Term::kMul == 2 ? __ldg(e4 + dim4 + d) : e0;
        const float4 q1 = Term::kNQ == 2 ? __ldg(r4 + d) : q0;
        Term::fwd(e0.x, e1.x, q0.x, q1.x, acc);
        Term::fwd(e0.y, e1.y, q0.y, q1.y, acc);
        Term::fwd(e0.z, e1.z, q0.z, q1.z, acc);
        Term::fwd(e0.w, e1.w, q0.w, q1.w, acc);
      }
    } else {
#pragma unroll 4
      for (size_t d = lane; d < a.dim; d += kWarp) {
        const T e0 = pe[d];
        const T e1 = Term::kMul == 2 ? pe[d + a.dim] : T(0);
        Term::fwd(e0, e1, p0[d], p1[d], acc);
      }
    }
#pragma unroll
    for (int o = 0; o < Term::kNOut; ++o) {
#pragma unroll
      for (int m = kWarp / 2; m > 0; m >>= 1) acc[o] += __shfl_xor_sync(0xffffffffu, acc[o], m);
    }
    if (lane == 0) {
      dst0[cell] = bad ? T(NAN) : acc[0];
      if (Term::kNOut == 2) dst1[cell] = bad ? T(NAN) : acc[Term::kNOut - 1];
    }
  }
}

// One thread per (entity position, d).  With slot == nullptr the result is stored to
// g_ent[position]; otherwise it goes to g_rows[slot[position]] (store when that slot has a
// single contributor in the whole step, atomic otherwise).
template <typename T, class Term>
__global__ void __launch_bounds__(256)
    cell_backward_ent_kernel(CellArgs<T> a, const T* __restrict__ gout0, const T* __restrict__ gout1,
                             T* __restrict__ g_ent, const int32_t* __restrict__ slot,
                             const int32_t* __restrict__ slot_count, T* __restrict__ g_rows) {
  const size_t total = a.be * a.ne * a.dim;
  const size_t nji = a.bsize / a.be, njj = a.num / a.ne;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const size_t pos = t / a.dim, d = t - pos * a.dim;
    const size_t r0 = pos / a.ne, r1 = pos - r0 * a.ne;
    size_t row = pos;
    if (a.idx) {
      const long long r = checked_row_id(a.idx, pos, a.n_rows, &g_cell_status);
      if (r < 0) continue;   // no gradient from (or for) a row that does not exist
      row = (size_t)r;
    }
    const T* pe = a.ent + row * a.dim * Term::kMul;
    const T e0 = pe[d];
    const T e1 = Term::kMul == 2 ? pe[d + a.dim] : T(0);
    T ge0 = T(0), ge1 = T(0), t0 = T(0), t1 = T(0);
    for (size_t ji = 0; ji < nji; ++ji) {
      const size_t i = ji * a.be + r0;
      for (size_t jj = 0; jj < njj; ++jj) {
        const size_t j = jj * a.ne + r1;
        const size_t qrow = (i % a.bc) * a.nc + (j % a.nc);
        T g[Term::kNOut];
        g[0] = gout0[i * a.num + j];
        if (Term::kNOut == 2) g[Term::kNOut - 1] = gout1[i * a.num + j];
        Term::bwd(g, e0, e1, Term::prep(a.first[qrow * a.dim + d]), a.second[qrow * a.dim + d], ge0, ge1, t0, t1);
      }
    }
    if (slot == nullptr) {
      T* out = g_ent + pos * a.dim * Term::kMul;
      out[d] = ge0;
      if (Term::kMul == 2) out[d + a.dim] = ge1;
    } else {
      const int32_t s = slot[pos];
      if (s < 0) continue;
      T* out = g_rows + (size_t)s * a.dim * Term::kMul;
      if (slot_count != nullptr && slot_count[s] == 1) {
        out[d] = ge0;
        if (Term::kMul == 2) out[d + a.dim] = ge1;
      } else {
        atomicAdd(out + d, ge0);
        if (Term::kMul == 2) atomicAdd(out + d + a.dim, ge1);
      }
    }
  }
}

template <typename T, class Term>
__global__ void __launch_bounds__(256)
    cell_backward_query_kernel(CellArgs<T> a, const T* __restrict__ gout0, const T* __restrict__ gout1,
                               T* __restrict__ g_first, T* __restrict__ g_second) {
  const size_t total = a.bc * a.nc * a.dim;
  const size_t nji = a.bsize / a.bc, njj = a.num / a.nc;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const size_t qrow = t / a.dim, d = t - qrow * a.dim;
    const size_t r0 = qrow / a.nc, r1 = qrow - r0 * a.nc;
    const T q0 = Term::prep(a.first[qrow * a.dim + d]), q1 = a.second[qrow * a.dim + d];
    T gq0 = T(0), gq1 = T(0), t0 = T(0), t1 = T(0);
    for (size_t ji = 0; ji < nji; ++ji) {
      const size_t i = ji * a.bc + r0;
      for (size_t jj = 0; jj < njj; ++jj) {
        const size_t j = jj * a.nc + r1;
        size_t row = (i % a.be) * a.ne + (j % a.ne);
        if (a.idx) {
          const long long r = checked_row_id(a.idx, row, a.n_rows, &g_cell_status);
          if (r < 0) continue;
          row = (size_t)r;
        }
        const T* pe = a.ent + row * a.dim * Term::kMul;
        T g[Term::kNOut];
        g[0] = gout0[i * a.num + j];
        if (Term::kNOut == 2) g[Term::kNOut - 1] = gout1[i * a.num + j];
        Term::bwd(g, pe[d], Term::kMul == 2 ? pe[d + a.dim] : T(0), q0, q1, t0, t1, gq0, gq1);
      }
    }
    g_first[qrow * a.dim + d] = gq0;
    if (Term::kNQ == 2) g_second[qrow * a.dim + d] = gq1;
  }
}

// Entity [B, 1, W] against queries [B, num, dim]: no element of a gradient is shared between entity rows,
// so the thread that owns element piece (b, d) computes the entity gradient (summed over the row's queries
// in registers) and the query gradients in one pass, with V-float accesses.
// (4096 rows of 1000 floats: 64 us + 43 us as one scalar pass per gradient.)
template <class Term, int V>
__global__ void __launch_bounds__(256)
    pair_backward_kernel(CellArgs<float> a, const float* __restrict__ gout0, const float* __restrict__ gout1,
                         float* __restrict__ g_ent, const int32_t* __restrict__ slot,
                         const int32_t* __restrict__ slot_count, float* __restrict__ g_rows, float* __restrict__ g_first,
                         float* __restrict__ g_second) {
  struct alignas(4 * V) Piece { float v[V]; };
  const size_t cols = a.dim / V, total = a.be * cols;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const size_t b = t / cols, d = (t - b * cols) * V;
    size_t row = b;
    bool bad = false;
    if (a.idx) {
      const long long r = checked_row_id(a.idx, b, a.n_rows, &g_cell_status);
      bad = r < 0;                 // no gradient from (or for) a row that does not exist
      row = bad ? 0 : (size_t)r;
    }
    const float* pe = a.ent + row * a.dim * Term::kMul + d;
    const Piece e0 = *reinterpret_cast<const Piece*>(pe);
    const Piece e1 = Term::kMul == 2 ? *reinterpret_cast<const Piece*>(pe + a.dim) : e0;
    Piece ge0 = {}, ge1 = {};
    for (size_t j = 0; j < a.num; ++j) {
      const size_t cell = b * a.num + j, at = cell * a.dim + d;
      const Piece q0 = *reinterpret_cast<const Piece*>(a.first + at);
      const Piece q1 = Term::kNQ == 2 ? *reinterpret_cast<const Piece*>(a.second + at) : q0;
      float g[Term::kNOut];
      g[0] = bad ? 0.f : gout0[cell];
      if (Term::kNOut == 2) g[Term::kNOut - 1] = bad ? 0.f : gout1[cell];
      Piece gq0 = {}, gq1 = {};
#pragma unroll
      for (int i = 0; i < V; ++i)
        Term::bwd(g, e0.v[i], e1.v[i], Term::prep(q0.v[i]), q1.v[i], ge0.v[i], ge1.v[i], gq0.v[i], gq1.v[i]);
      if (bad) gq0 = gq1 = Piece{};
      *reinterpret_cast<Piece*>(g_first + at) = gq0;
      if (Term::kNQ == 2) *reinterpret_cast<Piece*>(g_second + at) = gq1;
    }
    float* out;
    bool store = true;
    if (slot == nullptr) {
      out = g_ent + b * a.dim * Term::kMul + d;
    } else {
      const int32_t s = slot[b];
      if (s < 0 || bad) continue;
      out = g_rows + (size_t)s * a.dim * Term::kMul + d;
      store = slot_count != nullptr && slot_count[s] == 1;
    }
#pragma unroll
    for (int part = 0; part < Term::kMul; ++part) {
      const Piece& ge = part ? ge1 : ge0;
      float* o = out + part * a.dim;
      if (store) {
        *reinterpret_cast<Piece*>(o) = ge;
      } else if constexpr (V == 4) {
        atomicAdd(reinterpret_cast<float4*>(o), make_float4(ge.v[0], ge.v[1], ge.v[2], ge.v[3]));
      } else if constexpr (V == 2) {
        atomicAdd(reinterpret_cast<float2*>(o), make_float2(ge.v[0], ge.v[1]));
      } else {
        atomicAdd(o, ge.v[0]);
      }
    }
  }
}

template <class Term>
static int launch_cell_forward(const Shape& s, const ForwardArgs& f, cudaStream_t st) {
  const float* second = Term::kNQ == 2 ? f.second : f.first;
  CellArgs<float> a{f.ent, f.idx, f.first, second, s.bsize, s.num, s.be, s.ne, s.bc, s.nc, s.dim, (long long)s.n_rows};
  const int grid = grid_for(s.bsize * s.num, 8);
  if ((s.dim & 3) == 0 && aligned16(f.ent) && aligned16(f.first) && aligned16(second))
    cell_forward_kernel<float, Term, true><<<grid, 256, 0, st>>>(a, f.dst0, f.dst1);
  else
    cell_forward_kernel<float, Term, false><<<grid, 256, 0, st>>>(a, f.dst0, f.dst1);
  return check_launch("cell_forward_kernel");
}

template <class Term>
static int launch_cell_backward(const Shape& s, const BackwardArgs& b, cudaStream_t st) {
  const float* second = Term::kNQ == 2 ? b.second : b.first;
  float* g_second = Term::kNQ == 2 ? b.g_second : b.g_first;
  CellArgs<float> a{b.ent, b.idx, b.first, second, s.bsize, s.num, s.be, s.ne, s.bc, s.nc, s.dim, (long long)s.n_rows};
  if (s.be == s.bsize && s.bc == s.bsize && s.ne == 1 && s.nc == s.num) {
    float* gdst = b.slot ? b.g_rows : b.g_ent;
    uintptr_t bits = 0;
    for (const float* p : {b.ent, b.first, second, (const float*)gdst, (const float*)b.g_first, (const float*)g_second})
      bits |= reinterpret_cast<uintptr_t>(p);
    const int v = (s.dim & 3) == 0 && (bits & 15) == 0 ? 4 : (s.dim & 1) == 0 && (bits & 7) == 0 ? 2 : 1;
    auto kern = v == 4 ? pair_backward_kernel<Term, 4> : v == 2 ? pair_backward_kernel<Term, 2> : pair_backward_kernel<Term, 1>;
    kern<<<grid_for(s.be * (s.dim / v), 256), 256, 0, st>>>(a, b.gout0, b.gout1, b.g_ent, b.slot, b.slot_count, b.g_rows,
                                                            b.g_first, g_second);
    return check_launch("pair_backward_kernel");
  }
  cell_backward_ent_kernel<float, Term><<<grid_for(s.be * s.ne * s.dim, 256), 256, 0, st>>>(
      a, b.gout0, b.gout1, b.g_ent, b.slot, b.slot_count, b.g_rows);
  cell_backward_query_kernel<float, Term><<<grid_for(s.bc * s.nc * s.dim, 256), 256, 0, st>>>(
      a, b.gout0, b.gout1, b.g_first, g_second);
  return check_launch("cell_backward kernels", 2);
}

int cell_forward(int term, const Shape& s, const ForwardArgs& a, cudaStream_t st) {
  SMORE_DISPATCH_BOTH(term, launch_cell_forward<Term>(s, a, st));
}
int cell_backward(int term, const Shape& s, const BackwardArgs& a, cudaStream_t st) {
  SMORE_DISPATCH_BOTH(term, launch_cell_backward<Term>(s, a, st));
}

template <class Term>
static int launch_forward_f64(const Shape& s, const double* ent, const double* first,
                              const double* second, double* dst, cudaStream_t st) {
  if (Term::kNQ == 1) second = first;
  CellArgs<double> a{ent, nullptr, first, second, s.bsize, s.num, s.be, s.ne, s.bc, s.nc, s.dim, (long long)s.n_rows};
  cell_forward_kernel<double, Term, false><<<grid_for(s.bsize * s.num, 8), 256, 0, st>>>(a, dst, dst);
  return check_launch("cell_forward_kernel<double>");
}

template <class Term>
static int launch_backward_f64(const Shape& s, const double* gout, const double* ent,
                               const double* first, const double* second, double* g_ent,
                               double* g_first, double* g_second, cudaStream_t st) {
  if (Term::kNQ == 1) {
    second = first;
    g_second = g_first;
  }
  CellArgs<double> a{ent, nullptr, first, second, s.bsize, s.num, s.be, s.ne, s.bc, s.nc, s.dim, (long long)s.n_rows};
  cell_backward_ent_kernel<double, Term><<<grid_for(s.be * s.ne * s.dim, 256), 256, 0, st>>>(
      a, gout, gout, g_ent, nullptr, nullptr, nullptr);
  cell_backward_query_kernel<double, Term><<<grid_for(s.bc * s.nc * s.dim, 256), 256, 0, st>>>(
      a, gout, gout, g_first, g_second);
  return check_launch("cell_backward kernels<double>", 2);
}

}  // namespace smore

using namespace smore;

extern "C" {

int smore_dist_forward_f64(int dist_id, const double* ent, const double* first, const double* second,
                           double* dst, size_t bsize, size_t num, size_t be, size_t ne, size_t bc, size_t nc,
                           size_t dim, void* stream) {
  if (!ent || !first || !dst || (needs_second(dist_id) && !second))
    return fail(SMORE_ERR_NULL, "forward_f64: required pointer is NULL");
  const Shape s{bsize, num, be, ne, bc, nc, dim};
  if (int rc = validate_shape(s)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  SMORE_DISPATCH(dist_id, launch_forward_f64<Term>(s, ent, first, second, dst, st));
}

int smore_dist_backward_f64(int dist_id, const double* gout, const double* ent, const double* first,
                            const double* second, double* g_ent, double* g_first, double* g_second,
                            size_t bsize, size_t num, size_t be, size_t ne, size_t bc, size_t nc, size_t dim,
                            void* stream) {
  if (!gout || !ent || !first || !g_ent || !g_first || (needs_second(dist_id) && (!second || !g_second)))
    return fail(SMORE_ERR_NULL, "backward_f64: required pointer is NULL");
  const Shape s{bsize, num, be, ne, bc, nc, dim};
  if (int rc = validate_shape(s)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  SMORE_DISPATCH(dist_id, launch_backward_f64<Term>(s, gout, ent, first, second, g_ent, g_first, g_second, st));
}

int smore_cell_status(int* status) {   // not part of the public header; smore_async_status adds it in
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_cell_status, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status: cannot read the status word");
  *status = v;
  return SMORE_OK;
}

int smore_cell_status_clear(void) {
  const int zero = 0;
  if (cudaMemcpyToSymbol(g_cell_status, &zero, sizeof(int)) != cudaSuccess)
    return fail(SMORE_ERR_CUDA, "async_status_clear: cannot write the status word");
  return SMORE_OK;
}

}  // extern "C"

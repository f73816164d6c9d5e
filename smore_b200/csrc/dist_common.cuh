// Shapes, term dispatch and the entry points by which the three files of distance kernels call one another:
//   dist_kernels.cu    candidate rows of each query's own (row-stream kernels) and the C entry points
//   shared_kernels.cu  one candidate list for all queries, and the evaluation step
//   cell_kernels.cu    every other broadcast, one candidate per query, fp64
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "common.cuh"
#include "dist_terms.cuh"

namespace smore {

struct Shape {
  size_t bsize, num, be, ne, bc, nc, dim;
  size_t n_rows = 0;   // rows of the table when the entity operand is (table, idx); 0: ids unchecked
};

inline int validate_shape(const Shape& s) {
  if (!s.bsize || !s.num || !s.be || !s.ne || !s.bc || !s.nc || !s.dim)
    return fail(SMORE_ERR_BAD_SHAPE, "all sizes must be positive");
  if (s.bsize != std::max(s.be, s.bc) || s.num != std::max(s.ne, s.nc))
    return fail(SMORE_ERR_BAD_SHAPE, "output must be [max(be,bc), max(ne,nc)]");
  if (s.bsize % s.be || s.bsize % s.bc || s.num % s.ne || s.num % s.nc)
    return fail(SMORE_ERR_BAD_SHAPE, "operand sizes must divide the output sizes");
  if (s.dim > (size_t)1 << 30 || s.bsize * s.num > (size_t)1 << 40)
    return fail(SMORE_ERR_TOO_LARGE, "operand too large");
  return SMORE_OK;
}

inline int grid_for(size_t work_items, int per_block) {
  size_t blocks = (work_items + per_block - 1) / per_block;
  const size_t cap = (size_t)sm_count() * 32;
  return (int)std::max<size_t>(1, std::min(blocks, cap));
}

inline bool needs_second(int id) {
  return id == SMORE_DIST_BOX_OUT || id == SMORE_DIST_BOX_IN || id == SMORE_DIST_ROTATE ||
         id == SMORE_DIST_COMPLEX;
}

#define SMORE_DISPATCH(id, CALL)                                        \
  switch (id) {                                                         \
    case SMORE_DIST_BOX_OUT: { using Term = TermBoxOut; return CALL; }  \
    case SMORE_DIST_BOX_IN: { using Term = TermBoxIn; return CALL; }    \
    case SMORE_DIST_ROTATE: { using Term = TermRotate; return CALL; }   \
    case SMORE_DIST_L1: { using Term = TermL1; return CALL; }           \
    case SMORE_DIST_L2: { using Term = TermL2; return CALL; }           \
    case SMORE_DIST_COMPLEX: { using Term = TermComplex; return CALL; } \
    case SMORE_DIST_DISTMULT: { using Term = TermDistmult; return CALL; } \
    default: return fail(SMORE_ERR_BAD_DIST, "unknown distance id %d", id); \
  }

// the same with both box distances (SMORE_DIST_BOX_BOTH)
#define SMORE_DISPATCH_BOTH(id, CALL)                                          \
  do {                                                                         \
    if (id == SMORE_DIST_BOX_BOTH) { using Term = TermBoxBoth; return CALL; }  \
    SMORE_DISPATCH(id, CALL)                                                   \
  } while (0)

// Operands of one call; `term` is a distance id or SMORE_DIST_BOX_BOTH.
struct ForwardArgs {
  const float* ent;        // [be * ne, mul * dim], or the table when idx != nullptr
  const int64_t* idx;      // nullable [be * ne]
  const float *first, *second;   // [bc * nc, dim]; second == first where the distance has one operand
  float *dst0, *dst1;
};
struct BackwardArgs {
  const float *gout0, *gout1;
  const float* ent;
  const int64_t* idx;
  const float *first, *second;
  float* g_ent;              // dense entity gradient, or nullptr when slot != nullptr
  const int32_t* slot;       // row of g_rows per entity position, < 0: skip
  const int32_t* slot_count; // contributors per slot over the whole step; nullptr: accumulate everywhere
  float* g_rows;
  float *g_first, *g_second;
};

// one list for all queries (or one query list for all entity rows)
bool shared_covers(const Shape& s);
int shared_forward(int term, const Shape& s, const ForwardArgs& a, cudaStream_t st);
int shared_backward(int term, const Shape& s, const BackwardArgs& a, cudaStream_t st);

// anything
int cell_forward(int term, const Shape& s, const ForwardArgs& a, cudaStream_t st);
int cell_backward(int term, const Shape& s, const BackwardArgs& a, cudaStream_t st);

}  // namespace smore

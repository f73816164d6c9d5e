// Negative sampling on the GPU: the step before the row gathers.
//
// The reference's online sampler draws, for every query, `negative_sample_size` entity ids that are
// not answers of the query - uniformly, or with degree-proportional weights through an alias table
// (smore/cpp_sampler/src/lib/naive_sampler.cpp:28-50, alias_method.cpp:33-99, sampler.cpp:90-99 for
// one shared list per batch) - on host threads, with a std::mt19937 per thread seeded from the clock
// (utils.cpp:33-39), so its draws are not reproducible.  Here one thread draws one id with a
// counter-based generator (Philox 4x32-10 keyed by a seed, counted by step and position): the same
// (seed, offset) gives the same ids on every run and any number of GPUs can draw disjoint streams.
// The alias table is built on the host by the reference's procedure (two first-in-first-out work
// lists), so the tables - and with them the distribution - are identical to the reference's.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <deque>
#include <vector>

#include "common.cuh"

namespace smore {

struct Philox {
  uint32_t c[4];
};

__device__ __forceinline__ Philox philox4x32_10(uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1, uint32_t c2,
                                                uint32_t c3) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t m0 = (uint64_t)M0 * c0, m1 = (uint64_t)M1 * c2;     // one multiplication for both halves
    const uint32_t n0 = (uint32_t)(m1 >> 32) ^ c1 ^ k0, n1 = (uint32_t)m1, n2 = (uint32_t)(m0 >> 32) ^ c3 ^ k1,
                   n3 = (uint32_t)m0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += W0;
    k1 += W1;
  }
  return Philox{{c0, c1, c2, c3}};
}

// 53 random bits -> [0, 1)
__device__ __forceinline__ double unit_double(uint32_t hi, uint32_t lo) {
  const unsigned long long x = (((unsigned long long)hi << 32) | lo) >> 11;
  return (double)x * (1.0 / 9007199254740992.0);
}

// One slot of an alias table whose ids fit 32 bits: one 16-byte read per draw instead of two dependent 8-byte
// reads from three arrays.
struct __align__(16) AliasEntry {
  double prob_small;
  uint32_t small, large;
};

struct SampleArgs {
  unsigned long long seed, offset;
  unsigned long long n_entities;
  const double* prob_small;      // kArrays
  const int64_t* choice_small;
  const int64_t* choice_large;
  const AliasEntry* entries;     // kEntries
  const int64_t* answer_ptr;     // nullable pair: nothing is rejected
  const int64_t* answer_ids;     // per query ascending
  size_t n_queries, k;
};

constexpr int kMaxDraws = 64;      // redraws of one position before the last draw is kept
constexpr int kSampleThreads = 256;
constexpr int kStagedAnswers = 2048;
enum AliasKind { kUniform, kArrays, kEntries };

template <int KIND>
__device__ __forceinline__ long long draw_id(const SampleArgs& a, unsigned long long ctr, int attempt) {
  const Philox r = philox4x32_10((uint32_t)a.seed, (uint32_t)(a.seed >> 32), (uint32_t)ctr, (uint32_t)(ctr >> 32),
                                 (uint32_t)attempt, 0x534d4f52u);
  // alias_method.cpp:41-52: slot = floor(n * u1), then the small or the large choice of the slot
  unsigned long long slot = (unsigned long long)((double)a.n_entities * unit_double(r.c[0], r.c[1]));
  if (slot >= a.n_entities) slot = a.n_entities - 1;
  if (KIND == kArrays)
    return unit_double(r.c[2], r.c[3]) < a.prob_small[slot] ? a.choice_small[slot] : a.choice_large[slot];
  if (KIND == kEntries) {
    const int4 raw = __ldg(reinterpret_cast<const int4*>(a.entries + slot));
    return (uint32_t)(unit_double(r.c[2], r.c[3]) < __hiloint2double(raw.y, raw.x) ? raw.z : raw.w);
  }
  return (long long)slot;
}

// naive_sampler.cpp:40-46: an id that is one of the query's answers is drawn again
__device__ __forceinline__ bool is_answer(const int64_t* ans, int n, long long id) {
  int at = 0;
  for (int step = n > 0 ? 1 << (31 - __clz(n)) : 0; step > 0; step >>= 1)
    if (step <= n - at && ans[at + step - 1] < id) at += step;
  return at < n && ans[at] == id;
}

// A draw is a serial chain: the query's answers, the generator, the table, the search.  A CTA takes P * 256
// consecutive positions: the answers of the queries among them are brought to shared memory once, and a
// thread's P draws have their table reads and searches in flight together.
// (1024 x 1024 draws by in-degree over 2.5M ids, 30 answers per query, with one position at a time per thread,
// three table arrays and the search in global memory -> like this: 15.1 -> 13.4 us with the tables in L2,
// 24.3 -> 21.4 us without; P = 1 and 2 take 23.3 and 23.1 us.)
template <int KIND, int P>
__global__ void __launch_bounds__(kSampleThreads) sample_negatives_kernel(SampleArgs a, int64_t* __restrict__ out) {
  __shared__ int64_t staged[kStagedAnswers];
  const size_t total = a.n_queries * a.k, first = (size_t)blockIdx.x * (kSampleThreads * P);
  const size_t n_here = min((size_t)(kSampleThreads * P), total - first);
  // queries of the CTA's positions: q0 holds the first one, at offset `rel0` of its list
  const size_t q0 = first / a.k, rel0 = first - q0 * a.k;
  auto query_of = [&](int i) -> size_t {
    const size_t rel = rel0 + i;
    if (rel < a.k) return q0;
    if (rel - a.k < a.k) return q0 + 1;
    return q0 + (uint32_t)rel / (uint32_t)a.k;     // several queries: k and rel are below 2 * 256 * P
  };
  long long id[P];
#pragma unroll
  for (int u = 0; u < P; ++u) {      // (their table reads are in flight while the answers are brought in)
    const int i = threadIdx.x + u * kSampleThreads;
    id[u] = (size_t)i < n_here ? draw_id<KIND>(a, a.offset + first + i, 0) : 0;
  }
  const int64_t* ans[P] = {};
  int n_ans[P] = {};
  if (a.answer_ptr != nullptr) {
    const int64_t begin = a.answer_ptr[q0], end = a.answer_ptr[query_of((int)n_here - 1) + 1];
    const bool fits = end - begin <= kStagedAnswers;
    if (fits) {
      for (int i = threadIdx.x; i < (int)(end - begin); i += kSampleThreads) staged[i] = a.answer_ids[begin + i];
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const int i = threadIdx.x + u * kSampleThreads;
      if ((size_t)i >= n_here) continue;
      const size_t q = query_of(i);
      const int64_t from = a.answer_ptr[q];
      ans[u] = fits ? staged + (from - begin) : a.answer_ids + from;
      n_ans[u] = (int)(a.answer_ptr[q + 1] - from);
    }
  }
  // lower bounds of the P ids, step by step together
  int at[P] = {}, longest = 0;
#pragma unroll
  for (int u = 0; u < P; ++u) longest = max(longest, n_ans[u]);
  for (int step = longest > 0 ? 1 << (31 - __clz(longest)) : 0; step > 0; step >>= 1) {
#pragma unroll
    for (int u = 0; u < P; ++u)
      if (step <= n_ans[u] - at[u] && ans[u][at[u] + step - 1] < id[u]) at[u] += step;
  }
#pragma unroll
  for (int u = 0; u < P; ++u) {
    const int i = threadIdx.x + u * kSampleThreads;
    if ((size_t)i >= n_here) continue;
    if (at[u] < n_ans[u] && ans[u][at[u]] == id[u]) {
      for (int attempt = 1; attempt < kMaxDraws; ++attempt) {
        id[u] = draw_id<KIND>(a, a.offset + first + i, attempt);
        if (!is_answer(ans[u], n_ans[u], id[u])) break;
      }
    }
    out[first + i] = id[u];
  }
}

// shared negatives: is_negative[b, j] = 0 where negatives[j] is an answer of query b (naive_sampler.cpp:33-38)
__global__ void __launch_bounds__(256)
    negative_mask_kernel(const int64_t* __restrict__ negatives, size_t k, const int64_t* __restrict__ answer_ptr,
                         const int64_t* __restrict__ answer_ids, size_t n_queries, float* __restrict__ is_negative) {
  const size_t total = n_queries * k;
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < total; p += (size_t)gridDim.x * blockDim.x) {
    const size_t b = p / k, j = p - b * k;
    const int64_t* ans = answer_ids + answer_ptr[b];
    const long long n_ans = answer_ptr[b + 1] - answer_ptr[b];
    const long long id = negatives[j];
    long long lo = 0, hi = n_ans;
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (ans[mid] < id) lo = mid + 1; else hi = mid;
    }
    is_negative[p] = (lo < n_ans && ans[lo] == id) ? 0.f : 1.f;
  }
}

template <int KIND>
static int launch_sample(const SampleArgs& a, int64_t* negatives, cudaStream_t st) {
  // Positions per thread: as many as leave every SM its eight CTAs.
  const size_t total = a.n_queries * a.k, threads = (size_t)sm_count() * 2048;
  const int per = total > 2 * threads ? 4 : total > threads ? 2 : 1;
  const size_t ctas = (total + (size_t)kSampleThreads * per - 1) / ((size_t)kSampleThreads * per);
  if (ctas > (size_t)INT_MAX) return fail(SMORE_ERR_TOO_LARGE, "sample_negatives: too many draws in one call");
  auto kern = per == 4 ? sample_negatives_kernel<KIND, 4> : per == 2 ? sample_negatives_kernel<KIND, 2> : sample_negatives_kernel<KIND, 1>;
  kern<<<(unsigned)ctas, kSampleThreads, 0, st>>>(a, negatives);
  return check_launch("sample_negatives_kernel");
}

static int sampler_grid(size_t items) {
  return (int)std::max<size_t>(1, std::min<size_t>((items + 255) / 256, (size_t)sm_count() * 16));
}

}  // namespace smore

using namespace smore;

extern "C" {

int smore_alias_build(const double* weights, size_t n, double* prob_small, int64_t* choice_small,
                      int64_t* choice_large) {
  if (!weights || !prob_small || !choice_small || !choice_large) return fail(SMORE_ERR_NULL, "alias_build: NULL pointer");
  if (n == 0) return fail(SMORE_ERR_BAD_SHAPE, "alias_build: no choices");
  double total = 0.0;
  for (size_t i = 0; i < n; ++i) total += weights[i];
  if (!(total > 0.0)) return fail(SMORE_ERR_BAD_SHAPE, "alias_build: weights must sum to a positive value");
  // alias_method.cpp:55-99: scaled probabilities; two first-in-first-out lists of the entries above
  // and below one; slot i pairs the oldest large entry with the oldest small one
  const double factor = (double)n / total;
  std::vector<double> probs(n);
  std::deque<size_t> large, small;
  for (size_t i = 0; i < n; ++i) {
    probs[i] = weights[i] * factor;
    (probs[i] >= 1.0 ? large : small).push_back(i);
  }
  for (size_t i = 0; i < n; ++i) {
    if (large.empty()) {
      const size_t s = small.front();     // (the reference does not pop here either)
      prob_small[i] = 1.0;
      choice_small[i] = choice_large[i] = (int64_t)s;
      continue;
    }
    const size_t l = large.front();
    large.pop_front();
    size_t s = 0;
    double ps = 0.0;
    if (!small.empty()) {
      s = small.front();
      small.pop_front();
      ps = probs[s];
    }
    probs[l] -= 1.0 - ps;
    prob_small[i] = ps;
    choice_small[i] = (int64_t)s;
    choice_large[i] = (int64_t)l;
    (probs[l] < 1.0 ? small : large).push_back(l);
  }
  return SMORE_OK;
}

int smore_sample_negatives(uint64_t seed, uint64_t offset, size_t n_entities, const double* prob_small,
                           const int64_t* choice_small, const int64_t* choice_large, const int64_t* answer_ptr,
                           const int64_t* answer_ids, size_t n_queries, size_t k, int64_t* negatives, void* stream) {
  if (n_queries == 0 || k == 0) return SMORE_OK;
  if (!negatives) return fail(SMORE_ERR_NULL, "sample_negatives: NULL pointer");
  if (n_entities == 0) return fail(SMORE_ERR_BAD_SHAPE, "sample_negatives: no entities");
  const int tables = (prob_small != nullptr) + (choice_small != nullptr) + (choice_large != nullptr);
  if (tables != 0 && tables != 3) return fail(SMORE_ERR_NULL, "sample_negatives: give all three alias tables or none");
  if ((answer_ptr != nullptr) != (answer_ids != nullptr))
    return fail(SMORE_ERR_NULL, "sample_negatives: give answer_ptr and answer_ids together");
  const SampleArgs a{seed, offset, n_entities, prob_small, choice_small, choice_large, nullptr, answer_ptr, answer_ids,
                     n_queries, k};
  return tables ? launch_sample<kArrays>(a, negatives, (cudaStream_t)stream)
                : launch_sample<kUniform>(a, negatives, (cudaStream_t)stream);
}

int smore_sample_negatives_packed(uint64_t seed, uint64_t offset, size_t n_entities, const void* entries,
                                  const int64_t* answer_ptr, const int64_t* answer_ids, size_t n_queries, size_t k,
                                  int64_t* negatives, void* stream) {
  if (n_queries == 0 || k == 0) return SMORE_OK;
  if (!negatives || !entries) return fail(SMORE_ERR_NULL, "sample_negatives: NULL pointer");
  if (n_entities == 0 || n_entities > (size_t)UINT32_MAX) return fail(SMORE_ERR_BAD_SHAPE, "sample_negatives: 1 to 2^32 - 1 entities");
  if (!aligned16(entries)) return fail(SMORE_ERR_BAD_SHAPE, "sample_negatives: entries must be 16-byte aligned");
  if ((answer_ptr != nullptr) != (answer_ids != nullptr))
    return fail(SMORE_ERR_NULL, "sample_negatives: give answer_ptr and answer_ids together");
  const SampleArgs a{seed, offset, n_entities, nullptr, nullptr, nullptr, static_cast<const AliasEntry*>(entries), answer_ptr,
                     answer_ids, n_queries, k};
  return launch_sample<kEntries>(a, negatives, (cudaStream_t)stream);
}

int smore_negative_mask(const int64_t* negatives, size_t k, const int64_t* answer_ptr, const int64_t* answer_ids,
                        size_t n_queries, float* is_negative, void* stream) {
  if (n_queries == 0 || k == 0) return SMORE_OK;
  if (!negatives || !answer_ptr || !answer_ids || !is_negative) return fail(SMORE_ERR_NULL, "negative_mask: NULL pointer");
  negative_mask_kernel<<<sampler_grid(n_queries * k), 256, 0, (cudaStream_t)stream>>>(negatives, k, answer_ptr, answer_ids,
                                                                                     n_queries, is_negative);
  return check_launch("negative_mask_kernel");
}

}  // extern "C"

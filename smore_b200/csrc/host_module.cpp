// The host side of a training step in native code: lookups, the step's de-duplication plan, the
// distance ops and path projections with their backward passes, and the optimizer step.
//
// What it replaces: the same steps written as Python autograd functions over ctypes.  A step of a small
// model is bound by that host work, not by its kernels: GQE on FB15k-237 (512 x 128 rows of 64 floats)
// spent 650 us per step issuing 87 us of kernels.  Here an op is one call that allocates, launches and
// links one autograd node, and the backward pass runs on the engine's thread without the interpreter.
//
// The classes are what smore_b200.embedding's optimizers keep their step in:
//   Lookup     one lookup of the step (row ids on the device, where they sit in the plan)
//   StepPlan   the de-duplicated rows of the step's lookups and their gradient buffer
//   RowCore    one table: pending lookups, plans, optimizer hyper-state
// Nothing here synchronises with the device.  Kernels are called through the C ABI of smore_b200.h.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <memory>
#include <optional>
#include <string>
#include <vector>

#include "smore_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

constexpr int kBoxBoth = 7;
constexpr double kBeta1 = 0.9, kBeta2 = 0.999, kEps = 1e-8;

// becomes smore_b200._lib.SmoreError in Python
struct SmoreFailure : std::runtime_error {
  using std::runtime_error::runtime_error;
};

void check(int rc, const char* what) {
  if (rc != SMORE_OK)
    throw SmoreFailure(std::string(what) + " failed (" + std::to_string(rc) + "): " + smore_last_error());
}

void* stream_of(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

const float* fptr(const Tensor& t) { return t.defined() ? (const float*)t.data_ptr() : nullptr; }
float* fmut(const Tensor& t) { return t.defined() ? (float*)t.data_ptr() : nullptr; }

int row_parts(int id) { return id == SMORE_DIST_ROTATE || id == SMORE_DIST_COMPLEX ? 2 : 1; }
bool two_operands(int id) {
  return id == SMORE_DIST_BOX_OUT || id == SMORE_DIST_BOX_IN || id == SMORE_DIST_ROTATE || id == SMORE_DIST_COMPLEX ||
         id == kBoxBoth;
}

// ---- optional per-call timing (benchmarks): smore_b200._lib's timer, when one is installed ----------
PyObject* g_timer = nullptr;   // borrowed from _lib while installed

class Timed {
 public:
  explicit Timed(const char* name) {
    if (g_timer == nullptr) return;
    py::gil_scoped_acquire gil;
    range_ = py::reinterpret_borrow<py::object>(g_timer).attr("range")(name).release().ptr();
    py::reinterpret_borrow<py::object>(range_).attr("__enter__")();
  }
  ~Timed() {
    if (range_ == nullptr) return;
    py::gil_scoped_acquire gil;
    py::object r = py::reinterpret_steal<py::object>(range_);
    r.attr("__exit__")(py::none(), py::none(), py::none());
  }

 private:
  PyObject* range_ = nullptr;
};

// ---- the step's state --------------------------------------------------------------------------------
struct StepPlan;

struct Lookup {
  Tensor idx;                       // int64 [n] on the table's device
  int64_t n = 0, order = 0, offset = 0;
  std::string name;
  std::weak_ptr<StepPlan> plan;
  bool received = false;            // a gradient producer has run for this lookup
  int n_consumers = 0;              // ops that took this lookup's rows in the forward pass
};

struct StepPlan {
  std::vector<std::shared_ptr<Lookup>> lookups;
  int64_t n = 0;
  Tensor uniq, slot, counts, n_unique, g_rows;

  const int32_t* slot_of(const Lookup& lk) const { return (const int32_t*)slot.data_ptr() + lk.offset; }
  const int32_t* counts_ptr() const { return (const int32_t*)counts.data_ptr(); }
};

struct RowCore {
  Tensor table, dummy;
  int opt = 0;
  bool squeeze = false, may_fuse = false;   // may_fuse: updates inside the backward pass are possible
  int64_t step = 0, n_fwd = 0;
  std::vector<std::shared_ptr<Lookup>> pending;   // registered since the last plan was built
  std::vector<std::shared_ptr<StepPlan>> plans;   // of this step (normally one)
  std::optional<double> fused_lr;                 // set by announce: rows may be updated in the backward pass
  Tensor m, v;                                    // optimizer state for the announced update
  Tensor step_dev, step_scalars;                  // step counter on the device (captured steps)
  bool step_advanced = false;
  Tensor workspace;

  int64_t rows() const { return table.size(0); }
  int64_t width() const { return table.size(1); }

  void drop_plans() {
    plans.clear();
  }

  void zero_grad() {
    n_fwd = 0;
    pending.clear();
    drop_plans();
    fused_lr.reset();
    m = Tensor();
    v = Tensor();
    step_advanced = false;
  }

  void advance_device_step(double lr) {
    c10::cuda::CUDAGuard guard(table.device());
    check(smore_adam_step_scalars((int64_t*)step_dev.data_ptr(), lr, kBeta1, kBeta2, fmut(step_scalars), stream_of(table)),
          "smore_adam_step_scalars");
  }

  std::shared_ptr<Lookup> lookup(const Tensor& indices, const std::optional<std::string>& name) {
    auto lk = std::make_shared<Lookup>();
    Tensor idx = indices;
    if (idx.dim() != 1) idx = idx.reshape({-1});
    if (idx.scalar_type() != at::kLong) idx = idx.to(at::kLong);
    if (idx.device() != table.device()) idx = idx.to(table.device(), /*non_blocking=*/true);
    lk->idx = idx.contiguous();
    lk->n = lk->idx.numel();
    if (name) lk->name = *name;
    lk->order = n_fwd++;
    pending.push_back(lk);
    return lk;
  }

  std::shared_ptr<StepPlan> build_plan(std::vector<std::shared_ptr<Lookup>> lookups) {
    auto p = std::make_shared<StepPlan>();
    std::vector<const int64_t*> ids;
    std::vector<size_t> sizes;
    std::vector<Tensor> tensors;
    for (auto& lk : lookups) {
      lk->offset = p->n;
      lk->plan = p;
      p->n += lk->n;
      ids.push_back((const int64_t*)lk->idx.data_ptr());
      sizes.push_back((size_t)lk->n);
      tensors.push_back(lk->idx);
    }
    p->lookups = std::move(lookups);
    c10::cuda::CUDAGuard guard(table.device());
    at::AutoDispatchBelowADInplaceOrView below;
    Tensor all;
    if (ids.size() > 8) {       // more lists than one call takes
      all = at::cat(tensors);
      ids = {(const int64_t*)all.data_ptr()};
      sizes = {(size_t)p->n};
    }
    const auto i64 = table.options().dtype(at::kLong), i32 = table.options().dtype(at::kInt);
    p->uniq = at::empty({p->n}, i64);
    p->slot = at::empty({p->n}, i32);
    p->counts = at::empty({p->n}, i32);
    p->n_unique = at::empty({2}, i32);
    p->g_rows = at::empty({p->n, width()}, table.options());
    if (!workspace.defined())
      workspace = at::empty({(int64_t)smore_unique_rows_workspace_bytes((size_t)rows())}, table.options().dtype(at::kByte));
    Timed timed("unique_rows");
    check(smore_step_rows(ids.data(), sizes.data(), ids.size(), (size_t)rows(), (int64_t*)p->uniq.data_ptr(),
                          (int32_t*)p->slot.data_ptr(), (int32_t*)p->counts.data_ptr(), (int32_t*)p->n_unique.data_ptr(),
                          fmut(p->g_rows), (size_t)width(), workspace.data_ptr(), (size_t)workspace.numel(), stream_of(table)),
          "smore_step_rows");
    return p;
  }

  // the plan that covers `lk`, built on first use from every lookup made so far
  std::shared_ptr<StepPlan> plan_for(const std::shared_ptr<Lookup>& lk) {
    if (auto p = lk->plan.lock()) return p;
    auto p = build_plan(std::move(pending));
    pending.clear();
    plans.push_back(p);
    if (lk->plan.lock() != p)
      throw SmoreFailure("a lookup of an earlier step was used after zero_grad() or apply_grad()");
    return p;
  }

  bool fuses(const Lookup& lk, const std::shared_ptr<StepPlan>& p) const {
    return fused_lr.has_value() && may_fuse && m.defined() && v.defined() && lk.n_consumers == 1 && !lk.received &&
           plans.size() == 1 && p == plans[0];
  }

  void update(const Tensor& uniq, const Tensor& g_rows, const Tensor& n_unique, int64_t capacity, double lr, const Tensor& m_,
              const Tensor& v_) {
    c10::cuda::CUDAGuard guard(table.device());
    Timed timed("sparse_update_rows");
    if (step_dev.defined()) {
      check(smore_sparse_update_rows_dev(opt, fmut(table), fmut(m_), fmut(v_), (const int64_t*)uniq.data_ptr(), fptr(g_rows),
                                         (const int32_t*)n_unique.data_ptr(), (size_t)capacity, (size_t)width(), lr, kBeta1,
                                         kBeta2, kEps, fptr(step_scalars), squeeze, stream_of(table)),
            "smore_sparse_update_rows_dev");
      return;
    }
    check(smore_sparse_update_rows(opt, fmut(table), fmut(m_), fmut(v_), (const int64_t*)uniq.data_ptr(), fptr(g_rows),
                                   (const int32_t*)n_unique.data_ptr(), (size_t)capacity, (size_t)width(), lr, kBeta1, kBeta2,
                                   kEps, step, squeeze, stream_of(table)),
          "smore_sparse_update_rows");
  }

  // The whole of apply_grad when one plan covers the step and every lookup of it got a gradient; false
  // leaves the step to the caller (several plans, or lookups without a gradient).
  bool apply_single_plan(double lr, const Tensor& m_, const Tensor& v_) {
    if (plans.size() != 1) return false;
    auto& p = plans[0];
    for (auto& lk : p->lookups)
      if (!lk->received) return false;
    if (step_dev.defined() && !step_advanced) advance_device_step(lr);
    update(p->uniq, p->g_rows, p->n_unique, p->n, lr, m_, v_);
    drop_plans();
    pending.clear();
    return true;
  }
};

// ---- shapes -----------------------------------------------------------------------------------------
struct QueryView {
  bool covered = false, both_branches = false;   // both_branches: the two-branch union kernels
  int64_t bc = 0, nc = 0, dim = 0;
  std::vector<int64_t> out;
};

// How a query operand ([bc, nc, dim], or [B, U, 1, dim] with U union branches) meets the entity operand
// [be, ne, *] in ONE call.  A union against one shared list is B * U queries; a union against one row per
// query is U columns; two branches against per-query lists have kernels of their own (`union_kernels`:
// table rows only).  Anything else: not covered, the caller runs branch by branch.
QueryView view_query(int64_t be, int64_t ne, const Tensor& q, bool union_kernels) {
  QueryView v;
  v.dim = q.size(-1);
  if (q.dim() == 3) {
    v.covered = true;
    v.bc = q.size(0);
    v.nc = q.size(1);
    v.out = {std::max(be, v.bc), std::max(ne, v.nc)};
    return v;
  }
  if (q.dim() != 4 || q.size(2) != 1) return v;
  const int64_t B = q.size(0), U = q.size(1);
  if (U == 1) {
    v.bc = B;
    v.nc = 1;
    v.out = {std::max(be, B), 1, ne};
  } else if (be == 1) {
    v.bc = B * U;
    v.nc = 1;
    v.out = {B, U, ne};
  } else if (ne == 1 && be == B) {
    v.bc = B;
    v.nc = U;
    v.out = {B, U, 1};
  } else if (union_kernels) {
    v.both_branches = true;
    v.bc = B;
    v.nc = 1;
    v.out = {B, U, ne};
  } else {
    return v;
  }
  v.covered = true;
  return v;
}

void check_broadcast(int64_t be, int64_t ne, int64_t bc, int64_t nc) {
  for (auto [a, b] : {std::pair<int64_t, int64_t>{be, bc}, {ne, nc}})
    if (a < 1 || b < 1 || (a % b != 0 && b % a != 0))
      throw py::value_error("entity (" + std::to_string(be) + ", " + std::to_string(ne) + ") and query (" + std::to_string(bc) +
                            ", " + std::to_string(nc) + ") do not broadcast");
}

bool needs_graph(std::initializer_list<const Tensor*> inputs) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : inputs)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// The nodes here have no forward-mode rule: refuse instead of dropping the tangent.
void no_tangents(std::initializer_list<const Tensor*> inputs) {
  for (const Tensor* t : inputs)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(/*level=*/0).defined(),
                                "forward-mode automatic differentiation is not supported by this op");
}

template <class N>
void link(const std::shared_ptr<N>& node, std::initializer_list<const Tensor*> inputs, std::initializer_list<Tensor*> outputs) {
  torch::autograd::edge_list edges;
  for (const Tensor* t : inputs)
    edges.push_back(t->defined() ? torch::autograd::impl::gradient_edge(*t) : torch::autograd::Edge());
  node->set_next_edges(std::move(edges));
  for (Tensor* t : outputs)
    if (t->defined()) torch::autograd::set_history(*t, node);
}

Tensor grad_or_zeros(const Tensor& g, at::IntArrayRef shape, const at::TensorOptions& options) {
  return g.defined() ? g.contiguous() : at::zeros(shape, options);
}

// Scratch of one call: from the caching allocator, in stream order.
Tensor scratch(const Tensor& like, size_t bytes) {
  return at::empty({(int64_t)std::max<size_t>(bytes, 256)}, like.options().dtype(at::kByte));
}

// ---- distances on table rows ------------------------------------------------------------------------
PyObject* g_fused_hook = nullptr;   // smore_b200.ext_ops, whose _fused_backward launches the update inside the backward pass

// What _fused_backward gets: everything of one backward pass with the Adam step folded in.
struct FusedLaunch {
  std::shared_ptr<RowCore> core;
  std::shared_ptr<StepPlan> plan;
  std::shared_ptr<Lookup> lk;
  int dist_id;
  Tensor first, second, g0, g1, g_first, g_second;
  int64_t branches, bsize, num, dim;

  bool run() {
    const bool dev = core->step_dev.defined();
    auto fused = core->squeeze ? smore_rows_backward_fused_adam : smore_rows_backward_fused_adam_full;
    const int rc = fused(
        dist_id, fptr(g0), fptr(g1), fmut(core->table), (const int64_t*)lk->idx.data_ptr(), (size_t)core->rows(), fptr(first),
        fptr(second), plan->slot_of(*lk), plan->counts_ptr(), fmut(plan->g_rows), fmut(g_first), fmut(g_second),
        (size_t)branches, (size_t)bsize, (size_t)num, (size_t)dim, fmut(core->m), fmut(core->v),
        (int64_t*)plan->uniq.data_ptr(), *core->fused_lr, kBeta1, kBeta2, kEps, dev ? 1 : core->step + 1,
        dev ? fptr(core->step_scalars) : nullptr, stream_of(core->table));
    if (rc == SMORE_ERR_BAD_SHAPE) return false;   // not covered: nothing was enqueued
    check(rc, "smore_rows_backward_fused_adam");
    return true;
  }
};

struct RowsDistNode : public Node {
  std::shared_ptr<RowCore> core;
  std::shared_ptr<Lookup> lk;
  SavedVariable first, second;
  int dist_id = 0;
  bool both_branches = false;
  int64_t be = 0, ne = 0, bc = 0, nc = 0, dim = 0;
  std::vector<int64_t> out;

  std::string name() const override { return "SmoreRowsDistBackward"; }
  void release_variables() override {
    first.reset_data();
    second.reset_data();
  }

  variable_list apply(variable_list&& grads) override {
    const Tensor q0 = first.unpack(), q1 = two_operands(dist_id) ? second.unpack() : Tensor();
    c10::cuda::CUDAGuard guard(core->table.device());
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor g0 = grad_or_zeros(grads[0], out, core->table.options());
    const Tensor g1 = dist_id == kBoxBoth ? grad_or_zeros(grads[1], out, core->table.options()) : Tensor();
    auto plan = core->plan_for(lk);
    Tensor gq0 = at::empty_like(q0), gq1 = q1.defined() ? at::empty_like(q1) : Tensor();
    const int64_t bsize = std::max(be, bc), num = std::max(ne, nc);
    if (core->fuses(*lk, plan) && (both_branches || (be == bsize && ne == num && bc == bsize && nc == 1)) && num >= 16) {
      Timed timed(both_branches ? "rows_backward_union" : "rows_backward");
      auto launch = std::make_shared<FusedLaunch>(
          FusedLaunch{core, plan, lk, dist_id, q0, q1, g0, g1, gq0, gq1, both_branches ? 2 : 1, bsize, num, dim});
      bool ran;
      {
        py::gil_scoped_acquire gil;
        ran = py::reinterpret_borrow<py::object>(g_fused_hook).attr("_fused_backward")(launch).cast<bool>();
      }
      if (ran) {
        lk->received = true;
        return {Tensor(), gq0, gq1};
      }
    }
    // the first gradient producer of a lookup may store rows that nothing else touches; any later one
    // over the same positions (another union branch) has to add to what is there
    const int32_t* counts = lk->received ? nullptr : plan->counts_ptr();
    lk->received = true;
    void* st = stream_of(core->table);
    const int64_t* idx = (const int64_t*)lk->idx.data_ptr();
    const float* tab = fptr(core->table);
    if (both_branches) {
      Timed timed("rows_backward_union");
      check(smore_union_backward_rows(dist_id, fptr(g0), fptr(g1), tab, idx, core->rows(), fptr(q0), fptr(q1), plan->slot_of(*lk),
                                      counts, fmut(plan->g_rows), fmut(gq0), fmut(gq1), 2, bsize, num, dim, st),
            "smore_union_backward_rows");
      return {Tensor(), gq0, gq1};
    }
    Timed timed(num >= 16 ? "rows_backward" : "rows_backward_few");
    if (dist_id == kBoxBoth)
      check(smore_box_backward(fptr(g0), fptr(g1), tab, idx, core->rows(), fptr(q0), fptr(q1), nullptr, plan->slot_of(*lk), counts,
                               fmut(plan->g_rows), fmut(gq0), fmut(gq1), bsize, num, be, ne, bc, nc, dim, st),
            "smore_box_backward");
    else
      check(smore_dist_backward_rows(dist_id, fptr(g0), tab, idx, core->rows(), fptr(q0), fptr(q1), plan->slot_of(*lk), counts,
                                     fmut(plan->g_rows), fmut(gq0), fmut(gq1), bsize, num, be, ne, bc, nc, dim, st),
            "smore_dist_backward_rows");
    return {Tensor(), gq0, gq1};
  }
};

// Inner products against one shared list as tensor-core GEMMs, on gathered table rows (lk set) or on an
// entity tensor.  score[B, K] = query[B, W] . cand[K, W]^T
struct DotNode : public Node {
  std::shared_ptr<RowCore> core;     // table rows
  std::shared_ptr<Lookup> lk;
  SavedVariable cand, query;         // [K, W], [B, W]
  int precision = 0;
  bool two = false;
  std::vector<int64_t> entity_shape, first_shape;

  std::string name() const override { return "SmoreDotSharedBackward"; }
  void release_variables() override {
    cand.reset_data();
    query.reset_data();
  }

  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor()};
    const Tensor c = cand.unpack(shared_from_this()), q = query.unpack(shared_from_this());
    c10::cuda::CUDAGuard guard(c.device());
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor g = grads[0].contiguous();
    const int64_t K = c.size(0), W = c.size(1), B = q.size(0);
    Tensor gc = at::empty_like(c), gq = at::empty_like(q);
    Tensor ws = scratch(c, smore_dot_workspace_bytes(B, K, W, precision));
    {
      Timed timed("dot_backward");
      check(smore_dot_backward_shared(fptr(g), fptr(c), fptr(q), fmut(gc), fmut(gq), B, K, W, precision, ws.data_ptr(),
                                      ws.numel(), stream_of(c)),
            "smore_dot_backward_shared");
    }
    Tensor g_entity;
    if (core) {
      auto plan = core->plan_for(lk);
      const int32_t* counts = lk->received ? nullptr : plan->counts_ptr();
      lk->received = true;
      check(smore_scatter_add_rows(fptr(gc), plan->slot_of(*lk), counts, fmut(plan->g_rows), K, W, stream_of(c)),
            "smore_scatter_add_rows");
    } else {
      g_entity = gc.view(entity_shape);
    }
    if (!two) return {g_entity, gq.view(first_shape), Tensor()};
    std::vector<int64_t> both = first_shape;
    both.back() *= 2;
    const Tensor gv = gq.view(both);
    const int64_t dim = first_shape.back();
    return {g_entity, gv.narrow(-1, 0, dim), gv.narrow(-1, dim, dim)};
  }
};

bool dot_route(int dist_id, int dot_mode, int64_t be, int64_t K, int64_t W, const QueryView& qv, const Tensor& first) {
  if (dot_mode < 0 || (dist_id != SMORE_DIST_COMPLEX && dist_id != SMORE_DIST_DISTMULT)) return false;
  if (be != 1 || qv.nc != 1 || qv.both_branches || qv.bc < 128 || K < 128 || ((qv.bc | K | W) & 3)) return false;
  return first.is_cuda() && first.scalar_type() == at::kFloat && W == row_parts(dist_id) * qv.dim && smore_dot_available();
}

Tensor gather(const RowCore& core, const Tensor& idx) {
  Tensor out = at::empty({idx.numel(), core.width()}, core.table.options());
  check(smore_gather_rows(fptr(core.table), (const int64_t*)idx.data_ptr(), core.rows(), fmut(out), idx.numel(), core.width(),
                          stream_of(core.table)),
        "smore_gather_rows");
  return out;
}

Tensor dot_scores(const std::shared_ptr<RowCore>& core, const std::shared_ptr<Lookup>& lk, const Tensor& entity, const Tensor& first,
                  const Tensor& second, const QueryView& qv, int64_t K, int64_t W, int precision) {
  const Tensor& dev = core ? core->table : entity;
  no_tangents({&entity, &first, &second});
  if (core) lk->n_consumers += 1;
  c10::cuda::CUDAGuard guard(dev.device());
  Tensor cand, query, dst;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    cand = core ? gather(*core, lk->idx) : entity.contiguous().view({K, W});
    query = second.defined() ? at::cat({first, second}, -1).view({qv.bc, W}) : first.contiguous().view({qv.bc, W});
    dst = at::empty(qv.out, first.options());
    Tensor ws = scratch(cand, smore_dot_workspace_bytes(qv.bc, K, W, precision));
    Timed timed("dot_forward");
    check(smore_dot_forward_shared(fptr(cand), fptr(query), fmut(dst), qv.bc, K, W, precision, ws.data_ptr(), ws.numel(),
                                   stream_of(cand)),
          "smore_dot_forward_shared");
  }
  const Tensor& lead = core ? core->dummy : entity;
  if (needs_graph({&lead, &first, &second})) {
    auto node = std::make_shared<DotNode>();
    node->core = core;
    node->lk = lk;
    node->precision = precision;
    node->two = second.defined();
    if (!core) node->entity_shape = entity.sizes().vec();
    node->first_shape = first.sizes().vec();
    link(node, {&lead, &first, &second}, {&dst});
    node->cand = SavedVariable(cand, false);
    node->query = SavedVariable(query, false);
  }
  return dst;
}

// Scores of table rows named by a lookup, viewed as [be, ne, width].  Returns None when the query operand
// has to be taken branch by branch.
py::object rows_dist(const std::shared_ptr<RowCore>& core, const std::shared_ptr<Lookup>& lk, int dist_id, int64_t be, int64_t ne,
                     Tensor first, const std::optional<Tensor>& second_opt, bool union_kernels, int dot_mode) {
  Tensor second = second_opt ? *second_opt : Tensor();
  const Tensor& table = core->table;
  const QueryView qv = view_query(be, ne, first, union_kernels);
  if (!qv.covered) return py::none();
  if (dot_route(dist_id, dot_mode, be, ne, core->width(), qv, first))
    return py::cast(dot_scores(core, lk, Tensor(), first, second, qv, ne, core->width(), dot_mode));
  if (!first.is_cuda() || first.device() != table.device() || first.scalar_type() != at::kFloat)
    throw py::type_error("query operands must be float32 on the table's device");
  if (second.defined() && second.sizes() != first.sizes())
    throw py::value_error("the two query operands must have the same shape");
  if (core->width() != row_parts(dist_id) * qv.dim)
    throw py::value_error("table rows must be " + std::to_string(row_parts(dist_id)) + " x the query dim");
  check_broadcast(be, ne, qv.bc, qv.nc);
  no_tangents({&first, &second});
  lk->n_consumers += 1;
  const int64_t bsize = std::max(be, qv.bc), num = std::max(ne, qv.nc);
  const bool both = dist_id == kBoxBoth;
  c10::cuda::CUDAGuard guard(table.device());
  Tensor q0, q1, d0, d1;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    q0 = first.contiguous();
    q1 = second.defined() ? second.contiguous() : Tensor();
    d0 = at::empty(qv.out, table.options());
    if (both) d1 = at::empty(qv.out, table.options());
    void* st = stream_of(table);
    const int64_t* idx = (const int64_t*)lk->idx.data_ptr();
    Timed timed(qv.both_branches ? "rows_forward_union" : num >= 16 ? "rows_forward" : "rows_forward_few");
    if (qv.both_branches)
      check(smore_union_forward_rows(dist_id, fptr(table), idx, core->rows(), fptr(q0), fptr(q1), fmut(d0), fmut(d1), 2, bsize, num,
                                     qv.dim, st),
            "smore_union_forward_rows");
    else if (both)
      check(smore_box_forward(fptr(table), idx, core->rows(), fptr(q0), fptr(q1), fmut(d0), fmut(d1), bsize, num, be, ne, qv.bc,
                              qv.nc, qv.dim, st),
            "smore_box_forward");
    else
      check(smore_dist_forward_rows(dist_id, fptr(table), idx, core->rows(), fptr(q0), fptr(q1), fmut(d0), bsize, num, be, ne, qv.bc,
                                    qv.nc, qv.dim, st),
            "smore_dist_forward_rows");
  }
  if (needs_graph({&core->dummy, &first, &second})) {
    auto node = std::make_shared<RowsDistNode>();
    node->core = core;
    node->lk = lk;
    node->dist_id = dist_id;
    node->both_branches = qv.both_branches;
    node->be = be;
    node->ne = ne;
    node->bc = qv.bc;
    node->nc = qv.nc;
    node->dim = qv.dim;
    node->out = qv.out;
    link(node, {&core->dummy, &first, &second}, {&d0, &d1});
    node->first = SavedVariable(q0, false);
    if (q1.defined()) node->second = SavedVariable(q1, false);
  }
  if (both) return py::make_tuple(d0, d1);
  return py::cast(d0);
}

// ---- distances on tensors ---------------------------------------------------------------------------
struct DenseDistNode : public Node {
  SavedVariable entity, first, second;
  int dist_id = 0;
  int64_t be = 0, ne = 0, bc = 0, nc = 0, dim = 0;
  std::vector<int64_t> out;

  std::string name() const override { return "SmoreDistBackward"; }
  void release_variables() override {
    entity.reset_data();
    first.reset_data();
    second.reset_data();
  }

  variable_list apply(variable_list&& grads) override {
    const Tensor e = entity.unpack(), q0 = first.unpack(), q1 = two_operands(dist_id) ? second.unpack() : Tensor();
    c10::cuda::CUDAGuard guard(e.device());
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor g0 = grad_or_zeros(grads[0], out, e.options());
    // the kernels write every element, so the buffers need not be cleared first
    Tensor ge = at::empty_like(e), gq0 = at::empty_like(q0), gq1 = q1.defined() ? at::empty_like(q1) : Tensor();
    const int64_t bsize = std::max(be, bc), num = std::max(ne, nc);
    void* st = stream_of(e);
    if (dist_id == kBoxBoth) {
      const Tensor g1 = grad_or_zeros(grads[1], out, e.options());
      check(smore_box_backward(fptr(g0), fptr(g1), fptr(e), nullptr, 0, fptr(q0), fptr(q1), fmut(ge), nullptr, nullptr, nullptr,
                               fmut(gq0), fmut(gq1), bsize, num, be, ne, bc, nc, dim, st),
            "smore_box_backward");
    } else if (e.scalar_type() == at::kFloat) {
      check(smore_dist_backward(dist_id, fptr(g0), fptr(e), fptr(q0), fptr(q1), fmut(ge), fmut(gq0), fmut(gq1), bsize, num, be, ne,
                                bc, nc, dim, st),
            "smore_dist_backward");
    } else {
      auto d = [](const Tensor& t) { return t.defined() ? (double*)t.data_ptr() : nullptr; };
      check(smore_dist_backward_f64(dist_id, d(g0), d(e), d(q0), d(q1), d(ge), d(gq0), d(gq1), bsize, num, be, ne, bc, nc, dim, st),
            "smore_dist_backward_f64");
    }
    return {ge, gq0, gq1};
  }
};

// Distances of an entity tensor [be, ne, W].  None when the query operand has to be taken branch by branch.
py::object dense_dist(int dist_id, const Tensor& entity, const Tensor& first, const std::optional<Tensor>& second_opt, int dot_mode) {
  const Tensor second = second_opt ? *second_opt : Tensor();
  if (!entity.is_cuda()) throw SmoreFailure("operands must be CUDA tensors (there is no CPU path)");
  const bool both = dist_id == kBoxBoth;
  if (entity.scalar_type() != at::kFloat && (both || entity.scalar_type() != at::kDouble))
    throw py::type_error(both ? "float32 expected" : "float32 or float64 expected");
  for (const Tensor* t : {&first, &second})
    if (t->defined() && (t->device() != entity.device() || t->scalar_type() != entity.scalar_type()))
      throw py::type_error("all operands must share device and dtype");
  const int64_t be = entity.size(0), ne = entity.size(1), W = entity.size(2);
  const QueryView qv = view_query(be, ne, first, false);
  if (!qv.covered) return py::none();
  if (second.defined() && second.sizes() != first.sizes())
    throw py::value_error("the two query operands must have the same shape");
  if (dot_route(dist_id, dot_mode, be, ne, W, qv, first))
    return py::cast(dot_scores(nullptr, nullptr, entity, first, second, qv, ne, W, dot_mode));
  if (W != row_parts(dist_id) * qv.dim)
    throw py::value_error("entity rows must be " + std::to_string(row_parts(dist_id)) + " x the query dim");
  check_broadcast(be, ne, qv.bc, qv.nc);
  no_tangents({&entity, &first, &second});
  const int64_t bsize = std::max(be, qv.bc), num = std::max(ne, qv.nc);
  c10::cuda::CUDAGuard guard(entity.device());
  Tensor e, q0, q1, d0, d1;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    e = entity.contiguous();
    q0 = first.contiguous();
    q1 = second.defined() ? second.contiguous() : Tensor();
    d0 = at::empty(qv.out, entity.options());
    void* st = stream_of(entity);
    if (both) {
      d1 = at::empty(qv.out, entity.options());
      check(smore_box_forward(fptr(e), nullptr, 0, fptr(q0), fptr(q1), fmut(d0), fmut(d1), bsize, num, be, ne, qv.bc, qv.nc, qv.dim,
                              st),
            "smore_box_forward");
    } else if (e.scalar_type() == at::kFloat) {
      check(smore_dist_forward(dist_id, fptr(e), fptr(q0), fptr(q1), fmut(d0), bsize, num, be, ne, qv.bc, qv.nc, qv.dim, st),
            "smore_dist_forward");
    } else {
      auto d = [](const Tensor& t) { return t.defined() ? (double*)t.data_ptr() : nullptr; };
      check(smore_dist_forward_f64(dist_id, d(e), d(q0), d(q1), d(d0), bsize, num, be, ne, qv.bc, qv.nc, qv.dim, st),
            "smore_dist_forward_f64");
    }
  }
  if (needs_graph({&entity, &first, &second})) {
    auto node = std::make_shared<DenseDistNode>();
    node->dist_id = dist_id;
    node->be = be;
    node->ne = ne;
    node->bc = qv.bc;
    node->nc = qv.nc;
    node->dim = qv.dim;
    node->out = qv.out;
    link(node, {&entity, &first, &second}, {&d0, &d1});
    node->entity = SavedVariable(e, false);
    node->first = SavedVariable(q0, false);
    if (q1.defined()) node->second = SavedVariable(q1, false);
  }
  if (both) return py::make_tuple(d0, d1);
  return py::cast(d0);
}

// ---- lookups that are used as tensors ---------------------------------------------------------------
struct GatherNode : public Node {
  std::shared_ptr<RowCore> core;
  std::shared_ptr<Lookup> lk;

  std::string name() const override { return "SmoreLookupBackward"; }

  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor()};
    c10::cuda::CUDAGuard guard(core->table.device());
    at::AutoDispatchBelowADInplaceOrView below;
    accumulate(*core, lk, grads[0].contiguous());
    return {Tensor()};
  }

  static void accumulate(RowCore& core, const std::shared_ptr<Lookup>& lk, const Tensor& g) {
    auto plan = core.plan_for(lk);
    // a second producer for the same positions must add to what the first one stored
    const int32_t* counts = lk->received ? nullptr : plan->counts_ptr();
    lk->received = true;
    check(smore_scatter_add_rows(fptr(g), plan->slot_of(*lk), counts, fmut(plan->g_rows), lk->n, core.width(),
                                 stream_of(core.table)),
          "smore_scatter_add_rows");
  }
};

Tensor lookup_tensor(const std::shared_ptr<RowCore>& core, const std::shared_ptr<Lookup>& lk) {
  c10::cuda::CUDAGuard guard(core->table.device());
  lk->n_consumers += 1;
  Tensor out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = gather(*core, lk->idx);
  }
  if (needs_graph({&core->dummy})) {
    auto node = std::make_shared<GatherNode>();
    node->core = core;
    node->lk = lk;
    link(node, {&core->dummy}, {&out});
  }
  return out;
}

Tensor gather_rows(const std::shared_ptr<RowCore>& core, const Tensor& idx) {
  c10::cuda::CUDAGuard guard(core->table.device());
  at::AutoDispatchBelowADInplaceOrView below;
  return gather(*core, idx);
}

void accumulate_grad(const std::shared_ptr<RowCore>& core, const std::shared_ptr<Lookup>& lk, const Tensor& g) {
  c10::cuda::CUDAGuard guard(core->table.device());
  GatherNode::accumulate(*core, lk, g);
}

// ---- path projections -------------------------------------------------------------------------------
enum Geometry { kAdd = 0, kRotation = 1, kComplexProduct = 2, kProduct = 3 };

struct PathNode : public Node {
  std::shared_ptr<RowCore> core;     // the start is table rows
  std::shared_ptr<Lookup> lk;
  SavedVariable rel_ids, rel, off, start;
  int geometry = 0;
  bool relu_offset = false, has_off = false, has_start_offset = false, two = false;
  double phase_scale = 1.0;
  int64_t B = 0, H = 0, D = 0, W = 0;

  std::string name() const override { return "SmorePathBackward"; }
  void release_variables() override {
    rel_ids.reset_data();
    rel.reset_data();
    off.reset_data();
    start.reset_data();
  }

  // inputs: start (the table's dummy for table rows), start_offset, rel, off
  variable_list apply(variable_list&& grads) override {
    const Tensor ids = rel_ids.unpack(), r = rel.unpack(), o = has_off ? off.unpack() : Tensor();
    const Tensor s = core ? Tensor() : start.unpack();
    c10::cuda::CUDAGuard guard(r.device());
    at::AutoDispatchBelowADInplaceOrView below;
    if (!grads[0].defined() && (grads.size() < 2 || !grads[1].defined())) return {Tensor(), Tensor(), Tensor(), Tensor()};
    const Tensor g0 = grad_or_zeros(grads[0], {B, D}, r.options());
    const bool second_out = two || has_off;
    const Tensor g1 = second_out ? grad_or_zeros(grads[1], {B, D}, r.options()) : Tensor();
    Tensor g_rel = at::empty_like(r), g_off = has_off ? at::empty_like(o) : Tensor(), g_start;
    const float* rows = nullptr;
    const int64_t* row_ids = nullptr;
    const int32_t *slot = nullptr, *counts = nullptr;
    float* g_rows = nullptr;
    int64_t n_rows = 0;
    if (core) {
      auto plan = core->plan_for(lk);
      counts = lk->received ? nullptr : plan->counts_ptr();
      lk->received = true;
      slot = plan->slot_of(*lk);
      g_rows = fmut(plan->g_rows);
      rows = fptr(core->table);
      row_ids = (const int64_t*)lk->idx.data_ptr();
      n_rows = core->rows();
    } else {
      rows = fptr(s);
      if (geometry != kAdd) g_start = at::empty({B, W}, r.options());
    }
    {
      Timed timed("path_project_backward");
      check(smore_path_embed_backward(geometry, fptr(g0), fptr(g1), rows, row_ids, n_rows, fptr(r), fptr(o), r.size(0),
                                      (const int64_t*)ids.data_ptr(), ids.stride(0), B, H, D, relu_offset, phase_scale, fmut(g_rel),
                                      fmut(g_off), fmut(g_start), slot, counts, g_rows, stream_of(r)),
            "smore_path_embed_backward");
    }
    if (!core && geometry == kAdd) g_start = g0;
    return {g_start, has_start_offset ? g1 : Tensor(), g_rel, g_off};
  }
};

// All relation projections of a batch of path queries that start from rows of a table (core, lk) or from
// `start` [B, W].  Operands are checked by the caller (smore_b200.query_ops).
py::object path_embed(int geometry, const std::shared_ptr<RowCore>& core, const std::shared_ptr<Lookup>& lk,
                      const std::optional<Tensor>& start_opt, const std::optional<Tensor>& start_offset_opt, const Tensor& rel,
                      const std::optional<Tensor>& off_opt, const Tensor& rel_ids, bool relu_offset, double phase_scale) {
  const Tensor start = start_opt ? *start_opt : Tensor(), off = off_opt ? *off_opt : Tensor();
  const Tensor start_offset = start_offset_opt ? *start_offset_opt : Tensor();
  no_tangents({&start, &start_offset, &rel, &off});
  if (core) lk->n_consumers += 1;
  c10::cuda::CUDAGuard guard(rel.device());
  const bool two = geometry == kRotation || geometry == kComplexProduct;
  const bool has_off = geometry == kAdd && off.defined();
  Tensor s, so, out0, out1;
  int64_t B, W, D;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (!core) s = start.contiguous();
    so = start_offset.defined() ? start_offset.contiguous() : Tensor();
    B = core ? lk->n : s.size(0);
    W = core ? core->width() : s.size(1);
    D = two ? W / 2 : W;
    out0 = at::empty({B, D}, rel.options());
    if (two || has_off) out1 = at::empty({B, D}, rel.options());
    Timed timed("path_project");
    check(smore_path_embed_forward(geometry, core ? fptr(core->table) : fptr(s), core ? (const int64_t*)lk->idx.data_ptr() : nullptr,
                                   core ? core->rows() : 0, fptr(so), fptr(rel), fptr(off), rel.size(0),
                                   (const int64_t*)rel_ids.data_ptr(), rel_ids.stride(0), B, rel_ids.size(1), D, relu_offset,
                                   phase_scale, fmut(out0), fmut(out1), stream_of(rel)),
          "smore_path_embed_forward");
  }
  const Tensor& lead = core ? core->dummy : start;
  if (needs_graph({&lead, &start_offset, &rel, &off})) {
    auto node = std::make_shared<PathNode>();
    node->core = core;
    node->lk = lk;
    node->geometry = geometry;
    node->relu_offset = relu_offset;
    node->has_off = has_off;
    node->has_start_offset = geometry == kAdd && start_offset.defined();
    node->two = two;
    node->phase_scale = phase_scale;
    node->B = B;
    node->H = rel_ids.size(1);
    node->D = D;
    node->W = W;
    link(node, {&lead, &start_offset, &rel, &off}, {&out0, &out1});
    node->rel_ids = SavedVariable(rel_ids, false);
    node->rel = SavedVariable(rel, false);
    if (has_off) node->off = SavedVariable(off, false);
    if (!core) node->start = SavedVariable(s, false);
  }
  if (out1.defined()) return py::make_tuple(out0, out1);
  return py::cast(out0);
}

// ---- evaluation --------------------------------------------------------------------------------------
// Answer lists of a batch of queries (Python iterables of ids) packed into one pinned block and sent to the
// device with one copy: [answer_ptr (Q + 1) | hard_ptr (Q + 1) | ids].
struct Answers {
  std::vector<int64_t> hard_counts;
  int64_t Q = 0, n = 0, longest = 0, n_hard = 0;
  Tensor device;

  const int64_t* ptr() const { return (const int64_t*)device.data_ptr(); }
  const int64_t* hard_ptr() const { return ptr() + Q + 1; }
  const int64_t* ids() const { return ptr() + 2 * (Q + 1); }
};

py::object as_list(PyObject* iterable) {   // itself where it is a list or tuple
  py::object fast = py::reinterpret_steal<py::object>(PySequence_Fast(iterable, "answers must be iterables of candidate ids"));
  if (!fast) throw py::error_already_set();
  return fast;
}

void append_ids(PyObject* list, int64_t limit, std::vector<int64_t>& out) {
  const py::object fast = as_list(list);
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast.ptr());
  PyObject** items = PySequence_Fast_ITEMS(fast.ptr());
  for (Py_ssize_t i = 0; i < n; ++i) {
    int64_t v;
    if (PyLong_Check(items[i])) {
      v = PyLong_AsLongLong(items[i]);
    } else {
      if (PyUnicode_Check(items[i]) || PyBytes_Check(items[i])) throw py::type_error("answer ids must be numbers");
      py::object num = py::reinterpret_steal<py::object>(PyNumber_Long(items[i]));
      if (!num) throw py::error_already_set();
      v = PyLong_AsLongLong(num.ptr());
    }
    if (v == -1 && PyErr_Occurred()) throw py::error_already_set();
    if (v < 0 || v >= limit) throw py::value_error("answer ids must lie in [0, " + std::to_string(limit) + ")");
    out.push_back(v);
  }
}

Answers pack_answers(const py::object& easy_lists, const py::object& hard_lists, int64_t Q, int64_t n_candidates, const Tensor& like) {
  if ((int64_t)py::len(easy_lists) != Q || (int64_t)py::len(hard_lists) != Q)
    throw py::value_error("one easy and one hard answer list per query");
  const py::object easy = as_list(easy_lists.ptr()), hard = as_list(hard_lists.ptr());
  if (PySequence_Fast_GET_SIZE(easy.ptr()) != Q || PySequence_Fast_GET_SIZE(hard.ptr()) != Q)
    throw py::value_error("one easy and one hard answer list per query");
  Answers a;
  a.Q = Q;
  std::vector<int64_t> ids, ptr{0}, hard_ptr{0};
  for (int64_t q = 0; q < Q; ++q) {
    append_ids(PySequence_Fast_GET_ITEM(easy.ptr(), q), n_candidates, ids);
    const int64_t easy_end = (int64_t)ids.size();
    append_ids(PySequence_Fast_GET_ITEM(hard.ptr(), q), n_candidates, ids);
    a.hard_counts.push_back((int64_t)ids.size() - easy_end);
    a.longest = std::max(a.longest, (int64_t)ids.size() - ptr.back());
    ptr.push_back((int64_t)ids.size());
    hard_ptr.push_back(hard_ptr.back() + a.hard_counts.back());
  }
  a.n = (int64_t)ids.size();
  a.n_hard = hard_ptr.back();
  if (a.n == 0) return a;
  Tensor host = at::empty({2 * (Q + 1) + a.n}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
  int64_t* h = (int64_t*)host.data_ptr();
  h = std::copy(ptr.begin(), ptr.end(), h);
  h = std::copy(hard_ptr.begin(), hard_ptr.end(), h);
  std::copy(ids.begin(), ids.end(), h);
  a.device = host.to(like.device(), /*non_blocking=*/true);
  return a;
}

py::list split_ranks(const Tensor& ranks, const Answers& a) {
  py::list out;
  int64_t at = 0;
  for (int64_t n : a.hard_counts) {
    out.append(ranks.narrow(0, at, n));
    at += n;
  }
  return out;
}

py::list filtered_ranks(Tensor logits, const py::object& easy, const py::object& hard) {
  if (logits.dim() != 2 || logits.scalar_type() != at::kFloat || !logits.is_cuda())
    throw py::type_error("logits must be a 2-D float32 CUDA tensor");
  const int64_t Q = logits.size(0), N = logits.size(1);
  c10::cuda::CUDAGuard guard(logits.device());
  at::NoGradGuard no_grad;
  logits = logits.contiguous();
  const Answers a = pack_answers(easy, hard, Q, N, logits);
  Tensor ranks = at::empty({a.n_hard}, logits.options().dtype(at::kLong));
  if (a.n) {
    Tensor ws = scratch(logits, smore_filtered_ranks_workspace_bytes(a.n));
    Timed timed("filtered_ranks");
    check(smore_hard_ranks(fptr(logits), Q, N, a.ptr(), a.ids(), a.n, a.longest, a.hard_ptr(), (int64_t*)ranks.data_ptr(),
                           ws.data_ptr(), ws.numel(), stream_of(logits)),
          "smore_hard_ranks");
  }
  return split_ranks(ranks, a);
}

py::list score_and_rank(int dist_id, const Tensor& table, const Tensor& first, const std::optional<Tensor>& second_opt,
                        const py::object& easy, const py::object& hard, double gamma, double cen) {
  if (table.scalar_type() != at::kFloat || !table.is_cuda() || !table.is_contiguous())
    throw py::type_error("table must be a contiguous float32 CUDA tensor");
  c10::cuda::CUDAGuard guard(table.device());
  at::NoGradGuard no_grad;
  const int64_t Q = first.size(0), N = table.size(0);
  const Tensor q0 = first.reshape({Q, -1}).contiguous();
  const Tensor q1 = second_opt ? second_opt->reshape({Q, -1}).contiguous() : Tensor();
  const Answers a = pack_answers(easy, hard, Q, N, table);
  Tensor ranks = at::empty({a.n_hard}, table.options().dtype(at::kLong));
  if (a.n) {
    Tensor ws = scratch(table, smore_score_filtered_ranks_workspace_bytes(Q, a.n));
    Timed timed("score_filtered_ranks");
    check(smore_score_hard_ranks(dist_id, fptr(table), N, fptr(q0), fptr(q1), Q, q0.size(1), gamma, cen, a.ptr(), a.ids(), a.n,
                                 a.longest, a.hard_ptr(), (int64_t*)ranks.data_ptr(), ws.data_ptr(), ws.numel(),
                                 stream_of(table)),
          "smore_score_hard_ranks");
  }
  return split_ranks(ranks, a);
}

// ---- negative sampling -------------------------------------------------------------------------------
// Draws of smore_b200.sampler.NegativeSampler: `entries` the packed alias tables, or nothing for uniform draws.
Tensor sample_negatives(uint64_t seed, uint64_t offset, int64_t n_entities, const std::optional<Tensor>& entries,
                        const std::optional<Tensor>& answer_ptr, const std::optional<Tensor>& answer_ids, int64_t n_queries,
                        int64_t k, const at::Device& device) {
  c10::cuda::CUDAGuard guard(device);
  Tensor out = at::empty({n_queries, k}, at::TensorOptions().dtype(at::kLong).device(guard.current_device()));
  auto ids = [](const std::optional<Tensor>& t) { return t ? (const int64_t*)t->data_ptr() : nullptr; };
  if (entries)
    check(smore_sample_negatives_packed(seed, offset, n_entities, entries->data_ptr(), ids(answer_ptr), ids(answer_ids), n_queries,
                                        k, (int64_t*)out.data_ptr(), stream_of(out)),
          "smore_sample_negatives_packed");
  else
    check(smore_sample_negatives(seed, offset, n_entities, nullptr, nullptr, nullptr, ids(answer_ptr), ids(answer_ids), n_queries, k,
                                 (int64_t*)out.data_ptr(), stream_of(out)),
          "smore_sample_negatives");
  return out;
}

}  // namespace

PYBIND11_MODULE(_host, mod) {
  static PyObject* smore_error = nullptr;
  mod.def("bind", [](py::object error, py::object ops) {
    smore_error = error.release().ptr();        // both live as long as the process
    g_fused_hook = ops.release().ptr();
  });
  mod.def("set_timer", [](py::object timer) { g_timer = timer.is_none() ? nullptr : timer.ptr(); });
  py::register_local_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const SmoreFailure& e) {
      PyErr_SetString(smore_error ? smore_error : PyExc_RuntimeError, e.what());
    }
  });

  py::class_<Lookup, std::shared_ptr<Lookup>>(mod, "Lookup")
      .def_readonly("idx", &Lookup::idx)
      .def_readonly("n", &Lookup::n)
      .def_readonly("name", &Lookup::name)
      .def_readonly("order", &Lookup::order)
      .def_readonly("offset", &Lookup::offset)
      .def_readwrite("received", &Lookup::received)
      .def_readwrite("n_consumers", &Lookup::n_consumers)
      .def_property_readonly("plan", [](const Lookup& lk) { return lk.plan.lock(); });

  py::class_<StepPlan, std::shared_ptr<StepPlan>>(mod, "StepPlan")
      .def_readonly("lookups", &StepPlan::lookups)
      .def_readonly("n", &StepPlan::n)
      .def_readonly("uniq", &StepPlan::uniq)
      .def_readonly("slot", &StepPlan::slot)
      .def_readonly("counts", &StepPlan::counts)
      .def_readonly("n_unique", &StepPlan::n_unique)
      .def_readonly("g_rows", &StepPlan::g_rows)
      .def("slot_of", [](const StepPlan& p, const Lookup& lk) { return p.slot.narrow(0, lk.offset, lk.n); });

  py::class_<RowCore, std::shared_ptr<RowCore>>(mod, "RowCore")
      .def(py::init([](Tensor table, Tensor dummy, int opt, bool squeeze, bool may_fuse) {
        auto c = std::make_shared<RowCore>();
        c->table = std::move(table);
        c->dummy = std::move(dummy);
        c->opt = opt;
        c->squeeze = squeeze;
        c->may_fuse = may_fuse;
        return c;
      }))
      .def_readwrite("step", &RowCore::step)
      .def_readonly("n_fwd", &RowCore::n_fwd)
      .def_readonly("plans", &RowCore::plans)
      .def_readonly("pending", &RowCore::pending)
      .def_readonly("fused_lr", &RowCore::fused_lr)
      .def_readonly("step_advanced", &RowCore::step_advanced)
      .def_property_readonly("step_dev", [](const RowCore& c) -> std::optional<Tensor> {
        return c.step_dev.defined() ? std::optional<Tensor>(c.step_dev) : std::nullopt;
      })
      .def("use_device_step",
           [](RowCore& c) {
             c.step_dev = at::full({1}, c.step, c.table.options().dtype(at::kLong));
             c.step_scalars = at::zeros({2}, c.table.options());
           })
      .def("advance_device_step",
           [](RowCore& c, double lr) {
             if (!c.step_dev.defined() || c.step_advanced) return;
             c.advance_device_step(lr);
           })
      .def("zero_grad", &RowCore::zero_grad)
      .def("announce",
           [](RowCore& c, double lr, const Tensor& m, const Tensor& v) {
             c.fused_lr = lr;
             c.m = m;
             c.v = v;
             if (c.step_dev.defined() && !c.step_advanced) {
               c.advance_device_step(lr);
               c.step_advanced = true;
             }
           })
      .def("lookup", &RowCore::lookup)
      .def("lookup_tensor", &lookup_tensor)
      .def("gather_rows", &gather_rows)
      .def("accumulate_grad", &accumulate_grad)
      .def("plan_for", &RowCore::plan_for)
      .def("merged_plan",   // a plan over id lists given as tensors (ids < 0 are ignored)
           [](RowCore& c, const std::vector<Tensor>& ids) {
             std::vector<std::shared_ptr<Lookup>> lookups;
             for (auto& t : ids) {
               auto lk = std::make_shared<Lookup>();
               lk->idx = t;
               lk->n = t.numel();
               lk->order = -1;
               lookups.push_back(lk);
             }
             return c.build_plan(std::move(lookups));
           })
      .def("update",
           [](RowCore& c, const Tensor& uniq, const Tensor& g_rows, const Tensor& n_unique, int64_t capacity, double lr,
              const std::optional<Tensor>& m, const std::optional<Tensor>& v) {
             if (c.step_dev.defined() && !c.step_advanced) c.advance_device_step(lr);
             c.update(uniq, g_rows, n_unique, capacity, lr, m ? *m : Tensor(), v ? *v : Tensor());
           })
      .def("apply_single_plan",
           [](RowCore& c, double lr, const std::optional<Tensor>& m, const std::optional<Tensor>& v) {
             return c.apply_single_plan(lr, m ? *m : Tensor(), v ? *v : Tensor());
           })
      .def("end_step", [](RowCore& c) {
        c.drop_plans();
        c.pending.clear();
      });

  py::class_<FusedLaunch, std::shared_ptr<FusedLaunch>>(mod, "FusedLaunch")
      .def("run", &FusedLaunch::run)
      .def_property_readonly("counts", [](const FusedLaunch& f) { return f.plan->counts; });

  mod.def("rows_dist", &rows_dist);
  mod.def("dense_dist", &dense_dist);
  mod.def("path_embed", &path_embed);
  mod.def("filtered_ranks", &filtered_ranks);
  mod.def("score_and_rank", &score_and_rank);
  mod.def("sample_negatives", &sample_negatives);
}

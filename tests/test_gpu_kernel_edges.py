"""Sizes and values at which the kernels' tiles, pieces and routes change over (needs a B200): row lengths
that are no multiple of the piece size, ragged tiles, the remainders of the split matrix product, ties and
special values of the cheaper term rules, and the accepted forms of the native host side."""
import argparse
import copy

import numpy as np
import pytest
import torch

from tests.util import RTOL, RTOL_ATOMIC, close, forward_scale, make_operands

pytestmark = pytest.mark.gpu


def _cuda(*arrays):
    return [None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


# ---- distance kernels ------------------------------------------------------------------------------

@pytest.mark.parametrize("op", ["l1", "l2", "box_out", "box_in", "rotate", "complex", "distmult"])
@pytest.mark.parametrize("shape", [
    (4, 33, 4, 1, 250),      # 8-byte pieces
    (4, 33, 4, 1, 31),       # 4-byte pieces, one chunk and a tail
    (2, 40, 2, 1, 129),      # one float past a full chunk of 4-byte pieces
    (2, 17, 2, 1, 1001),     # odd and wide
    (2, 19, 2, 1, 1022),     # the widest rows of 8-byte pieces
    (3, 130, 3, 1, 412),     # 16-byte pieces with a tail of 12 floats
    (7, 1, 7, 1, 37),        # positives: one thread owns an element of both gradients
    (5, 1, 5, 1, 1000),
    (1, 1, 1, 1, 3),
    (65, 1, 1, 33, 37),      # one query list against every row: shared-list kernels, odd dim, ragged tiles
    (1, 65, 33, 1, 35),
    (1, 63, 32, 1, 32),
    (1, 64, 31, 1, 128),
    (1, 257, 100, 1, 100),   # query segments of a cluster end inside a chunk of 64
], ids=lambda s: "x".join(map(str, s)))
def test_distances_at_piece_and_tile_edges(oracle, op, shape):
    """Tolerances: the forward sums and the per-row gradients are re-associated sums of the same fp32 terms
    (1e-5 of the summed magnitudes); query gradients are accumulated by several CTAs (1e-4)."""
    from smore_b200 import extlib_cuda as ext
    be, ne, bc, nc, dim = shape
    ent, q0, q1 = make_operands(op, be, ne, bc, nc, dim, seed=sum(shape) + len(op))
    want = oracle.dist_forward(op, ent, q0, q1)
    d_ent, d_q0, d_q1 = _cuda(ent, q0, q1)
    dst = torch.full(want.shape, float("nan"), device="cuda")
    ext.dist_forward(op, d_ent, d_q0, d_q1, dst)
    close(dst.cpu().numpy(), want, RTOL, forward_scale(oracle, op, ent, q0, q1), "forward")
    gout = np.random.default_rng(3).standard_normal(want.shape).astype(np.float32)
    w = oracle.dist_backward(op, gout, ent, q0, q1)
    g = [torch.full_like(d_ent, float("nan")), torch.full_like(d_q0, float("nan")),
         None if q1 is None else torch.full_like(d_q1, float("nan"))]
    ext.dist_backward(op, _cuda(gout)[0], d_ent, d_q0, d_q1, *g)
    for got, ref, what in zip(g, w, ("g_entity", "g_first", "g_second")):
        if got is not None:
            close(got.cpu().numpy(), ref, RTOL_ATOMIC, what=what)


@pytest.mark.parametrize("op", ["box_out", "box_in"])
@pytest.mark.parametrize("shape", [(1, 64, 40, 1, 64), (4, 48, 4, 1, 64), (3, 20, 3, 1, 37)], ids=str)
def test_box_ties_and_signs_of_offsets(oracle, op, shape):
    """Entities on the center (as +0 and -0 too), on the box's face, offsets of either sign and zero: the
    rule for positive offsets takes over element by element."""
    from smore_b200 import ext_ops
    be, ne, bc, nc, dim = shape
    rng = np.random.default_rng(dim)
    ent = (rng.integers(-3, 4, (be, ne, dim)) * 0.125).astype(np.float32)
    center = (rng.integers(-2, 3, (bc, nc, dim)) * 0.125).astype(np.float32)
    offset = (rng.integers(-1, 3, (bc, nc, dim)) * 0.125).astype(np.float32)
    for a in (ent, center):
        a[(a == 0) & (rng.random(a.shape) < 0.5)] = -0.0
    gouts = [rng.standard_normal((max(be, bc), max(ne, nc))).astype(np.float32) for _ in range(2)]
    leaves = [t.requires_grad_() for t in _cuda(ent, center, offset)]
    d_out, d_in = ext_ops.box_dist_both(*leaves)
    np.testing.assert_array_equal((d_out if op == "box_out" else d_in).detach().cpu().numpy(),
                                  oracle.dist_forward(op, ent, center, offset))     # sums of multiples of 1/8
    out, g = (d_out, gouts[0]) if op == "box_out" else (d_in, gouts[1])
    got = torch.autograd.grad(out, leaves, _cuda(g)[0])
    for a, b in zip(got, oracle.dist_backward(op, g, ent, center, offset)):
        close(a.cpu().numpy(), b, RTOL_ATOMIC)


@pytest.mark.parametrize("K,B", [(70, 33), (64, 5)])
def test_box_scores_of_special_values_do_not_depend_on_the_kernel(oracle, K, B):
    """A NaN or an infinite box around an infinite distance adds nothing to the out-of-box distance, in the
    tiles of the shared-list kernels as in the single-distance kernels."""
    from smore_b200 import ext_ops
    ent, center, offset = make_operands("box_out", 1, K, B, 1, 40, seed=K)
    ent[0, 3, 7], ent[0, 9, 39], ent[0, 10, 0], ent[0, K - 1, 5] = np.nan, np.inf, -np.inf, np.nan
    center[2, 0, 4], offset[1, 0, :], offset[0, 0, 6] = np.nan, np.inf, np.nan
    d_out, d_in = ext_ops.box_dist_both(*_cuda(ent, center, offset))
    for got, op in ((d_out, "box_out"), (d_in, "box_in")):
        single = torch.empty_like(got)
        from smore_b200 import extlib_cuda
        extlib_cuda.dist_forward(op, *_cuda(ent, center, offset), single)
        got, single = got.cpu().numpy(), single.cpu().numpy()
        assert np.array_equal(np.isfinite(got), np.isfinite(single))
        close(np.nan_to_num(got, posinf=9e9), np.nan_to_num(single, posinf=9e9), RTOL, scale=100.0, what=op)


# ---- products in fp32 on the tensor cores ----------------------------------------------------------

@pytest.mark.parametrize("B,K,W", [(128, 128, 4), (132, 260, 36), (256, 256, 64), (260, 132, 68), (128, 1024, 1000),
                                   (1028, 516, 32), (516, 4100, 96), (2304, 2304, 520), (32768, 4100, 32)])
def test_split_products_at_tile_edges(monkeypatch, B, K, W):
    """Edges of the 128 x 256 x 32 tiles, of the chunks of 64, of the reduction cut in two, and (the last) of
    the parts a long candidate list is taken in.  The planes carry 24 bits and the partial sums are fp32:
    2^-22 of the summed magnitudes is above what 2 roundings per chunk of 64 leave at these lengths."""
    monkeypatch.setenv("SMORE_B200_DOT", "fp32")
    from smore_b200 import ext_ops
    g = torch.Generator(device="cuda").manual_seed(B + K + W)
    ent = torch.randn(1, K, W, device="cuda", generator=g).requires_grad_()
    q = torch.randn(B, 1, W, device="cuda", generator=g).requires_grad_()
    w = torch.randn(B, K, device="cuda", generator=g)
    out = ext_ops.distmult_sim(ent, q)
    g_ent, g_q = torch.autograd.grad(out, [ent, q], w)
    e64, q64, w64 = ent.detach()[0].double(), q.detach()[:, 0].double(), w.double()
    for got, a, b in ((out.detach(), q64, e64.t()), (g_ent[0], w64.t(), q64), (g_q[:, 0], w64, e64)):
        rel = ((got.double() - a @ b).norm() / (a @ b).norm()).item()
        assert rel <= 2.0 ** -21, rel


# ---- the step's rows -------------------------------------------------------------------------------

@pytest.mark.parametrize("n_rows", [33, 262144, 262145, 3000000])
@pytest.mark.parametrize("sizes", [(1,), (5000,), (700, 0, 3, 4099), (64,) * 11], ids=str)
def test_lists_of_a_step(n_rows, sizes):
    """Several id lists of one step, empty ones and more lists than one call takes among them, on either side
    of the table size up to which a CTA collects its bits on the SM; ids outside the table are left out."""
    from smore_b200 import embedding
    emb = embedding.SparseEmbedding(0, 8)
    emb.num_rows = n_rows
    emb.embedding = torch.nn.Parameter(torch.zeros(n_rows, 8, device="cuda"), requires_grad=False)
    opt = embedding.SGDEmbedOptimizer(argparse.Namespace(optim_mode=("aggr", "sgd", "gpu", False, 0)), emb, 0)
    gen = torch.Generator(device="cuda").manual_seed(sum(sizes))
    lists = [torch.randint(0, n_rows, (n,), device="cuda", generator=gen) for n in sizes]
    lookups = [opt.core.lookup(i, None) for i in lists]
    p = opt.core.plan_for(lookups[0])
    ids = torch.cat(lists)
    uniq, inverse, counts = torch.unique(ids, return_inverse=True, return_counts=True)
    n = uniq.numel()
    assert p.n_unique.tolist() == [n, 0]
    assert torch.equal(p.uniq[:n], uniq) and torch.equal(p.counts[:n].long(), counts)
    assert torch.equal(torch.cat([p.slot_of(lk) for lk in lookups]).long(), inverse)
    assert not p.g_rows[:n][counts > 1].any()


# ---- Adam inside the backward pass -----------------------------------------------------------------

def _adam_pair(n_rows, dim, rowwise, seed=0):
    from smore_b200 import embedding
    opts = []
    for _ in range(2):
        g = torch.Generator(device="cuda").manual_seed(seed)
        emb = embedding.SparseEmbedding(0, dim)
        emb.num_rows = n_rows
        emb.embedding = torch.nn.Parameter(torch.rand(n_rows, dim, device="cuda", generator=g) - 0.5, requires_grad=False)
        opt = embedding.AdamEmbedOptimizer(argparse.Namespace(optim_mode=("aggr", "adam", "gpu", rowwise, 0)), emb, 0,
                                           lazy_names=("rows",))
        opt.step = 7
        opt.state("state_sum_fo").normal_(0, 1e-3, generator=g)
        opt.state("state_sum_sq").uniform_(1e-6, 2e-6, generator=g)
        opts.append((emb, opt))
    return opts


@pytest.mark.parametrize("rowwise", [True, False], ids=["row_moment", "full_moment"])
@pytest.mark.parametrize("op,dim", [("l1", 400), ("rotate", 500), ("box", 412), ("distmult", 1000), ("box", 250), ("l2", 31)])
@pytest.mark.parametrize("branches", [1, 2])
def test_update_inside_backward(op, dim, rowwise, branches):
    """The same table, moments and query gradients as with the update in apply_grad, for rows of one and of
    several contributors."""
    from smore_b200 import ext_ops
    B, K, n_rows = 3, 40, 400
    width = dim * (2 if op == "rotate" else 1)
    g = torch.Generator(device="cuda").manual_seed(dim)
    ids = torch.randint(0, n_rows, (B, K), device="cuda", generator=g)
    qs = [torch.rand(B, branches, 1, dim, device="cuda", generator=g) * 0.4 for _ in range(1 if op in ("l1", "l2", "distmult") else 2)]
    grads, tables = [], []
    for announce, (emb, opt) in zip((True, False), _adam_pair(n_rows, width, rowwise)):
        opt.zero_grad()
        if announce:
            opt.announce_lr(1e-3)
        leaves = [q.clone().requires_grad_() for q in qs]
        rows = emb(ids.view(-1), "rows").view(B, K, -1)
        if op == "box":
            outs = [ext_ops.box_dist_out(rows, *leaves), ext_ops.box_dist_in(rows, *leaves)]
        else:
            fn = {"l1": ext_ops.l1_dist, "l2": ext_ops.l2_dist, "rotate": ext_ops.rotate_dist, "distmult": ext_ops.distmult_sim}[op]
            outs = [fn(rows, *leaves)]
        torch.autograd.backward(outs, [torch.full_like(o, 0.01 * (i + 1)) for i, o in enumerate(outs)])
        opt.apply_grad(1e-3)
        grads.append([q.grad for q in leaves])
        tables.append([emb.embedding.data, opt.state("state_sum_fo"), opt.state("state_sum_sq")])
    for a, b in zip(*grads):
        close(a.cpu().numpy(), b.cpu().numpy(), RTOL_ATOMIC)
    for a, b in zip(*tables):
        close(a.cpu().numpy(), b.cpu().numpy(), RTOL)


@pytest.mark.parametrize("rowwise", [True, False], ids=["row_moment", "full_moment"])
@pytest.mark.parametrize("other_op", ["distance", "gather", "path"])
def test_rows_with_two_consumers_get_both_gradients(rowwise, other_op):
    """A lookup whose rows a distance op and something else read is not updated inside the backward pass."""
    from smore_b200 import ext_ops, query_ops
    B, K, dim, n_rows = 2, 32, 64, 5000
    g = torch.Generator(device="cuda").manual_seed(1)
    ids = torch.randperm(n_rows, device="cuda", generator=g)[:B * K]
    q = torch.rand(B, 1, dim, device="cuda", generator=g)
    rel = torch.rand(3, dim, device="cuda", generator=g)
    rel_ids = torch.randint(0, 3, (B * K, 2), device="cuda", generator=g)
    results = []
    for announce, (emb, opt) in zip((True, False), _adam_pair(n_rows, dim, rowwise)):
        opt.zero_grad()
        if announce:
            opt.announce_lr(1e-3)
        rows = emb(ids, "rows")
        if other_op == "gather":
            other = rows.materialize().square().sum()
        elif other_op == "path":
            other = query_ops.embed_path("distmult", rows, rel, rel_ids).sum()
        else:
            other = ext_ops.l2_dist(rows.view(B, K, -1), q.clone().requires_grad_()).sum()
        # made last, so its backward pass runs first
        loss = 0.01 * ext_ops.l1_dist(rows.view(B, K, -1), q.clone().requires_grad_()).sum()
        torch.autograd.backward([other, loss])
        opt.apply_grad(1e-3)
        results.append([emb.embedding.data, opt.state("state_sum_fo"), opt.state("state_sum_sq")])
    for a, b in zip(*results):
        close(a.cpu().numpy(), b.cpu().numpy(), RTOL)


@pytest.mark.parametrize("dim", [33, 400])
def test_row_moment_update_divides_exactly(dim):
    """The quotient of the row-wise update is the correctly rounded one, as a division gives it, over the
    exponents a moment can have, and for infinite and NaN moments."""
    from smore_b200 import _lib
    n = 4096
    g = torch.Generator(device="cuda").manual_seed(dim)
    p = torch.zeros(n, dim, device="cuda")
    m = torch.randn(n, dim, device="cuda", generator=g) * 10.0 ** torch.randint(-12, 6, (n, dim), device="cuda", generator=g)
    v = 10.0 ** (torch.rand(n, 1, device="cuda", generator=g) * 60 - 40)
    v[0], v[1], v[2] = float("inf"), float("nan"), 0.0
    m[3, 0], m[4, 1], m[5, 2] = float("inf"), float("-inf"), float("nan")
    zero = torch.zeros(n, dim, device="cuda")
    lr, b1, b2, eps = 0.25, 0.5, 0.25, 1e-8       # powers of two; omb2 g^2 = 0, v_new = v / 4, m_new = m / 2
    m0, v0 = m.clone(), v.clone()
    ids = torch.arange(n, device="cuda")
    count = torch.tensor([n, 0], dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().smore_sparse_update_rows(
        _lib.OPT_IDS["adam"], p.data_ptr(), m.data_ptr(), v.data_ptr(), ids.data_ptr(), zero.data_ptr(), count.data_ptr(), n, dim,
        lr, b1, b2, eps, 1, 1, torch.cuda.current_stream().cuda_stream), "update")
    step_size = torch.tensor(-lr / (1 - b1), device="cuda", dtype=torch.float32)
    root = torch.tensor(float(np.float32(np.sqrt(1 - b2))), device="cuda")
    want = (step_size * (m0 * 0.5)) / (torch.sqrt(v0 * 0.25) / root + torch.tensor(eps, device="cuda", dtype=torch.float32))
    got, want = p.cpu().numpy(), want.cpu().numpy()
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    assert same.all(), (np.argwhere(~same)[:5], got[~same][:5], want[~same][:5])


@pytest.mark.parametrize("dim", [4, 128, 132, 256, 260, 1000, 1028])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 3000])
def test_full_moment_update_in_pieces(dim, n):
    """Rows of one piece, of several and with a last piece that is not full; batches that are not full;
    entries whose update is done already (negative ids).  Against float64: a handful of roundings each."""
    from smore_b200 import _lib
    rows = 4 * n
    g = torch.Generator(device="cuda").manual_seed(dim + n)
    table = torch.randn(rows, dim, device="cuda", generator=g)
    m, v = torch.randn(rows, dim, device="cuda", generator=g) * 1e-3, torch.rand(rows, dim, device="cuda", generator=g) * 1e-6
    grad = torch.randn(n, dim, device="cuda", generator=g) * 1e-3
    ids = torch.sort(torch.randperm(rows, device="cuda", generator=g)[:n])[0]
    done = torch.rand(n, device="cuda", generator=g) < 0.3
    before = [t.clone() for t in (table, m, v)]
    listed = torch.where(done, ~ids, ids)
    count = torch.tensor([n, 0], dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().smore_sparse_update_rows(
        _lib.OPT_IDS["adam"], table.data_ptr(), m.data_ptr(), v.data_ptr(), listed.data_ptr(), grad.data_ptr(), count.data_ptr(),
        n, dim, 1e-2, 0.9, 0.999, 1e-8, 3, 0, torch.cuda.current_stream().cuda_stream), "update")
    p64, m64, v64 = [t.double() for t in before]
    r, gr = ids[~done], grad[~done].double()
    m64[r] = 0.9 * m64[r] + 0.1 * gr
    v64[r] = 0.999 * v64[r] + 0.001 * gr * gr
    p64[r] -= 1e-2 / (1 - 0.9 ** 3) * m64[r] / ((v64[r] / (1 - 0.999 ** 3)).sqrt() + 1e-8)
    for got, want in zip((table, m, v), (p64, m64, v64)):
        close(got.cpu().numpy(), want.cpu().numpy(), RTOL)
    for got, old in zip((table, m, v), before):
        keep = torch.ones(rows, dtype=torch.bool, device="cuda")
        keep[r] = False
        assert torch.equal(got[keep], old[keep])


# ---- evaluation ------------------------------------------------------------------------------------

@pytest.mark.parametrize("Q,N", [(1, 63), (31, 64), (32, 65), (33, 4096), (64, 129), (70, 1000)])
@pytest.mark.parametrize("kind", [tuple, set, np.array, lambda ids: torch.tensor(ids, dtype=torch.int64)], ids=["tuple", "set", "numpy", "tensor"])
def test_ranks_at_tile_edges_and_forms_of_answers(Q, N, kind):
    """Ragged 32 x 64 scoring tiles; answers in every iterable form, the outer collection a view."""
    from smore_b200 import ext_ops, ranking
    g = torch.Generator(device="cuda").manual_seed(Q)
    table = torch.rand(N, 36, device="cuda", generator=g) - 0.5
    query = [torch.rand(Q, 1, 36, device="cuda", generator=g) - 0.5, torch.rand(Q, 1, 36, device="cuda", generator=g) * 0.1]
    rng = np.random.default_rng(N)
    ids = [[int(i) for i in rng.choice(N, 30, replace=False)] for _ in range(Q)]
    easy = {q: kind(ids[q][:q % 11]) for q in range(Q)}
    hard = {q: kind(ids[q][11:11 + q % 20]) for q in range(Q)}
    got = None if Q < 8 else ranking.score_and_rank("box", table, query, easy.values(), hard.values(), gamma=2.0, cen=0.02)
    logits = 2.0 - ext_ops.box_dist_out(table.unsqueeze(0), *query) - 0.02 * ext_ops.box_dist_in(table.unsqueeze(0), *query)
    for q, r in enumerate(ranking.filtered_ranks(logits, easy.values(), hard.values())):
        known = torch.zeros(N, dtype=torch.bool, device="cuda")
        known[[int(i) for i in easy[q]] + [int(i) for i in hard[q]]] = True
        h = torch.tensor([int(i) for i in hard[q]], dtype=torch.int64, device="cuda")
        own, others = logits[q][h][:, None], logits[q][~known][None, :]
        low, high = torch.sort((others > own).sum(1))[0] + 1, torch.sort((others >= own).sum(1))[0] + 1   # ties: either order
        assert r.shape == low.shape and (low <= r).all() and (r <= high).all()
        assert got is None or torch.equal(got[q], r)


def test_answers_that_are_no_ids_are_refused():
    from smore_b200 import ranking
    logits = torch.zeros(1, 8, device="cuda")
    for bad, error in (([8], ValueError), ([-1], ValueError), (["3"], TypeError), (3, TypeError)):
        with pytest.raises(error):
            ranking.filtered_ranks(logits, [[]], [bad])


# ---- negative sampling -----------------------------------------------------------------------------

@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("Q,k,per_query", [(1, 1, 0), (3, 5, 2), (1, 700, 9), (64, 33, 30), (2, 257, 1500), (40, 9000, 3),
                                           (700, 1024, 31)])
def test_draws_do_not_depend_on_the_launch(weighted, Q, k, per_query):
    """One, two and four positions per thread, CTAs that span several queries, answers that fit on the SM and
    that do not: every position draws what its counter gives, from packed tables as from three arrays."""
    from smore_b200 import _lib, sampler
    n = 5000
    rng = np.random.default_rng(Q + k)
    weights = rng.random(n) ** 4 + 1e-3 if weighted else None
    csr = sampler.answers_csr([rng.choice(n, per_query, replace=False) for _ in range(Q)], "cuda")
    s = sampler.NegativeSampler(n, "cuda", weights=weights, seed=11)
    s.offset = 5
    got = s.sample(Q, k, csr)
    stream = torch.cuda.current_stream().cuda_stream
    t = [None] * 3 if s.tables is None else [x.data_ptr() for x in s.tables]
    one = torch.empty_like(got)
    for q in (range(Q) if Q <= 64 else (0, 1, Q // 2, Q - 1)):       # a query by itself, from the arrays
        a, b = int(csr[0][q]), int(csr[0][q + 1])
        ptr = torch.tensor([0, b - a], device="cuda")
        ids = csr[1][a:max(b, a + 1)]
        for at in range(0, k, 300):                                   # and in pieces
            m = min(300, k - at)
            _lib.check(_lib.lib().smore_sample_negatives(11, 5 + q * k + at, n, *t, ptr.data_ptr(), ids.data_ptr(), 1, m,
                                                         one[q, at:].data_ptr(), stream), "sample")
        assert torch.equal(got[q], one[q]) and not torch.isin(got[q], csr[1][a:b]).any()


# ---- the native host side --------------------------------------------------------------------------

def test_forward_mode_is_refused():
    import torch.autograd.forward_ad as fwad
    from smore_b200 import ext_ops, query_ops
    e, q = torch.rand(2, 20, 8, device="cuda"), torch.rand(2, 1, 8, device="cuda")
    rel_ids = torch.zeros(2, 1, dtype=torch.int64, device="cuda")
    with fwad.dual_level():
        dual = fwad.make_dual(q, torch.ones_like(q))
        for call in (lambda: ext_ops.l1_dist(e, dual), lambda: query_ops.embed_path("add", dual[:, 0], q[:, 0], rel_ids)):
            with pytest.raises((RuntimeError, NotImplementedError)):
                call()


@pytest.mark.parametrize("rowwise", [True, False])
def test_copy_of_a_model_between_steps(rowwise):
    """A copied optimizer goes on by itself, on its own table and state."""
    (emb, opt), _ = _adam_pair(50, 16, rowwise)
    model = torch.nn.Module()
    model.emb, model.opt = emb, opt
    twin = copy.deepcopy(model)
    assert twin.opt.step == 7 and twin.opt.sparse_embed is twin.emb
    ids = torch.tensor([3, 4, 3], device="cuda")
    for m in (model, twin):
        m.opt.zero_grad()
        m.emb(ids).square().sum().backward()
        m.opt.apply_grad(1e-2)
    assert torch.equal(model.opt.table, twin.opt.table) and model.opt.table.data_ptr() != twin.opt.table.data_ptr()
    assert torch.equal(model.opt.state("state_sum_fo"), twin.opt.state("state_sum_fo"))

"""The work that a user of this library has it do, as cases that can be timed and compared.

Five kinds, all through the public entry points:

  step    one training step on an embedding table in GPU memory: lookups of positives, negatives and
          anchors (smore_b200.embedding), relation projections (smore_b200.query_ops), candidate scores
          (smore_b200.ext_ops), the backward pass from the loss's gradients, the row-wise Adam update
  op      a distance op on materialised tensors, forward and backward
  eval    queries scored against every entity and the filtered ranks of their answers
          (smore_b200.ranking), fused or through the logits
  sample  negative sampling (smore_b200.sampler)

Sizes are those of bench.py's workloads and of the tests; values are synthetic with the distributions of
those workloads (embeddings uniform in +-(gamma + 2) / dim, popularity of anchors and relations by a power
law, uniform negatives).
"""
import argparse
import math
import os

import numpy as np
import torch

from smore_b200 import embedding, ext_ops, query_ops, ranking, sampler

LR = 1e-4
FREEBASE_ROWS = 10756769          # one eighth of 86,054,151: the rows one of eight GPUs holds

# largest sizes of a case: floats in the table, term evaluations of a step, of an evaluation
MAX_TABLE = FREEBASE_ROWS * 400
MAX_STEP_TERMS = 1024 * 1024 * 1000
MAX_EVAL_TERMS = 32 * FREEBASE_ROWS * 400

# geometry -> (parts of an entity row, operands of a query, relation row parts, geometry of embed_path)
GEOMETRIES = {
    "vec": (1, 1, 1, "add"),
    "box": (1, 2, 1, "add"),
    "rotate": (2, 2, 1, "rotate"),
    "complex": (2, 2, 2, "complex"),
    "distmult": (1, 1, 1, "distmult"),
}
# arithmetic instructions of one term, forward and backward
TERM_FLOPS = {"vec": (2, 5), "box": (6, 14), "rotate": (6, 11), "complex": (4, 8), "distmult": (2, 4)}

OPS = {
    "box_dist_out": (1, 2, 4, 7),
    "box_dist_in": (1, 2, 4, 8),
    "rotate_dist": (2, 2, 6, 11),
    "l1_dist": (1, 1, 2, 5),
    "l2_dist": (1, 1, 3, 5),
}


def _step(name, geo, rows, relations, dim, B, K, gamma, hops=1, shared=False, branches=1, rowwise=False, announce=True,
          dot="fp32"):
    c = dict(kind="step", geo=geo, rows=rows, relations=relations, dim=dim, B=B, K=K, gamma=gamma, hops=hops,
             shared=shared, branches=branches, rowwise=rowwise, announce=announce, dot=dot)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's own self-check of a distance op: the smallest call, latency only
        dict(name="op_box_out_30x20", kind="op", op="box_dist_out", be=30, ne=1, bc=1, nc=20, dim=400),
        # candidates gathered by the caller, a dim that is no multiple of four, ragged counts
        dict(name="op_l2_ragged", kind="op", op="l2_dist", be=333, ne=101, bc=333, nc=1, dim=250),
        # GQE on FB15k-237: a small model's step, bound by launches and host work
        _step("gqe_fb15k237", "vec", 14505, 237, 64, 512, 128, 12.0, announce=False),
        # Query2box on FB15k with one negative list for the batch (--share_negative), two-hop queries
        _step("q2b_fb15k_shared", "box", 14951, 1345, 400, 1024, 512, 12.0, hops=2, shared=True),
        # RotatE on ogbl-wikikg2: 4000-byte rows, full second moment
        _step("rotate_wikikg", "rotate", 2500604, 535, 500, 1024, 1024, 24.0),
        # Query2box at Freebase scale, one GPU's part of the table: three-hop queries
        _step("q2b_freebase_3p", "box", FREEBASE_ROWS, 14824, 400, 1024, 1024, 2.0, hops=3, rowwise=True),
        # the same with union queries: two boxes per query
        _step("q2b_freebase_2u", "box", FREEBASE_ROWS, 14824, 400, 1024, 1024, 2.0, branches=2, rowwise=True),
        # DistMult against shared negatives: the tensor-core route in its default precision
        _step("distmult_wikikg", "distmult", 2500604, 535, 1000, 4096, 8192, 0.0, shared=True),
        # ComplEx, the same size, with SMORE_B200_DOT=tf32
        _step("complex_wikikg_tf32", "complex", 2500604, 535, 500, 4096, 8192, 0.0, shared=True, dot="tf32"),
        # evaluation at Freebase scale: 32 queries against the whole (part of the) table, ranks only
        dict(name="eval_box_freebase", kind="eval", geo="box", rows=FREEBASE_ROWS, dim=400, Q=32, gamma=2.0, fused=True),
        # evaluation on FB15k as the reference's test step does it: logits first, ranks from them
        dict(name="eval_box_fb15k", kind="eval", geo="box", rows=14951, dim=400, Q=32, gamma=12.0, fused=False),
        # negatives of one batch drawn by in-degree, the queries' answers left out
        dict(name="sample_wikikg", kind="sample", rows=2500604, B=1024, K=1024, weighted=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng, lo, hi):
    """Mostly multiples of four, as every published configuration has them; one in six is any number."""
    d = _log(rng, lo, hi)
    return d if rng.random() < 1 / 6 else max(lo, d // 4 * 4)


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["op"] * 2 + ["eval"] * 2 + ["sample"])
    if kind == "op":
        op = rng.choice(sorted(OPS))
        if rng.random() < 0.5:       # outer form: every entity row against every query
            return dict(kind="op", op=op, be=_log(rng, 8, 512), ne=1, bc=1, nc=_log(rng, 4, 256), dim=_dim(rng, 32, 800))
        B = _log(rng, 8, 512)
        return dict(kind="op", op=op, be=B, ne=_log(rng, 4, 256), bc=B, nc=1, dim=_dim(rng, 32, 800))
    if kind == "sample":
        return dict(kind="sample", rows=_log(rng, 10000, 2500604), B=_log(rng, 64, 1024), K=_log(rng, 32, 1024),
                    weighted=rng.random() < 0.5)
    if kind == "eval":
        geo = rng.choice(["vec", "box", "rotate"])
        dim = _log(rng, 64, 500) // 4 * 4
        Q = _log(rng, 8, 64)
        most = min(MAX_TABLE // (GEOMETRIES[geo][0] * dim), MAX_EVAL_TERMS // (Q * dim) // (1 if geo != "rotate" else 2))
        return dict(kind="eval", geo=geo, rows=_log(rng, 10000, min(FREEBASE_ROWS, most)), dim=dim, Q=Q,
                    gamma=rng.choice([2.0, 12.0, 24.0]), fused=rng.random() < 0.6)
    geo = rng.choice(["vec", "box", "box", "rotate", "complex", "distmult"])
    parts = GEOMETRIES[geo][0]
    dim = _dim(rng, 32, 1000 // parts)
    rowwise = rng.random() < 0.5
    rows = _log(rng, 10000, min(FREEBASE_ROWS, MAX_TABLE * 2 // 3 // (parts * dim)))
    relations = _log(rng, 200, 15000)
    gamma = rng.choice([2.0, 12.0, 24.0])
    hops = rng.randint(1, 3)
    branches = 2 if rng.random() < 0.25 else 1
    announce = rng.random() < 0.75
    shared = rng.random() < 0.35
    if shared and geo in ("complex", "distmult"):
        return _step(None, geo, rows, relations, dim, _log(rng, 256, 4096), _log(rng, 512, 8192), 0.0, hops, True, 1,
                     rowwise, announce, rng.choice(["fp32", "tf32"]))
    B, K = _log(rng, 128, 1024), _log(rng, 32, 1024)
    room = MAX_STEP_TERMS // (parts * dim * B * branches) // (8 if dim % 4 else 1)
    return _step(None, geo, rows, relations, dim, B, max(4, min(K, room)), gamma, hops, shared, branches, rowwise, announce)


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------

DEVICE = torch.device("cuda", 0)


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _uniform(gen, lo, hi, *shape):
    return torch.empty(*shape, device=DEVICE).uniform_(lo, hi, generator=gen)


def _power_law_ids(gen, n, size, s):
    """Ids in [0, n) whose popularity rank falls like rank^-s, spread over the table."""
    u = torch.rand(size, generator=gen, device=DEVICE, dtype=torch.float64)
    x = torch.exp(u * math.log(n)) if abs(s - 1.0) < 1e-9 else (1.0 + u * (float(n) ** (1.0 - s) - 1.0)) ** (1.0 / (1.0 - s))
    rank = x.floor().long().clamp_(1, n) - 1
    mult = 2654435761 % n
    while mult < 2 or math.gcd(mult, n) != 1:
        mult += 1
    return (rank * mult + 12345) % n


def _prepare_step(c, seed):
    gen = _generator(seed)
    parts, n_q, rel_parts, _ = GEOMETRIES[c["geo"]]
    width, B, K, dim = parts * c["dim"], c["B"], c["K"], c["dim"]
    r = (c["gamma"] + 2.0) / dim
    emb = embedding.SparseEmbedding(0, width)
    emb.num_rows = c["rows"]
    emb.embedding = torch.nn.Parameter(_uniform(gen, -r, r, c["rows"], width), requires_grad=False)
    args = argparse.Namespace(optim_mode=("aggr", "adam", "gpu", c["rowwise"], 0), share_optim_stats=False)
    opt = embedding.AdamEmbedOptimizer(args, emb, 0, lazy_names=("negative_entity", "positive_entity", "anchor_entity"))
    # a run in progress: moments of the size of its gradients
    size = 0.5 / (B * K)
    opt.step = 1000
    opt.state("state_sum_fo").normal_(0.0, size, generator=gen)
    opt.state("state_sum_sq").uniform_(0.5 * size * size, 1.5 * size * size, generator=gen)
    s = dict(case=c, emb=emb, opt=opt)
    s["rel"] = torch.nn.Parameter(_uniform(gen, -r, r, c["relations"], rel_parts * dim))
    s["off"] = torch.nn.Parameter(_uniform(gen, 0.0, r, c["relations"], dim)) if c["geo"] == "box" else None
    s["pos"] = torch.randint(0, c["rows"], (B,), generator=gen, device=DEVICE)
    s["neg"] = torch.randint(0, c["rows"], (1 if c["shared"] else B, K), generator=gen, device=DEVICE)
    s["anchors"] = [_power_law_ids(gen, c["rows"], (B,), 1.2) for _ in range(c["branches"])]
    s["relations"] = [_power_law_ids(gen, c["relations"], (B * c["hops"],), 1.0).view(B, c["hops"])
                      for _ in range(c["branches"])]
    # what a negative-sampling loss sends back: every positive 1 / 2B, every negative its share of 1 / 2B;
    # distances (a larger distance lowers the score) and similarities differ in sign
    sign = 1.0 if c["geo"] in ("complex", "distmult") else -1.0
    U = c["branches"]
    s["g_pos"] = _uniform(gen, -0.5 * sign / B, 0.0, B, U, 1) if sign > 0 else _uniform(gen, 0.0, 0.5 / B, B, U, 1)
    s["g_neg"] = sign * _uniform(gen, 0.0, 2.0 * size, B, U, K)
    if c["geo"] == "box":
        s["g_pos_in"], s["g_neg_in"] = 0.02 * s["g_pos"], 0.02 * s["g_neg"]
    return s


def _prepare_op(c, seed):
    gen = _generator(seed)
    parts, n_q, _, _ = OPS[c["op"]]
    r = 14.0 / c["dim"]
    lead = (max(c["be"], c["bc"]), max(c["ne"], c["nc"]))
    s = dict(case=c, entity=_uniform(gen, -r, r, c["be"], c["ne"], parts * c["dim"]).requires_grad_(),
             query=[_uniform(gen, -r, r, c["bc"], c["nc"], c["dim"]).requires_grad_()], grad=_uniform(gen, -1.0, 1.0, *lead))
    if n_q == 2:
        low = 0.0 if c["op"].startswith("box") else -r
        s["query"].append(_uniform(gen, low, r, c["bc"], c["nc"], c["dim"]).requires_grad_())
    return s


def _answers(rng, n, Q, easy, hard):
    """Distinct answer ids of every query, as Python lists: what a test set holds."""
    out_easy, out_hard = [], []
    for _ in range(Q):
        ids = rng.choice(n, size=easy + hard, replace=False) if n <= 65536 else np.unique(rng.integers(0, n, easy + hard))
        ids = [int(i) for i in ids]
        out_easy.append(ids[:easy])
        out_hard.append(ids[easy:])
    return out_easy, out_hard


def _prepare_eval(c, seed):
    gen = _generator(seed)
    parts, n_q, _, _ = GEOMETRIES[c["geo"]]
    r = (c["gamma"] + 2.0) / c["dim"]
    s = dict(case=c, table=_uniform(gen, -r, r, c["rows"], parts * c["dim"]),
             query=[_uniform(gen, -r, r, c["Q"], 1, c["dim"])])
    if n_q == 2:
        s["query"].append(_uniform(gen, 0.0 if c["geo"] == "box" else -r, r, c["Q"], 1, c["dim"]))
    s["easy"], s["hard"] = _answers(np.random.default_rng(seed), c["rows"], c["Q"], 10, 20)
    return s


def _prepare_sample(c, seed):
    rng = np.random.default_rng(seed)
    weights = rng.permutation(1.0 / np.arange(1, c["rows"] + 1) ** 0.75) if c["weighted"] else None
    s = dict(case=c, sampler=sampler.NegativeSampler(c["rows"], DEVICE, weights=weights, seed=int(seed)))
    easy, hard = _answers(rng, c["rows"], c["B"], 10, 20)
    s["answers"] = sampler.answers_csr([a + b for a, b in zip(easy, hard)], DEVICE)
    return s


def prepare(case, seed):
    return {"step": _prepare_step, "op": _prepare_op, "eval": _prepare_eval, "sample": _prepare_sample}[case["kind"]](case, seed)


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------

def _embed_queries(s):
    """Query operands [B, branches, 1, dim], the form the models hand to the distance ops."""
    c = s["case"]
    geometry = GEOMETRIES[c["geo"]][3]
    r = (c["gamma"] + 2.0) / c["dim"]
    branches = []
    for anchors, relations in zip(s["anchors"], s["relations"]):
        rows = s["emb"](anchors, "anchor_entity")
        out = query_ops.embed_path(geometry, rows, s["rel"], relations, off_table=s["off"],
                                   phase_scale=math.pi / r if geometry == "rotate" else 1.0)
        branches.append([t.unsqueeze(1) for t in (out if isinstance(out, tuple) else (out,))])
    parts = [torch.cat(p, dim=1) if len(p) > 1 else p[0] for p in zip(*branches)]
    return [p.unsqueeze(-2) for p in parts]


def _scores(geo, entity, query):
    if geo == "box":
        return [ext_ops.box_dist_out(entity, query[0], query[1]), ext_ops.box_dist_in(entity, query[0], query[1])]
    if geo == "rotate":
        return [ext_ops.rotate_dist(entity, query[0], query[1])]
    if geo == "complex":
        return [ext_ops.complex_sim(entity, query[0], query[1])]
    if geo == "distmult":
        return [ext_ops.distmult_sim(entity, query[0])]
    return [ext_ops.l1_dist(entity, query[0])]


def _run_step(s):
    c, opt = s["case"], s["opt"]
    os.environ["SMORE_B200_DOT"] = c["dot"]
    for p in (s["rel"], s["off"]):
        if p is not None:
            p.grad = None
    opt.zero_grad()
    if c["announce"]:
        opt.announce_lr(LR)
    pos = s["emb"](s["pos"], "positive_entity")
    neg = s["emb"](s["neg"].view(-1), "negative_entity")
    query = _embed_queries(s)
    d_pos = _scores(c["geo"], pos.unsqueeze(1), query)
    d_neg = _scores(c["geo"], neg.view(s["neg"].shape[0], c["K"], -1), query)
    grads = [s["g_pos"], s["g_neg"]] if len(d_pos) == 1 else [s["g_pos"], s["g_pos_in"], s["g_neg"], s["g_neg_in"]]
    torch.autograd.backward(d_pos + d_neg, grads)
    opt.apply_grad(LR)
    return dict(d_pos=d_pos, d_neg=d_neg, g_rel=s["rel"].grad, g_off=None if s["off"] is None else s["off"].grad,
                table=s["emb"].embedding, m=opt.state("state_sum_fo"), v=opt.state("state_sum_sq"))


def _run_op(s):
    out = getattr(ext_ops, s["case"]["op"])(s["entity"], *s["query"])
    return dict(out=out, grads=torch.autograd.grad(out, [s["entity"]] + s["query"], s["grad"]))


def _run_eval(s):
    c = s["case"]
    with torch.no_grad():
        if c["fused"]:
            return ranking.score_and_rank(c["geo"], s["table"], s["query"], s["easy"], s["hard"], c["gamma"], 0.02)
        d = _scores(c["geo"], s["table"].unsqueeze(0), s["query"])
        logits = c["gamma"] - d[0] if len(d) == 1 else c["gamma"] - d[0] - 0.02 * d[1]
        return dict(logits=logits, ranks=torch.cat(ranking.filtered_ranks(logits, s["easy"], s["hard"])))


def _run_sample(s):
    return s["sampler"].sample(s["case"]["B"], s["case"]["K"], s["answers"])


def run(state):
    return {"step": _run_step, "op": _run_op, "eval": _run_eval, "sample": _run_sample}[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------

def work(case):
    c = case
    if c["kind"] == "op":
        parts, n_q, fwd, bwd = OPS[c["op"]]
        cells = max(c["be"], c["bc"]) * max(c["ne"], c["nc"])
        operands = c["be"] * c["ne"] * parts * c["dim"] + n_q * c["bc"] * c["nc"] * c["dim"]
        # operands read, their gradients written; outputs written, the gradients of the outputs read
        return {"bytes": 4 * (2 * operands + 2 * cells), "flops": cells * c["dim"] * (fwd + bwd)}
    if c["kind"] == "sample":
        draws = c["B"] * c["K"]
        # an id written per draw; one entry of each alias table read (a 32-byte sector of DRAM each)
        return {"bytes": draws * (8 + (2 * 32 if c["weighted"] else 0)) + c["B"] * 30 * 8, "flops": draws * 100}
    if c["kind"] == "eval":
        parts, n_q, _, _ = GEOMETRIES[c["geo"]]
        nbytes = 4 * (c["rows"] * parts * c["dim"] + n_q * c["Q"] * c["dim"])
        if not c["fused"]:
            nbytes += 4 * c["Q"] * c["rows"]         # the logits
        return {"bytes": nbytes, "flops": c["Q"] * c["rows"] * c["dim"] * TERM_FLOPS[c["geo"]][0]}
    parts, n_q, rel_parts, _ = GEOMETRIES[c["geo"]]
    width, B, U = parts * c["dim"], c["B"], c["branches"]
    n_neg = c["K"] * (1 if c["shared"] else B)
    looked_up = n_neg + B + U * B
    rows = c["rows"] * -math.expm1(-looked_up / c["rows"])          # distinct rows, expected
    row = 4 * width
    # every distinct row: read by the forward pass; read again by the backward pass, whose inputs depend on
    # all scores; written by the update; first moment and second moment read and written
    per_row = 3 * row + 2 * row + (2 * 4 if c["rowwise"] else 2 * row)
    scores = B * U * (c["K"] + 1) * (2 if c["geo"] == "box" else 1)
    tables = 4 * c["relations"] * c["dim"] * (rel_parts + (1 if c["geo"] == "box" else 0))   # gradients written
    queries = 4 * B * U * c["dim"] * n_q * 4        # operands and their gradients, written and read
    terms = B * U * (c["K"] + 1) * c["dim"]
    return {"bytes": rows * per_row + 8 * looked_up + 2 * 4 * scores + tables + queries,
            "flops": terms * sum(TERM_FLOPS[c["geo"]])}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["kind"] == "eval" and case["fused"]:
        return "exact"             # ranks
    if case["kind"] == "step" and case["dot"] == "tf32":
        return {"rel": 1e-3}       # products of 10-bit mantissas
    return {"rel": 1e-5}           # 32-bit sums; ranks stay the same

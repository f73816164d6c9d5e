"""Evaluation of ranked answers: the part of the reference's test step that follows the scoring of
a query against every entity (smore/training/train_process.py:113-153).

    logits = gamma - dist(all_entities, query)          # the distance ops with be = 1, ne = N
    ranks = filtered_ranks(logits, easy_answers, hard_answers)
    logs  = ranking_metrics(ranks)                      # MRR, HITS1/3/10, HITS1max per query

`filtered_ranks` replaces argsort + scatter over the N logits by a count per answer
(smore_hard_ranks in libsmore_b200.so); there is no CPU path.
"""
import torch

from . import _lib


def filtered_ranks(logits, easy_answers, hard_answers):
    """Ranks of the hard answers in the filtered setting.

    logits        float32 CUDA tensor [Q, N] (one row of scores over all candidates per query)
    easy_answers  Q iterables of candidate ids that are filtered out but not scored
    hard_answers  Q iterables of candidate ids to rank
    Returns a list of Q int64 CUDA tensors: the ranks of each query's hard answers in ascending
    order, the quantity `cur_ranking[masks]` of train_process.py:140-141.
    """
    return _lib.host().filtered_ranks(logits, easy_answers, hard_answers)


_SCORE_IDS = {"box": _lib.BOX_BOTH_ID, "vec": _lib.DIST_IDS["l1"], "l1": _lib.DIST_IDS["l1"], "l2": _lib.DIST_IDS["l2"],
              "rotate": _lib.DIST_IDS["rotate"], "complex": _lib.DIST_IDS["complex"],
              "distmult": _lib.DIST_IDS["distmult"]}


def score_and_rank(geo, table, query, easy_answers, hard_answers, gamma=0.0, cen=0.0):
    """The evaluation step in one call: score Q queries against every row of `table` with the model's
    logit and return the filtered ranks of their hard answers, without materialising the [Q, N]
    logits (smore_score_hard_ranks).

    geo      "box" (gamma - d_out - cen * d_in), "vec" / "l1" / "rotate" (gamma - d), "l2" (gamma - sqrt(d)),
             "complex" / "distmult" (the similarity)
    table    float32 CUDA [N, W] - the whole entity table (W = dim, or 2 * dim for rotate / complex rows)
    query    one or two float32 CUDA tensors [Q, dim] (or [Q, 1, dim]): center (and offset), re and im, ...
    Returns what filtered_ranks returns for the logits the distance ops would have produced."""
    if geo not in _SCORE_IDS:
        raise ValueError("geo must be one of %s" % sorted(_SCORE_IDS))
    return _lib.host().score_and_rank(_SCORE_IDS[geo], table, query[0], query[1] if len(query) > 1 else None, easy_answers,
                                      hard_answers, float(gamma), float(cen))


def ranking_metrics(hard_ranks):
    """Per-query metrics of train_process.py:142-146 from the sorted filtered ranks of a query's hard
    answers: MRR, HITS1, HITS3, HITS10 (means over the answers) and HITS1max (best answer ranked 1)."""
    r = hard_ranks.to(torch.float32)
    if r.numel() == 0:
        return {"MRR": 0.0, "HITS1": 0.0, "HITS3": 0.0, "HITS10": 0.0, "HITS1max": 0.0}
    return {"MRR": torch.mean(1.0 / r).item(),
            "HITS1": torch.mean((r <= 1).float()).item(),
            "HITS3": torch.mean((r <= 3).float()).item(),
            "HITS10": torch.mean((r <= 10).float()).item(),
            "HITS1max": float(r[0].item() == 1)}

"""Timed workloads over the public Python entry points.

Sizes come from the repository's own configurations: 63 genes x 64 cells
(8 chains), 95 x 96 (1024 chains; fixed rates, or the sum score with
Langevin error moves), a mix of datasets of 16-127 genes and 16-256 cells
with 32 chains each, 255 x 512, and the gradient check's 4096 trees.

Chain workloads keep warmed-up chains and advance them by one launch a pass,
as a long run does between two checkpoints; a pass returns the best tree and
the chains' whole state.  The calls on host buffers (scores, gradients,
moves) take new arrays and return theirs.
"""
import math

import numpy as np
import torch

from bbscite_gb300 import data as D
from bbscite_gb300 import native as N

MOVES = {"none": N.ERROR_BETA_WALK, "beta": N.ERROR_BETA_WALK,
         "walk": N.ERROR_RANDOM_WALK, "langevin": N.ERROR_LANGEVIN}
SCORES = {"max": N.SCORE_MAX, "sum": N.SCORE_SUM}

# (genes x cells x chains x steps) of the largest chain workload listed
LARGEST = 255 * 512 * 1024 * 1000


def listed():
    return [
        # one tree scored at a time: a caller with its own search loop, where
        # the latency of a call counts
        dict(name="score one tree 95x96", kind="score", genes=95, cells=96,
             trees=1, attach=False),
        # a batch of trees with counts and attachments
        dict(name="score 4096 trees 95x96", kind="score", genes=95, cells=96,
             trees=4096, attach=True),
        # the widest rows
        dict(name="score 1500 trees 255x512", kind="score", genes=255,
             cells=512, trees=1500, attach=False),
        # the sum score and its adjoint, as the gradient check takes it
        dict(name="adjoint 4096 trees 95x96", kind="grad", genes=95, cells=96,
             trees=4096, posterior=False),
        # attachment posteriors of a few trees, odd sizes
        dict(name="posteriors 50 trees 61x201", kind="grad", genes=61,
             cells=201, trees=50, posterior=True),
        # realised moves and the proposed trees of a batch
        dict(name="moves 3000 trees 127x64", kind="moves", genes=127,
             cells=64, trees=3000),
        # the small command-line job from random trees: 8 chains, few blocks
        dict(name="job 63x64 8 chains", kind="job", genes=63, cells=64,
             chains=8, steps=2000, score="max", move="none"),
        # the largest size of the reference's FPGA build: fixed rates
        dict(name="plain 95x96 1024 chains", kind="plain", genes=95,
             cells=96, chains=1024, steps=8000, score="max", move="none",
             warm=20000, tune=True),
        # the same data with the sum score, learning both rates
        dict(name="langevin 95x96 1024 chains", kind="batch", genes=95,
             cells=96, chains=1024, steps=8000, score="sum", move="langevin",
             warm=20000, tune=True),
        # many uneven datasets in one launch
        dict(name="mix of 128 datasets", kind="mix", datasets=128, sizes=512,
             chains=32, steps=2000, warm=2000, tune=True),
        # beyond the FPGA's caps
        dict(name="plain 255x512 1024 chains", kind="plain", genes=255,
             cells=512, chains=1024, steps=1000, score="max", move="none",
             warm=4000, tune=True),
        dict(name="langevin 255x512 1024 chains", kind="batch", genes=255,
             cells=512, chains=1024, steps=1000, score="sum",
             move="langevin", warm=4000, tune=True),
    ]


def _spread(rng, lo, hi):
    """An integer in [lo, hi], even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo),
                                                          math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["score", "grad", "moves", "job", "plain", "plain",
                       "batch", "batch", "mix"])
    genes, cells = _spread(rng, 8, 255), _spread(rng, 8, 512)
    if kind == "mix":
        return dict(kind=kind, datasets=_spread(rng, 2, 96),
                    sizes=rng.randrange(1 << 20), chains=_spread(rng, 4, 32),
                    steps=_spread(rng, 100, 2000), warm=2000,
                    tune=rng.random() < 0.7)
    if kind == "score":
        trees = _spread(rng, 1, max(1, min(8192, 2 * 10**8 // (genes * cells))))
        return dict(kind=kind, genes=genes, cells=cells, trees=trees,
                    attach=rng.random() < 0.5)
    if kind == "grad":
        trees = _spread(rng, 1, max(1, min(4096, 4 * 10**7 // (genes * cells))))
        return dict(kind=kind, genes=genes, cells=cells, trees=trees,
                    posterior=trees * genes * cells < 10**6
                    and rng.random() < 0.5)
    if kind == "moves":
        return dict(kind=kind, genes=genes, cells=64,
                    trees=_spread(rng, 1, 8192))
    score = rng.choice(["max", "sum"])
    move = rng.choice(["none", "beta", "walk", "langevin"])
    if kind == "job":
        return dict(kind=kind, genes=genes, cells=cells,
                    chains=_spread(rng, 1, 64), steps=_spread(rng, 200, 3000),
                    score=score, move=move)
    chains = _spread(rng, 16, 4096)
    most = min(8000, LARGEST // (3 * genes * cells * chains))
    steps = _spread(rng, 50, max(60, most))
    return dict(kind=kind, genes=genes, cells=cells, chains=chains,
                steps=steps, score=score, move=move, warm=2 * steps,
                tune=rng.random() < 0.5)


def _dataset(rng, genes, cells):
    """Bit rows of a generated dataset and its error rates."""
    alpha = float(10 ** rng.uniform(-5, -2))
    beta = float(rng.uniform(0.05, 0.45))
    m, _, _ = D.generate_dataset(int(rng.integers(1 << 31)), genes, cells,
                                 alpha, beta, float(rng.uniform(0.0, 0.15)),
                                 0.02)
    mut, known = D.matrix_to_bits(m)
    return mut, known, alpha, beta


def _mix_sizes(case):
    """(genes, cells) of each dataset of a mix."""
    rng = np.random.default_rng(case["sizes"])
    return [(int(rng.integers(16, 128)), int(rng.integers(16, 257)))
            for _ in range(case["datasets"])]


def _params(rng, case, alpha, beta):
    more = {}
    if case["move"] != "none":
        more = dict(prob_beta_change=0.1)
    if case["move"] in ("walk", "langevin"):  # the rates are learned
        alpha, beta = 1e-2, 0.3
    return N.default_params(alpha_mean=alpha, beta_mean=beta,
                            seed=int(rng.integers(1 << 62)),
                            score_mode=SCORES[case["score"]],
                            error_move=MOVES[case["move"]], **more)


def _trees(rng, genes, trees):
    """Ancestor rows of random trees."""
    parents = N.random_parents(int(rng.integers(1 << 62)), genes, trees)
    return np.stack([N.parent_to_matrix(p)[1] for p in parents])


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "mix":
        data, params = [], []
        for genes, cells in _mix_sizes(case):
            mut, known, alpha, beta = _dataset(rng, genes, cells)
            data.append((mut, known, cells, genes))
            params.append(N.default_params(alpha_mean=alpha, beta_mean=beta,
                                           seed=int(rng.integers(1 << 62))))
        handle = N.Batch(data, params)
        handle.init_chains(case["chains"])
        handle.run(case["warm"])
        if case["tune"]:
            handle.autotune(64)
        return dict(case=case, handle=handle)
    genes, cells = case["genes"], case["cells"]
    mut, known, alpha, beta = _dataset(rng, genes, cells)
    if kind in ("plain", "batch", "job"):
        params = _params(rng, case, alpha, beta)
        if kind == "batch":
            handle = N.Batch([(mut, known, cells, genes)], params)
        else:
            handle = N.Context(mut, known, cells, genes, params)
        if kind != "job":
            handle.init_chains(case["chains"])
            handle.run(case["warm"])
            if case["tune"]:
                handle.autotune(32)
        return dict(case=case, handle=handle)
    state = dict(case=case)
    state["handle"] = N.Context(mut, known, cells, genes,
                                N.default_params(alpha_mean=alpha,
                                                 beta_mean=beta))
    trees = case["trees"]
    state["rows"] = _trees(rng, genes, trees)
    state["beta"] = rng.uniform(0.05, 0.45, trees).astype(np.float32)
    if kind == "grad":
        state["alpha"] = (10 ** rng.uniform(-5, -2, trees)).astype(np.float32)
    if kind == "moves":
        raw = np.zeros(trees, dtype=N.RAW_MOVE)
        raw["move_type"] = rng.choice(4, trees, p=[0.05, 0.5, 0.35, 0.1])
        raw["raw_v"] = rng.integers(0, genes, trees)
        w = rng.integers(0, genes - 1, trees)
        raw["raw_w"] = w + (w >= raw["raw_v"])
        for name in ("raw_descendant_of_v", "raw_nondescendant_of_v",
                     "acceptance_level"):
            raw[name] = rng.random(trees, dtype=np.float32) * np.float32(0.999)
        raw["beta_jump"] = rng.normal(0, 0.01, trees)
        state["raw"] = raw
    # exact() makes the same inputs again and needs their sources
    state["source"] = (mut, known, alpha, beta)
    return state


def run(state):
    case, handle = state["case"], state["handle"]
    kind = case["kind"]
    if kind == "score":
        scores, counts, attach = handle.score_trees(
            state["rows"], state["beta"], attach=case["attach"])
        return dict(scores=scores, counts=counts, attach=attach)
    if kind == "grad":
        logl, da, db, post = handle.sumscore_grad(
            state["rows"], state["alpha"], state["beta"],
            posterior=case["posterior"])
        return dict(logl=logl, dalpha=da, dbeta=db, posterior=post)
    if kind == "moves":
        params, rows, betas = handle.apply_moves(state["rows"], state["beta"],
                                                 raw=state["raw"])
        return dict(rows=rows, betas=betas,
                    **{k: params[k] for k in N.MOVE_PARAMS.names})
    if kind == "job":
        handle.init_chains(case["chains"])
    handle.run(case["steps"])
    if kind in ("plain", "job"):
        return dict(best=handle.best(), chains=handle.chains())
    image = np.frombuffer(handle.save_chains(), dtype=np.uint8)
    if kind == "batch":
        return dict(best=handle.best(0), chains=image)
    # of a mix: every dataset's best tree, one array of each kind
    best = [handle.best(d) for d in range(case["datasets"])]
    return dict(
        rows=np.concatenate([b["dm"].ravel() for b in best]),
        parents=np.concatenate([b["parent"] for b in best]),
        **{k: np.array([b[k] for b in best], dtype=np.float32)
           for k in ("alpha", "beta", "score")},
        chains=image)


def work(case):
    """Each row, state and result once; per (cell, node) pair of an
    evaluated tree one addition and one comparison for the max score, and
    for the sum score an addition, a power and three sums."""
    kind = case["kind"]
    if kind == "mix":
        chains = case["chains"]
        out = dict(bytes=0.0, flops=0.0)
        for genes, cells in _mix_sizes(case):
            n, row = genes + 1, 8 * N.words(genes + 1)
            out["bytes"] += 2.0 * cells * row + chains * (3.0 * n * row + 256)
            out["flops"] += 2.0 * chains * case["steps"] * cells * n
        return out
    n, cells = case["genes"] + 1, case["cells"]
    row = 8 * N.words(n)
    data = 2.0 * cells * row
    if kind == "moves":
        return dict(bytes=case["trees"] * (2.0 * n * row + 72), flops=0.0)
    if kind in ("score", "grad"):
        trees = case["trees"]
        out = 4.0 + 32 if kind == "score" else 12.0
        if case.get("attach"):
            out += 4.0 * cells
        if case.get("posterior"):
            out += 4.0 * cells * n
        per = 2.0 if kind == "score" else 5.0
        return dict(bytes=data + trees * (n * row + 8 + out),
                    flops=per * trees * cells * n)
    chains = case["chains"]
    per = 2.0 if case["score"] == "max" else 5.0
    return dict(bytes=data + chains * (3.0 * n * row + 2 * 128),
                flops=per * chains * case["steps"] * cells * n)


def _bits(rows, n):
    """Bit rows as a float64 0/1 tensor on the GPU."""
    rows = np.ascontiguousarray(rows)
    b = np.unpackbits(rows.view(np.uint8), axis=-1, bitorder="little")[..., :n]
    return torch.from_numpy(np.ascontiguousarray(b)).cuda().double()


def exact(case, seed):
    """Scores, gradients and posteriors in 64 bits; chains and moves have no
    such value (their trees are whole numbers that follow from a stream of
    decisions)."""
    kind = case["kind"]
    if kind not in ("score", "grad"):
        return None
    state = prepare(case, seed)
    mut, known, alpha, beta_mean = state["source"]
    genes, trees = case["genes"], case["trees"]
    n = genes + 1
    K, M = _bits(known, n)[:, :genes], _bits(mut, n)[:, :genes]
    zero, one = K - K * M, K * M
    pd, pm = zero.sum(1)[:, None], one.sum(1)[:, None]
    be = torch.from_numpy(state["beta"]).cuda().double()
    if kind == "grad":
        al = torch.from_numpy(state["alpha"]).cuda().double()
    else:
        al = torch.full_like(be, float(np.float32(alpha)))
    l00, l10 = torch.log1p(-al), torch.log(al)
    l01, l11 = torch.log(be), torch.log1p(-be)
    if kind == "score":
        # Beta prior of the mean and standard deviation 0.1
        mean = float(np.float32(beta_mean))
        sd = float(np.float32(0.1))
        pa = (1 - mean) * mean * mean / (sd * sd) - mean
        pb = pa * (1 / mean - 1)
        prior = (math.lgamma(pa + pb) - math.lgamma(pa) - math.lgamma(pb)
                 + (pa - 1) * torch.log(be) + (pb - 1) * torch.log1p(-be))
    step = max(1, 4 * 10**7 // (case["cells"] * n))
    outs = []
    for t0 in range(0, trees, step):
        t = slice(t0, min(trees, t0 + step))
        A = _bits(state["rows"][t], n)[:, :, :genes]   # trees x nodes x genes
        d = torch.einsum("cg,tng->tcn", zero, A)
        m = torch.einsum("cg,tng->tcn", one, A)
        v = [x[t][:, None, None] for x in (l00, l01, l10, l11)]
        s = (pd - d) * v[0] + d * v[1] + (pm - m) * v[2] + m * v[3]
        if kind == "score":
            outs.append((s.amax(2).sum(1) + prior[t],))
            continue
        lse = torch.logsumexp(s, 2)
        post = torch.exp(s - lse[:, :, None])
        e01, e11 = (post * d).sum((1, 2)), (post * m).sum((1, 2))
        e00, e10 = pd.sum() - e01, pm.sum() - e11
        outs.append((lse.sum(1), -e00 / (1 - al[t]) + e10 / al[t],
                     e01 / be[t] - e11 / (1 - be[t]),
                     post if case["posterior"] else None))
    outs = [None if any(x is None for x in p) else torch.cat(p).cpu().numpy()
            for p in zip(*outs)]
    if kind == "score":
        return dict(scores=outs[0], counts=None, attach=None)
    return dict(logl=outs[0], dalpha=outs[1], dbeta=outs[2],
                posterior=outs[3])

"""Chains that read proposals off a table of every node (rows of up to four
words): exact counts, scores and trees at the edges of the table's groups and
chunks, at rates whose integer codes tie, are near their margin or do not
exist, and without a trace (proposals rejected by a bound) as with one."""
import os
import subprocess

import numpy as np
import pytest

from bbscite_gb300 import data as D

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _setup(G, Cn, seed=3):
    m, _, _ = D.generate_dataset(seed * 1000 + G * 7 + Cn, G, Cn, 2e-3, 0.2,
                                 0.1, 0.02)
    return D.matrix_to_bits(m)


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn,launch,alpha,beta", [
    (2, 1, (1, 1, 1), 1e-3, 0.2),       # the smallest problem
    (7, 40, (2, 1, 2), 1e-3, 0.2),      # one group of eight nodes
    (8, 33, (1, 2, 1), 1e-5, 0.4),      # a ragged group, two warps
    (32, 129, (1, 1, 4), 1e-3, 0.2),    # five chunks, the last of one cell
    (95, 200, (3, 1, 2), 6e-5, 0.43),   # three chunks of 96
    (127, 256, (2, 4, 1), 1e-3, 0.2),   # the widest table, four warps
    (40, 64, (2, 1, 2), 0.2, 0.2),      # every fraction ties: ratio 1
    (40, 64, (2, 1, 2), 0.125, 0.5),    # few distinct logs
    (40, 64, (2, 1, 2), 0.7, 0.6),      # alpha + beta above 1: signs turn
    (30, 40, (2, 1, 2), 0.5, 0.5),      # no codes: every node scores alike
])
def test_max_chains_match_the_oracle(native, orc, G, Cn, launch, alpha, beta):
    mut, known = _setup(G, Cn)
    chains, steps = 3, 120
    p = native.default_params(alpha_mean=alpha, beta_mean=beta, seed=11)
    rng = np.random.default_rng(G)
    starts = np.stack([D.random_parent_vector(rng, G) for _ in range(chains)])
    out = []
    for trace in (True, False):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(chains, starts)
            c.set_launch(*launch)
            tr = c.run(steps, trace=trace)
            out.append((c.chains(), c.best()))
            if trace:
                t = tr
    (a, ab), (b, bb) = out
    for k in ("dm", "score", "counts", "beta"):
        np.testing.assert_array_equal(a[k], b[k])
    assert ab["score"] == bb["score"] and (ab["dm"] == bb["dm"]).all()
    for ch in range(chains):
        raws = np.zeros(steps, dtype=orc.RAW_MOVE)
        raws.view(np.uint8)[:] = np.frombuffer(t["move"][ch].tobytes(),
                                               dtype=np.uint8)
        res = orc.run_chain(alpha, beta, 0.1, 1.0, starts[ch], mut, known,
                            raws, score_mode=1, forced=t["accepted"][ch],
                            ambiguity=1e-5)
        np.testing.assert_array_equal(res["trace"]["counts"],
                                      t["proposed_counts"][ch])
        assert (res["dm"] == a["dm"][ch]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("score", ["max", "sum"])
@pytest.mark.parametrize("move", ["beta_walk", "langevin"])
@pytest.mark.parametrize("G,Cn,q", [(2, 3, 1), (31, 32, 1), (64, 70, 3),
                                    (95, 96, 3), (127, 128, 4)])
def test_untraced_chains_equal_traced_ones(native, score, move, G, Cn, q):
    """The sum score's bound and the near-tie margin of the max score reject
    proposals without evaluating them; a traced chain evaluates every one."""
    mut, known = _setup(G, Cn, 5)
    p = native.default_params(
        alpha_mean=1e-2, beta_mean=0.3, seed=29, prob_beta_change=0.15,
        score_mode=getattr(native, "SCORE_" + score.upper()),
        error_move=getattr(native, "ERROR_" + move.upper()))
    got = []
    for trace in (False, True):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(8)
            c.set_launch(q, 1, 1)
            for steps in (1, 37, 400):
                c.run(steps, trace=trace)
            got.append((c.chains(), c.best(), c.save_chains()))
    assert got[0][2] == got[1][2]
    assert got[0][1]["score"] == got[1][1]["score"]


@pytest.mark.gpu
@pytest.mark.parametrize("move", ["beta_walk", "langevin"])
@pytest.mark.parametrize("G,Cn", [(8, 12), (8, 13), (31, 12), (31, 13),
                                  (32, 12), (62, 9), (127, 4)])
def test_few_cells_give_the_same_in_company(native, move, G, Cn):
    """Sum-score chains of few cells alone, on either side of the sizes that
    take a table, and in a launch with a larger dataset, which decides for
    both; n - 1 nodes with every remainder of the sum's groups of four."""
    sets, params = [], []
    for k, (g, c) in enumerate([(G, Cn), (G, 40)]):
        mut, known = _setup(g, c, 5 + k)
        sets.append((mut, known, c, g))
        params.append(native.default_params(
            alpha_mean=1e-2, beta_mean=0.3, seed=31 + k, prob_beta_change=0.15,
            score_mode=native.SCORE_SUM,
            error_move=getattr(native, "ERROR_" + move.upper())))
    got = []
    for who in ([0], [0, 1]):
        with native.Batch([sets[k] for k in who],
                          [params[k] for k in who]) as b:
            b.init_chains(4)
            b.set_launch(2, 4, 1)
            for steps in (1, 50, 300):
                b.run(steps)
            got.append(b.best(0))
    assert got[0]["score"] == got[1]["score"]
    assert got[0]["alpha"] == got[1]["alpha"]
    assert (got[0]["dm"] == got[1]["dm"]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 4, 0, 1), (4, 2, 1, 1), (2, 4, 0, 4)])
def test_mixed_batches_equal_their_datasets_alone(native, shape):
    """Datasets of one launch with one to eight chunks of cells."""
    sizes = [(33, 17), (40, 250), (63, 64), (60, 129), (20, 31), (127, 200)]
    data = [_setup(G, Cn, 9 + i) + (Cn, G) for i, (G, Cn) in enumerate(sizes)]
    params = [native.default_params(alpha_mean=1e-3 * (i + 1), beta_mean=0.2,
                                    seed=70 + i) for i in range(len(sizes))]
    q, wpb, merge, wpc = shape
    with native.Batch(data, params) as b:
        b.init_chains(5)
        b.set_launch(q, wpb, merge)
        b.set_chain_warps(wpc)
        b.run(150)
        best = [b.best(d) for d in range(len(sizes))]
    for d, (G, Cn) in enumerate(sizes):
        with native.Context(*data[d], params[d]) as c:
            c.init_chains(5)
            c.run(150)
            one = c.best()
        assert one["score"] == best[d]["score"]
        assert (one["dm"] == best[d]["dm"]).all()


def test_layout_of_slots_with_tables(tmp_path):
    """Every piece of a slot with a table but no increments lies inside its
    slot, apart from the others and aligned, and the plan asks for the room."""
    from bbscite_gb300 import build as B
    exe = str(tmp_path / "table_probe")
    subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "-I" + B.INCLUDE,
                    "-I" + B.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "table_probe.cu"),
                    "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("tables ok "), r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn,launch", [
    (128, 40, (2, 1, 2)),     # 129 nodes, the table in shared memory
    (200, 150, (1, 3, 1)),    # two chunks
    (191, 97, (2, 1, 1)),     # 192 nodes, an odd last chunk
    (255, 512, (2, 4, 1)),    # nodes past the block's room in global memory
    (255, 300, (1, 3, 1)),    # four chunks, some nodes in global memory
])
def test_wide_max_chains_equal_traced_ones(native, G, Cn, launch):
    """Rows of five to eight words at fixed rates: chains on a table against
    traced ones, which evaluate every node through the ring."""
    mut, known = _setup(G, Cn, 7)
    p = native.default_params(alpha_mean=1e-3, beta_mean=0.2, seed=31)
    got = []
    for trace in (False, True):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(5)
            c.set_launch(*launch)
            for steps in (1, 60, 200):
                c.run(steps, trace=trace)
            got.append((c.chains(), c.best(), c.save_chains()))
    assert got[0][2] == got[1][2]
    assert got[0][1]["score"] == got[1][1]["score"]


@pytest.mark.gpu
@pytest.mark.parametrize("score", ["max", "sum"])
@pytest.mark.parametrize("G,Cn,chains", [(8, 70, 700), (31, 96, 40),
                                         (63, 200, 3), (95, 96, 1200),
                                         (127, 130, 400), (127, 400, 5)])
def test_default_shapes_give_the_chains_of_one_warp(native, score, G, Cn,
                                                    chains):
    """The shape chosen without tuning, few and many chains, one and more
    passes over the cells, leaves every chain as one-warp blocks of one cell
    per lane do."""
    mut, known = _setup(G, Cn, 7)
    p = native.default_params(alpha_mean=1e-2, beta_mean=0.3, seed=41,
                              prob_beta_change=0.1,
                              score_mode=getattr(native,
                                                 "SCORE_" + score.upper()))
    images = []
    for shape in (None, (1, 1, 1)):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(chains)
            if shape:
                c.set_launch(*shape)
            c.run(40)
            images.append(c.save_chains())
    assert images[0] == images[1]


@pytest.mark.gpu
def test_blocks_whose_counts_do_not_fit_are_refused(native):
    """Eight chains of 96 nodes and 96 cells at three cells per lane have no
    room for their counts, although they would without a table."""
    mut, known = _setup(95, 96, 7)
    with native.Context(mut, known, 96, 95) as c:
        c.init_chains(8)
        c.set_launch(3, 1, 8)
        with pytest.raises(native.BbsError):
            c.run(10)
        c.set_launch(3, 1, 7)
        c.run(10)


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn", [(20, 64), (20, 65), (63, 97), (127, 128),
                                  (40, 129)])
def test_untuned_sum_batches_equal_their_chains_alone(native, G, Cn):
    """Two, three and four cells per lane by default, and more cells than one
    pass takes."""
    mut, known = _setup(G, Cn, 9)
    p = native.default_params(alpha_mean=1e-2, beta_mean=0.3, seed=43,
                              prob_beta_change=0.1,
                              score_mode=native.SCORE_SUM)
    with native.Batch([(mut, known, Cn, G)], p) as b:
        b.init_chains(6)
        b.run(120)
        batch = b.best(0)
    with native.Context(mut, known, Cn, G, p) as c:
        c.init_chains(6)
        c.set_launch(1, 1, 1)
        c.run(120)
        one = c.best()
    assert one["score"] == batch["score"]
    assert (one["dm"] == batch["dm"]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["far", "high"])
def test_the_sum_scores_bound_is_a_bound(tmp_path, kind):
    """Proposals bounded and summed by the chain kernels' own functions, at
    cells far below their reference with nodes at the end of the range of
    normal floats, and at gains beyond what a lane counts
    (tests/cpp/bound_probe.cu)."""
    from bbscite_gb300 import build as B
    exe = str(tmp_path / "bound_probe")
    subprocess.run([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "-I" + B.INCLUDE,
                    "-I" + B.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "bound_probe.cu"),
                    "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe, kind], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("bound ok "), r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("move", ["beta_walk", "langevin"])
@pytest.mark.parametrize("G,Cn,q,alpha", [(95, 96, 3, 1e-4), (95, 96, 3, 1e-5),
                                          (111, 60, 2, 1e-4),
                                          (126, 128, 4, 1e-5)])
def test_first_steps_at_small_rates_equal_traced_ones(native, move, G, Cn, q,
                                                      alpha):
    """Random trees and rates far below them: the first steps pass cells whose
    best node lies far below their reference."""
    mut, known = _setup(G, Cn, 5)
    p = native.default_params(
        alpha_mean=alpha, beta_mean=0.3, seed=59, prob_beta_change=0.05,
        score_mode=native.SCORE_SUM,
        error_move=getattr(native, "ERROR_" + move.upper()))
    got = []
    for trace in (False, True):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(1000)
            c.set_launch(q, 1, 1)
            for steps in (30, 100):
                c.run(steps, trace=trace)
            got.append(c.save_chains())
    assert got[0] == got[1]


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn,warps,chain_warps", [
    (95, 96, 8, 1), (127, 128, 6, 1), (127, 128, 7, 1), (127, 96, 4, 4)])
def test_untuned_sum_batches_take_any_warps(native, G, Cn, warps, chain_warps):
    """Warps set without cells per lane: where as many cells per lane as a pass
    takes leave the block no room, two do."""
    mut, known = _setup(G, Cn, 9)
    p = native.default_params(alpha_mean=1e-2, beta_mean=0.3, seed=43,
                              prob_beta_change=0.1,
                              score_mode=native.SCORE_SUM)
    got = []
    for shape in (None, (warps, chain_warps)):
        with native.Batch([(mut, known, Cn, G)], p) as b:
            if shape:
                b.set_launch(warps_per_block=warps)
            b.init_chains(10)
            if shape:
                b.set_chain_warps(chain_warps)
                assert b.launch()[0] == 2
            b.run(60)
            got.append(b.save_chains())
    assert got[0] == got[1]


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn,chains,part", [
    (63, 64, 8, dict(chains_per_block=8)),
    (20, 33, 1024, dict(chains_per_block=6)),
    (95, 96, 1024, dict(cells_per_lane=1)),
    (111, 128, 40, dict(warps_per_chain=4)),
])
def test_parts_of_a_shape_are_accepted(native, G, Cn, chains, part):
    """A shape of which the caller sets a part runs, whatever the default for
    the rest."""
    mut, known = _setup(G, Cn, 9)
    for score in (native.SCORE_MAX, native.SCORE_SUM):
        p = native.default_params(alpha_mean=1e-3, beta_mean=0.2, seed=43,
                                  score_mode=score)
        got = []
        for kw in ({}, part):
            with native.Context(mut, known, Cn, G, p) as c:
                c.init_chains(chains)
                if kw:
                    c.set_launch(**kw)
                c.run(20)
                got.append(c.save_chains())
        assert got[0] == got[1]


def _ms_a_run(native, mut, known, Cn, G, chains, steps, runs=1, launch=None,
              **kw):
    """Device time of `runs` runs of `steps` steps, the least of several."""
    p = native.default_params(seed=5, **kw)
    with native.Context(mut, known, Cn, G, p) as c:
        c.init_chains(chains)
        if launch:
            c.set_launch(*launch)
        c.run(500)
        times = []
        for _ in range(5):
            t = 0.0
            for _ in range(runs):
                c.run(steps)
                t += c.last_run_ms()
            times.append(t)
    return min(times)


# rates whose codes tie at every sixth count: log(1 - alpha) - log(beta) is a
# sixth of log(1 - beta) - log(alpha)
TIES = dict(alpha_mean=0.000511870, beta_mean=0.3)


@pytest.mark.gpu
def test_wide_chains_with_codes_that_tie_cost_no_more_than_the_ring(native):
    """255 x 512 at rates whose codes tie, against the same chains with error
    moves that never come, which take the ring."""
    mut, known = _setup(255, 512, 7)
    ties = _ms_a_run(native, mut, known, 512, 255, 128, 100, **TIES)
    ring = _ms_a_run(native, mut, known, 512, 255, 128, 100,
                     prob_beta_change=1e-6, **TIES)
    assert ties <= 1.3 * ring, (ties, ring)


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn,launch", [
    (150, 100, (1, 4, 1)),   # codes, the proposals they leave from the rows
    (200, 150, (2, 3, 1)),   # the ring
])
def test_wide_chains_with_codes_that_tie_equal_traced_ones(native, G, Cn,
                                                           launch):
    mut, known = _setup(G, Cn, 7)
    p = native.default_params(seed=31, **TIES)
    got = []
    for trace in (False, True):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(5)
            c.set_launch(*launch)
            for steps in (2, 60, 200):
                c.run(steps, trace=trace)
            got.append(c.save_chains())
    assert got[0] == got[1]


@pytest.mark.gpu
@pytest.mark.parametrize("share", [0.0, 1.0, 50.0])
@pytest.mark.parametrize("move", ["beta_walk", "langevin"])
@pytest.mark.parametrize("G,Cn,launch", [
    (127, 33, (1, 2, 1)),    # the most nodes, a last cell of its own
    (126, 64, (2, 1, 2)),    # an odd number of nodes
    (95, 97, (2, 1, 1)),     # two chunks, the last of one cell
    (63, 200, (1, 2, 1)),    # four chunks
    (112, 128, (1, 4, 1)),   # four warps
])
def test_chains_on_tables_of_counts_equal_traced_ones(native, share, move, G,
                                                      Cn, launch):
    """Error moves as many as tree moves and fifty times as many, and none at
    rates without codes: tables of counts against evaluations from the rows."""
    mut, known = _setup(G, Cn, 5)
    p = native.default_params(
        alpha_mean=1e-2 if share else 0.5, beta_mean=0.3 if share else 0.5,
        seed=29, prob_beta_change=share,
        error_move=getattr(native, "ERROR_" + move.upper()))
    got = []
    for trace in (False, True):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(8)
            c.set_launch(*launch)
            for steps in (3, 37, 300):
                c.run(steps, trace=trace)
            got.append(c.save_chains())
    assert got[0] == got[1]


@pytest.mark.gpu
def test_mixed_batches_on_tables_of_counts_equal_their_datasets_alone(native):
    """A launch group most of whose datasets are better off with counts runs
    the others on counts too."""
    sizes = [(100, 90), (120, 64), (127, 200), (97, 40)]
    data = [_setup(G, Cn, 9 + i) + (Cn, G) for i, (G, Cn) in enumerate(sizes)]
    params = [native.default_params(alpha_mean=1e-2, beta_mean=0.3,
                                    prob_beta_change=0.1 if i == 1 else 2.0,
                                    error_move=native.ERROR_RANDOM_WALK,
                                    seed=70 + i) for i in range(len(sizes))]
    with native.Batch(data, params) as b:
        b.init_chains(5)
        b.run(150)
        best = [b.best(d) for d in range(len(sizes))]
    for d, (G, Cn) in enumerate(sizes):
        with native.Context(*data[d], params[d]) as c:
            c.init_chains(5)
            c.set_launch(1, 1, 1)
            c.run(150)
            one, alpha = c.best(), c.best_alpha()
        assert alpha == best[d]["alpha"]
        for k in ("score", "beta"):
            assert one[k] == best[d][k]
        assert (one["dm"] == best[d]["dm"]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn,chains,launch,share,most", [
    # many small chains: a step with one error move in eleven, and without
    (8, 24, 2432, None, 0.1, 1.5),
    # error moves as many as tree moves
    (95, 96, 1024, (3, 1, 7), 1.0, 4.8),
])
def test_error_moves_cost_what_they_should(native, G, Cn, chains, launch, share,
                                           most):
    """Against the same chains at fixed rates."""
    mut, known = _setup(G, Cn, 5)
    kw = dict(alpha_mean=1e-2, beta_mean=0.2)
    fixed = _ms_a_run(native, mut, known, Cn, G, chains, 200, launch=launch,
                      **kw)
    moved = _ms_a_run(native, mut, known, Cn, G, chains, 200, launch=launch,
                      prob_beta_change=share,
                      error_move=native.ERROR_LANGEVIN, **kw)
    assert moved <= most * fixed, (moved, fixed)


@pytest.mark.gpu
@pytest.mark.parametrize("steps,most", [(1, 1.4), (4, 1.2)])
def test_short_runs_make_no_table_for_a_few_steps(native, steps, most):
    """Runs of a few steps at 255 x 512, against chains that take the ring."""
    mut, known = _setup(255, 512, 7)
    kw = dict(alpha_mean=1e-3, beta_mean=0.2)
    table = _ms_a_run(native, mut, known, 512, 255, 128, steps, 40, **kw)
    ring = _ms_a_run(native, mut, known, 512, 255, 128, steps, 40,
                     prob_beta_change=1e-6, **kw)
    assert table <= most * ring, (table, ring)


@pytest.mark.gpu
@pytest.mark.parametrize("score", ["max", "sum"])
@pytest.mark.parametrize("G,Cn,launch", [(63, 64, (2, 1, 2)), (95, 97, (2, 1, 1)),
                                         (200, 40, (2, 1, 1)),
                                         (255, 512, (2, 4, 1))])
def test_short_runs_equal_one_long_one(native, score, G, Cn, launch):
    mut, known = _setup(G, Cn, 5)
    p = native.default_params(alpha_mean=1e-3, beta_mean=0.2, seed=29,
                              score_mode=getattr(native,
                                                 "SCORE_" + score.upper()))
    got = []
    for runs in ([36], [1, 2, 3, 4, 6, 7, 13]):
        with native.Context(mut, known, Cn, G, p) as c:
            c.init_chains(6)
            c.set_launch(*launch)
            for steps in runs:
                c.run(steps)
            got.append(c.save_chains())
    assert got[0] == got[1]

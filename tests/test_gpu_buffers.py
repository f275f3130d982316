"""The calls on host buffers give the same results whether an array crosses
through the pinned mirror (small arrays) or straight from the caller's memory:
a batch equals its trees taken a few at a time."""
import numpy as np
import pytest

from bbscite_gb300 import data as D


@pytest.mark.gpu
@pytest.mark.parametrize("G,trees", [(63, 127), (63, 129), (95, 600),
                                     (255, 40)])
def test_large_and_small_arrays_give_the_same(native, G, trees):
    Cn = 33
    m, _, _ = D.generate_dataset(G, G, Cn, 1e-3, 0.2, 0.1, 0.02)
    mut, known = D.matrix_to_bits(m)
    parents = native.random_parents(5, G, trees)
    dm = np.stack([native.parent_to_matrix(x)[1] for x in parents])
    rng = np.random.default_rng(2)
    al = rng.uniform(1e-4, 1e-2, trees).astype(np.float32)
    be = rng.uniform(0.1, 0.4, trees).astype(np.float32)
    raw = np.zeros(trees, dtype=native.RAW_MOVE)
    raw["move_type"] = rng.integers(0, 4, trees)
    raw["raw_v"] = rng.integers(0, G // 2, trees)
    raw["raw_w"] = rng.integers(G // 2, G, trees)
    raw["raw_descendant_of_v"] = raw["raw_nondescendant_of_v"] = 0.4
    with native.Context(mut, known, Cn, G) as c:
        def calls(t):
            return (*c.score_trees(dm[t], be[t], attach=True),
                    *c.sumscore_grad(dm[t], al[t], be[t], posterior=True),
                    *c.apply_moves(dm[t], be[t], raw=raw[t]))
        whole = calls(slice(0, trees))
        parts = [calls(slice(k, min(trees, k + 7)))
                 for k in range(0, trees, 7)]
    for i, w in enumerate(whole):
        np.testing.assert_array_equal(w, np.concatenate([p[i] for p in parts]))


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn", [(2, 1), (3, 33), (63, 129), (128, 64),
                                  (159, 65), (255, 200)])
def test_many_trees_score_as_few_do(native, orc, G, Cn):
    """Calls above and below the number of trees that get a block each, on
    random trees, a star (its order does not fit the ring), a path, rates
    whose codes tie (beta = alpha) and rows that are no tree; a few against
    the oracle."""
    trees, n = 340, G + 1
    m, _, _ = D.generate_dataset(G, G, Cn, 1e-2, 0.2, 0.1, 0.02)
    mut, known = D.matrix_to_bits(m)
    parents = native.random_parents(9, G, trees)
    parents[3] = n - 1                                  # a star
    parents[5] = np.minimum(np.arange(n) + 1, n - 1)    # a path
    dm = np.stack([native.parent_to_matrix(x)[1] for x in parents])
    dm[7, 0, G // 128] ^= np.uint64(1 << (G // 2 % 64))  # no tree
    rng = np.random.default_rng(2)
    be = rng.uniform(0.1, 0.4, trees).astype(np.float32)
    p = native.default_params(alpha_mean=1e-2, beta_mean=0.2)
    be[11] = np.float32(1e-2)                           # every ratio ties
    with native.Context(mut, known, Cn, G, p) as c:
        whole = c.score_trees(dm, be, attach=True)
        parts = [c.score_trees(dm[k:k + 34], be[k:k + 34], attach=True)
                 for k in range(0, trees, 34)]
        bare = c.score_trees(dm, be)
    for i in range(3):
        np.testing.assert_array_equal(
            whole[i], np.concatenate([x[i] for x in parts]))
    np.testing.assert_array_equal(whole[0], bare[0])
    np.testing.assert_array_equal(whole[1], bare[1])
    for t in (0, 3, 5, 7, 11):
        _, st, oc, oatt = orc.logscore_tree(1e-2, 0.2, 0.1, dm[t], mut, known,
                                            float(be[t]))
        assert whole[0][t] == np.float32(st)
        assert (whole[1][t] == oc).all() and (whole[2][t] == oatt).all()


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn,trees", [(2, 1, 3), (31, 33, 2), (32, 257, 5),
                                        (95, 96, 40), (255, 70, 3)])
def test_adjoint_and_posteriors_match_fp64(native, orc, G, Cn, trees):
    """Odd node and cell counts of the adjoint's chunks and of the tile its
    posteriors leave through; the tolerances are those of the FP32 score
    (1e-5 relative) and of the adjoint (1e-4)."""
    m, _, _ = D.generate_dataset(G + Cn, G, Cn, 1e-3, 0.2, 0.1, 0.02)
    mut, known = D.matrix_to_bits(m)
    parents = native.random_parents(4, G, trees)
    dm = np.stack([native.parent_to_matrix(x)[1] for x in parents])
    al = np.full(trees, 1e-5, dtype=np.float32)  # far-off cells too
    al[0] = 1e-2
    be = np.linspace(0.1, 0.4, trees).astype(np.float32)
    with native.Context(mut, known, Cn, G) as c:
        lg, da, db, post = c.sumscore_grad(dm, al, be, posterior=True)
        bare = c.sumscore_grad(dm, al, be)
    for i, x in enumerate((lg, da, db)):
        np.testing.assert_array_equal(x, bare[i])
    for t in range(trees):
        f, ga, gb, po = orc.sumscore_grad_f64(float(al[t]), float(be[t]),
                                              dm[t], mut, known, posterior=True)
        assert abs(lg[t] - f) <= 1e-5 * abs(f) + 1e-4
        assert abs(da[t] - ga) <= 1e-4 * abs(ga) + 1e-2
        assert abs(db[t] - gb) <= 1e-4 * abs(gb) + 1e-3
        assert np.abs(post[t] - po).max() <= 1e-3
        np.testing.assert_allclose(post[t].sum(1), 1.0, rtol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn", [(62, 65), (63, 64), (63, 65), (95, 97),
                                  (127, 66)])
def test_walked_trees_score_as_few_do(native, orc, G, Cn):
    """Both sides of the sizes from which rows of up to four words are
    walked, odd and even ends of the walk's pairs, and the most nodes."""
    test_many_trees_score_as_few_do(native, orc, G, Cn)


@pytest.mark.gpu
@pytest.mark.parametrize("G,Cn", [(91, 100), (92, 128), (174, 64)])
def test_posteriors_whose_tiles_nearly_fill_48_kb(native, orc, G, Cn):
    """The tile alone below 48 KB, with the kernel's static shared memory
    above."""
    test_adjoint_and_posteriors_match_fp64(native, orc, G, Cn, 3)

"""The calls on host buffers give the same results whether an array crosses
through the pinned mirror (up to 64 KB) or straight from the caller's memory:
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

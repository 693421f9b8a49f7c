"""Octrees at the edges of the level builder and of the leaf ordering, bit for bit against the CPU
restatement: deep chains below the shallow key sort, more branches than first reserved, levels larger
than one cluster takes, leaves too large to be ordered by comparisons, and the smallest systems."""
import numpy as np
import pytest

import fastmultipole_b200 as fm
from fastmultipole_b200 import _lib as L
import oracle_lib as O
from test_gpu_fmm import compare_lists, compare_trees, opt_pair

pytestmark = pytest.mark.gpu


def points(x, seed=0):
    rng = np.random.default_rng(seed)
    b = np.zeros((len(x), 5))
    b[:, :3] = x
    b[:, 3] = 1e-3 * rng.random(len(x))
    b[:, 4] = rng.standard_normal(len(x))
    return b


def pairs(n, gap, seed):
    """n tight pairs: each needs a chain of one-child branches down to the gap."""
    rng = np.random.default_rng(seed)
    x = rng.random((n, 3))
    return np.concatenate([x, x + gap])[rng.permutation(2 * n)]


RNG = np.random.default_rng(4)
CASES = {
    "one_body": (RNG.random((1, 3)), 1),
    "two_bodies": (RNG.random((2, 3)), 1),
    "nine_bodies": (RNG.random((9, 3)), 1),
    "below_the_shallow_sort": (pairs(50, 2.0 ** -17, 1), 1),
    "more_branches_than_reserved": (pairs(1500, 2.0 ** -15, 2), 1),
    "levels_beyond_one_cluster": (RNG.random((40001, 3)), 1),
    "ragged_small_leaves": (RNG.random((5003, 3)) ** 3, 3),
    "leaf_of_1024": (RNG.random((1024, 3)), 1024),
    "leaf_of_1025": (RNG.random((1025, 3)), 1024),
    "leaves_beyond_comparison": (RNG.random((30011, 3)), 900),
    "line": (np.stack([np.linspace(0, 1, 777), np.zeros(777), np.zeros(777)], 1), 2),
}


@pytest.mark.parametrize("shrink", [True, False])
@pytest.mark.parametrize("name", list(CASES))
def test_tree_and_lists(name, shrink):
    x, ls = CASES[name]
    b = points(x)
    ctx = fm.Context(0)  # first build of a context: nothing reserved yet
    og, oo = opt_pair(expansion_order=2, leaf_size_source=ls, multipole_acceptance=0.5, shrink_recenter=shrink)
    for _ in range(2):
        fm.solve_buffers(b, L.FMM_POINT_SOURCE, og, ctx=ctx)
        ref = O.fmm(b, O.POINT_SOURCE, oo, want_tree=True)
        compare_trees(fm.get_tree(ctx, 1), ref["source_tree"])
        compare_lists(*fm.get_lists(ctx), ref["m2l"], ref["direct"])
    ctx.close()


def test_max_influence_of_ancestors():
    """Every branch's influence is the largest of its children's."""
    b = points(np.random.default_rng(8).random((3000, 3)))
    ctx = fm.Context(0)
    og = fm.make_options(expansion_order=6, leaf_size_source=8, error_tolerance=fm.PowerRelativeGradient(1e-5))
    fm.solve_buffers(b, L.FMM_POINT_SOURCE, og, ctx=ctx)
    t = fm.get_tree(ctx, 1)
    for k in range(t["n_branches"]):
        c0, nc = t["child_start"][k], t["n_children"][k]
        if nc:
            assert t["max_influence"][k] == t["max_influence"][c0:c0 + nc].max()
    assert t["max_influence"].min() > 0
    ctx.close()


@pytest.mark.parametrize("n,ls", [(60001, 1), (60001, 3), (200003, 40)])
def test_ancestors_enclose_finished_children(n, ls):
    """Every branch's geometry is the one its children's gives, bit for bit, build after build: a
    parent is formed by whichever child is last to finish, from what other SMs wrote."""
    b = points(np.random.default_rng(n + ls).random((n, 3)) ** 2)
    ctx = fm.Context(0)
    og = fm.make_options(expansion_order=1, leaf_size_source=ls, farfield=False, nearfield=False)
    for _ in range(5):
        fm.solve_buffers(b, L.FMM_POINT_SOURCE, og, ctx=ctx)
        t = fm.get_tree(ctx, 1)
        parents = np.flatnonzero(t["n_children"])
        first = t["child_start"][parents]
        kids = np.concatenate([np.arange(c, c + k) for c, k in zip(first, t["n_children"][parents])])
        at = np.concatenate([[0], np.cumsum(t["n_children"][parents])[:-1]])
        rep = np.repeat(np.arange(len(parents)), t["n_children"][parents])
        for c, w, r in (("target_center", "target_box", "target_radius"), ("source_center", "source_box", "source_radius")):
            lo = np.minimum.reduceat(np.minimum(t[c][kids], t[c][kids] - t[w][kids]), at)
            hi = np.maximum.reduceat(np.maximum(t[c][kids], t[c][kids] + t[w][kids]), at)
            cen = (lo + hi) * 0.5
            d = t[c][kids] - cen[rep]
            rad = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]) + t[r][kids]
            np.testing.assert_array_equal(t[c][parents], cen)
            np.testing.assert_array_equal(t[w][parents], hi - cen)
            np.testing.assert_array_equal(t[r][parents], np.maximum.reduceat(rad, at))
    ctx.close()


def test_traversals_of_changing_size():
    """One context, systems whose traversals outgrow what the previous build's let expect, and back."""
    ctx = fm.Context(0)
    rng = np.random.default_rng(9)
    for n, ls in ((900, 4), (60, 4), (30000, 4), (2500, 40), (12000, 3), (1, 1), (5000, 2)):
        b = points(rng.random((n, 3)) ** 2, n)
        og, oo = opt_pair(expansion_order=1, leaf_size_source=ls, multipole_acceptance=0.4)
        fm.solve_buffers(b, L.FMM_POINT_SOURCE, og, ctx=ctx)
        ref = O.fmm(b, O.POINT_SOURCE, oo, want_tree=True)
        compare_trees(fm.get_tree(ctx, 1), ref["source_tree"])
        compare_lists(*fm.get_lists(ctx), ref["m2l"], ref["direct"])
    ctx.close()

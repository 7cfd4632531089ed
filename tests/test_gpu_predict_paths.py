"""Margins where the prediction path changes shape: row counts around a warp's
32 rows, the part size of the upload and the trees-per-thread rule, node forms
with and without the 8-byte form (categorical splits, children apart), many
outputs, a tree limit and both kinds of missing value. Compared bit for bit with sums
in tree order over leaves found by a plain walk."""
import numpy as np
import pytest

from gpu_helpers import leaf_ids

pytestmark = pytest.mark.gpu


def _forest(sb, rng, trees, f, apart=False):
    """Trees of two levels; `apart` puts the children of the root at nodes 1 and 4."""
    nodes = np.zeros(7 * trees, sb.api.NODE_DTYPE)
    nodes["left"] = nodes["right"] = -1
    nodes["leaf_value"] = rng.standard_normal(7 * trees).astype(np.float32)
    nodes["sum_hess"] = 1.0
    kids = {0: (1, 4), 1: (2, 3), 4: (5, 6)} if apart else {0: (1, 2), 1: (3, 4), 2: (5, 6)}
    for i, (l, r) in kids.items():
        at = np.arange(trees) * 7 + i
        nodes["left"][at], nodes["right"][at] = l, r
        nodes["split_feature"][at] = rng.integers(0, f, trees)
        nodes["split_cond"][at] = rng.standard_normal(trees).astype(np.float32)
        nodes["default_left"][at] = rng.random(trees) < 0.5
    return np.arange(trees + 1, dtype=np.int64) * 7, nodes


def _margins(off, nodes, x, base, k, limit):
    out = np.full((len(x), k), np.float32(base), np.float32)
    for t in range(limit):
        nd = nodes[off[t]:off[t + 1]]
        out[:, t % k] = out[:, t % k] + nd["leaf_value"][leaf_ids(nd, [], x)]
    return out.reshape(-1)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 16_383, 16_384, 16_387])
@pytest.mark.parametrize("apart", [False, True])
def test_row_counts(sb, ctx, n, apart):
    rng = np.random.default_rng(n)
    off, nodes = _forest(sb, rng, 9, 5, apart)
    x = rng.standard_normal((n, 5)).astype(np.float32)
    x[rng.random(x.shape) < 0.2] = np.nan
    m = sb.BoostedModel.from_arrays(off, nodes, np.zeros(10, np.int64), [], 0.25, 0, 5, ctx=ctx)
    some = np.unique(np.concatenate([np.arange(min(n, 40)), np.arange(max(0, n - 40), n), np.arange(8180, min(n, 8200))]))
    got = m.predict_margin(sb.DMatrix(x))
    assert np.array_equal(got[some], _margins(off, nodes, x[some], 0.25, 1, 9))
    assert np.array_equal(m.predict(sb.DMatrix(x)), got)  # squared error: the identity


@pytest.mark.parametrize("k,trees", [(1, 1), (1, 255), (1, 257), (3, 300), (16, 48), (17, 51)])
@pytest.mark.parametrize("limit", [0, 5])
def test_outputs_and_limits(sb, ctx, k, trees, limit):
    rng = np.random.default_rng(k * 1000 + trees)
    off, nodes = _forest(sb, rng, trees, 7)
    x = rng.standard_normal((70, 7)).astype(np.float32)
    m = sb.BoostedModel.from_arrays(off, nodes, np.zeros(trees + 1, np.int64), [], -0.5, 0 if k == 1 else k, 7,
                                    objective="multi:softprob" if k > 1 else "reg:squarederror", ctx=ctx)
    got = m.predict_margin_limited(sb.DMatrix(x), limit)
    assert np.array_equal(got, _margins(off, nodes, x, -0.5, k, min(limit, trees) if limit else trees))


def test_missing_value_that_is_a_number(sb, ctx):
    """`missing` = -1: such entries take the default direction; NaN is not
    missing then, and compares false (right)."""
    rng = np.random.default_rng(8)
    off, nodes = _forest(sb, rng, 40, 4)
    x = rng.standard_normal((65, 4)).astype(np.float32)
    x[rng.random(x.shape) < 0.2] = -1.0
    x[rng.random(x.shape) < 0.2] = np.nan
    m = sb.BoostedModel.from_arrays(off, nodes, np.zeros(41, np.int64), [], 0.0, 0, 4, ctx=ctx)
    seen = np.where(np.isnan(x), np.float32(np.inf), np.where(x == -1.0, np.float32(np.nan), x))  # right / default
    assert np.array_equal(m.predict_margin(sb.DMatrix(x, missing=-1.0)), _margins(off, nodes, seen, 0.0, 1, 40))


def test_wide_rows(sb, ctx):
    """Rows too wide to stage in shared memory."""
    rng = np.random.default_rng(9)
    off, nodes = _forest(sb, rng, 30, 2_000)
    x = rng.standard_normal((50, 2_000)).astype(np.float32)
    m = sb.BoostedModel.from_arrays(off, nodes, np.zeros(31, np.int64), [], 0.0, 0, 2_000, ctx=ctx)
    assert np.array_equal(m.predict_margin(sb.DMatrix(x)), _margins(off, nodes, x, 0.0, 1, 30))

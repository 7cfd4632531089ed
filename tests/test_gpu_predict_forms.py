"""Margins on either side of the rules that choose how a request is walked:
rows staged in shared memory or read from global memory (features against the
trees of a block), 8- and 16-byte nodes, uploads whole or in parts, the width
of the ordered sum. Compared bit for bit with sums in tree order over leaves
found by a plain walk."""
import numpy as np
import pytest

from gpu_helpers import leaf_ids
from test_gpu_predict_paths import _forest, _margins

pytestmark = pytest.mark.gpu


def _categorical(nodes, trees, f, rng):
    """The right child of every root splits on a code set of the last feature."""
    at = np.arange(trees) * 7 + 2
    nodes["split_feature"][at] = f - 1
    nodes["is_categorical"][at] = 1
    nodes["cat_end"][at] = 3
    return np.stack([rng.permutation(6)[:3] for _ in range(trees)]).astype(np.uint32)


# one row walks 128 trees per block, 2 rows 64, 16 rows 8, from 17 on 4
@pytest.mark.parametrize("n,f", [(1, 512), (1, 513), (2, 256), (2, 257), (16, 32), (16, 33), (33, 16), (33, 17)])
@pytest.mark.parametrize("form", ["compact", "apart", "categorical"])
def test_staging_and_node_forms(sb, ctx, n, f, form):
    rng = np.random.default_rng(100 * n + f)
    trees = 9
    off, nodes = _forest(sb, rng, trees, f, form == "apart")
    x = rng.standard_normal((n, f)).astype(np.float32)
    cats, cat_off = np.zeros((trees, 0), np.uint32), np.zeros(trees + 1, np.int64)
    if form == "categorical":
        cats, cat_off = _categorical(nodes, trees, f, rng), np.arange(trees + 1, dtype=np.int64) * 3
        x[:, f - 1] = rng.integers(0, 6, n)
    x[rng.random(x.shape) < 0.2] = np.nan
    m = sb.BoostedModel.from_arrays(off, nodes, cat_off, cats.reshape(-1), 0.25, 0, f, ctx=ctx)
    want = np.full(n, np.float32(0.25), np.float32)
    for t in range(trees):
        nd = nodes[off[t]:off[t + 1]]
        want = want + nd["leaf_value"][leaf_ids(nd, cats[t], x)]
    assert np.array_equal(m.predict_margin(sb.DMatrix(x)), want)


# (rows, features, trees, uploads): short of the bytes, of the pairs, and past both in 2 and in 8 parts
@pytest.mark.parametrize("n,f,trees,parts", [(16_384, 61, 1000, 1), (16_384, 64, 610, 1), (16_385, 64, 611, 3),
                                             (66_000, 40, 250, 8), (100_000, 20, 9, 1)])
def test_uploads_in_parts(sb, ctx, n, f, trees, parts):
    rng = np.random.default_rng(n + f)
    off, nodes = _forest(sb, rng, trees, f)
    x = rng.standard_normal((n, f)).astype(np.float32)
    x[rng.random(x.shape) < 0.2] = np.nan
    m = sb.BoostedModel.from_arrays(off, nodes, np.zeros(trees + 1, np.int64), [], 0.25, 0, f, ctx=ctx)
    d = sb.DMatrix(x)
    m.predict_margin(d)
    before = ctx.launch_count()
    got = m.predict_margin(d)
    assert ctx.launch_count() - before == 2 * parts  # leaf values and sum of each part
    some = np.unique(np.concatenate([[0, n - 1], np.arange(8_190, 8_194), np.arange(16_382, min(n, 16_386)),
                                     rng.integers(0, n, 20)]))
    assert np.array_equal(got[some], _margins(off, nodes, x[some], 0.25, 1, trees))


@pytest.mark.parametrize("k,trees", [(1, 64), (1, 65), (2, 63), (4, 64), (4, 65), (5, 64)])
def test_width_of_the_sum(sb, ctx, k, trees):
    rng = np.random.default_rng(10 * trees + k)
    off, nodes = _forest(sb, rng, trees, 6)
    x = rng.standard_normal((65, 6)).astype(np.float32)
    w = rng.random(trees).astype(np.float32)
    m = sb.BoostedModel.from_arrays(off, nodes, np.zeros(trees + 1, np.int64), [], -0.5, 0 if k == 1 else k, 6,
                                    objective="multi:softprob" if k > 1 else "reg:squarederror", weights=w, ctx=ctx)
    nodes = nodes.copy()
    nodes["leaf_value"] *= np.repeat(w, 7)
    assert np.array_equal(m.predict_margin(sb.DMatrix(x)), _margins(off, nodes, x, -0.5, k, trees))


@pytest.mark.parametrize("k,trees", [(1, 129), (3, 64), (5, 65), (16, 130), (17, 193)])
def test_served_outputs(sb, ctx, k, trees):
    """The serving loop's sum, with more outputs than its blocks have warps."""
    rng = np.random.default_rng(trees + k)
    off, nodes = _forest(sb, rng, trees, 6)
    m = sb.BoostedModel.from_arrays(off, nodes, np.zeros(trees + 1, np.int64), [], -0.5, 0 if k == 1 else k, 6,
                                    objective="multi:softprob" if k > 1 else "reg:squarederror", ctx=ctx)
    xs = [rng.standard_normal((n, 6)).astype(np.float32) for n in (1, 33, 70)]
    srv = sb.Server(m, mem_bytes=64 << 20, n_slots=2)
    try:
        tickets = [srv.submit(x) for x in xs]
        for x, t in zip(xs, tickets):
            assert np.array_equal(srv.wait(t, timeout_ms=60000)[0], _margins(off, nodes, x, -0.5, k, trees))
    finally:
        srv.close()

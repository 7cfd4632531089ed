"""Contributions where two leaves of one parent share a table: complete trees
(every leaf in a pair), chains (one pair, the other leaves alone), stumps and
lone roots among them, with few features (the parent's split repeats an
earlier one) and many, and row counts around a block's 64. Within 1e-4 of the
oracle's, the bound of every contribution here, and adding up to the margins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tree(sb, rng, f, depth, chain):
    nodes = []

    def grow(d, cover):
        i = len(nodes)
        nodes.append(np.zeros((), sb.api.NODE_DTYPE))
        nodes[i]["left"] = nodes[i]["right"] = -1
        nodes[i]["sum_hess"] = cover
        if d == 0:
            nodes[i]["leaf_value"] = rng.standard_normal() * 0.1
            return i
        q, right = rng.uniform(0.2, 0.8), rng.random() < 0.5
        nodes[i]["split_feature"] = rng.integers(f)
        nodes[i]["split_cond"] = rng.standard_normal() * 0.5
        nodes[i]["default_left"] = rng.random() < 0.5
        nodes[i]["left"] = grow(0 if chain and right else d - 1, cover * q)
        nodes[i]["right"] = grow(0 if chain and not right else d - 1, cover * (1 - q))
        return i

    grow(depth, 1e4)
    return np.array(nodes, sb.api.NODE_DTYPE)


@pytest.mark.parametrize("f,depth,chain,classes,n", [
    (3, 8, False, 0, 65), (3, 6, True, 3, 64), (12, 9, False, 0, 33), (40, 8, False, 0, 70), (40, 10, True, 0, 1),
    (40, 10, False, 0, 5), (5, 1, False, 0, 63), (230, 8, False, 0, 2)])
def test_contribs_of_paired_leaves(sb, ctx, orc, f, depth, chain, classes, n):
    rng = np.random.default_rng(100 * f + depth)
    trees = [_tree(sb, rng, f, d, chain) for d in (depth, 0, depth, 1, depth, depth)]
    off = np.concatenate([[0], np.cumsum([len(t) for t in trees])]).astype(np.int64)
    arrays = (off, np.concatenate(trees), np.zeros(len(off), np.int64), np.zeros(0, np.uint32),
              np.ones(len(trees), np.float32))
    objective = "multi:softprob" if classes else "reg:squarederror"
    m = sb.BoostedModel.from_arrays(*arrays[:4], 0.25, classes, f, objective=objective, ctx=ctx)
    x = rng.standard_normal((n, f)).astype(np.float32)
    x[rng.random(x.shape) < 0.1] = np.nan
    k = max(classes, 1)
    got = np.asarray(m.predict_contribs(sb.DMatrix(x))).reshape(n, k, f + 1)
    want = np.asarray(orc.predict_contribs(arrays, x, 0.25, classes)).reshape(n, k, f + 1)
    assert np.max(np.abs(got - want)) < 1e-4
    margins = np.asarray(orc.predict_margin(arrays, x, 0.25, classes)).reshape(n, k)
    assert np.max(np.abs(got.astype(np.float64).sum(axis=2) - margins)) < 1e-4

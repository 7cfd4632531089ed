"""The split search's screening and its short cut against the oracle where
they can go wrong: bins per lane from one to nine and beyond the register
form, equal gains (duplicate and empty bins, copied features), gains of the
size of consider's 1e-6 step, missing values on either side, L1, a weight cap
and monotone bounds."""
import numpy as np
import pytest

from gpu_helpers import assert_trees_equal, hist_layout

pytestmark = pytest.mark.gpu


def _check(sb, ctx, orc, x, y, rounds=3, ftypes=None, **kw):
    p = sb.TrainingParams(**{"objective": "reg:squarederror", "seed": 2, **kw})
    d = sb.DMatrix(x, labels=y, feature_types=ftypes)
    assert_trees_equal(sb.train(p, d, rounds, ctx=ctx).export(), orc.train(x, y, p, rounds, ftypes=ftypes)["model"].export())


def _data(n, f, seed, nan=0.1):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, f)).astype(np.float32)
    y = (np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2 % f] + 0.1 * rng.standard_normal(n)).astype(np.float32)
    x[rng.random(x.shape) < nan] = np.nan
    return x, y


@pytest.mark.parametrize("max_bin", [2, 31, 32, 33, 64, 95, 256, 287, 288, 400])
def test_bins_per_lane(sb, ctx, orc, max_bin):
    x, y = _data(5_000, 9, max_bin)
    _check(sb, ctx, orc, x, y, max_bin=max_bin, max_depth=5)


@pytest.mark.parametrize("kw", [
    {"alpha": 0.7}, {"max_delta_step": 0.05}, {"min_child_weight": 0.0, "lambda_": 0.0}, {"gamma": 2.0},
    {"monotone_constraints": [1, -1, 0, 1]}, {"monotone_constraints": [1, 1, 1, 1], "max_delta_step": 0.1},
    {"interaction_constraints": [[0, 1], [2, 3, 4]]}, {"colsample_bynode": 0.5},
])
@pytest.mark.parametrize("grow", ["depthwise", "lossguide"])
def test_parameters(sb, ctx, orc, kw, grow):
    x, y = _data(4_000, 8, 5)
    kw = dict(kw, max_depth=6) if grow == "depthwise" else dict(kw, max_depth=0, max_leaves=40, grow_policy=grow)
    _check(sb, ctx, orc, x, y, **kw)


@pytest.mark.parametrize("scale", [1.0, 1e-2, 1e-3, 1e-4])
def test_ties_and_tiny_gains(sb, ctx, orc, scale):
    """Copied and negated features tie exactly; few distinct values leave most
    bins empty; small labels bring every gain to the size of the 1e-6 step."""
    rng = np.random.default_rng(11)
    a = rng.integers(0, 40, (3_000, 4)).astype(np.float32)
    x = np.concatenate([a, a, -a, rng.standard_normal((3_000, 3)).astype(np.float32)], axis=1)
    y = (scale * (np.sin(a[:, 0] / 7) + 0.3 * (a[:, 1] > 20))).astype(np.float32)
    _check(sb, ctx, orc, x, y, rounds=2, max_depth=5, min_child_weight=0.0)


def test_many_features_and_categories(sb, ctx, orc):
    """More pool positions than a block's threads, categorical winners."""
    rng = np.random.default_rng(4)
    x, y = _data(2_000, 300, 4)
    ft = np.zeros(300, np.uint8)
    for c in (5, 270, 299):
        x[:, c] = rng.integers(0, 20, 2_000)
        ft[c] = 1
    y = y + 2.0 * np.isin(x[:, 270], [1, 5, 7]).astype(np.float32)
    _check(sb, ctx, orc, x, y.astype(np.float32), rounds=2, ftypes=ft, max_depth=5, max_bin=32)

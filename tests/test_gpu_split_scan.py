"""Levels whose features above 288 bins are scanned by a launch of their own
(enough of them to fill the chip), beside narrow and categorical features,
against the oracle."""
import numpy as np
import pytest

from gpu_helpers import assert_trees_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nan", [0.0, 0.1])
@pytest.mark.parametrize("kw", [{}, {"colsample_bytree": 0.5}, {"monotone_constraints": [1, -1, 0, 1]}, {"max_bin": 700}])
def test_wide_features_ahead(sb, ctx, orc, nan, kw):
    rng = np.random.default_rng(17)
    n, f = 6_000, 82  # 79 wide features x 64 nodes: 5,056 warps of 2,368 that run at once
    x = rng.standard_normal((n, f)).astype(np.float32)
    x[:, 7] = rng.integers(0, 50, n)
    x[:, 80] = rng.integers(0, 12, n)
    x[:, 81] = rng.integers(0, 12, n)
    y = (np.sin(2 * x[:, 0]) + x[:, 1] * x[:, 2] + np.isin(x[:, 80], [2, 3, 9]) + 0.5 * rng.standard_normal(n)).astype(np.float32)
    x[rng.random(x.shape) < nan] = np.nan
    ft = np.zeros(f, np.uint8)
    ft[80:] = 1
    p = sb.TrainingParams(**{"objective": "reg:squarederror", "max_bin": 300, "max_depth": 7, "min_child_weight": 0.0,
                             "seed": 3, **kw})
    got = sb.train(p, sb.DMatrix(x, labels=y, feature_types=ft), 2, ctx=ctx).export()
    assert_trees_equal(got, orc.train(x, y, p, 2, ftypes=ft)["model"].export())

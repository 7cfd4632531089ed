"""Contributions of trees whose longest paths lie at the lengths the table
kernel is unrolled to (8 and 10 features): within 1e-4 of the oracle's, the
bound of every contribution here, and adding up to the margins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 7, 8, 9, 10])
def test_contribs_by_path_length(sb, ctx, orc, depth):
    rng = np.random.default_rng(depth)
    f = 24
    x = rng.standard_normal((6000, f)).astype(np.float32)
    x[rng.random(x.shape) < 0.05] = np.nan
    y = np.nan_to_num(x) @ rng.standard_normal(f).astype(np.float32)
    p = sb.TrainingParams(objective="reg:squarederror", max_depth=depth, eta=0.3)
    r = orc.train(x, y.astype(np.float32), p, 4)
    arrays, base = r["model"].export(), r["model"].base_score
    m = sb.BoostedModel.from_arrays(*arrays[:4], base, 0, f, objective=p.objective, ctx=ctx)
    xt = x[:67]
    got = m.predict_contribs(sb.DMatrix(xt))
    assert np.max(np.abs(got - orc.predict_contribs(arrays, xt, base, 0))) < 1e-4
    sums = got.reshape(len(xt), f + 1).astype(np.float64).sum(axis=1)
    assert np.max(np.abs(sums - orc.predict_margin(arrays, xt, base, 0))) < 1e-4

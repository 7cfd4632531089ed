"""Where the device adds a booster's labels: integers, from the row count on at
which the launch pays. The base score is the sequential f64 mean either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [131_071, 131_072, 140_001])
@pytest.mark.parametrize("kind", ["classes", "reals", "one real at the end"])
def test_launches_and_base_score(sb, ctx, n, kind):
    rng = np.random.default_rng(n)
    y = (rng.standard_normal(n) if kind == "reals" else rng.random(n) < 0.3).astype(np.float32)
    if kind.startswith("one"):
        y[-1] = 0.3
    g = sb.GHistIndex(sb.DMatrix(np.zeros((n, 1), np.float32)), ctx=ctx)
    before = ctx.launch_count()
    b = sb.Booster(g, sb.TrainingParams(max_depth=1), y, ctx=ctx)
    assert ctx.launch_count() - before == (2 if n >= 131_072 and kind != "reals" else 1)  # the margins' fill
    total = 0.0
    for v in y.astype(np.float64).tolist():
        total += v
    assert np.float32(b.model().base_score()) == np.float32(total / n)

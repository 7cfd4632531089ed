"""The base score of a booster (init_margin, train.rs:496-511) is the labels'
sequential f64 mean, whether the device or the host adds them: class labels,
counts, magnitudes at which f64 stops being exact, and other values, below and
above the row count from which the device takes integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65_535, 65_536, 70_001])
@pytest.mark.parametrize("kind", ["classes", "counts", "huge", "reals"])
def test_base_score_is_the_sequential_mean(sb, ctx, n, kind):
    rng = np.random.default_rng(n)
    y = {"classes": rng.random(n) < 0.3, "counts": rng.integers(-40, 1000, n),
         "huge": rng.integers(1, 1 << 20, n) * 2.0 ** 33 + 1.0, "reals": rng.standard_normal(n) + 0.1}[kind]
    y = y.astype(np.float32)
    x = np.zeros((n, 1), np.float32)
    m = sb.train(sb.TrainingParams(max_depth=1), sb.DMatrix(x, labels=y), 0, ctx=ctx)
    total = 0.0
    for v in y.astype(np.float64).tolist():
        total += v
    assert np.float32(m.base_score()) == np.float32(total / n)

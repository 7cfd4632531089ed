"""Cuts where the planning of a feature's key levels can go wrong: as many
distinct values as bins and one more, fewer rows than bins, values that share
their upper key bits, many copies of one value, signed zeros, infinities and
subnormals. Cuts and bins equal the oracle's."""
import numpy as np
import pytest

from test_gpu_bin import _compare

pytestmark = pytest.mark.gpu


def _columns(rng, n, max_bin):
    tight = (np.float32(1.0).view(np.uint32) + rng.integers(0, 5000, n).astype(np.uint32)).view(np.float32)
    wide = rng.integers(0, 0x7F800000, n, dtype=np.uint32).view(np.float32) * rng.choice([-1, 1], n).astype(np.float32)
    special = rng.choice(np.array([-np.inf, -1e-41, -0.0, 0.0, 1e-45, 1e-41, 3.0, np.inf], np.float32), n)
    skewed = np.where(rng.random(n) < 0.97, np.float32(2.5), rng.standard_normal(n)).astype(np.float32)
    cols = [tight, wide, special, skewed, rng.standard_normal(n).astype(np.float32)]
    for distinct in (1, max_bin, max_bin + 1):  # enumerated up to max_bin distinct values, ranked above
        v = np.arange(n) % distinct
        cols.append(rng.permutation(v).astype(np.float32) - 3)
    cols.append(np.full(n, np.nan, np.float32))
    return np.stack(cols, axis=1)


@pytest.mark.parametrize("max_bin", [2, 3, 64, 256, 1023, 1024])
@pytest.mark.parametrize("n", [1, 5, 1030, 40_000])
def test_cuts_and_bins(sb, ctx, orc, n, max_bin):
    x = _columns(np.random.default_rng(n + max_bin), n, max_bin)
    x[:, 4][np.random.default_rng(1).random(n) < 0.3] = np.nan
    _compare(sb, ctx, orc, x, max_bin=max_bin)

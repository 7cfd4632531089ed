"""The histogram kernel at the sizes where its row division, its feature
packing and its flush can go wrong: row counts around a warp's block of 32 and
a CTA's share, tiles whose features fill a lane's column or overflow it, and
both CTA sizes. Fixed-point sums are integers, so every one is compared
exactly with the oracle fed the same quantised pairs."""
import numpy as np
import pytest

from gpu_helpers import assert_trees_equal, hist_layout, mixed_data, random_gpair

pytestmark = pytest.mark.gpu

N = 9_000


def _matrix(f, seed):
    """Continuous columns (257 bins at max_bin 256) with holes."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((N, f)).astype(np.float32)
    x[rng.random(x.shape) < 0.05] = np.nan
    return x


# features: below / at / above the 96 columns of 257 bins that 32 lanes hold,
# two tiles, and one position per lane
@pytest.mark.parametrize("f", [1, 31, 33, 64, 65, 96, 97, 100, 129, 200])
@pytest.mark.parametrize("layout", ["tiled", "lanes"])
def test_packing_edges_exact(sb, ctx, orc, f, layout):
    x = _matrix(f, f)
    g = random_gpair(N, seed=f)
    gq, _, _ = orc.quantize(g, 16)
    d = orc.data(x, max_bin=256)
    with hist_layout(layout):
        gh = sb.GHistIndex(sb.DMatrix(x), max_bin=256, ctx=ctx)
    backend = sb.GpuBackend("fixed", quantize_bits=16, ctx=ctx)
    sel = np.arange(0, N, 2, dtype=np.uint32)
    assert np.array_equal(backend.build(gh, sel, g), d.hist(sel, gq, threads=1))


@pytest.mark.parametrize("max_bin", [16, 256])  # 256-thread CTAs, 1024-thread CTAs
@pytest.mark.parametrize("layout", ["tiled", "lanes"])
@pytest.mark.parametrize("m", [0, 1, 31, 32, 33, 63, 65, 1023, 1024, 1025, 4737, N])
def test_row_counts_exact(sb, ctx, orc, max_bin, layout, m):
    x = _matrix(40, 7)
    g = random_gpair(N, seed=m + 1)
    gq, _, _ = orc.quantize(g, 16)
    sel = np.sort(np.random.default_rng(m).permutation(N)[:m]).astype(np.uint32)
    with hist_layout(layout):
        gh = sb.GHistIndex(sb.DMatrix(x), max_bin=max_bin, ctx=ctx)
    got = sb.GpuBackend("fixed", quantize_bits=16, ctx=ctx).build(gh, sel, g)
    assert np.array_equal(got, orc.data(x, max_bin=max_bin).hist(sel, gq, threads=1))


@pytest.mark.parametrize("max_bin,depth", [(16, 3), (16, 9), (256, 3), (256, 8)])
@pytest.mark.parametrize("layout", ["tiled", "lanes"])
def test_levels_of_many_nodes_exact(sb, ctx, orc, max_bin, depth, layout):
    """From one node to more nodes than CTAs: whole-range CTAs on the shallow
    levels, equal shares across nodes on the deep ones; column sampling sends
    codes to the words that the flush leaves out."""
    x, ft = mixed_data(12_000, 70, seed=3, n_cat=2, card=12)
    y = (np.nan_to_num(x[:, 0]) - 0.5 * np.nan_to_num(x[:, 5]) + 0.2 * (x[:, -1] == 3)).astype(np.float32)
    p = sb.TrainingParams(objective="reg:squarederror", max_depth=depth, max_bin=max_bin, min_child_weight=0.0,
                          subsample=0.9, colsample_bytree=0.6, seed=5)
    with hist_layout(layout):
        m = sb.train(p, sb.DMatrix(x, labels=y, feature_types=ft), 2, ctx=ctx)
    assert_trees_equal(m.export(), orc.train(x, y, p, 2, ftypes=ft)["model"].export())

"""Which wide matrices take the LANES layout: enough rows to a histogram entry,
and memory left beside its wider codes."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,f,max_bin,layout", [
    (200_000, 70, 256, "lanes"), (200_000, 70, 64, "lanes"), (200_000, 70, 1024, "tiled"), (199_999, 70, 256, "tiled"),
    (200_000, 64, 1024, "tiled"), (260_000, 65, 1000, "tiled"), (261_000, 65, 1000, "lanes")])
def test_rows_to_an_entry(sb, ctx, n, f, max_bin, layout, monkeypatch):
    monkeypatch.setenv("SB_HIST_AUTOTUNE", "0")
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, f), dtype=np.float32)
    g = sb.GHistIndex(sb.DMatrix(x), max_bin=max_bin, ctx=ctx)
    lanes = f > 64 and n >= 200_000 and n >= 4 * (g.total_bins + f)
    assert layout == ("lanes" if lanes else "tiled"), g.total_bins
    assert g.layout()["layout"] == layout


CHILD = """
import sys, torch
sys.path.insert(0, sys.argv[1])
import __graft_entry__ as ge
sb = ge.load_package()
n, f = 2_000_000, 65
x = torch.randn(n, f, device="cuda")
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
hog = torch.empty(free - (int(sys.argv[2]) << 20), dtype=torch.uint8, device="cuda") if int(sys.argv[2]) else None
g = sb.GHistIndex.from_device(x.data_ptr(), n, f, max_bin=63)
print("LAYOUT", g.layout()["layout"])
"""


# LANES codes take 368 MB more than TILED's 144 MB, which with the feature-major
# bins leave 404 MB less: the line is at 8 * 368 + 404 = 3,348 MB, less some 100 MB
# of the build's own temporary arrays.
@pytest.mark.parametrize("left_mb,layout", [(0, "lanes"), (2_600, "tiled"), (4_400, "lanes")])
def test_memory_left(left_mb, layout):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD, root, str(left_mb)], capture_output=True, text=True, timeout=300)
    assert "LAYOUT " + layout in r.stdout, (r.stdout, r.stderr[-2000:])

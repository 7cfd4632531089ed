"""bench.py reports the histogram's measured traffic only for the form of row
codes that it was measured with."""
import json


def test_traffic_belongs_to_the_layout(tmp_path, monkeypatch):
    import bench
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    layout = {"layout": "lanes", "code_bytes": 2, "row_stride": 128, "rows_per_instruction": 1}
    assert bench.traffic_per_launch(layout, 100.0) is None  # no summary
    (tmp_path / "profiles").mkdir()
    out = tmp_path / "profiles" / "k_hist_traffic.json"
    out.write_text(json.dumps({"layout": layout, "traffic_over_algorithmic": 1.5}))
    assert bench.traffic_per_launch(layout, 100.0) == 150.0
    assert bench.traffic_per_launch(dict(layout, layout="tiled", row_stride=104), 100.0) is None
    out.write_text(json.dumps({"bytes_per_launch": 968721270}))
    assert bench.traffic_per_launch(layout, 100.0) is None

"""The bench line's figures from a committed capture say whether the capture
is of the present device code (CPU)."""

import json

import bench


def _issue(tmp_path, **change):
    w = bench.make_workload("pt")
    t = json.loads((bench.ROOT / "profiles" / "roofline_traffic.json").read_text())
    w.opts = dict(t["pt"]["sass_options"])
    t["pt"].update(change)
    (tmp_path / "t.json").write_text(json.dumps(t))
    return bench.ncu_rooflines(w, 23.0, 1965.0, path=tmp_path / "t.json")[1]


def test_a_capture_of_other_code_says_so(tmp_path):
    assert _issue(tmp_path, code=bench.code_digest("sphere_pt_f32"))["capture_of_this_code"] is True
    assert _issue(tmp_path, code="0" * 16)["capture_of_this_code"] is False
    assert _issue(tmp_path, code=None)["capture_of_this_code"] is False


def test_digest_sees_code_and_no_comments(tmp_path, monkeypatch):
    src = tmp_path / "loom_b200" / "csrc"
    (src / "gen").mkdir(parents=True)
    (src / "engine").mkdir()
    for f in ("gen/k.cu", "engine/common.cuh", "engine/regroup.cuh"):
        (src / f).write_text("int a; // one\n")
    monkeypatch.setattr(bench, "ROOT", tmp_path)
    first = bench.code_digest("k")
    (src / "gen" / "k.cu").write_text("int  a;\n/* two */\n")
    assert bench.code_digest("k") == first
    (src / "engine" / "regroup.cuh").write_text("int b; // one\n")
    assert bench.code_digest("k") != first

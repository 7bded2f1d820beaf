"""The benchmark's default takes the learned cut only while the batched kernel
is the one the recorded gain was measured on (no GPU)."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def test_learned_cut_only_on_the_kernel_it_was_measured_on(tmp_path, monkeypatch):
    calls = []
    monkeypatch.setattr(bench, "build_script", lambda d, blocks, cost_model=None, **kw:
                        calls.append(cost_model is not None))
    with open(os.path.splitext(bench.MODEL_PATHS[2])[0] + ".json") as f:
        summary = json.load(f)
    assert summary["eval_soc2m"]["gain"] > 1.0  # it won, on an earlier kernel
    with open(bench.MODEL_PATHS[2], "rb") as f:
        (tmp_path / "m.npz").write_bytes(f.read())
    monkeypatch.setitem(bench.MODEL_PATHS, 2, str(tmp_path / "m.npz"))
    now = bench.kernel_code_hash()[:16]
    for kernel, learned, want in [(None, "auto", False), ("0" * 16, "auto", False),
                                  (now, "auto", True), (now, "off", False), (None, "on", True)]:
        s = dict(summary, kernel=kernel) if kernel else summary
        (tmp_path / "m.json").write_text(json.dumps(s))
        bench.default_batched_script(None, blocks=148, lanes=8, per_item=2, learned=learned)
        assert calls.pop() is want

"""bench.py's result line: short enough for a log's tail, with every number it reports, the tables in a file."""
import json

import bench


def _line():
    curve = [[0.1234567890123456] * 13] * 51
    run = {"value": 3.0000000001, "curves": {"columns": ["t"] * 13, "fp64": curve, "mixed": curve},
           "rel_l2_mixed_vs_fp64": dict.fromkeys("abcdefgh", 1.23456789e-7),
           "curve_max_rel_err_mixed_vs_fp64": dict.fromkeys("abcdefghijkl", 1e-9),
           "fp64": {"value": 1.5, "sweep_shapes": [{}] * 3}, "within_bars": True}
    return {"metric": "Gcell-updates/s", "value": 2.0661234567891, "n_gpus": 1, "steps": 20, "e2e": None,
            "config": {"workload": "w", "n": 256}, "gpu_launches": 123,
            "sweep_shapes": [{"dir": d, "variant": 2, "window": [16, 16], "segment": 64} for d in "xyz"],
            "forms": {"c2_256_curves": run, "c3_512": run, "mixed": {"stats_rel_err_vs_fp64": {"TKE": 1e-8}, "value": 3.1}}}


def test_line_is_short_and_complete(tmp_path):
    line, path = _line(), tmp_path / "forms.json"
    text = bench.short_line(line, str(path))
    assert "\n" not in text and len(text) < 2000
    out = json.loads(text)
    assert out["value"] == 2.066123 and out["steps"] == 20 and out["gpu_launches"] == 123 and out["e2e"] is None
    assert out["sweep_shapes"] == [[2, 64]] * 3
    assert out["forms"]["c3_512"]["value"] == 3.0 and out["forms"]["c3_512"]["within_bars"] is True
    assert out["forms"]["c3_512"]["rel_l2_mixed_vs_fp64"]["a"] == 1.234568e-7
    assert "curves" not in out["forms"]["c3_512"]
    assert json.loads(path.read_text()) == line["forms"]
    assert json.loads(bench.short_line(line, "")) == out


def test_executed_instructions_follow_the_shapes():
    def shapes(v, L):
        return [{"variant": v, "segment": L}] * 3

    assert abs(bench.fp64_instr_per_cell_update(192, shapes(0, 48)) - 5137.7) < 0.2
    assert abs(bench.fp64_instr_per_cell_update(192, shapes(0, 16)) / 5358.8 - 1) < 0.004   # counted with 16 faces
    assert bench.fp64_instr_per_cell_update(256, shapes(2, 64)) > bench.fp64_instr_per_cell_update(256, shapes(2, 256))
    assert bench.fp64_instr_per_cell_update(250, shapes(0, 48)) is None
    assert bench.fp64_instr_per_cell_update(256, shapes(3, 48)) is None

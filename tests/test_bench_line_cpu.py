"""The line that bench.py prints for the default run, on the CPU: the headline's
whole record and a summary of every workload, short enough for a log's last lines
to keep it whole."""
import json
import sys

from conftest import ROOT

sys.path.insert(0, ROOT)
import bench  # noqa: E402


def _record(name, value):
    """A workload's record with everything a run can put into it."""
    text = "x" * 300
    call = {"value": value, "unit": bench.UNIT, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2, "api": text,
            "timing": text}
    return {"metric": bench.METRIC, "value": value, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 1.0 / 3.0, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": text, "config": {"workload": name, "form": "mixed", "desc": text},
            "error_vs_fp64_full": {"max_abs_over_rms": 1e-7 * value, "reference": text}, "plain_fp64":
            {"speedup_of_chosen_form": 6.0, "path": text}, "other_forms": {"a": {"t": text}, "b": {"t": text}},
            "gpu_launches": 9, "roofline": {"frac": 0.8, "note": text}, "cpu_baseline": {"value": 0.7, "sample": text},
            "e2e": dict(call), "e2e_structured_api": dict(call), "dropin_e2e_default_tolerance": dict(call),
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}}


def test_headline_line_is_short_and_whole():
    lines = {n: _record(n, float(i + 1)) for i, n in enumerate(bench.ALL_WORKLOADS)}
    head = bench.headline_record(lines)
    text = json.dumps(head)
    assert "\n" not in text and len(text) <= 8000
    own = lines[bench.HEADLINE]
    for k, v in own.items():
        if k != "config":
            assert head[k] == v, k
    assert head["config"]["workload"].startswith(bench.HEADLINE)
    for n, l in lines.items():
        s = head["summary"][n]
        assert s["value"] == l["value"] and s["e2e"] == l["e2e"]["value"] and s["form"] == "mixed"
        assert s["roofline_frac"] == 0.8 and s["ms_per_step"] == l["ms_per_step"]
    assert head["summary"]["max_err_full_all"] == max(l["error_vs_fp64_full"]["max_abs_over_rms"]
                                                      for l in lines.values())
    assert own["config"]["workload"] == bench.HEADLINE      # the records themselves stay as they are

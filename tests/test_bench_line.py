"""bench.py's line on stdout: the headline and its checks in under 2.5 KB whatever the other timings hold; those
follow on stderr."""
import json

import bench


def test_the_headline_fits_a_short_tail(capsys):
    line = {k: "x" * 60 for k in bench.HEADLINE}
    line["config"] = {"workload": "w" * 200, "grid": [41, 181, 361], "l2": "x" * 60}
    line["roofline"] = {"bound": "hbm", "frac": 0.5, "step": {"what": "y" * 900}}
    line["e2e"] = {"value": 1.0, "what": "z" * 250}
    line["cpu_baseline"] = {"value": 1.0, "sample": "s" * 300}
    extra = {"adjoint": {"a": "b" * 4000}, "accuracy_vs_fp64": {"step10": ["c" * 4000]}}
    bench.report({**line, **extra})
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < 2500
    head = json.loads(out)
    assert set(head) == set(bench.HEADLINE) and "step" not in head["roofline"]
    rest = json.loads(err)["details"]
    assert rest["adjoint"] == extra["adjoint"] and rest["accuracy_vs_fp64"] == extra["accuracy_vs_fp64"]
    assert rest["roofline_step"]["what"] == "y" * 900

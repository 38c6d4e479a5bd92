"""The benchmark's result line stays short: what it says about a series of 60
registrations is a summary and the worst pairs, and numbers are printed at
eight significant digits (CPU)."""
import json

import numpy as np


def test_final_costs_are_summed_up(capsys):
    import bench
    rng = np.random.default_rng(1)
    f = rng.uniform(20.0, 2000.0, 60)
    res = [(None, None, v * (1 + 1.1e-5 * k), 9) for k, v in enumerate(f)]
    plain = [(None, None, v, 9) for v in f]
    rep = bench.final_cost_report(res, plain, [(v, 1e-6 * v, v) for v in f])
    o = rep["vs_oracle"]
    assert o["pairs"] == 60 and o["plain_pairs_passing"] == 60
    assert o["batched_pairs_passing"] == 10   # 1.1e-5 k <= 1e-4
    assert [p["pair"] for p in o["worst_pairs"]] == [59, 58, 57]
    bench.print_line({"value": 12345.678901234567, "n": 60, "ok": True, "none": None, "final_cost": rep})
    text = capsys.readouterr().out
    assert text.count("\n") == 1 and len(text) < 3000
    line = json.loads(text)
    assert line["value"] == 12345.679 and line["ok"] is True and line["none"] is None and line["n"] == 60

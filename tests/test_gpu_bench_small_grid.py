"""bench.py on a grid whose pressure solve runs on chip: the line names that
kernel and gives no HBM rate for it (its vectors do not go through HBM)."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_line_of_a_small_grid():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--n", "32", "--steps", "2", "--warmup", "3",
                        "--class-steps", "2", "--adj-steps", "0", "--precision-steps", "0", "--no-cpu-baseline"],
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["value"] > 0 and out["e2e"]["value"] > 0 and out["gpu_launches"] > 0
    assert out["pcg_hbm_gbs"] is None and out["pcg_roofline"] is None
    cls = out["kernel_classes"]
    assert "k_cg_dir" not in cls and "k_cg_upd" not in cls
    assert cls["k_cg_res"]["launches"] == cls["steps"] and 0 < cls["k_cg_res"]["us_per_iteration"] < 100
    roof = out["roofline"]
    assert roof["traffic"] is None            # captured at one grid, not scaled to others
    if roof["kernel"].startswith("k_cg"):
        assert roof["kernel"].startswith("k_cg_res") and roof["achieved"] is None and roof["frac"] is None

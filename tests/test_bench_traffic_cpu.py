"""bench.py reports the DRAM traffic of the kernel it names, from the recorded
capture, and none when the capture is of another kernel."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402

PROF = {"pcg_launches": 4, "pcg_ms": 0.8, "pcg_iters": 2240, "pcg_iters_timed": 160, "pcg_cells": 65536}


@pytest.mark.parametrize("kernel,want", [("k_pcg_column<8>, 16 CTAs", 123), ("k_pcg_cluster<float, 8>", None)])
def test_traffic_is_of_the_named_kernel(monkeypatch, tmp_path, kernel, want):
    os.makedirs(tmp_path / "profiles")
    (tmp_path / "profiles" / "pcg_traffic.json").write_text(json.dumps({"kernel": kernel, "dram_bytes_per_launch": 123}))
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    r = bench.roofline(PROF, None)
    assert r["kernel"].startswith("k_pcg_column") and r["traffic"] == want

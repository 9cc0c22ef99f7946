"""bench.py's count of launches and its kernel's traffic: an event holds one
launch, so the steps between events are ones that a launch can take."""

import json
import os
from types import SimpleNamespace

import pytest

import bench
from latticeboltzmann_gb300 import _lib


@pytest.mark.parametrize("most,steps,chunk", [(4, 20, 4), (4, 6, 2), (4, 9, 1), (4, 15, 1), (4, 18, 2), (2, 9, 1),
                                              (2, 6, 2), (8, 6, 6), (6, 9, 3), (3, 9, 3), (1, 7, 1)])
def test_steps_of_an_event_are_one_launch(monkeypatch, most, steps, chunk):
    monkeypatch.setattr(_lib, "load", lambda: SimpleNamespace(lbgb_max_steps_per_launch=lambda *a: most))
    assert bench.steps_per_event(SimpleNamespace(nx=1, ny=1, bcode=0, code=0), steps) == chunk


def test_march_traffic():
    rows = json.load(open(os.path.join(bench.ROOT, "profiles", "k_march_traffic.json")))
    assert {r["storage"] for r in rows} == {"f32", "f32dev", "f16dev", "bf16dev"}
    for r in rows:
        # one read and one write of the lattice, the strips' outermost lanes read twice
        full = 72 if r["storage"] in ("f32", "f32dev") else 36
        assert full < r["dram_bytes_per_launch"] / r["cells"] < full * (1 + 32 / 30) / 2 + 3
        assert r["kernel"] == "k_march" and r["steps_per_launch"] == 4 and "--clock-control none" in r["source"]
    n = 8192 * 8192
    assert bench.step_kernel(n, 4) == "k_march" and bench.step_kernel(n, 1) == "k_step_pipe"
    assert bench.step_kernel(256 * 256, 6) == "k_march / k_tile"
    got, row = bench.profiled_traffic("f32", "cavity", n, "k_march", 4)
    assert row["storage"] == "f32" and got == pytest.approx(4 * row["dram_bytes_per_launch"])
    assert bench.profiled_traffic("f32", "cavity", n, "k_march", 2) == (None, None)
    assert bench.profiled_traffic("f32", "cavity", n, "k_step_pipe", 1)[1]["kernel"] == "k_step_pipe"

"""The benchmark's host side (no GPU): what its line holds where the reference is not at hand."""

from __future__ import annotations

import json
from types import SimpleNamespace

import pytest

import bench
from oracle import harness as H


@pytest.fixture
def no_reference(tmp_path, monkeypatch):
    monkeypatch.setattr(H, "REF", tmp_path)
    monkeypatch.setattr(H, "_libs", {})


def test_the_reference_arm_says_that_it_is_unavailable(no_reference, capsys):
    bench.run_reference(SimpleNamespace(steps=1, warmup=0, cpu_window=65), 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libtgref.so" in line["unavailable"]


def test_the_line_keeps_its_measurements_without_the_reference(no_reference):
    baseline = bench.cpu_baseline(65)
    assert baseline["value"] is None and "libtgref.so" in baseline["unavailable"]
    assert "unavailable" in bench.dropin_leg(65)


@pytest.mark.parametrize("side, kernels", [
    (513, ["fbm", "crater_footprint", "scan_block", "crater_bin_scatter", "crater_lean_shape",
           "crater_extras", "boulder_count", "scan_block", "boulder_scatter", "boulder_bake"]),
    (4097, ["fbm", "crater_footprint", "crater_wide_count", "scan_block", "scan_block", "scan_add",
            "crater_bin_scatter", "crater_lean_shape", "crater_extras", "boulder_count",
            "scan_block", "scan_block", "scan_add", "boulder_scatter", "boulder_bake"])])
def test_a_steps_launches_are_the_profilers_list(side, kernels):
    assert bench.step_launches(((side + 31) // 32) ** 2) == len(kernels)


def test_operations_are_those_of_the_cases():
    from perf import cases

    assert bench.NOISE_OPS_PER_CELL_OCTAVE == cases._OCTAVE
    assert bench.CRATER_OPS_PER_PAIR == cases._CRATER

"""The bench's reference arm is the reference's own build or nothing: no figure of this repository's code in its place."""
import argparse
import json

import bench


def test_without_the_build_the_arm_says_unavailable(monkeypatch, capsys):
    monkeypatch.setattr(bench, "reference_binary", lambda: None)
    assert bench.run_reference(argparse.Namespace(gpus=1, steps=2, warmup=3), 1, 0) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_a_run_that_fails_gives_no_figure(monkeypatch, capsys):
    monkeypatch.setattr(bench, "reference_binary", lambda: ("exe", "conf"))
    for failing in (0, 3, 4):  # in the warm-up and in the timed runs
        runs = iter([(1e6, 0.1)] * failing + [None])
        monkeypatch.setattr(bench, "run_reference_binary", lambda *a, **k: next(runs))
        assert bench.run_reference(argparse.Namespace(gpus=1, steps=2, warmup=3), 1, 0) == 0
        line = json.loads(capsys.readouterr().out)
        assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_with_the_build_its_own_clock_counts(monkeypatch, capsys):
    monkeypatch.setattr(bench, "reference_binary", lambda: ("exe", "conf"))
    monkeypatch.setattr(bench, "run_reference_binary", lambda *a, **k: (1e6, 0.5))
    assert bench.run_reference(argparse.Namespace(gpus=1, steps=2, warmup=3), 1, 0) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["ms_per_step"] == 500.0 and line["cpu_baseline"]["kind"] == "reference"


def test_the_batched_arm_too(monkeypatch, capsys):
    monkeypatch.setattr(bench, "reference_batched_rate", lambda *a, **k: None)
    monkeypatch.setattr(bench, "batched_draws", lambda: {})
    assert bench.run_reference_batched(argparse.Namespace(gpus=1, steps=2, warmup=3), 1, 0) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line

"""Bench bookkeeping that needs no GPU: the algorithmic FP64 work behind the
roofline figure, and the crops of the timed CPU baseline."""

import json
import sys
from pathlib import Path
from types import SimpleNamespace

import bench
from oracle import ref


def anchors_in_tile(tw: int, th: int, cw: int, ch: int, step: int) -> int:
    """Anchors of one transform family in a tile of tw x th blocks: positions
    on the family's step grid (within the 8x8 tile) whose footprint fits."""
    xs = [x for x in range(0, 8, step) if x + cw <= min(8, tw)]
    ys = [y for y in range(0, 8, step) if y + ch <= min(8, th)]
    return len(xs) * len(ys)


def test_candidate_cost_operations_match_the_candidate_set():
    bx, by = bench.WIDTH // 8, bench.HEIGHT // 8
    total = 0
    for w, h, cw, ch, step in bench.FAMILIES:
        anchors = sum(anchors_in_tile(min(8, bx - tx), min(8, by - ty), cw, ch, step)
                      for ty in range(0, by, 8) for tx in range(0, bx, 8))
        # Forward and inverse separable DCT of 3 channels: (W + H) multiply-adds
        # per coefficient, each multiply and add counted as one operation.
        total += anchors * 3 * 2 * (w * h) * (w + h) * 2
    assert bench.candidate_cost_fp64_ops(bx, by) == total
    # The figure quoted with the roofline for the 4032x3024 workload.
    assert total == 70_894_559_232


def test_reference_crops_tile_the_workload_image():
    crops = bench.reference_crops(16)
    assert len(crops) == 16
    for x, y in crops:
        assert 0 <= x <= bench.WIDTH - bench.CROP_W
        assert 0 <= y <= bench.HEIGHT - bench.CROP_H
    # Distinct crops while the image holds enough of them.
    cols, rows = bench.WIDTH // bench.CROP_W, bench.HEIGHT // bench.CROP_H
    assert len(set(bench.reference_crops(cols * rows))) == cols * rows


def test_executed_operations_of_the_candidate_set():
    """Per 8 outputs of a line of length L: 16 L forward, 4 L + 8 in the folded
    inverse."""
    bx, by = bench.WIDTH // 8, bench.HEIGHT // 8
    total = 0
    for (w, h), anchors in bench.candidate_anchors(bx, by):
        lines = sum(16 * n + 4 * n + 8 for n in (w, h))
        total += anchors * 3 * (w * h // 8) * lines
    assert bench.candidate_cost_executed_ops(bx, by) == total
    assert bench.candidate_cost_fp64_ops(bx, by) / 2 < total < bench.candidate_cost_fp64_ops(bx, by)


def missing(*args):
    raise FileNotFoundError("not here")


def test_line_is_printed_without_the_optional_legs(monkeypatch, capsys):
    """Legs that stand on the reference's files: their absence is reported in
    the line, which keeps what was measured."""
    monkeypatch.setattr(sys, "argv", ["bench.py", "--no-batched"])
    for name in ("RANK", "WORLD_SIZE"):
        monkeypatch.delenv(name, raising=False)
    monkeypatch.setattr(bench, "run_gpu", lambda args: {"value": 12.0})
    monkeypatch.setattr(bench, "learned_leg", lambda *args: {
        "value_12mp": 13.0} | bench.or_unavailable("bd_rate", missing))
    monkeypatch.setattr(bench, "reference_missing", lambda: None)
    monkeypatch.setattr(bench, "ReferencePool", lambda: SimpleNamespace(close=lambda: None))
    monkeypatch.setattr(bench, "cpu_baseline_leg", missing)
    monkeypatch.setattr(bench, "reference_gpu_leg", missing)
    bench.main()
    line = json.loads(capsys.readouterr().out.strip())
    assert line["value"] == 12.0 and line["learned_form"]["value_12mp"] == 13.0
    assert "not here" in line["learned_form"]["bd_rate"]["unavailable"]
    for name in ("cpu_baseline", "reference_gpu"):
        assert "not here" in line[name]["unavailable"]


def test_reference_arm_says_what_is_missing(monkeypatch):
    monkeypatch.setenv("RANK", "0")
    monkeypatch.setattr(ref, "LIBRARY_PATH", Path("/nowhere/libgjxl_ref.so"))
    out = bench.run_reference(None)
    assert out["impl"] == "reference" and "libgjxl_ref.so" in out["unavailable"]

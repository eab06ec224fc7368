"""The span copy (cubam_b200/csrc/spans.cuh) checked on the host, where a word outside a span's own is a page fault."""

import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_span_copy_stays_inside_its_spans(tmp_path):
    from cubam_b200 import build

    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    exe = tmp_path / "span_copy_check"
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Wno-deprecated-gpu-targets", str(HERE / "span_copy_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)
    assert r.stdout.startswith("0 failures")

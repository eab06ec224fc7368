"""The sizes of members that the split inflater takes (cubam_b200/csrc/split_slots.cuh), checked on the host."""

import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_every_size_taken_is_counted_in_32_bits(tmp_path):
    from cubam_b200 import build

    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    exe = tmp_path / "split_slots_check"
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Wno-deprecated-gpu-targets", str(HERE / "split_slots_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)
    assert r.stdout.startswith("0 failures")

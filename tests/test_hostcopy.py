"""The threaded device-to-host reads (host code, csrc/hostcopy.cuh): compiled
with the host compiler against a stand-in CUDA runtime and checked by
tests/hostcopy_check.cpp (every byte once, one wait for the stream's queued
work before the first piece, threads that cannot be created, no page-locked
memory, a failing copy)."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_threaded_reads_on_a_stand_in_runtime(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    shutil.copy(ROOT / "tests" / "fake_cuda_runtime.h", tmp_path / "cuda_runtime.h")
    shutil.copy(ROOT / "magnelio_b200" / "csrc" / "hostcopy.cuh", tmp_path / "hostcopy.cuh")
    exe = tmp_path / "hostcopy_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", "-I", str(tmp_path),
                    str(ROOT / "tests" / "hostcopy_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-2000:]
    assert res.stdout.startswith("ok"), res.stdout

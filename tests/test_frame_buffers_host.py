"""Ownership of the output frames' page-locked buffers (anuga_core_gb300/csrc/
frame_buffers.h, compiled by g++ on the host with the heap in their place;
tests/cpp/check_frame_buffers.cpp): no buffer has two owners, whatever callers
give back, no steady loop page-locks memory, and what is page-locked stays
bounded."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_frame_buffer_ownership(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "check_frame_buffers")
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-o", exe,
                    os.path.join(HERE, "cpp", "check_frame_buffers.cpp")], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "failures 0" in r.stdout, r.stdout + r.stderr

"""The friction term's cube root and 7/3 power (de_plain.cuh dcbrt and
h_pow_7_3, compiled by g++ on the host) against the long double library over
the whole exponent range, with the error bounds their forms have
(tests/cpp/check_cbrt.cpp derives them)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_cube_root_within_its_bound(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "check_cbrt")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "cpp", "check_cbrt.cpp")], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "failures 0" in r.stdout, r.stdout + r.stderr

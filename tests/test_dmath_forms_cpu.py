"""Short integer forms of the double math (gr_dmath.h, gr_exact.h, compiled for
the host) against the long forms or the IEEE operations they stand for."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


# fp64i_check also with the single-precision estimates a few units off
@pytest.mark.parametrize("src,ulps", [("dmath_short_check", 0), ("fp64i_check", 0), ("fp64i_check", -4), ("fp64i_check", 4)])
def test_host_check(tmp_path, src, ulps):
    exe = tmp_path / src
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DGRF_HOST_ULPS=({ulps})", "-I",
                    os.path.join(ROOT, "eigenrand_gb300", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", src + ".cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0 of" in r.stdout

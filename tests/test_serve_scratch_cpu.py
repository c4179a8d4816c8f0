"""Host-side checks of how the serving loop admits requests with scratch (no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_admission_with_scratch(tmp_path):
    exe = tmp_path / "admit_scratch_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "admit_scratch_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

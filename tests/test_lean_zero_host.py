"""The products of qsl_gb300/csrc/lean.cuh that take zeros, and those by constants
that are powers of two, equal the host's IEEE arithmetic bit for bit."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_zeros_and_powers_of_two_match_ieee(tmp_path):
    exe = os.path.join(str(tmp_path), "lean_zero_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "qsl_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "lean_zero_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "lean zero ok" in r.stdout

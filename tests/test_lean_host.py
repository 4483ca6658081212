"""The products and the division of qsl_gb300/csrc/lean.cuh equal the host's
IEEE round-to-nearest arithmetic bit for bit on every operand they accept."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lean_arithmetic_matches_ieee(tmp_path):
    exe = os.path.join(str(tmp_path), "lean_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "qsl_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "lean_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "4000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "lean ok" in r.stdout


def test_single_precision_division_step_matches_ieee(tmp_path):
    exe = os.path.join(str(tmp_path), "fdiv_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "qsl_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "fdiv_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "fdiv ok" in r.stdout


def test_squares_match_ieee(tmp_path):
    exe = os.path.join(str(tmp_path), "square_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "qsl_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "square_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "4000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "square ok" in r.stdout

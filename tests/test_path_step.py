"""Host check of single fixed-point path steps (no GPU): tests/cpp/step_test.cpp."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_path_step(tmp_path):
    exe = str(tmp_path / "step_test")
    csrc = os.path.join(ROOT, "compfinance_gb300", "csrc")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", csrc, os.path.join(ROOT, "tests", "cpp", "step_test.cpp"),
                           *(os.path.join(csrc, f) for f in ("fx_tables.cpp", "inv_normal64.cpp", "host_math.cpp")),
                           "-ffp-contract=off", "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and all(x.startswith("ok") for x in r.stdout.splitlines()), r.stdout + r.stderr

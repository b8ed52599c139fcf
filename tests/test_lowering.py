"""Host check of the fixed-point lowering (no GPU): tests/cpp/lowering_test.cpp."""
import os
import platform
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lowering(tmp_path):
    exe = str(tmp_path / "lowering_test")
    csrc = os.path.join(ROOT, "compfinance_gb300", "csrc")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", csrc, os.path.join(ROOT, "tests", "cpp", "lowering_test.cpp"),
                           *(os.path.join(csrc, f) for f in ("fx_tables.cpp", "inv_normal64.cpp", "host_math.cpp")),
                           "-ffp-contract=off", "-o", exe])
    # the time of a 128-bit division is known on x86 only
    r = subprocess.run([exe] + (["time"] if platform.machine() == "x86_64" else []), capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and all(x.startswith("ok") for x in r.stdout.splitlines()), r.stdout + r.stderr

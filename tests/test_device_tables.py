"""Host check of the device tables' uploads against a stand-in for the CUDA runtime (no GPU):
tests/cpp/tables_test.cpp."""
import os
import subprocess

from compfinance_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "compfinance_gb300", "csrc")


def test_device_tables(tmp_path):
    exe = str(tmp_path / "tables_test")
    inc = os.path.join(B._cuda_home(), "include")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", CSRC, "-I", inc, "-ffp-contract=off",
                           os.path.join(ROOT, "tests", "cpp", "tables_test.cpp"),
                           *(os.path.join(CSRC, f) for f in ("device_buf.cpp", "fx_plan.cpp", "fx_tables.cpp",
                                                             "inv_normal64.cpp", "host_math.cpp")), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and all(x.startswith("ok") for x in r.stdout.splitlines()), r.stdout + r.stderr

"""Host check of the accumulators' two words (no GPU): tests/cpp/split_test.cpp."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_split_words_and_sums(tmp_path):
    exe = str(tmp_path / "split_test")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "compfinance_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "split_test.cpp"), "-ffp-contract=off", "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and all(x.startswith("ok") for x in r.stdout.splitlines()), r.stdout + r.stderr

"""The overflow check of the mixed form's 32-bit weight sums leaves no sum that
can wrap before the next check, whatever order the fused kernel's warps run
in.  CPU only: the same constants are compiled into the library."""
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_sum_can_wrap_between_checks():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "sums_check")
        subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(HERE, "sums_check.cpp"), "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    assert r.stdout.strip().endswith("0 failures"), r.stdout

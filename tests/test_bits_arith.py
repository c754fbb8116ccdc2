"""The integer and fused forms of FP64 operations in
cpic_gb300/csrc/cpic_bits.h give the FP64 operations' results bit for bit.
CPU only: the same header is compiled for the device."""
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))


def test_arithmetic_matches_fp64():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "bits_arith_check")
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                        os.path.join(HERE, "bits_arith_check.cpp"), "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    assert r.stdout.strip().startswith("0 mismatches"), r.stdout

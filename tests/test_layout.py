"""The tile sizes chosen by cpic_gb300/csrc/cpic_layout.h keep the kernels'
indices in range on every grid, narrow ones among them.  CPU only: the same
header is compiled into the library."""
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))


def test_field_tiles_stay_on_the_grid():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "layout_check")
        subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(HERE, "layout_check.cpp"), "-o", exe],
                       check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    assert r.stdout.strip().endswith("0 failures"), r.stdout

"""The word of a minimizer bin (spades-rs_b200/csrc/spk_bins.h) on the CPU: a bin
with more records than its field counts is reported before a rank repeats."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_bin_word(tmp_path):
    exe = str(tmp_path / "bins_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", os.path.join(HERE, "bins_test.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "bins ok" in r.stdout, r.stdout + r.stderr

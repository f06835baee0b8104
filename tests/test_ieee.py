"""The branch-free IEEE reciprocal, quotient and square root of the serial
kernels (csrc/pd_ieee.h) against the processor's own operators."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_refinements_equal_the_ieee_operators(tmp_path):
    exe = str(tmp_path / "ieee_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "native", "ieee_check.cpp")], check=True)
    r = subprocess.run([exe, "3000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("ok")

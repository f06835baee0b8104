"""The seeds of csrc/pd_ieee.h: the square root within the bound its header
states (CPU), and the device's own seeds (GPU), whose accuracy the serial
mode's bit-exactness rests on."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_roots_from_any_seed_within_the_stated_bound(tmp_path):
    exe = str(tmp_path / "ieee_root_bound")
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "native", "ieee_root_bound.cpp")], check=True)
    r = subprocess.run([exe, "6000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("ok")


@pytest.mark.gpu
def test_device_seeds_and_results(tmp_path):
    """Every leading 21 bits of a significand with several tails: the seeds are
    within the bounds of the header, and what the refinements report as exact
    equals the device's IEEE operators."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "ieee_device")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-fmad=false",
                    "--expt-relaxed-constexpr", "-o", exe, os.path.join(HERE, "native", "ieee_device.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok")

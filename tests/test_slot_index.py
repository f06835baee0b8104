"""Index arithmetic of the serial slice kernels (csrc/pd_slots.h), checked on
the CPU: a small C++ program walks every slot of every lane of lattice blocks
with padding lanes, several types and neighbouring blocks."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_slot_of_every_lane_stays_in_its_tables(tmp_path):
    exe = str(tmp_path / "slot_index_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-o", exe,
                    os.path.join(HERE, "native", "slot_index_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("ok ")

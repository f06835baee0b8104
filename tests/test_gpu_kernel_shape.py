"""Kernel shapes of the throughput modes: the shape an environment was tuned to
can be pinned on another one, the sixteen-warp shape only where the tuner may
choose it, and the tuner's cache keeps to that limit."""
import os
import subprocess
import sys

import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import _abi, configs
from peridyn_b200.environment import GeneralEnvironment

from .cases import ep_cube

pytestmark = pytest.mark.gpu

HI = {"fp64": 2, "fp32c": 4}
LO = {"fp64": 1, "fp32c": 2}


def _workload(law):
    if law == "ep":
        return ep_cube(1e8)
    return configs.lps_cube((9, 8, 7)) if law == "lps" else configs.pmb_cube(n=8, peak=20.0)


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("law", ["pmb", "lps", "ep"])
def test_a_sixteen_warp_shape_can_be_pinned(monkeypatch, precision, law):
    """env.set_kernel_shape(*other.kernel_shape()), before and after finalize:
    the same bits."""
    u = LO[precision] if law == "ep" else HI[precision]
    w = _workload(law)
    monkeypatch.setenv("PD_KERNEL_SHAPE", f"16,{u}")
    env = pb.Env(1, w["materials"], [], [], w["dt"], precision=precision)
    pb.velocity_verlet_step(env, nsteps=12)
    monkeypatch.delenv("PD_KERNEL_SHAPE")
    assert env.kernel_shape() == (16, u)
    for finalized in (True, False):
        b = GeneralEnvironment(1, w["materials"], [], [], w["dt"], precision=precision, finalize=finalized)
        b.set_kernel_shape(*env.kernel_shape())
        if not finalized:
            _abi.check(_abi.lib().pd_env_finalize(b._h))
        pb.velocity_verlet_step(b, nsteps=12)
        assert b.kernel_shape() == (16, u)
        for s, t in zip(env.get_state(), b.get_state()):
            assert np.array_equal(s, t)
        # refused: the unroll that has no sixteen-warp kernel, warps in between
        for bad in ((16, LO[precision] + HI[precision] - u), (12, u), (32, u)):
            assert _abi.lib().pd_env_set_kernel_shape(b._h, *bad) == _abi.PD_ERR_ARG
        b.close()
    env.close()


def test_sixteen_warps_are_refused_above_the_limit():
    w = configs.pmb_cube(dims=(41, 40, 40))  # 65,600 particles
    env = pb.Env(1, w["materials"], [], [], w["dt"], precision="fp32c")
    assert _abi.lib().pd_env_set_kernel_shape(env._h, 16, 4) == _abi.PD_ERR_ARG
    env.set_kernel_shape(8, 4)
    env.close()

def test_tuned_shapes_are_not_shared_across_the_limit():
    """65,600 and 65,536 particles lie in one class of sizes; only the smaller
    body may run, and is timed with, sixteen warps per slice."""
    code = ("import peridyn_b200 as pb\n"
            "from peridyn_b200 import configs\n"
            "for dims in ((41, 40, 40), (64, 32, 32)):\n"
            "    w = configs.pmb_cube(dims=dims)\n"
            "    env = pb.Env(1, w['materials'], [], [], w['dt'], precision='fp32c')\n"
            "    pb.velocity_verlet_step(env, nsteps=2)\n")
    env = dict(os.environ, PD_TUNE_LOG="1")
    env.pop("PD_KERNEL_SHAPE", None)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    lines = [s for s in r.stderr.splitlines() if s.startswith("pd autotune")]
    assert [s.split()[2] for s in lines] == ["N=65600:", "N=65536:"]
    assert " 16,4=" not in lines[0] and " 16,4=" in lines[1]

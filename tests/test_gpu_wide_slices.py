"""The throughput modes with sixteen warps per slice (chosen by the
autotuner for small environments, forced here): slot lists of 32 to 320
entries, so that the warps' ranges are short, rounded and partly empty.
Displacements and velocities against the oracle within the throughput modes'
bounds (relative L2: FP64 1e-10, FP32C 1e-4)."""
import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import lattice

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "fp32c": 1e-4}


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("layout", ["auto", "explicit"])
@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("law,factor", [("pmb", 1.2), ("lps", 1.8), ("pmb", 2.4), ("lps", 2.7), ("pmb", 3.015),
                                        ("lps", 3.015), ("ep", 2.7), ("pmb", 4.2)])
def test_sixteen_warps_per_slice(oracle, monkeypatch, layout, precision, law, factor):
    if layout == "explicit":
        monkeypatch.setenv("PD_FAMILY_LAYOUT", "explicit")
    hi = {"fp64": 2, "fp32c": 4}[precision]
    lo = {"fp64": 1, "fp32c": 2}[precision]
    monkeypatch.setenv("PD_KERNEL_SHAPE", f"16,{lo if law == 'ep' else hi}")
    x, vol = lattice.cuboid(11, 9, 7, 1.0e-3, jitter=1.0e-5, seed=9)
    gen = pb.GeneralMaterial(x.copy(order="F"), lattice.gaussian_pulse(x, 20.0, 3.0e-3), x, vol,
                             np.ones(x.shape[1], dtype=np.int64), factor * 1.0e-3, max_neigh=400)
    spc = {"pmb": lambda: pb.BondBasedSpecific([14.9e9], [0.05], [2200.0]),
           "lps": lambda: pb.OrdinaryStateBasedSpecific([20e9], [9e9], [0.05], [2000.0]),
           "ep": lambda: pb.ElastoPlasticSolidSpecific([46.7e9], [28e9], [0.05], [2700.0], [1e8])}[law]()
    m = pb.PeridynamicsMaterial(gen, spc)
    env = pb.Env(1, [m], [], [], 1.0e-8, precision=precision)
    ora = oracle.OracleEnv([m], [], [], 1.0e-8)
    pb.velocity_verlet_step(env, nsteps=40)
    assert env.kernel_shape()[0] == 16
    for _ in range(40):
        ora.vv_step()
    assert _rel(env.y - x, ora.y - x) <= TOL[precision]
    assert _rel(env.v, ora.v) <= TOL[precision]
    env.close()

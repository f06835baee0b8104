"""The FP64 throughput mode far from SI lengths.  A bond's reciprocal weight is
one inverse root of a sixth power of its length, so the records are held in a
power-of-two unit near the bonds' length; the results are those of the
oracle within the mode's bound (relative L2 1e-10) at every scale at which the
materials' own constants are finite."""
import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import lattice

pytestmark = pytest.mark.gpu


def _rel(a, b):
    s = np.abs(b).max()
    return float(np.linalg.norm(a / s - b / s) / np.linalg.norm(b / s))


def _block(law, scale, first_type=1, offset=0.0, dims=(9, 7, 6)):
    """Strained by up to 1e-3, one corner pulled well past the critical stretch."""
    x, vol = lattice.cuboid(*dims, 1.0, jitter=0.02, seed=3)
    rng = np.random.default_rng(5)
    y = x * (1.0 + 1e-3 * np.array([[1.0], [-0.3], [0.2]])) + rng.normal(0.0, 2e-5, x.shape)
    corner = np.linalg.norm(x - x.max(axis=1, keepdims=True), axis=0) < 1.5
    y[:, corner] += 0.6
    x, y = x + offset, y + offset
    x, y = np.asfortranarray(x * scale), np.asfortranarray(y * scale)
    n = x.shape[1]
    gen = pb.GeneralMaterial(y, np.zeros((3, n), order="F"), x, np.full(n, vol.mean()) * scale ** 3,
                             np.full(n, first_type, dtype=np.int64), 2.5 * scale, max_neigh=150)
    spc = {"pmb": lambda: pb.BondBasedSpecific([14.9e9], [0.05], [2200.0]),
           "lps": lambda: pb.OrdinaryStateBasedSpecific([20e9], [9e9], [0.05], [2000.0]),
           "ep": lambda: pb.ElastoPlasticSolidSpecific([46.7e9], [28e9], [0.05], [2700.0], [3e7])}[law]()
    return pb.PeridynamicsMaterial(gen, spc)


def _compare(oracle, mats, tol=1e-10):
    env = pb.Env(1, mats, [], [], 1.0, precision="fp64")
    ora = oracle.OracleEnv(mats, [], [], 1.0)
    pb.update_acc(env)
    ora.update_acc()
    assert np.isfinite(ora.f).all() and np.abs(ora.f).max() > 0.0
    assert _rel(env.f, ora.f) <= tol
    for b, B in enumerate(ora.blocks):
        assert np.array_equal(env._family(b)[1], B.intact.astype(bool))
        assert B.intact.sum() < (B.family > 0).sum()
    env.close()
    # a step size that moves the particles by about 1e-4 spacings a step
    spacing = max(m.general.horizon for m in mats) / 2.5
    dt = float(np.sqrt(1e-4 * spacing / np.abs(ora.f).max()))
    env = pb.Env(1, mats, [], [], dt, precision="fp64")
    ora = oracle.OracleEnv(mats, [], [], dt)
    pb.update_acc(env)
    ora.update_acc()
    pb.velocity_verlet_step(env, nsteps=20)
    for _ in range(20):
        ora.vv_step()
    x = np.concatenate([m.general.x for m in mats], axis=1)
    assert _rel(env.y - x, ora.y - x) <= tol
    assert _rel(env.v, ora.v) <= tol
    env.close()


@pytest.mark.parametrize("layout", ["auto", "explicit"])
@pytest.mark.parametrize("law,scale", [("pmb", 1e-3), ("lps", 1e-3), ("pmb", 1e-55), ("lps", 1e-55), ("pmb", 1e55),
                                       ("lps", 1e55), ("ep", 1e-3), ("ep", 1e-33), ("ep", 1e38)])
def test_lengths_far_from_one(oracle, monkeypatch, layout, law, scale):
    if layout == "explicit":
        monkeypatch.setenv("PD_FAMILY_LAYOUT", "explicit")
    _compare(oracle, [_block(law, scale)])


@pytest.mark.parametrize("laws,scale", [(("lps", "ep"), 1e-33), (("pmb", "ep"), 1e38)])
def test_blocks_of_two_laws(oracle, laws, scale):
    _compare(oracle, [_block(laws[0], scale), _block(laws[1], scale, 2, 40.0)])


@pytest.mark.parametrize("scale", [1e-3, 1e-55])
def test_halo_records_carry_the_displacement_itself(scale):
    """Packed on one environment, unpacked on another: the same state, in the
    environment's unit whatever the records' is."""
    import ctypes

    import torch

    from peridyn_b200 import _abi

    L = _abi.lib()
    mats = [_block("lps", scale)]
    src = pb.Env(1, mats, [], [], 1.0, precision="fp64")
    dst = pb.Env(1, mats, [], [], 1.0, precision="fp64")
    y, v, f, _ = src.get_state()
    rng = np.random.default_rng(1)
    y = np.asfortranarray(y + rng.normal(0.0, 1e-3 * scale, y.shape))
    v = np.asfortranarray(rng.normal(0.0, scale, y.shape))
    _abi.check(L.pd_env_set_state(src._h, _abi.dptr(y), _abi.dptr(v), _abi.dptr(f)))
    pb.update_acc(src)
    pb.update_acc(dst)
    n = y.shape[1]
    idx = torch.arange(n, dtype=torch.int64, device="cuda")
    buf = torch.zeros(9 * n, dtype=torch.float64, device="cuda")
    _abi.check(L.pd_env_pack_halo(src._h, ctypes.c_void_p(idx.data_ptr()), n, ctypes.c_void_p(buf.data_ptr())))
    torch.cuda.synchronize()
    x = mats[0].general.x
    assert np.array_equal(buf.cpu().numpy().reshape(n, 9)[:, :3], (y - x).T)
    _abi.check(L.pd_env_unpack_halo(dst._h, ctypes.c_void_p(idx.data_ptr()), n, ctypes.c_void_p(buf.data_ptr())))
    for a, b in zip(src.get_state()[:3], dst.get_state()[:3]):
        assert np.array_equal(a, b)
    src.close()
    dst.close()

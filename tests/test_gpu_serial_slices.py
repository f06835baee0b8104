"""The serial mode's block-per-slice force and dilatation kernels at the
edges of their split, bit-identical to the oracle's serial loop: slot counts
around the runs each warp takes and above what a block holds in shared
memory (the particle loop takes those slices), more and fewer slices than
SMs, both laws with one and two types, undisturbed bonds (zero stretch),
bonds outside the branch-free arithmetic's range, and an accumulator that
holds -0.0."""
import ctypes

import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import _abi, lattice

pytestmark = pytest.mark.gpu


def _body(law, dims, factor, ntypes=1, scale=1.0, jitter=2.0e-5):
    """A cuboid whose first planes move; the rest starts undisturbed."""
    h = 1.0e-3 * scale
    x, vol = lattice.cuboid(*dims, h, jitter=jitter * scale, seed=5)
    v = lattice.gaussian_pulse(x, 40.0 * scale, 2.0 * h)
    t = np.where(x[0] < np.median(x[0]), 1, ntypes).astype(np.int64)
    gen = pb.GeneralMaterial(x.copy(order="F"), v, x, vol, t, factor * h, max_neigh=700)
    pairs = ntypes * (ntypes + 1) // 2
    rho = [2200.0, 2500.0][:ntypes]
    if law == "pmb":
        spc = pb.BondBasedSpecific([14.9e9] * pairs, [0.003, 0.004, 0.005][:pairs], rho)
    else:
        spc = pb.OrdinaryStateBasedSpecific([20e9, 21e9, 22e9][:pairs], [9e9, 8e9, 7e9][:pairs],
                                            [0.003, 0.004, 0.005][:pairs], rho)
    return pb.PeridynamicsMaterial(gen, spc)


def _same(env, ora):
    y, v, f, _ = env.get_state()
    assert np.array_equal(f, ora.f)
    assert np.array_equal(v, ora.v)
    assert np.array_equal(y, ora.y)
    for b, B in enumerate(ora.blocks):
        assert np.array_equal(env._family(b)[1], B.intact.astype(bool))


@pytest.mark.parametrize("layout", ["auto", "explicit"])
@pytest.mark.parametrize("law,dims,factor,ntypes,scale", [
    ("pmb", (3, 1, 1), 1.5, 1, 1.0),      # two slots, one slice
    ("lps", (7, 3, 3), 1.1, 2, 1.0),      # fewer slots than warps
    ("pmb", (9, 8, 8), 2.0, 2, 1.0),      # 26..32 slots
    ("lps", (9, 8, 8), 2.3, 1, 1.0),      # 33..64 slots
    ("lps", (26, 16, 15), 3.015, 2, 1.0),  # more slices than SMs
    ("pmb", (22, 18, 17), 3.015, 1, 1.0),
    ("pmb", (12, 11, 10), 4.2, 1, 1.0),   # 304 slots inside: above the block's capacity
    ("lps", (12, 11, 10), 4.2, 1, 1.0),
    ("lps", (6, 5, 5), 3.015, 1, 1e-32),  # lengths below 2^-100
    ("pmb", (6, 5, 5), 3.015, 1, 1e-32),
])
def test_slice_kernels_match_the_serial_loop(oracle, monkeypatch, layout, law, dims, factor, ntypes, scale):
    if layout == "explicit":
        monkeypatch.setenv("PD_FAMILY_LAYOUT", "explicit")
    m = _body(law, dims, factor, ntypes, scale)
    dt = 2.0e-8
    env = pb.Env(1, [m], [], [], dt)
    ora = oracle.OracleEnv([m], [], [], dt)
    pb.update_acc(env)
    ora.update_acc()
    pb.velocity_verlet_step(env, nsteps=12)
    for _ in range(12):
        ora.vv_step()
    _same(env, ora)
    env.close()


@pytest.mark.parametrize("law", ["pmb", "lps"])
def test_accumulating_into_negative_zeros(oracle, law):
    """force_density_T! adds into f: an entry of -0.0 stays -0.0 where every
    term is a negative zero or absent."""
    import torch

    x, vol = lattice.cuboid(6, 6, 5, 1.0e-3, centered=False)
    y = np.asfortranarray(x * np.array([[1.0 + 1.0e-4], [1.0], [1.0]]))
    gen = pb.GeneralMaterial(y, np.zeros_like(x, order="F"), x, vol, np.ones(x.shape[1], dtype=np.int64), 3.015e-3,
                             max_neigh=200)
    spc = (pb.BondBasedSpecific([14.9e9], [0.005], [2200.0]) if law == "pmb" else
           pb.OrdinaryStateBasedSpecific([20e9], [9e9], [0.004], [2000.0]))
    m = pb.PeridynamicsMaterial(gen, spc)
    env = pb.Env(1, [m], [], [], 1.0e-8)
    ora = oracle.OracleEnv([m], [], [], 1.0e-8)
    f0 = np.zeros_like(x, order="F")
    f0[:, ::3] = -0.0
    ora.f[:] = f0
    ora.force_density_T(ora.blocks[0])
    yd = torch.from_numpy(np.ascontiguousarray(y.T)).cuda()
    fd = torch.from_numpy(np.ascontiguousarray(f0.T)).cuda()
    _abi.check(_abi.lib().pd_force_density_device(env._h, 0, ctypes.c_void_p(fd.data_ptr()),
                                                  ctypes.c_void_p(yd.data_ptr()), None))
    f = fd.cpu().numpy().T
    assert np.array_equal(f, ora.f)
    assert np.array_equal(np.signbit(f), np.signbit(ora.f))
    env.close()


@pytest.mark.parametrize("conditions", [1, 4, 9])  # fused integration: at most 8
def test_several_conditions_on_the_same_particles(oracle, conditions):
    m = _body("lps", (14, 6, 5), 3.015)
    x = m.general.x
    lo, hi = x[0].min(), x[0].max()
    bcs = [pb.FixBC(x[0] < lo + 2.0e-3, dims=(True, False, True)),
           pb.ToFroBC(x[0] > hi - 2.0e-3, [0.5, 0.0, -0.25], 5.0, applyafter=3),
           pb.ContainerBC(x[1] < x[1].mean(), limits=None),
           pb.ContainerBC(x[0] > lo + 5.0e-3, limits=np.array([[lo, hi], [x[1].min(), x[1].max()],
                                                               [x[2].min(), x[2].max()]]))]
    bcs += [pb.FixBC((x[0] < lo + 1.5e-3) & (x[1] < x[1].min() + k * 1.0e-3), dims=(False, True, False))
            for k in range(1, 6)]
    bcs = bcs[:conditions]
    env = pb.Env(1, [m], [], bcs, 2.0e-8)
    ora = oracle.OracleEnv([m], [], bcs, 2.0e-8)
    ora.apply_bc_at0()
    pb.apply_bc_at0(env, 0)
    for n in (1, 9, 6):
        pb.velocity_verlet_step(env, nsteps=n)
        for _ in range(n):
            ora.vv_step()
    _same(env, ora)
    assert np.array_equal(env.p, ora.p)
    env.close()


@pytest.mark.parametrize("max_iter,f_tol", [(1, 1e-3), (2, 1e-3), (3, 1e-3), (7, 1e-3), (40, 1e-3), (40, 1e30),
                                            (40, "fifth")])
def test_minimize_stops_where_the_loop_does(oracle, max_iter, f_tol):
    """Iterations run in batches between two reads of the progress; the state
    is the one of the iteration that converged."""
    def build():
        m = _body("lps", (11, 5, 5), 3.015, jitter=0.0)
        x = m.general.x
        m.general.velocity[:] = 0.0
        bcs = [pb.FixBC(x[0] < x[0].min() + 1.5e-3), pb.MoveBC(x[0] > x[0].max() - 1.5e-3, [10.0, 0.0, 0.0])]
        return m, bcs

    if f_tol == "fifth":  # a tolerance the fifth iteration is the first to meet
        m, bcs = build()
        ora = oracle.OracleEnv([m], [], bcs, 1.0e-7)
        ora.apply_bc_at0()
        seen = []
        for n in range(1, 8):
            m, bcs = build()
            o = oracle.OracleEnv([m], [], bcs, 1.0e-7)
            o.apply_bc_at0()
            o.minimize(1.0e-7, 10.0, max_iter=n, x_tol=1e-30, f_tol=1e-30)
            free = (bcs[0].bool == 0) & (bcs[1].bool == 0)
            seen.append(np.abs(o.f[:, free]).max())
        k = int(np.argmin(seen))
        f_tol = np.nextafter(seen[k], np.inf)
    m, bcs = build()
    env = pb.Env(1, [m], [], bcs, 1.0e-7)
    ora = oracle.OracleEnv([m], [], bcs, 1.0e-7)
    ora.apply_bc_at0()
    pb.apply_bc_at0(env, 0)
    for _ in range(2):
        it = pb.minimize(env, pb.QSDrag(1.0e-7, 10.0, max_iter=max_iter, x_tol=1e30, f_tol=f_tol))
        assert it == ora.minimize(1.0e-7, 10.0, max_iter=max_iter, x_tol=1e30, f_tol=f_tol)
        _same(env, ora)
        assert np.array_equal(env.p, ora.p)
    env.close()

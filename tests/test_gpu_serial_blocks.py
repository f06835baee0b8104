"""The serial mode's slice kernels in environments of several blocks, some
with several types, whose particle counts leave padding lanes and whose
stencils reach into the neighbouring block's records: bit-identical to the
oracle's serial loop."""
import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import lattice

pytestmark = pytest.mark.gpu


def block(law, dims, ntypes, first_type, offset, factor=2.3, seed=5):
    h = 1.0e-3
    x, vol = lattice.cuboid(*dims, h, jitter=2.0e-5, seed=seed)
    x = np.asfortranarray(x + np.array([[offset], [0.0], [0.0]]))
    v = lattice.gaussian_pulse(x, 40.0, 2.0e-3)
    t = (first_type + (np.arange(x.shape[1]) * 7 // 5) % ntypes).astype(np.int64)
    gen = pb.GeneralMaterial(x.copy(order="F"), v, x, vol, t, factor * h, max_neigh=200)
    pairs = ntypes * (ntypes + 1) // 2
    r = np.linspace(1.0, 1.2, pairs)
    rho = list(np.linspace(2000.0, 2600.0, ntypes))
    cs = list(0.003 * r)
    if law == "ep":
        return pb.PeridynamicsMaterial(gen, pb.ElastoPlasticSolidSpecific(list(46.7e9 * r), list(28e9 * r), cs, rho,
                                                                          list(2e7 * r)))
    if law == "pmb":
        return pb.PeridynamicsMaterial(gen, pb.BondBasedSpecific(list(14.9e9 * r), cs, rho))
    return pb.PeridynamicsMaterial(gen, pb.OrdinaryStateBasedSpecific(list(20e9 * r), list(9e9 * r), cs, rho))


def three_blocks(law, sizes, factor=2.3):
    other = "lps" if law == "pmb" else "pmb"
    return [block(other, sizes[0], 3, 1, 0.0, factor), block(law, sizes[1], 2, 4, 0.03, factor, seed=6),
            block(law, sizes[2], 5, 6, 0.06, factor, seed=7)]


@pytest.mark.parametrize("law", ["pmb", "lps"])
@pytest.mark.parametrize("sizes", [((7, 3, 3), (5, 5, 5), (3, 3, 3)), ((8, 4, 4), (9, 7, 5), (4, 4, 2)),
                                   ((3, 1, 1), (26, 16, 15), (1, 2, 3))])
def test_blocks_of_several_types(oracle, law, sizes):
    mats = three_blocks(law, sizes)
    env = pb.Env(1, mats, [], [], 2.0e-8)
    ora = oracle.OracleEnv(mats, [], [], 2.0e-8)
    pb.update_acc(env)
    ora.update_acc()
    pb.velocity_verlet_step(env, nsteps=15)
    for _ in range(15):
        ora.vv_step()
    y, v, f, _ = env.get_state()
    assert np.array_equal(f, ora.f)
    assert np.array_equal(v, ora.v)
    assert np.array_equal(y, ora.y)
    for b, B in enumerate(ora.blocks):
        assert np.array_equal(env._family(b)[1], B.intact.astype(bool))
    env.close()


@pytest.mark.parametrize("entry", ["pd_force_density_device_static", "pd_force_density_device"])
@pytest.mark.parametrize("law", ["pmb", "lps"])
@pytest.mark.parametrize("dims,factor", [((9, 7, 5), 2.3), ((36, 32, 32), 1.1)])  # a block per slice, a thread each
def test_one_block_of_several_through_device_pointers(oracle, law, dims, factor, entry):
    """Each block by itself, in turn; the other blocks' positions are NaN."""
    import ctypes

    import torch

    from peridyn_b200 import _abi

    mats = three_blocks(law, ((7, 3, 3), dims, (3, 3, 3)), factor)
    env = pb.Env(1, mats, [], [], 2.0e-8)
    ora = oracle.OracleEnv(mats, [], [], 2.0e-8)
    rng = np.random.default_rng(4)
    ora.y[:] = ora.y + rng.normal(0.0, 1e-6, size=ora.y.shape)
    f0 = np.asfortranarray(rng.normal(0.0, 1.0, size=ora.y.shape))
    ora.f[:] = f0
    for b, B in enumerate(ora.blocks):
        own = slice(B.off, B.off + B.n)
        y = np.full_like(ora.y, np.nan)
        y[:, own] = ora.y[:, own]
        yd = torch.from_numpy(np.ascontiguousarray(y.T)).cuda()
        fd = torch.from_numpy(np.ascontiguousarray(f0.T)).cuda()
        _abi.check(getattr(_abi.lib(), entry)(env._h, b, ctypes.c_void_p(fd.data_ptr()),
                                              ctypes.c_void_p(yd.data_ptr()), None))
        f = fd.cpu().numpy().T
        ora.force_density_T(B)
        assert np.array_equal(f[:, own], ora.f[:, own])
        assert np.array_equal(np.delete(f, np.r_[own], axis=1), np.delete(f0, np.r_[own], axis=1))
        assert np.array_equal(env._family(b)[1], B.intact.astype(bool))
    env.close()


@pytest.mark.parametrize("law", ["pmb", "lps"])
@pytest.mark.parametrize("factor,dims", [(1.1, (36, 32, 32)),   # 6 slots, 1152 slices: threads
                                         (1.1, (24, 25, 24)),   # 450 slices: warps per slice
                                         (1.5, (46, 42, 40)),   # 18 slots, 2415 slices: threads
                                         (2.1, (52, 51, 46))])  # 32 slots, 3812 slices: dilatation by threads
def test_short_slot_lists_on_many_slices(oracle, law, factor, dims):
    """A thread per particle or a block per slice: the same numbers."""
    m = block(law, dims, 2, 1, 0.0, factor=factor)
    env = pb.Env(1, [m], [], [], 2.0e-8)
    ora = oracle.OracleEnv([m], [], [], 2.0e-8)
    pb.velocity_verlet_step(env, nsteps=6)
    for _ in range(6):
        ora.vv_step()
    y, v, f, _ = env.get_state()
    assert np.array_equal(f, ora.f)
    assert np.array_equal(v, ora.v)
    assert np.array_equal(y, ora.y)
    assert np.array_equal(env._family(0)[1], ora.blocks[0].intact.astype(bool))
    env.close()


@pytest.mark.parametrize("larger", ["ep", "others"])
def test_many_alternating_blocks(oracle, larger):
    """More runs of blocks than are launched one by one (the elasto-plastic
    force has the thread form only): one launch in the form of the larger part."""
    mats, t = [], 1
    for k in range(12):
        law, nt = ("ep", "pmb", "ep", "lps")[k % 4], 1 + k % 3
        n = 6 if (law == "ep") == (larger == "ep") else 3
        mats.append(block(law, (4 + k % 4, n, 3), nt, t, 0.02 * k, seed=k))
        t += nt
    env = pb.Env(1, mats, [], [], 2.0e-8)
    ora = oracle.OracleEnv(mats, [], [], 2.0e-8)
    pb.velocity_verlet_step(env, nsteps=10)
    for _ in range(10):
        ora.vv_step()
    y, v, f, _ = env.get_state()
    assert np.array_equal(f, ora.f)
    assert np.array_equal(y, ora.y)
    env.close()


@pytest.mark.parametrize("peak", [0.0, 0.1, 40.0])
@pytest.mark.parametrize("law,factor", [("lps", 2.3), ("pmb", 2.6)])
def test_bodies_that_are_undeformed_at_first(oracle, law, factor, peak):
    """Many slices of a body that is undeformed throughout, for the first steps
    only, or from the start, between two small ones that move; an odd number of
    evaluations, so both buffers of the bond flags are read."""
    mats = [block("pmb", (5, 4, 3), 1, 1, -0.02), block(law, (48, 44, 37), 2, 2, 0.0, factor=factor),
            block("lps", (6, 5, 4), 1, 4, 0.06)]
    gen = mats[1].general
    gen.velocity[:] = lattice.gaussian_pulse(gen.x, peak, 4.0e-3) if peak else 0.0
    env = pb.Env(1, mats, [], [], 2.0e-8)
    ora = oracle.OracleEnv(mats, [], [], 2.0e-8)
    for n in (9, 4):
        pb.velocity_verlet_step(env, nsteps=n)
        for _ in range(n):
            ora.vv_step()
        y, v, f, _ = env.get_state()
        assert np.array_equal(f, ora.f)
        assert np.array_equal(v, ora.v)
        assert np.array_equal(y, ora.y)
        for b, B in enumerate(ora.blocks):
            assert np.array_equal(env._family(b)[1], B.intact.astype(bool))
    assert bool(ora.blocks[1].deformed) == (peak > 0.0)
    env.close()

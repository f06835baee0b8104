"""Paths of the stepping code that the larger tests pass by: a quasi-static
batch that converges in an elasto-plastic body (whose plastic strains change
buffers with every evaluation that ran), and the FP32 state-based walk that
takes slots two by two, against the one-slot walk."""
import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import configs, lattice

pytestmark = pytest.mark.gpu


def _pulled_bar():
    x, vol = lattice.cuboid(11, 5, 5, 1.0e-3)
    y = np.asfortranarray(x * np.array([[1.0 + 4.0e-3], [1.0], [1.0]]))
    gen = pb.GeneralMaterial(y, np.zeros_like(x, order="F"), x, vol, np.ones(x.shape[1], dtype=np.int64), 3.015e-3,
                             max_neigh=200)
    m = pb.PeridynamicsMaterial(gen, pb.ElastoPlasticSolidSpecific([46.7e9], [28e9], [0.05], [2700.0], [3e7]))
    bcs = [pb.FixBC(x[0] < x[0].min() + 1.5e-3), pb.MoveBC(x[0] > x[0].max() - 1.5e-3, [10.0, 0.0, 0.0])]
    return m, bcs


@pytest.mark.parametrize("stop", [None, 2, 3, 5, 6, 8])
def test_elasto_plastic_minimize_stops_where_the_loop_does(oracle, stop):
    """stop: the iteration that is the first to meet the tolerance (None: the
    iterations run out), so that a batch of iterations ends inside or at its
    end, after an odd or an even number of evaluations."""
    step = 3.0e-8
    f_tol, max_iter = 1e-30, 9
    if stop:  # |f| falls at first from iteration to iteration
        seen = []
        for n in (stop - 1, stop):
            m, bcs = _pulled_bar()
            o = oracle.OracleEnv([m], [], bcs, 1.0e-7)
            o.apply_bc_at0()
            o.minimize(step, 10.0, max_iter=n, x_tol=1e-30, f_tol=1e-30)
            seen.append(np.abs(o.f[:, (bcs[0].bool == 0) & (bcs[1].bool == 0)]).max())
        assert seen[1] < seen[0]
        f_tol, max_iter = np.nextafter(seen[1], np.inf), 40
    m, bcs = _pulled_bar()
    env = pb.Env(1, [m], [], bcs, 1.0e-7)
    m2, bcs2 = _pulled_bar()
    ora = oracle.OracleEnv([m2], [], bcs2, 1.0e-7)
    ora.apply_bc_at0()
    pb.apply_bc_at0(env, 0)
    for k in range(2):
        it = pb.minimize(env, pb.QSDrag(step, 10.0, max_iter=max_iter, x_tol=1e30, f_tol=f_tol))
        assert it == ora.minimize(step, 10.0, max_iter=max_iter, x_tol=1e30, f_tol=f_tol)
        assert k or it == (stop or max_iter)
        y, v, f, p = env.get_state()
        assert np.array_equal(f, ora.f) and np.array_equal(y, ora.y) and np.array_equal(p, ora.p)
        assert np.array_equal(env.plastic_strain(0), ora.blocks[0].edp)
    assert np.abs(ora.blocks[0].edp).max() > 0.0
    pb.velocity_verlet_step(env, nsteps=3)  # the buffers carry on
    for _ in range(3):
        ora.vv_step()
    assert np.array_equal(env.f, ora.f)
    assert np.array_equal(env.plastic_strain(0), ora.blocks[0].edp)
    env.close()


@pytest.mark.parametrize("unroll", [2, 4])
@pytest.mark.parametrize("dims", [(9, 8, 7), (13, 12, 11)])
def test_paired_slots_equal_single_slots(monkeypatch, unroll, dims):
    """One warp per slice walks the same slots in the same order in both
    layouts; explicit slices take them one by one, stencil slices two by two
    but for a word's last ones."""
    w = configs.lps_cube(dims, cs=0.004, peak=30.0)
    states = []
    for layout in ("auto", "explicit"):
        if layout == "explicit":
            monkeypatch.setenv("PD_FAMILY_LAYOUT", "explicit")
        else:
            monkeypatch.delenv("PD_FAMILY_LAYOUT", raising=False)
        env = pb.Env(1, w["materials"], [], [], w["dt"], precision="fp32c")
        env.set_kernel_shape(1, unroll)
        pb.update_acc(env)
        pb.velocity_verlet_step(env, nsteps=40)
        states.append(env.get_state() + tuple(env._family(0)) + (env.theta(0),))
        env.close()
    for a, b in zip(*states):
        assert np.array_equal(a, b)

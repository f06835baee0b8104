"""Two-block contact search at the edges of its selection buffers: more
candidates than a warp's buffer (1024), more rows than half of it (the
counting path takes those), reverse lists above and below it, one row, and
blocks out of reach.  Neighbour lists and forces bit-identical to the
oracle.  The throughput modes' contact array across list changes."""
import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import _abi

pytestmark = pytest.mark.gpu


def _cloud(n, side, centre, seed, type_id):
    rng = np.random.default_rng(seed)
    x = np.asfortranarray(rng.uniform(-0.5 * side, 0.5 * side, size=(3, n)) + np.asarray(centre).reshape(3, 1))
    v = np.asfortranarray(rng.uniform(-1.0, 1.0, size=(3, n)))
    gen = pb.GeneralMaterial(x.copy(order="F"), v, x, np.full(n, 1.0e-9), np.full(n, type_id, dtype=np.int64), 1.0e-4,
                             max_neigh=200)
    return pb.PeridynamicsMaterial(gen, pb.BondBasedSpecific([10e9], [0.5], [2000.0]))


def _models(n1, n2, side, gap, rows):
    a = _cloud(n1, side, (0.0, 0.0, 0.0), 1, 1)
    b = _cloud(n2, side, (gap, 0.0, 0.0), 2, 2)
    return a, b, pb.NonLinearSpringContactModel(2.0, 1.0e15, a, b, distanceD=1.0, distanceX=3.0, max_neighs=rows)


@pytest.mark.parametrize("n1,n2,side,gap,rows", [
    (1200, 1500, 1.2e-3, 0.0, 512),   # all pairs in reach: buffers cut, long reverse lists
    (1200, 1500, 1.2e-3, 0.0, 600),   # the counting path
    (40, 1500, 1.2e-3, 0.0, 50),
    (1, 1030, 1.0e-3, 0.0, 1030),
    (700, 900, 6.0e-3, 5.0e-3, 50),   # partly in reach
    (33, 70, 3.0e-3, 0.0, 1),
    (20, 30, 1.0e-3, 0.1, 10),        # out of reach
])
def test_search_and_forces(oracle, n1, n2, side, gap, rows):
    a, b, cm = _models(n1, n2, side, gap, rows)
    env = pb.Env(1, [a, b], [cm], [], 1.0e-9)
    ora = oracle.OracleEnv([a, b], [cm], [], 1.0e-9)
    for _ in range(2):
        pb.update_neighs(env)
        ora.update_neighs()
        assert np.array_equal(env.contact_neighs(0), ora.contacts[0].neighs)
        pb.velocity_verlet_step(env, nsteps=2)
        for _ in range(2):
            ora.vv_step()
        y, v, f, _ = env.get_state()
        assert np.array_equal(f, ora.f) and np.array_equal(v, ora.v) and np.array_equal(y, ora.y)
    env.close()


@pytest.mark.parametrize("precision,unroll", [("fp64", 2), ("fp32c", 4)])
def test_lists_that_shrink_leave_no_force_behind(precision, unroll):
    """Stepping after an update that drops particles from the lists computes
    what an environment computes that never had them, bit for bit."""
    a, b, cm = _models(300, 400, 3.0e-3, 1.5e-3, 50)
    y0 = np.asfortranarray(np.hstack([a.general.x, b.general.x]))
    zero = np.zeros_like(y0, order="F")
    far = y0.copy(order="F")
    far[0, 300:] += 2.0e-3

    def run(shifts):
        env = pb.Env(1, [a, b], [cm], [], 1.0e-9, precision=precision)
        env.set_kernel_shape(2, unroll)
        env.set_deformed([True, True], hold=True)
        for y in shifts:
            env.set_state(y=y, v=zero, f=zero)
            _abi.check(_abi.lib().pd_env_reset_bonds(env._h))
            pb.update_neighs(env)
            pb.velocity_verlet_step(env, nsteps=40)  # a graph replay and direct steps
        out = env.get_state()
        touched = int((env.contact_neighs(0) > 0).any(axis=0).sum())
        env.close()
        return out, touched

    (y, v, f, p), few = run([far])
    (y2, v2, f2, p2), same = run([y0, far])
    _, many = run([y0])
    assert 0 < few == same < many
    assert np.array_equal(f, f2) and np.array_equal(v, v2) and np.array_equal(y, y2) and np.array_equal(p, p2)

"""Read-out of large states into buffers of every kind -- fresh, read into
before, at an odd offset, pinned --, whose pages the library maps first where
they are not mapped: the same values, and nothing beyond them written."""
import ctypes

import numpy as np
import pytest

import peridyn_b200 as pb
from peridyn_b200 import _abi, lattice

pytestmark = pytest.mark.gpu


def test_large_reads_into_any_buffer():
    import torch

    L = _abi.lib()
    x, _ = lattice.cuboid(90, 90, 89, 1.0e-3)  # 720,900 particles: 17 MB of positions
    n = x.shape[1]
    gen = pb.GeneralMaterial(x.copy(order="F"), np.zeros_like(x, order="F"), x, np.full(n, 1e-9),
                             np.ones(n, dtype=np.int64), 1.1e-3, max_neigh=20)
    env = pb.Env(1, [pb.PeridynamicsMaterial(gen, pb.BondBasedSpecific([14.9e9], [0.05], [2200.0]))], [], [], 1e-9)
    want = np.asfortranarray(x).ravel(order="F")

    def read(buf, offset):
        p = ctypes.cast(buf + 8 * offset, _abi.c_dp)
        _abi.check(L.pd_env_get_state(env._h, p, None, None, None))

    fresh = np.empty(3 * n + 64)
    pinned = torch.empty(3 * n + 64, dtype=torch.float64).pin_memory().numpy()
    for buf in (fresh, fresh, pinned, pinned):
        for offset in (0, 1, 37):
            buf[offset + 3 * n:] = -7.0
            buf[:offset] = -5.0
            read(buf.ctypes.data, offset)
            assert np.array_equal(buf[offset:offset + 3 * n], want)
            assert (buf[offset + 3 * n:] == -7.0).all() and (buf[:offset] == -5.0).all()
    dam = np.full(n + 8, 3.0)
    _abi.check(L.pd_env_damage(env._h, _abi.dptr(dam)))
    assert (dam[:n] == 0.0).all() and (dam[n:] == 3.0).all()
    env.close()

"""Metropolis sweeps of spins without bonds whose material numbers do not fit
beside the atom index in one 31-bit word (3,000 systems of 175 spins: 20 bits of
index, 12 of material): the sweep must find every spin's own move width."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_materials_beyond_a_word(vgpu_lib):
    from vampire_b200 import batch as B
    from vampire_b200 import system as S
    from vampire_b200 import vgpu as V
    m, k = 175, 3000
    assert (k - 1) << int(m * k).bit_length() >= 1 << 31
    base = S.build("sc", m, 1, 1, 3.0, [S.Material()], [[1e-21]], S.SimParams(H_applied=0.0), spin_seed=1)
    base.nl = base.nl[:0]
    base.jlist = base.jlist[:0]
    base.nl_start[:] = 0
    base.nl_end[:] = -1
    temps = np.linspace(10.0, 900.0, k)
    zero = (0.0, 0.0, 0.0)
    params = [{"temperature": T, "H_start": zero, "H_end": zero, "n_ramp": 0} for T in temps]
    rng = np.random.default_rng(2)
    n = m * k
    rnd = np.concatenate([rng.standard_normal(3 * n), rng.random(n)])
    with B.Batch([base] * k, params, precision="fp64") as b:
        nc = C.c_int32()
        V.check(V.lib().vgpu_mc_setup(b.handle, C.cast(None, V._I32), C.byref(nc)), b.handle)
        V.check(V.lib().vgpu_mc_set_replay(b.handle, rnd.ctypes.data_as(V._D)), b.handle)
        V.check(V.lib().vgpu_mc_sweep(b.handle, C.c_uint64(1)), b.handle)
        got = np.concatenate(b.spins(), axis=1)
    # no field and no anisotropy: every move is accepted, of the width at the system's temperature
    sigma = 0.08 * (temps * 1.3806503e-23 / 9.27400915e-24) ** 0.2
    T = np.tile(base.spins, (1, k)) + rnd[:3 * n].reshape(3, n) * np.repeat(sigma, m)
    want = T / np.sqrt((T * T).sum(0))
    assert np.abs(got - want).max() < 1e-12

"""The workspace that gradients keep between calls is bounded over all handles
of the process (1 GiB) and goes back with its system."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_handles_share_the_bound(vgpu_lib):
    """Three handles whose states take 0.7 GiB each (1,800 steps of 32,768
    spins): only one keeps them, and the next one when that has gone."""
    import torch
    from vampire_b200 import adjoint as A
    from vampire_b200 import vgpu as V
    s = A.system(11.2e-21, 6.69e-24, (0.1, 0.0, 0.4), 32)
    steps = 1800
    target = np.full(steps, 0.9)

    def grad(sim):
        g, loss = np.zeros(5), C.c_double()
        sim._check(V.lib().vgpu_adjoint_llg(sim.handle, C.c_uint64(steps), target.ctypes.data_as(V._D),
                                            C.c_double(1e-16), C.c_int32(0), C.byref(loss), g.ctypes.data_as(V._D)))
        return np.r_[loss.value, g]

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    gib = 1 << 30
    states = steps * 3 * s.n * 4
    sims = [V.Simulation(s) for _ in range(3)]
    try:
        for sim in sims:
            sim.synchronize()
            sim.llg_heun(1)  # loads the kernels
            sim.set_spins(s.spins)
        start = free()
        want = grad(sims[0])
        assert start - free() >= states
        for sim in sims[1:]:
            got = grad(sim)  # with checkpoints: the forward states again, the same sums in another order
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
            assert start - free() <= gib + (32 << 20)
        sims[0].close()
        assert start - free() < states  # given back with the system
        grad(sims[1])
        assert start - free() >= states
    finally:
        for sim in sims:
            sim.close()
    assert start - free() <= 0

"""The workspace that gradients keep between calls is bounded over all handles
of the process (8 GiB) and goes back with its system."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_handles_share_the_bound(vgpu_lib):
    """14 handles whose states take 0.7 GiB each (1,800 steps of 32,768 spins):
    ten keep them, two more the checkpoints, the rest nothing; the last one keeps
    its states when the first has gone."""
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
    sims = [V.Simulation(s) for _ in range(14)]
    try:
        for sim in sims:
            sim.synchronize()
            sim.llg_heun(1)  # loads the kernels
            sim.set_spins(s.spins)
        start = free()
        want = grad(sims[0])
        assert start - free() >= states
        for sim in sims[1:]:
            got = grad(sim)  # the same sums in another order
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
            assert start - free() <= 8 * gib + (32 << 20)
        assert start - free() >= 10 * states
        sims[0].close()
        before = free()
        grad(sims[-1])
        assert before - free() >= states
    finally:
        for sim in sims:
            sim.close()
    assert start - free() <= 0

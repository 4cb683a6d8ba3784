"""Resident launches whose waits for the neighbours' spins run out (their limit
is 1 s): every call that runs such a launch reports it, and the handle works on
afterwards."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,L", [("fp32", 14), ("fp32", 52), ("fp64", 9)])
def test_steps(vgpu_lib, prec, L):
    from vampire_b200 import system as S
    from vampire_b200 import vgpu as V
    s = S.config_sc_llg(L, temperature=300.0)
    with V.Simulation(s, precision=prec, noise_seed=4) as sim:
        sim.set_option(V.OPT_STAGED_RECORDS, 1)  # the passes
        sim.llg_heun(5)
        want = sim.spins()
    with V.Simulation(s, precision=prec, noise_seed=4) as sim:
        sim.set_option(V.OPT_RESIDENT_WAIT_TEST, 1)
        with pytest.raises(V.VGPUError) as e:
            sim.llg_heun(3)
            sim.synchronize()
        assert e.value.code == V.ERR_TIMEOUT
        sim.set_option(V.OPT_RESIDENT_WAIT_TEST, 0)
        sim.set_spins(s.spins)
        sim.step = 0
        sim.llg_heun(5)
        assert np.array_equal(sim.spins(), want)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_trajectory_and_adjoint(vgpu_lib, prec):
    from vampire_b200 import adjoint as A
    from vampire_b200 import vgpu as V
    s = A.system(11.2e-21, 6.69e-24, (0.1, 0.0, 0.4), 9)
    steps = 20
    target = np.full(steps, 0.9)

    def trajectory(sim):
        mz = np.zeros(steps)
        sim._check(V.lib().vgpu_mz_trajectory(sim.handle, C.c_uint64(steps), mz.ctypes.data_as(V._D)))
        return mz

    def gradient(sim):
        g, loss = np.zeros(5), C.c_double()
        sim._check(V.lib().vgpu_adjoint_llg(sim.handle, C.c_uint64(steps), target.ctypes.data_as(V._D),
                                            C.c_double(1e-16), C.c_int32(0), C.byref(loss), g.ctypes.data_as(V._D)))
        return np.r_[loss.value, g]

    with V.Simulation(s, precision=prec) as sim:
        want = trajectory(sim), gradient(sim)
    with V.Simulation(s, precision=prec) as sim:
        for call in (trajectory, gradient):
            sim.set_option(V.OPT_RESIDENT_WAIT_TEST, 1)
            with pytest.raises(V.VGPUError) as e:
                call(sim)
            assert e.value.code == V.ERR_TIMEOUT
            sim.set_option(V.OPT_RESIDENT_WAIT_TEST, 0)
            sim.synchronize()  # reported once
        assert np.array_equal(trajectory(sim), want[0])
        # the same sums, added to the result in another order
        assert np.abs(gradient(sim) - want[1]).max() <= 1e-12 * np.abs(want[1]).max()

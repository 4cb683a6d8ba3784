"""The adjoint with resident threads against the launch-by-launch one (asked for
by a pass option): the same trajectory and loss, gradients to rounding, with
runs shorter and longer than the 64 steps held at once, checkpoint intervals
that do and do not divide the steps, systems that end inside a warp, and the
per-material gradients of a DMI alloy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(s, prec, steps, every, pairs, passes):
    from vampire_b200 import vgpu as V
    rng = np.random.default_rng(steps)
    target = np.ascontiguousarray(0.8 + 0.1 * rng.random(steps))
    M = s.materials.size
    g, pair, loss = np.zeros(5), np.zeros(1 + M * M), C.c_double()
    mz = np.zeros(steps)
    with V.Simulation(s, precision=prec) as sim:
        if passes:
            sim.set_option(V.OPT_STAGED_RECORDS, 1)
        before = sim.spins()
        sim._check(V.lib().vgpu_mz_trajectory(sim.handle, C.c_uint64(steps), mz.ctypes.data_as(V._D)))
        args = (sim.handle, C.c_uint64(steps), target.ctypes.data_as(V._D), C.c_double(1e-16), C.c_int32(every),
                C.byref(loss), g.ctypes.data_as(V._D))
        if pairs:
            sim._check(V.lib().vgpu_adjoint_llg_materials(*args, pair.ctypes.data_as(V._D)))
        else:
            sim._check(V.lib().vgpu_adjoint_llg(*args))
        assert np.array_equal(before, sim.spins())  # the handle's spins are left alone
    return mz, loss.value, g, pair


def _compare(s, prec, steps, every, pairs=False):
    mz, loss, g, pair = _run(s, prec, steps, every, pairs, False)
    mz0, loss0, g0, pair0 = _run(s, prec, steps, every, pairs, True)
    # sums of the same FP64 terms in another order
    assert np.abs(mz - mz0).max() < 1e-13
    assert abs(loss - loss0) < 1e-11 * abs(loss0)
    # gradients: the same operations, contracted differently; a few thousand
    # roundings of the adjoint vector, random in sign
    tol = 1e-5 if prec == "fp32" else 1e-11
    for a, b in ((g[:1], g0[:1]), (g[1:2], g0[1:2]), (g[2:], g0[2:])):
        assert np.abs(a - b).max() <= tol * np.abs(b).max() + 1e-300
    assert np.abs(pair - pair0).max() <= tol * np.abs(pair0).max() + 1e-300


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("L,steps,every", [(3, 1, 0), (5, 2, 1), (7, 37, 0), (8, 64, 64), (6, 130, 100), (20, 65, 65),
                                           (33, 20, 7)])
def test_steps_and_checkpoints(vgpu_lib, prec, L, steps, every):
    from vampire_b200 import adjoint as A
    _compare(A.system(11.2e-21, 6.69e-24, (0.1, 0.0, 0.4), L), prec, steps, every)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("pairs", [False, True])
def test_alloy(vgpu_lib, prec, pairs):
    from vampire_b200 import system as S
    s = S.config_fcc_tensor(5, temperature=0.0)
    s.params.H_applied = 0.3
    _compare(s, prec, 30, 0, pairs)


def test_workspace_between_calls(vgpu_lib):
    """One handle, calls of different length and checkpointing in turn: each
    equals the same call on a handle of its own."""
    from vampire_b200 import adjoint as A
    from vampire_b200 import vgpu as V
    s = A.system(11.2e-21, 6.69e-24, (0.1, 0.0, 0.4), 6)

    def grad(sim, steps, every):
        target = np.full(steps, 0.9)
        g, loss = np.zeros(5), C.c_double()
        sim._check(V.lib().vgpu_adjoint_llg(sim.handle, C.c_uint64(steps), target.ctypes.data_as(V._D),
                                            C.c_double(1e-16), C.c_int32(every), C.byref(loss), g.ctypes.data_as(V._D)))
        return np.r_[loss.value, g]

    with V.Simulation(s, precision="fp64") as sim:
        for steps, every in ((10, 0), (90, 7), (3, 0), (150, 0), (90, 90)):
            with V.Simulation(s, precision="fp64") as fresh:
                want = grad(fresh, steps, every)
            assert np.abs(grad(sim, steps, every) - want).max() <= 1e-12 * np.abs(want).max()

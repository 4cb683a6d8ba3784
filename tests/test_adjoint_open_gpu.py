"""Adjoint gradients and trajectories of systems with rows of different width
(open surfaces, vacancies) against the FP64 CPU adjoint: such a row is filled
up with bonds to the padding atom, whose entry has to be zero in everything
that is gathered.  One handle makes calls of different length and checkpoint
interval, so that its workspace holds other data each time, and the device
memory it is cut from is filled beforehand."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = ((10, 0), (90, 7), (3, 0), (150, 0), (90, 90), (10, 0))


def _system(name):
    from vampire_b200 import adjoint as A
    from vampire_b200 import system as S
    p = S.SimParams(dt_SI=1e-16, temperature=0.0, H_applied=1.0, H_vec=(0.1, 0.0, 0.4), thermal=False)
    rng = np.random.default_rng(8)
    if name == "alloy":
        L = (4, 3, 5)
        n = 4 * L[0] * L[1] * L[2]
        keep = rng.random(n) > 0.1
        mats = [S.Material(alpha=0.05, mu_s_muB=1.72, Kc=1e-24), S.Material(alpha=0.1, mu_s_muB=2.3, Kc=0.5e-24)]
        J = np.array([[11.2e-21, 5e-21], [5e-21, 9e-21]])
        m = int(keep.sum())
        return S.build("fcc", *L, 3.54, mats, J, p, periodic=(False,) * 3, keep=keep,
                       types=(rng.random(m) < 0.5).astype(np.int32), dmi_SI=0.1 * J, spins=A.tilted_spins(m, 6))
    L, keep = (7, 5, 9), None
    if name == "sc_vacancies":
        keep = rng.random(7 * 5 * 9) > 0.15
    n = 315 if keep is None else int(keep.sum())
    mats, J, types = [S.Material(alpha=0.1, mu_s_muB=1.72, Ku=6.69e-24)], [[11.2e-21]], None
    if name == "sc_two_materials":
        mats.append(S.Material(alpha=0.05, mu_s_muB=2.3, Ku=2e-24))
        J, types = [[11.2e-21, 4e-21], [4e-21, 7e-21]], np.arange(n) % 2
    s = S.build("sc", *L, 3.0, mats, J, p, periodic=(False,) * 3, keep=keep, types=types,
                spins=A.tilted_spins(n, 6))
    if name.endswith("_bond"):
        # a coupling of its own for every pair of neighbours
        w = rng.uniform(0.5, 1.5, (n, n))
        w = w + w.T
        i = np.repeat(np.arange(n), s.nl_end - s.nl_start + 1)
        iso = s.jlist * w[i, s.nl]
        if name == "iso_bond":
            s.jlist = iso
        else:
            sym = rng.uniform(-0.2, 0.2, (n, n, 3, 3))
            sym = sym + sym.transpose(1, 0, 3, 2)
            s.jlist = (iso[:, None, None] * (np.eye(3) + sym[i, s.nl])).reshape(-1)
            s.exch_type = S.EXCH_TENSORIAL
    return s


def _dirty():
    """Device memory with data in it, given back for the next allocations."""
    import torch
    x = [torch.full((1 << k,), 7.5, device="cuda") for k in range(10, 27)]
    torch.cuda.synchronize()
    del x
    torch.cuda.empty_cache()


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("passes", [False, True])
@pytest.mark.parametrize("name,fmt", [("sc", "iso_tab"), ("sc_vacancies", "iso_tab"), ("sc_two_materials", "iso_tab"),
                                      ("iso_bond", "iso_bond"), ("tensor_bond", "tensor_bond"), ("alloy", "dmi_tab")])
def test_short_rows(vgpu_lib, name, fmt, passes, prec):
    from oracle import oracle as O
    from vampire_b200 import vgpu as V
    s = _system(name)
    o = O.OracleSystem(s)
    # FP64: sums in another order.  FP32: the trajectory's rounding, a few 1e-5
    # of the loss (an offset of 0.05 from the target) and of the gradients.
    tol = 1e-3 if prec == "fp32" else 1e-9
    _dirty()
    with V.Simulation(s, precision=prec) as sim:
        assert sim.exchange_format() == fmt
        if passes:
            sim.set_option(V.OPT_STAGED_RECORDS, 1)
        for steps, every in CALLS:
            want_mz = o.mz_trajectory(s.spins, steps)
            mz = np.zeros(steps)
            sim._check(V.lib().vgpu_mz_trajectory(sim.handle, C.c_uint64(steps), mz.ctypes.data_as(V._D)))
            assert np.abs(mz - want_mz).max() < (1e-5 if prec == "fp32" else 1e-12)
            target = np.ascontiguousarray(want_mz - 0.05)
            g, loss = np.zeros(5), C.c_double()
            sim._check(V.lib().vgpu_adjoint_llg(sim.handle, C.c_uint64(steps), target.ctypes.data_as(V._D),
                                                C.c_double(1e-16), C.c_int32(every), C.byref(loss),
                                                g.ctypes.data_as(V._D)))
            want_loss, want = o.adjoint(s.spins, target, 1e-16, every=every)
            assert abs(loss.value - want_loss) <= tol * want_loss
            for k in (slice(0, 1), slice(1, 2), slice(2, 5)):
                assert np.abs(g[k] - want[k]).max() <= tol * np.abs(want[k]).max(), (steps, every, g, want)

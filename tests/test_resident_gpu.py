"""Steps in one resident launch against one launch per pass: the same spins bit
for bit.  Asking for a pass option (staged records on, the default) selects the
passes.  Every exchange format and pass variant, both precisions, systems that
end inside a warp, a block or exactly at one, several atoms per thread, a
dipole update inside the run, and a batch."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def _pair(s, prec, steps, midpoint=False, cells=None, seed=17):
    from vampire_b200 import vgpu
    out = []
    for passes in (False, True):
        with vgpu.Simulation(s, precision=prec, noise_seed=seed) as sim:
            if passes:
                sim.set_option(vgpu.OPT_STAGED_RECORDS, 1)
            if cells is not None:
                sim.dipole_setup(cells)
            for k in steps:
                sim.llg_midpoint(k) if midpoint else sim.llg_heun(k)
            assert sim.step == sum(steps)
            out.append(sim.spins())
    return out


@pytest.mark.parametrize("name", ["sc10_t300", "sc6_open_t300", "fcc4_dmi_t300", "tet_iso_bond_t300",
                                  "tet_vec_bond_t300", "tet_ten_bond_t300", "sc6_vec_t300", "sc6_aniso_ho",
                                  "sc6_biquadratic_t300", "fcc4_neel_rot"])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("midpoint", [False, True])
def test_formats_and_variants(vgpu_lib, name, prec, midpoint):
    s, _ = load_golden(name)
    s.params.temperature = 300.0
    got, want = _pair(s, prec, (1, 7, 2), midpoint)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 1, 1), (33, 1, 1), (16, 16, 1), (257, 1, 1), (9, 19, 3), (64, 32, 2),
                                  (63, 62, 61), (67, 66, 65)])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_sizes(vgpu_lib, dims, prec):
    from vampire_b200 import system as S
    s = S.build("sc", *dims, 3.0, [S.Material(alpha=0.1, mu_s_muB=1.72, Ku=6.69e-24)], [[11.2e-21]],
                S.SimParams(temperature=400.0, H_applied=0.2), periodic=(False, False, True) if dims[2] > 2 else
                (False,) * 3, spin_seed=3)
    got, want = _pair(s, prec, (6,))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("L", [5, 16, 31, 36])
def test_alloy_sizes(vgpu_lib, L):
    from vampire_b200 import system as S
    s = S.config_fcc_tensor(L)
    got, want = _pair(s, "fp32", (4,))
    assert np.array_equal(got, want)


def test_three_materials_with_table(vgpu_lib):
    """Several materials, so the coupling comes from the table per bond."""
    from vampire_b200 import system as S
    mats = [S.Material(alpha=0.1 * (k + 1), mu_s_muB=1.0 + k, Ku=1e-24 * k) for k in range(3)]
    J = np.array([[6e-21, 2e-21, -1e-21], [2e-21, 5e-21, 3e-21], [-1e-21, 3e-21, 4e-21]])
    s = S.build("sc", 13, 11, 12, 3.0, mats, J, S.SimParams(temperature=200.0), types=np.arange(13 * 11 * 12) % 3,
                spin_seed=9)
    for prec in ("fp32", "fp64"):
        got, want = _pair(s, prec, (5,))
        assert np.array_equal(got, want)


def test_dipole_updates_inside_the_run(vgpu_lib):
    from vampire_b200 import system as S
    s = S.config_fcc_tensor(8, dipole=True)
    s.cells["update_rate"] = 3
    got, want = _pair(s, "fp64", (2, 8, 1), cells=s.cells)
    # the direct sum's and the moments' FP64 order may differ between runs
    assert np.abs(got - want).max() < 1e-13


def test_applied_field_of_each_call(vgpu_lib):
    """Parameters set between calls reach the next resident launch."""
    from vampire_b200 import system as S
    from vampire_b200 import vgpu
    s = S.config_sc_llg(9, temperature=300.0)
    out = []
    for passes in (False, True):
        with vgpu.Simulation(s, noise_seed=2) as sim:
            if passes:
                sim.set_option(vgpu.OPT_STAGED_RECORDS, 1)
            for H in (0.1, -2.0, 5.0):
                s.params.H_applied = H
                sim.set_params(s.params)
                sim.llg_heun(3)
            out.append(sim.spins())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_spins_set_between_calls(vgpu_lib, prec):
    """A launch starts from the spins it finds, not from the words that the one
    before left behind (many blocks, so that some start late)."""
    from vampire_b200 import system as S
    from vampire_b200 import vgpu
    s = S.config_sc_llg(36, temperature=300.0)
    starts = [S.random_spins(s.n, k) for k in range(6)]
    out = []
    for passes in (False, True):
        with vgpu.Simulation(s, precision=prec, noise_seed=5) as sim:
            if passes:
                sim.set_option(vgpu.OPT_STAGED_RECORDS, 1)
            got = []
            for sp in starts:
                sim.set_spins(sp)
                sim.llg_heun(2)
                got.append(sim.spins())
            out.append(got)
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_batch(vgpu_lib, prec):
    from vampire_b200 import batch as B
    from vampire_b200 import vgpu
    systems, params = B.nanoparticle_ensemble(9, seed=4, n_ramp=50)
    out = []
    for passes in (False, True):
        with B.Batch(systems, params, noise_seed=8, precision=prec) as b:
            if passes:
                vgpu.check(vgpu.lib().vgpu_set_option(b.handle, vgpu.OPT_STAGED_RECORDS, 1), b.handle)
            b.llg_heun(60)
            out.append(np.concatenate(b.spins(), axis=1))
    assert np.array_equal(out[0], out[1])


def test_two_handles_in_two_threads(vgpu_lib):
    """Resident launches of independent handles from two host threads."""
    import threading

    from vampire_b200 import system as S
    from vampire_b200 import vgpu
    s = S.config_sc_llg(30, temperature=300.0)
    with vgpu.Simulation(s, noise_seed=1) as sim:
        sim.set_option(vgpu.OPT_STAGED_RECORDS, 1)
        sim.llg_heun(60)
        want = sim.spins()
    got = [None, None]

    def work(k):
        with vgpu.Simulation(s, noise_seed=1) as sim:
            for _ in range(20):
                sim.llg_heun(3)
            got[k] = sim.spins()

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert np.array_equal(got[0], want) and np.array_equal(got[1], want)


@pytest.mark.parametrize("name", ["sc6_open_t300", "sc20_t0", "fcc4_dmi_t0"])
def test_steps_recorded_into_a_graph(vgpu_lib, name):
    """Steps recorded on the handle's stream and replayed twice do at T = 0 what
    twice as many steps do (the replays cannot reuse a resident launch)."""
    import torch
    from vampire_b200 import vgpu
    s, _ = load_golden(name)
    s.params.temperature = 0.0
    with vgpu.Simulation(s) as sim:
        sim.llg_heun(2 + 2 * 6)
        want = sim.spins()
    with vgpu.Simulation(s) as sim:
        sim.llg_heun(2)
        sim.synchronize()
        stream = torch.cuda.ExternalStream(sim.stream_ptr())
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream, capture_error_mode="relaxed"):
            sim.llg_heun(6)
        with torch.cuda.stream(stream):
            g.replay()
            g.replay()
        torch.cuda.synchronize()
        got = sim.spins()
    assert np.array_equal(got, want)

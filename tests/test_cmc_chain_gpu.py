"""The parallel solution of the constrained Monte Carlo acceptance chain
against the sequential rule (oracle/vref.c vref_cmc_pairs): phases of one pair
up to past one chunk of 4,096 pairs, from spins near saturation (decisions
hardly depend on the running moment) and from random spins (a moment of the
size of single pairs, so almost every decision depends on the ones before)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [0.3, 30.0])
@pytest.mark.parametrize("K", [1, 3, 4, 31, 1025, 4095, 4096, 4097, 4394])
def test_chain_equals_sequential_rule(vgpu_lib, K, width):
    from oracle import oracle as O
    from vampire_b200 import system as S
    from vampire_b200 import vgpu
    s = S.config_sc_llg(26, temperature=500.0)
    rng = np.random.default_rng(K)
    v = rng.standard_normal((3, s.n)) * width
    v[2] += 1.0
    s.spins = v / np.sqrt((v * v).sum(0))
    with vgpu.Simulation(s, precision="fp64") as sim:
        sim.cmc_setup(20.0, 35.0, init_spins=False)
        P, pv = sim.cmc_frame()
        atoms = rng.permutation(np.flatnonzero(sim.mc_colours() == 0))[: 2 * K].reshape(K, 2)
        rnd = np.concatenate([rng.standard_normal(3 * K), rng.random(K)])
        M = (s.spins * s.mu_s_muB()).sum(axis=1)
        if M @ pv < 0.0:
            M = -M
        sim.cmc_pairs(atoms, rnd, moment=M)
        want, M_o, cnt = O.OracleSystem(s).cmc_pairs(s.spins, atoms, rnd, P, pv, M)
        got = sim.spins()
        Mg, c = sim.cmc_state()
    assert np.abs(got - want).max() < 1e-12
    assert np.abs(Mg - M_o).max() < 1e-9
    assert c[0] == K and list(c[1:4].astype(int)) == list(np.asarray(cnt).astype(int))

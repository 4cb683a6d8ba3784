"""Monte Carlo trials on trial rows: every row width (2, 6, 8 and 12 bonds a
row, 14 on the neighbour list itself), chains with narrower rows at their ends,
colours that end inside a warp, and colours of several trials per thread,
against the oracle's acceptance rule with replayed numbers; and the sweeps of a
system whose terms are all of the plain instance against the general one (a
cubic term of constant zero selects it), the same spins bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(n, reach, kc=0.0):
    """Open chain of two mixed materials: bonds to the `reach` atoms on each side."""
    from vampire_b200 import system as S
    mats = [S.Material(mu_s_muB=1.5, Ku=1e-24), S.Material(mu_s_muB=2.0, Ku=0.0)]
    rng = np.random.default_rng(n + reach)
    s = S.build("sc", n, 1, 1, 3.0, mats, [[4e-21, -2e-21], [-2e-21, 3e-21]], S.SimParams(temperature=300.0),
                periodic=(False, False, False), types=rng.integers(0, 2, n))
    off = np.array([d for d in range(-reach, reach + 1) if d])
    nbr = np.arange(n)[:, None] + off
    ok = (nbr >= 0) & (nbr < n)
    cnt = ok.sum(1)
    s.nl = nbr[ok].astype(s.nl.dtype)
    end = np.cumsum(cnt)
    s.nl_start = (end - cnt).astype(s.nl_start.dtype)
    s.nl_end = (end - 1).astype(s.nl_end.dtype)
    s.jlist = S.exchange_lists(s.nl_start, s.nl_end, s.nl, s.type, s.materials,
                               np.array([[4e-21, -2e-21], [-2e-21, 3e-21]]), s.exch_type)
    s.cubic = kc is not None
    return s


SIZES = [(2, 1), (65, 1), (97, 3), (1000, 3), (333, 4), (130, 6), (999, 6), (500, 7), (700001, 1)]


@pytest.mark.parametrize("n,reach", SIZES)
def test_rows_match_oracle(vgpu_lib, n, reach):
    from oracle import oracle as O
    from vampire_b200 import vgpu
    s = _chain(n, reach, None)
    rng = np.random.default_rng(5)
    with vgpu.Simulation(s, precision="fp64") as sim:
        sim.mc_setup()
        rnd = np.concatenate([rng.standard_normal(3 * n), rng.random(n)])
        sim.mc_set_replay(rnd)
        sim.mc_sweep(1)
        want, rej = O.OracleSystem(s).mc_colour_sweep(s.spins.copy(), sim.mc_colours(), rnd)
        got = sim.spins()
        moves, rejects = sim.mc_counters()
    assert np.abs(got - want).max() < 1e-12
    assert moves == n and rejects == rej


@pytest.mark.parametrize("n,reach", SIZES)
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_plain_instance_equals_general(vgpu_lib, n, reach, prec):
    from vampire_b200 import vgpu
    out = []
    for kc in (None, 0.0):
        with vgpu.Simulation(_chain(n, reach, kc), precision=prec, noise_seed=3) as sim:
            sim.mc_setup()
            sim.mc_sweep(3)
            out.append((sim.spins(), sim.mc_counters()))
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]

"""Masked sums over masks the reductions treat differently: one bin, two bins
(registers per bin), more bins in runs (replicas), interleaved, and mixed
within a warp beyond four bins; sizes with partial warps and blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _masks(n):
    i = np.arange(n)
    return {"one": (np.zeros(n), 1), "alternating two": (i % 2, 2), "runs": (np.minimum(i // 50, 6), 7),
            "interleaved five": (i % 5, 5), "interleaved nineteen": (i % 19, 19),
            "runs and noise": (np.where(i % 97 == 0, 3, i * 3 // n), 4)}


@pytest.mark.parametrize("dims", [(3, 3, 3), (7, 9, 11), (12, 10, 9)])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_masked_sums(vgpu_lib, dims, prec):
    from oracle import oracle as O
    from vampire_b200 import system as S
    from vampire_b200 import vgpu
    s = S.build("sc", *dims, 3.0, [S.Material(alpha=0.1, mu_s_muB=1.72, Ku=6.69e-24)], [[11.2e-21]],
                S.SimParams(H_applied=0.3), periodic=(True, False, True), spin_seed=11)
    if prec == "fp32":
        s.spins = s.spins.astype(np.float32).astype(np.float64)
    o = O.OracleSystem(s)
    tol = 2e-6 if prec == "fp32" else 1e-11
    for name, (mask, size) in _masks(s.n).items():
        mask = mask.astype(np.int32)
        with vgpu.Simulation(s, precision=prec) as sim:
            mid = sim.add_mask(mask, size)
            sim.stats_update(magnetization=True, energy=True)
            m, _, _ = sim.magnetization(mid)
            e, _, _ = sim.energy(mid)
            sim.stats_update(magnetization=True)
            m1, mean, cnt = sim.magnetization(mid)
        want_m, want_e = o.magnetization(s.spins, mask, size), o.energy(s.spins, mask, size)
        assert cnt == 2
        for got in (m, m1, 0.5 * mean):
            assert np.abs(got - np.ravel(want_m)).max() < (1e-12 if prec == "fp64" else tol), name
        assert np.abs(e - np.ravel(want_e)).max() < tol * (np.abs(want_e).max() + 1.0), name


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_torque_of_many_materials(vgpu_lib, prec):
    """Quantities over several merge blocks (3 M + 1 = 37), rows of a partial last block."""
    from vampire_b200 import system as S
    from vampire_b200 import vgpu
    M = 12
    s = S.build("sc", 9, 10, 11, 3.0, [S.Material(alpha=0.1, mu_s_muB=1.0 + 0.1 * k) for k in range(M)],
                np.full((M, M), 5e-21), S.SimParams(H_applied=0.3), types=np.arange(990) % M, spin_seed=3)
    with vgpu.Simulation(s, precision=prec) as sim:
        sp, H = sim.spins(), sim.fields()
        for _ in range(2):
            sim.torque_update()
        t = sim.torque()
    c = np.cross(sp.T, H.T)
    mu = s.materials["mu_s_SI"] / 9.27400915e-24
    if prec == "fp32":
        mu = mu.astype(np.float32).astype(np.float64)  # moments are held in the handle's precision
    tq = c * (mu * 9.27400915e-24)[s.type][:, None]
    want = np.stack([tq[s.type == k].sum(0) for k in range(M)])
    # the field is read back exactly; sums of FP64 products
    assert np.abs(t["material"] - want).max() < 1e-12 * np.abs(tq).sum()
    assert np.abs(t["material_mean"] - want).max() < 1e-12 * np.abs(tq).sum()
    assert np.abs(t["total"] - want.sum(0)).max() < 1e-12 * np.abs(tq).sum()
    assert abs(t["max"] - np.sqrt((c * c).sum(1)).max()) < 1e-12 * t["max"] and t["count"] == 2

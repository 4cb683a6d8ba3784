"""Macrocell fields of FP32 handles on grids of at most 8 cells per axis equal the
FP64 handle's on the same (FP32) spins to the rounding of the stored field: 2^-24
of every component, so of its 2-norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 2), (2, 2, 2), (4, 4, 4), (8, 7, 6), (8, 8, 8), (3, 8, 1)])
def test_field_to_its_own_rounding(vgpu_lib, shape):
    from vampire_b200 import system as S
    from vampire_b200 import vgpu as V
    s = S.build("sc", *(2 * g for g in shape), 3.0, [S.Material(mu_s_muB=1.72)], [[5e-21]], S.SimParams(dt_SI=1e-16),
                spin_seed=sum(shape), periodic=(False,) * 3)
    s.spins = s.spins.astype(np.float32).astype(np.float64)
    S.dipole_cells(s, size=6.0, atomic_volume=27.0, update_rate=0)
    out = []
    for prec in ("fp32", "fp64"):
        with V.Simulation(s, precision=prec) as sim:
            sim.dipole_setup(s.cells)
            sim.dipole_update()
            out.append(sim.dipole_cells()[1:])
    for got, want in zip(*out):
        assert np.linalg.norm(got - want) <= 2.0 ** -24 * np.linalg.norm(want)

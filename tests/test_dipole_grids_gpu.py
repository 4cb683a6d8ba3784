"""The macrocell field on grids at the edges of the line transforms (8 to 128
padded points, odd extents, odd numbers of lines), with holes, and with enough
cells for the one-thread-per-cell finish, against FP64 sums by numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = 9.27400915e-01


def _cells(shape, solver, holes=0.0):
    from vampire_b200 import system as S
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 100 * ny + 10000 * nz)
    keep = None
    if holes:
        cell = rng.random((nz, ny, nx)) >= holes
        cell[0, 0, 0] = cell[-1, -1, -1] = True
        keep = np.repeat(np.repeat(np.repeat(cell, 2, 0), 2, 1), 2, 2).ravel()
    s = S.build("sc", 2 * nx, 2 * ny, 2 * nz, 3.0, [S.Material(alpha=0.1, mu_s_muB=1.72)], [[5e-21]],
                S.SimParams(dt_SI=1e-16), spin_seed=5, periodic=(False,) * 3, keep=keep)
    S.dipole_cells(s, size=6.0, atomic_volume=27.0, solver=solver, cutoff=1.5, update_rate=0)
    return s


def _terms(r):
    n = np.sqrt((r * r).sum(0))
    n = np.where(n == 0, np.inf, n)
    e = r / np.where(np.isinf(n), 1.0, n)
    a, b = (0, 0, 0, 1, 1, 2), (0, 1, 2, 1, 2, 2)
    return np.stack([(3 * e[p] * e[q] - (p == q)) / n ** 3 for p, q in zip(a, b)])


def _field(s, shape, near):
    """B of every cell: convolution of the moments with the point-dipole tensor,
    and with `near` the atomistic tensors within 1.5 cells (identical full cells)."""
    G = np.array(shape)
    nc = int(G.prod())
    mu = s.materials["mu_s_SI"][0] / 9.27400915e-24
    m = np.stack([np.bincount(s.cells["atom_cell"], weights=s.spins[q], minlength=nc) for q in range(3)]) * mu
    P = 2 * G
    off = [np.fft.fftfreq(p, 1.0 / p).round() for p in P]
    z, y, x = np.meshgrid(off[2], off[1], off[0], indexing="ij")
    T = _terms(np.stack([x, y, z]) * 6.0)
    if near:
        atoms = np.stack(np.meshgrid([0, 3.0], [0, 3.0], [0, 3.0], indexing="ij")).reshape(3, 8)
        for o in np.argwhere(np.ones((5, 5, 5))) - 2:
            if (o * o).sum() <= 2 and np.all(np.abs(o) < G):
                r = atoms[:, None, :] + 6.0 * o[:, None, None] - atoms[:, :, None]
                T[:, o[2], o[1], o[0]] = _terms(r.reshape(3, -1)).sum(1) / 64.0
    Tk = np.fft.rfftn(T, axes=(1, 2, 3))
    Mk = np.fft.rfftn(m.reshape(3, G[2], G[1], G[0]), s=tuple(P[::-1]), axes=(1, 2, 3))
    sym = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
    B = np.stack([np.fft.irfftn(sum(Tk[sym[a][b]] * Mk[b] for b in range(3)), s=tuple(P[::-1]), axes=(0, 1, 2))
                  for a in range(3)])
    return K * B[:, :G[2], :G[1], :G[0]].reshape(3, -1)


@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 1, 8), (9, 16, 3), (1, 17, 33), (33, 7, 5), (40, 3, 9), (2, 65, 2)])
@pytest.mark.parametrize("prec,far", [("fp64", 1), ("fp32", 1), ("fp32", 0)])
def test_grids(vgpu_lib, shape, prec, far):
    """FP64 transforms to 1e-12, FP32 ones and the direct FP32 terms to 1e-5
    (moments of FP32 spins included)."""
    from vampire_b200 import vgpu
    for solver in ("macrocell", "tensor"):
        s = _cells(shape, solver)
        with vgpu.Simulation(s, precision=prec) as sim:
            sim.set_option(vgpu.OPT_DIPOLE_FFT, far)
            sim.dipole_setup(s.cells)
            assert sim.dipole_method() == far
            for _ in range(2):  # the second update reuses the grids
                sim.dipole_update()
            _, b, _ = sim.dipole_cells()
        want = _field(s, shape, solver == "tensor")
        assert np.abs(b - want).max() < (1e-12 if prec == "fp64" else 1e-5) * np.abs(want).max()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_empty_cells(vgpu_lib, prec):
    from vampire_b200 import vgpu
    shape = (9, 6, 7)
    s = _cells(shape, "macrocell", holes=0.3)
    with vgpu.Simulation(s, precision=prec) as sim:
        sim.dipole_setup(s.cells)
        assert sim.dipole_method() == vgpu.DIPOLE_FAR_FFT
        _, b, hd = sim.dipole_cells()
    full = s.cells["cell_natoms"] > 0
    want = _field(s, shape, False)
    assert not full.all() and np.all(b[:, ~full] == 0) and np.all(hd[:, ~full] == 0)
    assert np.abs(b - want)[:, full].max() < (1e-12 if prec == "fp64" else 1e-5) * np.abs(want[:, full]).max()


def test_many_cells(vgpu_lib):
    """68,921 cells: a thread per cell in the finish, near pairs in groups of four."""
    from vampire_b200 import vgpu
    shape = (41, 41, 41)
    s = _cells(shape, "tensor")
    with vgpu.Simulation(s, precision="fp64") as sim:
        sim.dipole_setup(s.cells)
        _, b, _ = sim.dipole_cells()
    want = _field(s, shape, True)
    assert np.abs(b - want).max() < 1e-12 * np.abs(want).max()

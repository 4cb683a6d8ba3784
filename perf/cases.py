"""The work that users of this framework have it do, as cases that can be timed.

Each case is one kind of call over the sizes that programs use it at:

* ``llg``      a stretch of LLG steps between two statistics outputs (iron-like
               simple-cubic ferromagnets and the FCC two-material alloy with
               tensor exchange, DMI and, on request, the macrocell dipole
               field), in FP32 and FP64, Heun or midpoint;
* ``mc``       Metropolis sweeps of temperature replicas (a Curie sweep);
* ``cmc``      constrained Monte Carlo steps (anisotropy against direction);
* ``dipole``   dynamics whose demagnetising field is renewed every step, and
               the field map read out;
* ``batch``    an ensemble of nanoparticles on a hysteresis loop;
* ``adjoint``  the gradient of a trajectory loss (one fitting iteration);
* ``measure``  energy, magnetisation and torque of the current state.

``prepare`` makes what a program holds before the call (an uploaded system with
its solver, masks and output buffers), ``run`` makes the call.  Outputs have the
precision of the handle: the library hands FP32 results out in FP64 containers,
which are narrowed again here.  ``exact`` is the same computation in 64 bits by
plain torch and numpy, on the same couplings and the same random words.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from vampire_b200 import adjoint as A
from vampire_b200 import batch as B
from vampire_b200 import system as S
from vampire_b200 import vgpu as V

MU_B = 9.27400915e-24
KB = 1.3806503e-23


# ----------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------

def _llg(name, lattice, nx, ny, nz, steps, every, temperature=300.0, open_=False, exchange="iso", dipole=False,
         precision="fp32", integrator="heun"):
    return {"name": name, "kind": "llg", "lattice": lattice, "nx": nx, "ny": ny, "nz": nz, "open": open_,
            "exchange": exchange, "dipole": dipole, "precision": precision, "integrator": integrator,
            "temperature": temperature, "steps": steps, "every": every}


def listed():
    return [
        # the smallest systems (single nanoparticles, unit tests of a material file): launches and latency only
        _llg("llg_sc_10x9x11_open", "sc", 10, 9, 11, 20, 10, open_=True),
        # the simple-cubic ferromagnet of the first benchmark configuration
        _llg("llg_sc_20", "sc", 20, 20, 20, 100, 100),
        # an open thin block of ragged size, statistics every 10 steps
        _llg("llg_sc_61x53x47_open", "sc", 61, 53, 47, 50, 10, temperature=600.0, open_=True),
        # the alloy at odd size: partly filled macrocells, so the dipole far field is the direct sum
        _llg("llg_fcc_alloy_21_dipole", "fcc", 21, 21, 21, 100, 50, exchange="dmi", dipole=True),
        # the alloy of the headline benchmark at a million spins
        _llg("llg_fcc_alloy_64_dipole", "fcc", 64, 64, 64, 20, 20, exchange="dmi", dipole=True),
        # the precision used to check against the reference program
        _llg("llg_fcc_alloy_20_fp64", "fcc", 20, 20, 20, 20, 20, exchange="dmi", precision="fp64"),
        # a Curie sweep: SC 50^3 at 31 temperatures as replicas, <|m|> every 10 sweeps
        {"name": "mc_sc_50_replicas_31", "kind": "mc", "nx": 50, "ny": 50, "nz": 50, "replicas": 31,
         "t_lo": 50.0, "t_hi": 1500.0, "sweeps": 10, "every": 10},
        # constrained Monte Carlo at a size used for anisotropy curves
        {"name": "cmc_sc_24", "kind": "cmc", "nx": 24, "ny": 24, "nz": 24, "temperature": 400.0, "phi": 30.0,
         "theta": 20.0, "steps": 2},
        # 125,000 macrocells: the cell count of the headline benchmark's dipole solver
        {"name": "dipole_sc_100", "kind": "dipole", "nx": 100, "ny": 100, "nz": 100, "steps": 10},
        # the ensemble of the batched benchmark
        {"name": "batch_256", "kind": "batch", "systems": 256, "ensemble": 7, "steps": 200, "every": 100},
        # one fitting iteration on the system of the adjoint benchmark
        {"name": "adjoint_sc_32", "kind": "adjoint", "L": 32, "steps": 1000, "precision": "fp32"},
        # energies, magnetisation and torque of an open alloy block
        {"name": "measure_fcc_40x37x30_open", "kind": "measure", "nx": 40, "ny": 37, "nz": 30, "open": True,
         "updates": 5},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["llg", "llg", "llg", "mc", "cmc", "dipole", "batch", "adjoint", "measure"])
    if kind == "llg":
        lattice = rng.choice(["sc", "fcc"])
        atoms = _logint(rng, 300, 250000)
        edge = max(3, round((atoms / (1 if lattice == "sc" else 4)) ** (1 / 3)))
        nx, ny, nz = (max(3, edge + rng.randint(-(edge // 5), edge // 5)) for _ in range(3))
        exchange = "iso" if lattice == "sc" else "dmi"
        steps = rng.choice([10, 20, 50, 100]) if atoms < 100000 else rng.choice([10, 20])
        precision = rng.choice(["fp32", "fp32", "fp32", "fp64"])
        c = _llg("", lattice, nx, ny, nz, steps, rng.choice([10, steps]), temperature=float(rng.randint(0, 900)),
                 open_=rng.random() < 0.4, exchange=exchange, dipole=rng.random() < 0.3, precision=precision,
                 integrator=rng.choice(["heun", "heun", "heun", "midpoint"]))
        del c["name"]
        return c
    if kind == "mc":
        e = _logint(rng, 6, 50)
        r = _logint(rng, 1, 31)
        n = [max(4, e + rng.randint(-2, 2)) for _ in range(3)]
        return {"kind": "mc", "nx": n[0], "ny": n[1], "nz": n[2], "replicas": r, "t_lo": float(rng.randint(0, 300)),
                "t_hi": float(rng.randint(400, 1500)), "sweeps": 10, "every": rng.choice([1, 10])}
    if kind == "cmc":
        e = _logint(rng, 6, 40)
        n = [max(4, e + rng.randint(-2, 2)) for _ in range(3)]
        return {"kind": "cmc", "nx": n[0], "ny": n[1], "nz": n[2], "temperature": float(rng.randint(50, 900)),
                "phi": float(rng.randint(0, 90)), "theta": float(rng.randint(0, 90)), "steps": rng.choice([1, 2, 5])}
    if kind == "dipole":
        e = _logint(rng, 8, 100)
        n = [2 * max(2, (e + rng.randint(-e // 5, 0)) // 2) for _ in range(3)]
        return {"kind": "dipole", "nx": n[0], "ny": n[1], "nz": n[2], "steps": rng.choice([2, 5, 10])}
    if kind == "batch":
        return {"kind": "batch", "systems": _logint(rng, 8, 256), "ensemble": rng.randint(1, 1000),
                "steps": rng.choice([50, 100, 200]), "every": rng.choice([10, 50])}
    if kind == "adjoint":
        return {"kind": "adjoint", "L": rng.randint(6, 32), "steps": _logint(rng, 50, 1000),
                "precision": rng.choice(["fp32", "fp32", "fp64"])}
    e = _logint(rng, 5, 40)
    n = [max(3, e + rng.randint(-e // 4, 0)) for _ in range(3)]
    return {"kind": "measure", "nx": n[0], "ny": n[1], "nz": n[2], "open": rng.random() < 0.5, "updates": 5}


# ----------------------------------------------------------------------------
# systems: the couplings belong to the case, the spins and noise to the seed
# ----------------------------------------------------------------------------

@functools.lru_cache(maxsize=4)
def _lattice(lattice, nx, ny, nz, open_, exchange, dipole, temperature):
    per = (not open_,) * 3
    if lattice == "sc":
        m = S.Material(alpha=0.1, mu_s_muB=1.72, Ku=6.69e-24)
        p = S.SimParams(dt_SI=1e-16, temperature=temperature, H_applied=0.1)
        s = S.build("sc", nx, ny, nz, 3.0, [m], [[11.2e-21]], p, periodic=per)
        if dipole:
            S.dipole_cells(s, size=6.0, atomic_volume=27.0)
        return s
    mats = [S.Material(alpha=0.05, mu_s_muB=1.72, Kc=1e-24) for _ in range(2)]
    J = np.array([[11.2e-21, 5e-21], [5e-21, 11.2e-21]])
    p = S.SimParams(dt_SI=1e-16, temperature=temperature, H_applied=0.0)
    types = (np.random.default_rng(nx * 10007 + ny * 101 + nz).random(4 * nx * ny * nz) < 0.5).astype(np.int32)
    s = S.build("fcc", nx, ny, nz, 3.54, mats, J, p, periodic=per, types=types,
                dmi_SI=0.1 * J if exchange == "dmi" else None)
    if dipole:
        S.dipole_cells(s, size=2 * 3.54, atomic_volume=3.54 ** 3 / 4.0)
    return s


@functools.lru_cache(maxsize=2)
def _replicas(nx, ny, nz, replicas, t_lo, t_hi):
    base = S.build("sc", nx, ny, nz, 3.0, [S.Material(alpha=0.1, mu_s_muB=1.72, Ku=6.69e-24)], [[11.2e-21]],
                   S.SimParams(dt_SI=1e-16, H_applied=0.0))
    return S.replicas(base, np.linspace(t_lo, t_hi, replicas))


@functools.lru_cache(maxsize=2)
def _ensemble(systems, ensemble):
    return B.nanoparticle_ensemble(systems, seed=ensemble)


def _magnetised(n, seed, width):
    """Spins spread about +z, as an equilibrated ferromagnet holds them."""
    s = np.random.default_rng(seed).standard_normal((3, n)) * width
    s[2] += 1.0
    return s / np.sqrt((s * s).sum(0))


def _inputs(case, seed):
    """(system with the seed's spins, noise seed) of every kind but the batch."""
    k = case["kind"]
    if k == "llg":
        s = _lattice(case["lattice"], case["nx"], case["ny"], case["nz"], case["open"], case["exchange"],
                     case["dipole"], case["temperature"])
        if s.cells is not None:
            s.cells["update_rate"] = 100
        spins = _magnetised(s.n, seed, 0.5)
    elif k == "mc":
        s = _replicas(case["nx"], case["ny"], case["nz"], case["replicas"], case["t_lo"], case["t_hi"])
        spins = _magnetised(s.n, seed, 0.5)
    elif k == "cmc":
        s = _lattice("sc", case["nx"], case["ny"], case["nz"], False, "iso", False, case["temperature"])
        spins = _magnetised(s.n, seed, 0.3)
    elif k == "dipole":
        s = _lattice("sc", case["nx"], case["ny"], case["nz"], True, "iso", True, 300.0)
        s.cells["update_rate"] = 1
        spins = _magnetised(s.n, seed, 0.5)
    elif k == "measure":
        s = _lattice("fcc", case["nx"], case["ny"], case["nz"], case["open"], "dmi", False, 300.0)
        spins = _magnetised(s.n, seed, 0.5)
    else:
        s = _adjoint_system(case["L"])
        spins = A.tilted_spins(s.n, seed)
    s.spins = np.ascontiguousarray(spins)
    return s, int(seed)


@functools.lru_cache(maxsize=2)
def _adjoint_system(L):
    return A.system(11.2e-21, 6.69e-24, (0.0, 0.0, 0.4), L, 0)


def _target(case, seed):
    """The trajectory a fit compares with: a precession-damped rise of m_z."""
    t = np.arange(1, case["steps"] + 1) * 1e-16
    w = 1.0 + 0.1 * np.random.default_rng(seed).random()
    return math.cos(math.radians(30.0)) + 0.2 * (1.0 - np.exp(-t * w * 1e13))


# ----------------------------------------------------------------------------
# the calls
# ----------------------------------------------------------------------------

def _out_buffers(n, precision):
    out = torch.empty(3 * n, dtype=torch.float64 if precision == "fp64" else torch.float32, device="cuda")
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return out, idx


def _take_spins(handle, st):
    """The spins into the program's own device buffer, x|y|z blocks."""
    V.check(V.lib().vgpu_halo_pack(handle, C.c_int(V.STATE_SPIN), C.c_void_p(st["idx"].data_ptr()),
                                   C.c_int32(st["idx"].numel()), C.c_void_p(st["out"].data_ptr())), handle)
    return st["out"]


def prepare(case, seed):
    k = case["kind"]
    if k == "batch":
        systems, params = _ensemble(case["systems"], case["ensemble"])
        rng = np.random.default_rng(seed)
        for s in systems:
            s.spins = np.ascontiguousarray(_magnetised(s.n, rng.integers(1 << 30), 0.2))
        b = B.Batch(systems, params, noise_seed=int(seed))
        b.autotune(trial_steps=20)
        out, idx = _out_buffers(b.n, "fp32")
        return {"case": case, "batch": b, "out": out, "idx": idx}
    s, noise = _inputs(case, seed)
    precision = case.get("precision", "fp32")
    sim = V.Simulation(s, precision=precision, noise_seed=noise)
    st = {"case": case, "sim": sim}
    if k == "adjoint":
        st["target"] = np.ascontiguousarray(_target(case, seed))
        return st
    st["out"], st["idx"] = _out_buffers(s.n, precision)
    if s.cells is not None and (k == "dipole" or case.get("dipole")):
        sim.dipole_setup(s.cells)
    if k == "mc":
        st["mask"] = sim.add_mask(*s.masks["replica"])
        sim.mc_setup()
    elif k == "cmc":
        sim.mc_setup()
        sim.cmc_setup(case["phi"], case["theta"], init_spins=False)
    elif k == "llg":
        st["mask"] = sim.add_mask(*s.masks["system"])
    elif k == "measure":
        st["mask"] = sim.add_mask(*s.masks["system"])
        st["mask2"] = sim.add_mask(*s.masks["material"])
    sim.synchronize()
    return st


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "batch":
        b = state["batch"]
        b.run(case["steps"], record_every=case["every"])
        return {"history": b.history().astype(np.float32), "spins": _take_spins(b.handle, state)}
    sim = state["sim"]
    if k == "llg":
        real = np.float64 if case["precision"] == "fp64" else np.float32
        step = sim.llg_midpoint if case["integrator"] == "midpoint" else sim.llg_heun
        for _ in range(case["steps"] // case["every"]):
            step(case["every"])
            sim.stats_update(magnetization=True)
        spins = _take_spins(sim.handle, state)
        m, mean, _ = sim.magnetization(state["mask"])
        return {"spins": spins, "m": m.astype(real), "mean": mean.astype(real)}
    if k == "mc":
        for _ in range(case["sweeps"] // case["every"]):
            sim.mc_sweep(case["every"])
            sim.stats_update(magnetization=True)
        spins = _take_spins(sim.handle, state)
        m, _, _ = sim.magnetization(state["mask"])
        return {"spins": spins, "m": m.astype(np.float32)}
    if k == "cmc":
        sim.cmc_sweep(case["steps"])
        spins = _take_spins(sim.handle, state)
        moment, counters = sim.cmc_state()
        return {"spins": spins, "moment": moment, "counters": counters.astype(np.int64)}
    if k == "dipole":
        sim.llg_heun(case["steps"])
        spins = _take_spins(sim.handle, state)
        _, b, hd = sim.dipole_cells()
        return {"spins": spins, "B": b.astype(np.float32), "Hd": hd.astype(np.float32)}
    if k == "measure":
        for _ in range(case["updates"]):
            sim.stats_update(magnetization=True, energy=True)
            sim.torque_update()
        m, _, _ = sim.magnetization(state["mask"])
        e, _, _ = sim.energy(state["mask"])
        m2, _, _ = sim.magnetization(state["mask2"])
        e2, _, _ = sim.energy(state["mask2"])
        t = sim.torque()
        return {"m": m.astype(np.float32), "e": e.astype(np.float32), "m2": m2.astype(np.float32),
                "e2": e2.astype(np.float32), "torque_max": np.float32(t["max"]),
                "torque": t["material"].astype(np.float32)}
    tg = state["target"]
    g, loss = np.zeros(5), C.c_double()
    sim._check(V.lib().vgpu_adjoint_llg(sim.handle, C.c_uint64(tg.size), tg.ctypes.data_as(V._D), C.c_double(1e-16),
                                        C.c_int32(0), C.byref(loss), g.ctypes.data_as(V._D)))
    real = np.float64 if case["precision"] == "fp64" else np.float32
    # couplings, anisotropy and field gradients in their own units, so each an output of its own
    return {"loss": np.asarray([loss.value], dtype=real), "dJ": g[0:1].astype(real), "dKu": g[1:2].astype(real),
            "dH": g[2:5].astype(real)}


# ----------------------------------------------------------------------------
# what one pass cannot do without
# ----------------------------------------------------------------------------

def _counts(case):
    """(atoms, bonds) of the case."""
    k = case["kind"]
    if k == "batch":
        systems, _ = _ensemble(case["systems"], case["ensemble"])
        return sum(s.n for s in systems), sum(s.num_bonds for s in systems)
    if k == "adjoint":
        return case["L"] ** 3, 6 * case["L"] ** 3
    cells = case["nx"] * case["ny"] * case["nz"]
    if k == "measure" or case.get("lattice") == "fcc":
        return 4 * cells, 48 * cells
    return cells * case.get("replicas", 1), 6 * cells * case.get("replicas", 1)


def work(case):
    """Bytes: per pass over the atoms the states it reads and writes and one
    4-byte word per bond (none of it cached between passes); flops: 6 per
    isotropic bond, 18 with the antisymmetric part, about 100 per atom for the
    equation of motion and its noise."""
    n, nb = _counts(case)
    k = case["kind"]
    w = 8 if case.get("precision") == "fp64" else 4
    per_bond = 18 if (k == "measure" or case.get("exchange") == "dmi") else 6
    step_bytes = (3 * w * 2 + 3 * w * 3) * n + 2 * 4 * nb
    step_flops = 2 * (per_bond * nb + 100 * n)
    if k == "llg" or k == "batch":
        t = case["steps"]
        return {"bytes": t * step_bytes + (t // case["every"]) * 3 * w * n, "flops": t * step_flops}
    if k == "mc":
        t = case["sweeps"]
        return {"bytes": t * (24 * n + 4 * nb) + (t // case["every"]) * 12 * n, "flops": t * (6 * nb + 120 * n)}
    if k == "cmc":
        t = case["steps"]
        return {"bytes": t * 2 * (24 * n + 4 * nb), "flops": t * 2 * (6 * nb + 200 * n)}
    if k == "dipole":
        t = case["steps"]
        nc = math.prod((case[a] + 1) // 2 for a in ("nx", "ny", "nz"))
        # per update: spins and cell ids read, moments to fields through one transform each way
        up_bytes = 16 * n + nc * (24 + 48)
        up_flops = 6 * 5 * 8 * nc * max(1.0, math.log2(8 * nc)) + 8 * nc * 66 + nc * 33 * 15
        return {"bytes": t * (step_bytes + up_bytes), "flops": t * (step_flops + up_flops)}
    if k == "measure":
        return {"bytes": case["updates"] * (2 * (12 * n + 4 * nb) + 24 * n),
                "flops": case["updates"] * (2 * per_bond * nb + 80 * n)}
    # forward once, and backward through stored states with two transposed gathers a step
    return {"bytes": case["steps"] * (2 * step_bytes + 12 * w * n), "flops": case["steps"] * 3 * step_flops}


# ----------------------------------------------------------------------------
# the same in 64 bits
# ----------------------------------------------------------------------------

_M32 = 0xFFFFFFFF


def _mulhilo(a, m):
    lo = (a * m) & _M32
    hi = (m * (a >> 16) + ((m * (a & 0xFFFF)) >> 16)) >> 16
    return hi & _M32, lo


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words."""
    x, y, z, w = c0, c1, c2, c3
    for _ in range(10):
        h0, l0 = _mulhilo(x, 0xD2511F53)
        h1, l1 = _mulhilo(z, 0xCD9E8D57)
        x, y, z, w = h1 ^ y ^ k0, l1, h0 ^ w ^ k1, l0
        k0 = (k0 + 0x9E3779B9) & _M32
        k1 = (k1 + 0xBB67AE85) & _M32
    return x, y, z, w


def _u01(x, precision):
    if precision == "fp64":
        return (x.double() + 0.5) / 4294967296.0
    return ((x >> 8).double() + 0.5) / 16777216.0


def _gaussians(words, precision):
    """Box-Muller: two Gaussians of the first pair of words, one of the second."""
    u = [_u01(x, precision) for x in words]
    r1, r2 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    a1, a2 = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    return torch.stack([r1 * torch.cos(a1), r1 * torch.sin(a1), r2 * torch.cos(a2)])


def _words(ids, counter, purpose, seed):
    full = lambda v: torch.full_like(ids, v)  # noqa: E731
    klo = seed & _M32 if isinstance(seed, int) else seed
    khi = (seed >> 32) & _M32 if isinstance(seed, int) else torch.zeros_like(ids)
    return _philox(ids, full(counter & _M32), full((counter >> 32) & _M32), full(purpose),
                   klo if not isinstance(klo, int) else full(klo), khi if not isinstance(khi, int) else full(khi))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Ref:
    """A spin system in 64 bits: exchange gather, anisotropy, fields, steps."""

    def __init__(self, s, seed, precision, thermal=True, noise_ids=None, noise_keys=None):
        dev = self.dev = _device()
        self.n, self.s, self.seed, self.precision = s.n, s, seed, precision
        t = lambda v, d=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=d, device=dev)  # noqa: E731
        deg = (s.nl_end - s.nl_start + 1).astype(np.int64)
        self.z = z = int(deg.max()) if s.n else 0
        ok = np.arange(z)[None, :] < deg[:, None]
        slot = np.where(ok, s.nl_start[:, None].astype(np.int64) + np.arange(z)[None, :], 0)
        self.ok = ok
        self.nl = t(np.where(ok, s.nl[slot], s.n), torch.int64)
        self.tensor = s.exch_type == S.EXCH_TENSORIAL
        if self.tensor:
            j = s.jlist.reshape(-1, 9)
            self.J = [[t(np.where(ok[:, q], j[slot[:, q], c], 0.0)) for c in range(9)] for q in range(z)]
        else:
            self.J = [t(np.where(ok[:, q], s.jlist[slot[:, q]], 0.0)) for q in range(z)]
        self.typ = t(s.type, torch.int64)
        m, p = s.materials, s.params
        at = lambda v: t(v)[self.typ]  # noqa: E731
        self.A, self.Bc, self.alpha = (at(m[f]) for f in ("one_oneplusalpha_sq", "alpha_oneplusalpha_sq", "alpha"))
        self.ku2, self.kc4, self.mu = at(m["ku2"]), at(m["kc4"]), at(m["mu_s_SI"] / MU_B)
        self.mu_SI = at(m["mu_s_SI"])
        self.e = t(m["ku_vector"])[self.typ].T
        self.uniaxial, self.cubic = s.uniaxial, s.cubic
        temps = m["temperature"] if p.local_temperature else np.full(len(m), p.temperature)
        self.temps = temps
        self.sigma = at(np.sqrt(temps) * m["H_th_sigma"]) if thermal and p.thermal else None
        self.h = t(np.asarray(p.H_vec, dtype=np.float64) * p.H_applied)[:, None].expand(3, s.n)
        self.dt, self.step = p.dt, 0
        self.ids = torch.arange(s.n, dtype=torch.int64, device=dev) if noise_ids is None else noise_ids
        self.keys = int(seed) if noise_keys is None else noise_keys
        self.ramp = None
        self.cells = None
        self.S = t(s.spins)

    def gather(self, S):
        Sp = torch.cat([S, torch.zeros(3, 1, dtype=S.dtype, device=S.device)], 1)
        h = torch.zeros_like(S)
        for q in range(self.z):
            g = Sp[:, self.nl[:, q]]
            j = self.J[q]
            if self.tensor:
                h = h + torch.stack([j[0] * g[0] + j[1] * g[1] + j[2] * g[2], j[3] * g[0] + j[4] * g[1] + j[5] * g[2],
                                     j[6] * g[0] + j[7] * g[1] + j[8] * g[2]])
            else:
                h = h + j * g
        return h

    def aniso(self, S):
        h = torch.zeros_like(S)
        if self.uniaxial:
            h = h + 2.0 * self.ku2 * (S * self.e).sum(0) * self.e
        if self.cubic:
            h = h + 2.0 * self.kc4 * S ** 3
        return h

    def external(self):
        h = self.h
        if self.ramp is not None:
            dh, n_ramp = self.ramp
            h = h + dh * (min(self.step, n_ramp) / n_ramp)
        if self.sigma is not None:
            h = h + self.sigma * _gaussians(_words(self.ids, self.step, 0, self.keys), self.precision)
        if self.cells is not None:
            h = h + self.cells.B[:, self.cells.cell]
        return h

    def rhs(self, S, H):
        c = torch.linalg.cross(S, H, dim=0)
        return self.A * c + self.Bc * torch.linalg.cross(S, c, dim=0)

    def rotate(self, M, S, H):
        b = -0.5 * self.dt * self.A
        F = H + self.alpha * torch.linalg.cross(M, H, dim=0)
        ff, fs = b * b * (F * F).sum(0), b * b * (F * S).sum(0)
        return (S * (1.0 - ff) + 2.0 * (b * torch.linalg.cross(F, S, dim=0) + F * fs)) / (1.0 + ff)

    def advance(self, integrator="heun"):
        ext = self.external()
        S = self.S
        H = self.gather(S) + self.aniso(S) + ext
        if integrator == "midpoint":
            M = 0.5 * (S + self.rotate(S, S, H))
            self.S = self.rotate(M, S, self.gather(M) + self.aniso(M) + ext)
        else:
            f0 = self.rhs(S, H)
            P = S + f0 * self.dt
            P = P / torch.sqrt((P * P).sum(0))
            f1 = self.rhs(P, self.gather(P) + self.aniso(P) + ext)
            Q = S + 0.5 * self.dt * (f0 + f1)
            self.S = Q / torch.sqrt((Q * Q).sum(0))
        self.step += 1
        if self.cells is not None and self.step % self.cells.rate == 0:
            self.cells.update(self.S, self.mu)

    def magnetization(self, mask=None, size=1):
        mask = torch.zeros(self.n, dtype=torch.int64, device=self.dev) if mask is None else mask
        v = torch.zeros(size, 4, dtype=torch.float64, device=self.dev)
        v.index_add_(0, mask, torch.cat([self.S * self.mu, self.mu[None]]).T.contiguous())
        mag = torch.sqrt((v[:, :3] ** 2).sum(1, keepdim=True))
        return torch.cat([v[:, :3] / mag, mag / v[:, 3:]], 1).reshape(-1)


def _dip_terms(rx, ry, rz):
    ri = 1.0 / torch.sqrt(rx * rx + ry * ry + rz * rz)
    ex, ey, ez, r3 = rx * ri, ry * ri, rz * ri, ri ** 3
    return [(3 * ex * ex - 1) * r3, 3 * ex * ey * r3, 3 * ex * ez * r3, (3 * ey * ey - 1) * r3, 3 * ey * ez * r3,
            (3 * ez * ez - 1) * r3]


class _Cells:
    """The macrocell dipole field of the tensor solver (atomistic tensors for
    pairs within the cutoff, point dipoles beyond) by direct sums; the far sums
    of more than 20,000 cells of one full regular grid by convolution."""

    def __init__(self, cells, dev, S, mu):
        t = lambda v, d=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=d, device=dev)  # noqa: E731
        self.dev, self.rate, self.size = dev, cells["update_rate"], cells["macro_cell_size"]
        self.cell = t(cells["atom_cell"], torch.int64)
        nat = np.asarray(cells["cell_natoms"])
        self.nc = nc = nat.size
        self.pos = t(cells["cell_pos_mom"]).reshape(nc, 4)[:, :3].T.contiguous()
        self.has = t(nat > 0, torch.bool)
        self.self_ = torch.where(self.has, 8.0 * math.pi / (3.0 * t(np.maximum(cells["cell_volume"], 1e-30))), 0.0)
        # atoms of each cell, padded
        order = np.argsort(cells["atom_cell"], kind="stable")
        start = np.concatenate([[0], np.cumsum(np.bincount(cells["atom_cell"], minlength=nc))])
        mx = int(nat.max())
        k = np.arange(mx)[None, :]
        ok = k < nat[:, None]
        atoms = np.where(ok, order[np.minimum(start[:-1, None] + k, order.size - 1)], 0)
        xyz, ok = t(cells["coords"]), t(ok, torch.bool)
        ax = xyz[:, t(atoms, torch.int64)]
        pi, pj = [], []
        step = max(1, (1 << 25) // nc)
        for i0 in range(0, nc, step):
            i1 = min(nc, i0 + step)
            d = self.pos[:, None, :] - self.pos[:, i0:i1, None]
            rij = 1.0 / torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
            near = (1.0 / rij) / self.size <= cells["cutoff"]
            near &= self.has[None, :] & self.has[i0:i1, None]
            q = near.nonzero()
            pi.append(q[:, 0] + i0)
            pj.append(q[:, 1])
        self.pi, self.pj = torch.cat(pi), torch.cat(pj)
        nat_t = t(nat)
        parts = []
        chunk = max(1, (1 << 24) // (mx * mx))
        for a in range(0, self.pi.numel(), chunk):
            i, j = self.pi[a:a + chunk], self.pj[a:a + chunk]
            r = ax[:, j][:, :, None, :] - ax[:, i][:, :, :, None]
            valid = ok[i][:, :, None] & ok[j][:, None, :]
            valid &= ~((i == j)[:, None, None] & torch.eye(mx, dtype=torch.bool, device=dev)[None])
            far = torch.where(valid, r[0], 1e30)
            tt = [torch.where(valid, v, 0.0).sum((1, 2)) / (nat_t[i] * nat_t[j]) for v in _dip_terms(far, r[1], r[2])]
            d = self.pos[:, j] - self.pos[:, i]
            bare = _dip_terms(torch.where(i == j, 1.0, d[0]), d[1], d[2])
            parts.append(torch.stack([u - torch.where(i == j, 0.0, v) for u, v in zip(tt, bare)]))
        self.T = torch.cat(parts, 1)
        self.fft = None
        if nc > 20000:
            g = torch.round((self.pos - self.pos.min(1, keepdim=True).values) / self.size).long()
            self.G = [int(v) + 1 for v in g.max(1).values]
            full = math.prod(self.G) == nc and bool(self.has.all())
            off = (self.pos - self.pos.min(1, keepdim=True).values - g.double() * self.size).abs().max()
            if not full or float(off) > 1e-6:
                raise ValueError("more than 20,000 cells that are not one full grid")
            self.lin = (g[2] * self.G[1] + g[1]) * self.G[0] + g[0]
            P = [2 * v for v in self.G]
            ax_ = [torch.fft.fftfreq(p, 1.0 / p, dtype=torch.float64, device=dev).round() * self.size for p in P]
            rz, ry, rx = torch.meshgrid(ax_[2], ax_[1], ax_[0], indexing="ij")
            zero = (rx == 0) & (ry == 0) & (rz == 0)
            self.fft = [torch.fft.rfftn(torch.where(zero, 0.0, v)) for v in _dip_terms(torch.where(zero, 1.0, rx), ry, rz)]
            self.P = P
        self.update(S, mu)

    def update(self, S, mu):
        nc, has = self.nc, self.has
        m = torch.zeros(3, nc, dtype=torch.float64, device=self.dev).index_add_(1, self.cell, S * mu)
        f = torch.zeros(3, nc, dtype=torch.float64, device=self.dev)
        sym = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
        if self.fft is not None:
            G, P = self.G, self.P
            box = torch.zeros(3, nc, dtype=torch.float64, device=self.dev)
            box[:, self.lin] = m
            M = torch.fft.rfftn(box.reshape(3, G[2], G[1], G[0]), s=(P[2], P[1], P[0]), dim=(1, 2, 3))
            for a in range(3):
                h = torch.fft.irfftn(sum(self.fft[sym[a][b]] * M[b] for b in range(3)), s=(P[2], P[1], P[0]))
                f[a] = h[:G[2], :G[1], :G[0]].reshape(-1)[self.lin]
        else:
            step = max(1, (1 << 25) // nc)
            for i0 in range(0, nc, step):
                i1 = min(nc, i0 + step)
                d = self.pos[:, None, :] - self.pos[:, i0:i1, None]
                same = (torch.arange(i0, i1, device=self.dev)[:, None] == torch.arange(nc, device=self.dev)[None])
                out = same | ~has[None, :] | ~has[i0:i1, None]
                tt = _dip_terms(torch.where(out, 1e30, d[0]), torch.where(out, 0.0, d[1]), torch.where(out, 0.0, d[2]))
                for a in range(3):
                    f[a, i0:i1] = sum(tt[sym[a][b]] @ m[b] for b in range(3))
        mj = m[:, self.pj]
        for a in range(3):
            f[a].index_add_(0, self.pi, sum(self.T[sym[a][b]] * mj[b] for b in range(3)))
        k = 9.27400915e-01
        self.B = torch.where(has, f * k, 0.0)
        self.Hd = torch.where(has, (f - 0.5 * self.self_ * m) * k, 0.0)


def _greedy(s):
    """First-fit colours of the exchange graph in atom order."""
    colour = [-1] * s.n
    st, en, nl = s.nl_start.tolist(), s.nl_end.tolist(), s.nl.tolist()
    for i in range(s.n):
        used = {colour[j] for j in nl[st[i]:en[i] + 1]}
        c = 0
        while c in used:
            c += 1
        colour[i] = c
    return np.array(colour)


def _mc_tables(temps):
    kbt = np.where(temps > 0, MU_B / (np.maximum(temps, 1e-300) * KB), np.inf)
    sig = np.where(temps < 1.0, 0.02, (1.0 / kbt) ** 0.2 * 0.08)
    return sig, kbt


def _site_delta(r, i, Sold, Snew, h):
    """Energy change (Tesla) of moving the spins of atoms i in their exchange field."""
    d = -((Snew - Sold) * (h + r.h[:, i])).sum(0)
    if r.uniaxial:
        e = r.e[:, i]
        d = d - r.ku2[i] * ((Snew * e).sum(0) ** 2 - (Sold * e).sum(0) ** 2)
    return d


def _exact_mc(case, seed):
    s, noise = _inputs(case, seed)
    r = _Ref(s, noise, "fp32", thermal=False)
    base = _lattice("sc", case["nx"], case["ny"], case["nz"], False, "iso", False, 300.0)
    colour = torch.as_tensor(np.tile(_greedy(base), case["replicas"]), device=r.dev)
    sig, kbt = _mc_tables(np.asarray(r.temps, dtype=np.float64))
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=r.dev)[r.typ]  # noqa: E731
    sig, beta = t(sig), t(np.where(np.isfinite(kbt), kbt, 1e300))
    ratio = r.mu_SI * 1.07828231e23
    lists = [(colour == c).nonzero()[:, 0] for c in range(int(colour.max()) + 1)]
    for sweep in range(case["sweeps"]):
        for i in lists:
            h = r.gather(r.S)[:, i]
            w = _words(i, sweep, 1, noise)
            g = _gaussians(w, "fp32")
            u = _u01(((w[1] & 0xFF) << 8) | ((w[2] & 0xFF) << 16) | (w[3] << 24) & _M32, "fp32")
            old = r.S[:, i]
            new = old + g * sig[i]
            new = new / torch.sqrt((new * new).sum(0))
            d = _site_delta(r, i, old, new, h) * ratio[i]
            acc = (d < 0) | (torch.exp(torch.clamp(-d * beta[i], min=-1e4, max=0.0)) >= u)
            r.S[:, i] = torch.where(acc, new, old)
    mask = torch.as_tensor(s.masks["replica"][0], dtype=torch.int64, device=r.dev)
    return {"spins": r.S.reshape(-1), "m": r.magnetization(mask, case["replicas"])}


def _splitmix(x):
    x = (x + 0x9E3779B97F4A7C15) & (2 ** 64 - 1)
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & (2 ** 64 - 1)
    return x ^ (x >> 31)


def _exact_cmc(case, seed):
    s, noise = _inputs(case, seed)
    if s.n * case["steps"] > 200000:
        return None
    r = _Ref(s, noise, "fp64", thermal=False)
    colour = _greedy(s)
    sig, kbt = _mc_tables(np.array([case["temperature"]]))
    sig, beta = float(sig[0]), float(kbt[0])
    ph, th = math.radians(case["phi"]), math.radians(case["theta"])
    ry = np.array([[math.cos(ph), 0, -math.sin(ph)], [0, 1, 0], [math.sin(ph), 0, math.cos(ph)]])
    rz = np.array([[math.cos(th), math.sin(th), 0], [-math.sin(th), math.cos(th), 0], [0, 0, 1]])
    P = torch.as_tensor(ry @ rz, dtype=torch.float64, device=r.dev)
    pv = (ry @ rz)[2]
    ratio = float(s.materials["mu_s_SI"][0] * 1.07828231e23)
    nc = int(colour.max()) + 1
    lists = [torch.as_tensor(np.flatnonzero(colour == c), device=r.dev) for c in range(nc)]
    counts = [0, 0, 0, 0]
    M = np.zeros(3)
    for sweep in range(case["steps"]):
        M = (ratio * r.S.sum(1)).cpu().numpy()
        for phase in range(2 * nc):
            lst = lists[phase % nc]
            n = lst.numel()
            K = n // 2
            if K == 0:
                continue
            key = _splitmix(noise ^ _splitmix(sweep * 1024 + phase))
            mul = 1 + _splitmix(key) % n
            while math.gcd(mul, n) != 1:
                mul = mul % n + 1
            add = _splitmix((key + 1) & (2 ** 64 - 1)) % n
            k = torch.arange(K, dtype=torch.int64, device=r.dev)
            i1, i2 = lst[(mul * (2 * k) + add) % n], lst[(mul * (2 * k + 1) + add) % n]
            hi = (phase << 20) & _M32
            g = _gaussians(_words(k, sweep | (hi << 32), 4, noise), "fp64")
            u = _u01(_words(k, sweep | (hi << 32), 5, noise)[0], "fp64")
            S1, S2 = r.S[:, i1], r.S[:, i2]
            T1 = S1 + g * sig
            T1 = T1 / torch.sqrt((T1 * T1).sum(0))
            a1, b1, a2 = P @ S1, P @ T1, P @ S2
            x = (a1 - b1)[:2] + a2[:2]
            on = (x * x).sum(0) < 1.0
            z = torch.where(a2[2] >= 0, 1.0, -1.0) * torch.sqrt(torch.clamp(1.0 - (x * x).sum(0), min=1e-300))
            T2 = P.T @ torch.cat([x, z[None]])
            h = r.gather(r.S)
            d = _site_delta(r, i1, S1, T1, h[:, i1]) * ratio + _site_delta(r, i2, S2, T2, h[:, i2]) * ratio
            f = (torch.exp(-d * beta) * (a2[2] / z).abs()).cpu().numpy()
            dm = (ratio * (T1 + T2 - S1 - S2)).T.cpu().numpy()
            on_, u_ = on.cpu().numpy(), u.cpu().numpy()
            acc = np.zeros(K, dtype=bool)
            mz, dz = float(M @ pv), dm @ pv
            for q in range(K):
                if not on_[q]:
                    counts[3] += 1
                    continue
                new = mz + dz[q]
                if f[q] * (new / mz) ** 2 >= u_[q] and new > 0.0:
                    acc[q] = True
                    mz = new
                    counts[1] += 1
                else:
                    counts[2] += 1
            counts[0] += K
            M = M + dm[acc].sum(0)
            sel = torch.as_tensor(acc, device=r.dev)
            r.S[:, i1[sel]] = T1[:, sel]
            r.S[:, i2[sel]] = T2[:, sel]
    return {"spins": r.S.reshape(-1), "moment": torch.as_tensor(M), "counters": torch.as_tensor(counts)}


def _exact_batch(case, seed):
    systems, params = _ensemble(case["systems"], case["ensemble"])
    rng = np.random.default_rng(seed)
    spins = [_magnetised(s.n, rng.integers(1 << 30), 0.2) for s in systems]
    n = [s.n for s in systems]
    off, boff = np.concatenate([[0], np.cumsum(n)]), np.concatenate([[0], np.cumsum([s.num_bonds for s in systems])])
    cat = np.concatenate
    mats = cat([s.materials for s in systems])
    mats["temperature"] = [p["temperature"] for p in params]
    sysno = np.repeat(np.arange(len(n)), n)
    j = S.SpinSystem(n=int(off[-1]), nl_start=cat([s.nl_start + b for s, b in zip(systems, boff)]),
                     nl_end=cat([s.nl_end + b for s, b in zip(systems, boff)]),
                     nl=cat([s.nl + o for s, o in zip(systems, off)]), jlist=cat([s.jlist for s in systems]),
                     exch_type=S.EXCH_ISOTROPIC, type=sysno.astype(np.int32), materials=mats, spins=cat(spins, 1),
                     params=S.SimParams(dt_SI=1e-16, local_temperature=True), uniaxial=True)
    dev = _device()
    ids = torch.as_tensor(np.arange(j.n) - off[sysno], dtype=torch.int64, device=dev)
    keys = torch.as_tensor(int(seed) + sysno, dtype=torch.int64, device=dev)
    r = _Ref(j, int(seed), "fp32", noise_ids=ids, noise_keys=keys)
    at = lambda k: torch.as_tensor(np.array([p[k] for p in params])[sysno].T.copy(), device=dev)  # noqa: E731
    r.h = at("H_start")
    r.ramp = (at("H_end") - r.h, max(p["n_ramp"] for p in params))
    hist = []
    mask = torch.as_tensor(sysno, dtype=torch.int64, device=dev)
    for t in range(case["steps"]):
        r.advance()
        if (t + 1) % case["every"] == 0:
            hist.append(r.magnetization(mask, len(n)).reshape(len(n), 4))
    return {"history": torch.stack(hist), "spins": r.S.reshape(-1)}


def _exact_adjoint(case, seed):
    if case["L"] ** 3 * case["steps"] > 4e7:
        return None
    s, noise = _inputs(case, seed)
    r = _Ref(s, noise, "fp64", thermal=False)
    target = _target(case, seed)
    N, w, wt = case["steps"], 1e-16, (r.mu / r.mu.sum())
    ku2, h, J = r.ku2, r.h.clone(), list(r.J)
    states = [r.S]
    mz = []
    for _ in range(N):
        r.advance()
        states.append(r.S)
        mz.append((r.S[2] * wt).sum())
    diff = torch.stack(mz).cpu().numpy() - target
    scale = torch.ones((), dtype=torch.float64, device=r.dev, requires_grad=True)
    ku = torch.ones((), dtype=torch.float64, device=r.dev, requires_grad=True)
    dh = torch.zeros(3, 1, dtype=torch.float64, device=r.dev, requires_grad=True)
    lam = torch.zeros_like(r.S)
    g = [0.0, 0.0, torch.zeros(3, 1, dtype=torch.float64, device=r.dev)]
    for t in range(N - 1, -1, -1):
        lam = lam.clone()
        lam[2] += 2.0 * w * float(diff[t]) * wt
        x = states[t].detach().requires_grad_(True)
        with torch.enable_grad():
            r.J, r.ku2, r.h = [scale * v for v in J], ku * ku2, h + dh
            r.S = x
            r.advance()
            out = torch.autograd.grad((r.S * lam).sum(), [x, scale, ku, dh])
        lam = out[0].detach()
        g = [a + b.detach() for a, b in zip(g, out[1:])]
    # dL/dKu from the scale of the reduced constant ku2 = Ku / mu_s
    return {"loss": torch.as_tensor([w * float((diff * diff).sum())], dtype=torch.float64),
            "dJ": g[0].reshape(1), "dKu": (g[1] / 6.69e-24).reshape(1), "dH": g[2].reshape(3)}


def _exact_measure(case, seed):
    s, noise = _inputs(case, seed)
    r = _Ref(s, noise, "fp32", thermal=False)
    hx = r.gather(r.S)
    e = torch.stack([-(r.S * hx).sum(0), -0.5 * r.kc4 * (r.S ** 4).sum(0), -(r.S * r.h).sum(0)]) * r.mu
    tq = torch.linalg.cross(r.S, hx + r.aniso(r.S) + r.h, dim=0)
    out = {}
    for key, mask, size in (("", torch.zeros_like(r.typ), 1), ("2", r.typ, 2)):
        v = torch.zeros(3, size, dtype=torch.float64, device=r.dev).index_add_(1, mask, e)
        ex = 0.5 * v[0]
        out["m" + key] = r.magnetization(mask, size)
        out["e" + key] = torch.stack([ex + v[1] + v[2], ex, v[1], v[2], torch.zeros_like(ex)]).reshape(-1)
    out["torque_max"] = torch.sqrt((tq * tq).sum(0)).max()
    out["torque"] = torch.zeros(2, 3, dtype=torch.float64, device=r.dev).index_add_(0, r.typ, (tq * r.mu_SI).T.contiguous())
    return out


@torch.no_grad()
def exact(case, seed):
    k = case["kind"]
    if k == "mc":
        return _exact_mc(case, seed)
    if k == "cmc":
        return _exact_cmc(case, seed)
    if k == "batch":
        return _exact_batch(case, seed)
    if k == "adjoint":
        return _exact_adjoint(case, seed)
    if k == "measure":
        return _exact_measure(case, seed)
    s, noise = _inputs(case, seed)
    r = _Ref(s, noise, case.get("precision", "fp32"))
    if s.cells is not None:
        if len(s.cells["cell_natoms"]) > 20000 and k == "llg" and any(case[a] % 2 for a in ("nx", "ny", "nz")):
            return None  # direct sums over that many cells take minutes
        r.cells = _Cells(s.cells, r.dev, r.S, r.mu)
    mean = 0.0
    for t in range(case["steps"]):
        r.advance(case.get("integrator", "heun"))
        if k == "llg" and (t + 1) % case["every"] == 0:
            mean = mean + r.magnetization()
    if k == "dipole":
        return {"spins": r.S.reshape(-1), "B": r.cells.B, "Hd": r.cells.Hd}
    return {"spins": r.S.reshape(-1), "m": r.magnetization(), "mean": mean}

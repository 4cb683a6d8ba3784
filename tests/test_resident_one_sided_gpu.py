"""Systems with one-sided bonds (i feels j, j does not feel i) run one launch per
pass: resident threads wait on their neighbours' words, and only mutual bonds
keep a neighbour from running ahead of a reader.  They also hold no memory for
such words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(L, one_sided):
    from vampire_b200 import system as S
    s = S.config_sc_llg(L, temperature=0.0)
    if one_sided:
        i = np.repeat(np.arange(s.n), s.nl_end - s.nl_start + 1)
        drop = (np.random.default_rng(L).random(s.nl.size) < 0.1) & (i < s.nl)
        keep = ~drop
        cnt = np.bincount(i[keep], minlength=s.n)
        s.nl, s.jlist = s.nl[keep], s.jlist[keep]
        end = np.cumsum(cnt)
        s.nl_start = (end - cnt).astype(s.nl_start.dtype)
        s.nl_end = (end - 1).astype(s.nl_end.dtype)
    return s


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("one_sided", [False, True])
def test_steps(vgpu_lib, prec, one_sided):
    from oracle import oracle as O
    from vampire_b200 import vgpu as V
    s = _system(14, one_sided)
    with V.Simulation(s, precision=prec) as sim:
        before = sim.profile_read()["kernel_launches"]
        sim.llg_heun(5)
        got = sim.spins()
        launches = sim.profile_read()["kernel_launches"] - before
    want = O.OracleSystem(s).llg_heun(s.spins, 5)
    assert np.abs(got - want).max() < (1e-5 if prec == "fp32" else 1e-12)
    assert (launches >= 10) == one_sided


def test_memory(vgpu_lib):
    """140,608 spins in FP64: two states of 32 bytes a spin are 9 MB."""
    import torch
    from vampire_b200 import vgpu as V
    held = []
    for one_sided in (False, True):
        s = _system(52, one_sided)
        for _ in range(2):  # the first upload also loads the library's kernels
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            with V.Simulation(s, precision="fp64") as sim:
                sim.synchronize()
                used = free - torch.cuda.mem_get_info()[0]
        held.append(used)
    assert held[0] - held[1] >= 6 << 20

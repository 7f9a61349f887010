"""The block chains of the AMR sweeps, cut to 1, 2, 4 or 8 blocks (EMG_AMR_CHAIN),
against the oracle bit for bit: structure, data and counters, for the Euler and the
five-equation system, global and subcycled steps, with one periodic axis. The rule
that picks the cut (emg_amr::shorten_chains) gives hierarchies of this size single
blocks, so without the variable no chain of several would run here (needs a B200)."""
import functools

import numpy as np
import pytest

from emergence_b200 import workloads as W
from emergence_b200.physics import Bc, FluxMode
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

STEPS = 3


def _problem(system, dim):
    if system == "euler":
        s, cfg, lo, hi, bc, init = W.amr_explosion(dim=dim, base=6 if dim == 2 else 3, levels=3 if dim == 2 else 2, radius=0.25,
                                                   regrid_every=2)
        return s, cfg, lo, hi, [[Bc.Periodic, Bc.Periodic], bc[1], bc[2]], init
    s, cfg, lo, hi, bc, init = W.two_phase_amr_bubble(dim=dim, base=6 if dim == 2 else 3, b=16 if dim == 2 else 8,
                                                      levels=3 if dim == 2 else 2, regrid_every=2)
    return s, cfg, lo, hi, [bc[0], [Bc.Periodic, Bc.Periodic], bc[2]], init


def _steps(a, subcycle):
    for _ in range(STEPS):
        if subcycle:
            a.step_subcycled(a.dt_cfl_subcycled())
        else:
            a.step(a.dt_cfl())
    return a.structure(), a.download(), a.counters()


@functools.lru_cache(maxsize=None)
def _oracle(system, dim, subcycle):
    s, cfg, lo, hi, bc, init = _problem(system, dim)
    o = O.OracleAmr(s, cfg, lo, hi, bc, init, mode=FluxMode.Weno, subcycle=subcycle)
    start = o.structure(), o.download()
    return start, _steps(o, subcycle)


def _longest_run(structure, axis):
    """Blocks of the longest row of same-level leaves along an axis."""
    leaves = {tuple(r[:4]) for r in structure[structure[:, 4] == 1].tolist()}
    best = 0
    for r in leaves:
        n, q = 0, list(r)
        while tuple(q) in leaves:
            n, q[1 + axis] = n + 1, q[1 + axis] + 1
        best = max(best, n)
    return best


@pytest.mark.parametrize("cap", [1, 2, 4, 8])
@pytest.mark.parametrize("subcycle", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("system", ["euler", "five"])
def test_results_do_not_depend_on_the_cut(system, dim, subcycle, cap, monkeypatch):
    from emergence_b200 import GpuAmr
    start, (so, uo, co) = _oracle(system, dim, subcycle)
    assert all(_longest_run(so, d) >= min(cap, 3) for d in range(dim))  # chains of several blocks
    monkeypatch.setenv("EMG_AMR_CHAIN", str(cap))
    s, cfg, lo, hi, bc, init = _problem(system, dim)
    g = GpuAmr(s, cfg, lo, hi, bc, mode=FluxMode.Weno, blocks=start, subcycle=subcycle)
    sg, ug, cg = _steps(g, subcycle)
    assert np.array_equal(sg, so)
    rows = slice(None) if subcycle else so[:, 4] == 1  # a global step leaves ancestors to the next restriction
    assert np.array_equal(ug[rows], uo[rows]), float(np.nanmax(np.abs(ug[rows] - uo[rows])))
    assert cg == co
